"""The mean update and the copy of lambda between voxel order and bricked order, in whole
sectors: grids of every remainder of 2 voxels in x, 4 in y and 8 in z, images and
gradients against the FP64 oracle, and the image of a pass over no muons.

Tolerances: 1e-10 and 1e-9 in FP64, as in test_gpu_parity.py and test_gpu_adjoint.py;
mixed 2e-5 (three iterations, as in test_gpu_once.py) and 1e-4 for a gradient, whose sums are of
both signs (as in test_gpu_once_moments.py).
"""
import numpy as np
import pytest

import muontomography_gb300 as M
from muontomography_gb300 import workloads as W

pytestmark = pytest.mark.gpu

GRIDS = [(1, 1, 1), (2, 1, 3), (3, 5, 2), (5, 4, 7), (6, 7, 9), (9, 3, 4), (33, 2, 5), (8, 13, 16), (31, 17, 11), (64, 6, 13)]


def scan(nx, ny, nz):
    g = M.Grid(nx, ny, nz, -300.0, -300.0, -300.0, 600.0 / nx, 600.0 / ny, 600.0 / nz)
    return W.Workload("scan", g, [M.Block((-100.0, -100.0, -100.0), (100.0, 100.0, 100.0), M.X0_MM["iron"])], 4_000, 95, True, 3)


def rel_l2(a, b):
    return float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300))


@pytest.mark.parametrize("nx,ny,nz", GRIDS)
@pytest.mark.parametrize("precision,tol,gtol", [("fp64", 1e-10, 1e-9), ("mixed", 2e-5, 1e-4)])
@pytest.mark.parametrize("lists", ["muon_major", "recompute"])
def test_images_and_gradients(gpu, oracle, nx, ny, nz, precision, tol, gtol, lists):
    wl = scan(nx, ny, nz)
    rays = wl.tracks()
    cfg = wl.em_config(update_with_mean=True, precision=precision, path_lists=lists)
    ref = oracle.Mlsd(wl.grid, cfg, rays, np.full(wl.grid.nvox, 1e-7))
    ref.iterate(3)
    want = ref.image()
    rng = np.random.default_rng(5)
    lam = wl.lam() * rng.uniform(0.6, 1.4, wl.grid.nvox) + 2e-7
    with M.MutoMLSD(cfg) as rec:
        rec.load_tracks(rays)
        rec.prepare()
        rec.iterate(3)
        assert rel_l2(rec.image().reshape(-1, order="F"), want) < tol
        lam = np.where(rec.multiplicity() > 0, lam, 0.0)
        x = np.log(np.where(lam > 0, lam, 1.0))
        f, g = rec.nll_grad(x)
        rec.set_image(want.reshape(wl.grid.nx, wl.grid.ny, wl.grid.nz, order="F"))
        rec.iterate(1)  # (the gradient left the sums at zero)
        img = rec.image().reshape(-1, order="F")
    f_ref, g_ref = ref.nll(lam, grad=True)
    assert abs(f - f_ref) <= gtol * abs(f_ref) and rel_l2(g, g_ref) < gtol
    ref.iterate(1)
    assert rel_l2(img, ref.image()) < tol


@pytest.mark.parametrize("nx,ny,nz", GRIDS)
def test_without_muons(gpu, nx, ny, nz):
    wl = scan(nx, ny, nz)
    rays = wl.tracks()
    rays[:, 2:4] += 1.0e5
    rays[:, 5:7] += 1.0e5
    with M.MutoMLSD(wl.em_config(update_with_mean=True, precision="mixed")) as rec:
        assert not rec.reconstruct(rays).any()
