"""The mixed form's one-pass mean kernel in two passes (grids whose lambda and sums outgrow
L2): images against the FP64 form, and the sums of g_ij where one layer holds most of
every muon's sum lambda L.

Tolerances: as in test_gpu_once.py (2e-5 after three iterations) and
test_gpu_once_moments.py (1e-4 for the sums of a heavy layer).
"""
import numpy as np
import pytest

import muontomography_gb300 as M
from muontomography_gb300 import workloads as W

pytestmark = pytest.mark.gpu

IRON, LEAD = M.X0_MM["iron"], M.X0_MM["lead"]


def rel_l2(a, b):
    return float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300))


def scan(nx, ny, nz, mm, n_muons, seed):
    x, y, z = nx * mm / 2, ny * mm / 2, nz * mm / 2
    g = M.Grid(nx, ny, nz, -x, -y, -z, mm, mm, mm)
    blocks = [M.Block((-0.3 * x, -0.3 * y, -0.4 * z), (0.4 * x, 0.4 * y, 0.3 * z), IRON),
              M.Block((0.5 * x, -0.2 * y, -0.6 * z), (0.8 * x, 0.3 * y, 0.6 * z), LEAD)]
    return W.Workload("scan", g, blocks, n_muons, seed, True, 3)


def g_sums(wl, rays, x, precision):
    with M.MutoMLSD(wl.em_config(update_with_mean=True, precision=precision, num_iteration=0)) as rec:
        rec.load_tracks(rays)
        rec.prepare()
        value, grad = rec.nll_grad(x)
        return value, grad / np.exp(x), rec.status()


def heavy_layer(wl, height):
    g = wl.grid
    x = np.full(g.nvox, np.log(1.0e-7))
    x[np.arange(g.nvox) // (g.nx * g.ny) == int(height * g.nz)] = np.log(0.05)
    return x


def images(wl, rays, precision):
    with M.MutoMLSD(wl.em_config(update_with_mean=True, precision=precision, compute_cost=True)) as rec:
        rec.load_tracks(rays)
        rec.prepare()
        rec.iterate(1)
        before = rec.launch_count()
        rec.iterate(2)
        return rec.image().reshape(-1, order="F"), rec.launch_count() - before, rec.status()


# (330^2 x 160: 139 MB of lambda and sums, 280 pairs a path; 300^2 x 100: 76 MB, 175)
def test_two_passes_beyond_l2(gpu):
    small = scan(300, 300, 100, 6.0, 4_001, 85)
    img, one, _ = images(small, small.tracks(), "mixed")
    for n_muons in (1, 4_001):
        wl = scan(330, 330, 160, 6.0, n_muons, 86)
        rays = wl.tracks()
        img, two, st = images(wl, rays, "mixed")
        img64, _, st64 = images(wl, rays, "fp64")
        assert rel_l2(img, img64) < 2e-5
        if st["n_scat_in_grid"]:
            assert st["muon_group"] == 32 and two == one + 2
            assert abs(st["cost"] - st64["cost"]) <= 1e-5 * abs(st64["cost"])


@pytest.mark.parametrize("height", [0.95, 0.08])
def test_two_passes_one_heavy_layer(gpu, height):
    wl = scan(330, 330, 160, 6.0, 3_001, 87)
    rays = wl.tracks()
    x = heavy_layer(wl, height)
    v64, g64, _ = g_sums(wl, rays, x, "fp64")
    v, g, _ = g_sums(wl, rays, x, "mixed")
    assert rel_l2(g, g64) < 1e-4 and abs(v - v64) <= 1e-4 * abs(v64)
