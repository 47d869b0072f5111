"""Images of the mixed form in and out, on the host up to 16 384 voxels and on the device
beyond: the 32-bit value of every voxel, of single scans and of a batch's.
"""
import numpy as np
import pytest

import muontomography_gb300 as M
from muontomography_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,nz", [(1, 1, 1), (25, 25, 25), (64, 16, 16), (29, 113, 5), (26, 26, 26)])
def test_values_come_back(gpu, nx, ny, nz):
    g = M.Grid(nx, ny, nz, -300.0, -300.0, -300.0, 600.0 / nx, 600.0 / ny, 600.0 / nz)
    wl = W.Workload("scan", g, [], 50, 99, True, 1)
    rng = np.random.default_rng(nx)
    img = np.asfortranarray(10.0 ** rng.uniform(-12, 3, (nx, ny, nz)))
    img.reshape(-1)[0] = 0.0
    with M.MutoMLSD(wl.em_config(update_with_mean=True, precision="mixed")) as rec:
        rec.load_tracks(wl.tracks())
        rec.prepare()
        assert np.array_equal(rec.image(), np.full((nx, ny, nz), np.float64(np.float32(1.0e-7))))
        rec.set_image(img)
        assert np.array_equal(rec.image(), img.astype(np.float32).astype(np.float64))


def test_a_batch_of_both(gpu, oracle):
    wls = [W.small(n_muons=400, seed=100 + k, n=n) for k, n in enumerate((12, 26, 25))]
    rays = [w.tracks() for w in wls]
    cfg = wls[0].em_config(update_with_mean=True, precision="mixed", num_iteration=2)
    cfg.pop("grid")
    images = M.Batch(cfg, [w.grid for w in wls]).reconstruct_all(rays)
    for w, r, img in zip(wls, rays, images):
        ref = oracle.Mlsd(w.grid, w.em_config(update_with_mean=True), r, np.full(w.grid.nvox, 1e-7))
        ref.iterate(2)
        got = np.asarray(img).reshape(-1, order="F")
        assert np.array_equal(got, got.astype(np.float32))
        assert np.linalg.norm(got - ref.image()) < 2e-5 * np.linalg.norm(ref.image())
