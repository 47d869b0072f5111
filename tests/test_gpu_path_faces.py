"""EM paths just below a grid's upper x face.  A muon that moves at most 1e-6 mm along x
there is walked with index nx, so its flat voxel indices x + nx (y + ny z) are the next
row's, and past the image in the last row and plane: the first count as what they are,
the second for nothing (src/MutoMLSD.cpp reads past its vector).  In every form of the
lists, with grids that fill whole bricks and grids that do not.

Tolerances: FP64 1e-11 (sums of another order, three iterations), mixed 2e-5 (as in the
other tests of the mixed lists); medians and percentiles 1e-10 and 1e-4, as in theirs.
"""
import numpy as np
import pytest

import muontomography_gb300 as M
from muontomography_gb300 import workloads as W


def face_muons(grid, rng, n):
    """Muons with a kink in y at mid height, 4e-7 voxels below the upper x face, moving 2.5e-7 mm a half."""
    h = grid.dz * grid.nz / 2
    hi_x, hi_y = grid.x_min + grid.nx * grid.dx, grid.y_min + grid.ny * grid.dy
    y = rng.uniform(grid.y_min + 60.0, hi_y - 60.0, n)
    y[: n // 2] = hi_y - 0.4 * grid.dy  # within the last row
    s1 = np.where(np.arange(n) < n // 2, rng.uniform(-0.02, 0.02, n) * grid.dy / h, rng.uniform(-0.1, 0.1, n))
    s2 = s1 + rng.choice([-1.0, 1.0], n) * rng.uniform(0.02, 0.05, n) * np.where(np.arange(n) < n // 2, grid.dy / h, 1.0)
    sx = -2.5e-7 / h
    rays = np.zeros((n, 14))
    rays[:, 0] = rays[:, 1] = rng.uniform(1.0, 5.0, n)
    x = hi_x - 4.0e-7 * grid.dx
    rays[:, 2], rays[:, 3], rays[:, 4] = x, y + s1 * h, h
    rays[:, 5], rays[:, 6], rays[:, 7] = x + 5.0e-7, y - s2 * h, -h
    for at, s in ((8, s1), (11, s2)):
        d = np.stack([np.full(n, sx), s, np.ones(n)], 1)
        rays[:, at:at + 3] = d / np.linalg.norm(d, axis=1, keepdims=True)
    return rays


def scan(n):
    wl = W.small(n_muons=900, seed=111, n=n)
    rng = np.random.default_rng(n)
    rays = np.concatenate([wl.tracks(), face_muons(wl.grid, rng, 80)])
    return wl, np.ascontiguousarray(rays[np.concatenate([[0], 1 + rng.permutation(len(rays) - 1)])])


SIZES = [5, 6, 8, 9, 16]


@pytest.mark.parametrize("n", SIZES)
def test_such_paths_leave_the_image(oracle, n):
    wl, rays = scan(n)
    ref = oracle.Mlsd(wl.grid, wl.em_config(), rays, np.full(wl.grid.nvox, 1e-7))
    assert ref.counts()["n_bad_index"] >= 30
    idx = ref.export()["idx"]
    assert wl.grid.nvox <= idx.max() <= wl.grid.nvox + n * n


@pytest.mark.gpu
@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("precision,tol", [("fp64", 1e-11), ("mixed", 2e-5)])
@pytest.mark.parametrize("lists", ["muon_major", "voxel_major", "recompute"])
def test_they_count_as_in_the_oracle(gpu, oracle, n, precision, tol, lists):
    wl, rays = scan(n)
    cfg = wl.em_config(update_with_mean=True, mean_percentile=100, precision=precision, num_iteration=3, path_lists=lists)
    ref = oracle.Mlsd(wl.grid, cfg, rays, np.full(wl.grid.nvox, 1e-7))
    ref.iterate(3)
    with M.MutoMLSD(cfg) as rec:
        img = rec.reconstruct(rays).reshape(-1, order="F")
        assert rec.status()["n_scat_in_grid"] == ref.counts()["n_scat_in_grid"]
        if lists != "recompute":
            paths, want = rec.export_paths(), ref.export()
            assert np.array_equal(paths["off"], want["off"]) and np.array_equal(paths["idx"], want["idx"])
    assert np.linalg.norm(img - ref.image()) <= tol * np.linalg.norm(ref.image())


@pytest.mark.gpu
@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("precision,tol", [("fp64", 1e-10), ("mixed", 1e-4)])
@pytest.mark.parametrize("layout", ["index", "columns"])
@pytest.mark.parametrize("over", [{}, {"update_with_mean": True, "mean_percentile": 60}, {"muon_pass": "tile"}])
def test_in_the_voxel_major_copy(gpu, oracle, n, precision, tol, layout, over):
    wl, rays = scan(n)
    cfg = wl.em_config(precision=precision, num_iteration=3, muon_layout=layout, **over)
    ref = oracle.Mlsd(wl.grid, cfg, rays, np.full(wl.grid.nvox, 1e-7))
    ref.iterate(3)
    with M.MutoMLSD(cfg) as rec:
        img = rec.reconstruct(rays).reshape(-1, order="F")
        assert np.array_equal(rec.multiplicity(), np.bincount(ref.export()["idx"], minlength=wl.grid.nvox)[:wl.grid.nvox])
    assert np.linalg.norm(img - ref.image()) <= tol * np.linalg.norm(ref.image())


@pytest.mark.gpu
@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("variant", ["8x8", "split", "split8_overlap", "staged"])
def test_in_the_other_forms(gpu, oracle, n, variant):
    wl, rays = scan(n)
    cfg = wl.em_config(update_with_mean=True, mean_percentile=100, precision="mixed", num_iteration=3,
                       path_lists="muon_major", fused_variant=variant)
    ref = oracle.Mlsd(wl.grid, cfg, rays, np.full(wl.grid.nvox, 1e-7))
    ref.iterate(3)
    with M.MutoMLSD(cfg) as rec:
        img = rec.reconstruct(rays).reshape(-1, order="F")
    assert np.linalg.norm(img - ref.image()) <= 2e-5 * np.linalg.norm(ref.image())
