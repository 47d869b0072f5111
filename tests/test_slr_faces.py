"""Straight lines just below a grid's upper x and y faces: the walk gives such a line
the index nx (or ny) on its whole way, which is no voxel of the image.  SLRIter's
passes leave these voxels out, in every row and plane of the grid.

Tolerance: 1e-12, the bar of the other SLRIter tests: sums of positive FP64 values in
another order, and reciprocals to a few ulp.
"""
import numpy as np
import pytest

import muontomography_gb300 as M
from muontomography_gb300 import workloads as W


def face_lines(grid, rng, n, axis):
    """Ends (top, bottom) of n lines 5e-5 mm below the upper face of `axis`, moving 5e-7 mm along it."""
    hi = [grid.x_min + grid.nx * grid.dx, grid.y_min + grid.ny * grid.dy]
    top, bottom = np.empty((n, 3)), np.empty((n, 3))
    top[:, 2], bottom[:, 2] = grid.z_min + grid.nz * grid.dz, grid.z_min
    other = 1 - axis
    lo = (grid.x_min, grid.y_min)[other]
    top[:, other] = rng.uniform(lo, hi[other], n)
    bottom[:, other] = np.clip(top[:, other] + rng.uniform(-200.0, 200.0, n), lo + 1.0, hi[other] - 1.0)
    top[:3, other] = bottom[:3, other] = hi[other] - 1.0  # the last row
    top[3:6, other] = bottom[3:6, other] = lo + 1.0
    top[:, axis] = hi[axis] - 5.0e-5
    bottom[:, axis] = top[:, axis] + 5.0e-7
    return top, bottom


def face_rays(grid, rng, n, axis):
    top, bottom = face_lines(grid, rng, n, axis)
    rays = np.zeros((n, 14))
    rays[:, 0] = rays[:, 1] = rng.uniform(1.0, 5.0, n)
    rays[:, 2:5], rays[:, 5:8] = top, bottom
    for at in (8, 11):
        d = np.concatenate([rng.normal(0.0, 0.02, (n, 2)), np.ones((n, 1))], 1)
        rays[:, at:at + 3] = d / np.linalg.norm(d, axis=1, keepdims=True)
    return rays


@pytest.mark.parametrize("axis", [0, 1])
def test_walk_below_an_upper_face_has_the_index_past_it(oracle, axis):
    g = W.small(n=6).grid
    top, bottom = face_lines(g, np.random.default_rng(1), 40, axis)
    xyz, _, count = oracle.siddon_batch(g, top, bottom, 40)
    assert count.min() >= 6
    for i in range(40):
        assert (xyz[i, :count[i], axis] == (g.nx, g.ny)[axis]).all()


def expected(oracle, grid, rays, passes, weighted, energy):
    """SLRIter with the voxels outside the image left out (the equal shares count them)."""
    n = rays.shape[0]
    z_hi, z_lo = grid.z_min + grid.nz * grid.dz, grid.z_min
    t1, t2 = (z_hi - rays[:, 4]) / rays[:, 10], (z_lo - rays[:, 7]) / rays[:, 13]
    p1, p2 = rays[:, 2:5] + t1[:, None] * rays[:, 8:11], rays[:, 5:8] + t2[:, None] * rays[:, 11:14]
    total = np.sqrt(((p1 - p2) ** 2).sum(1))
    ang = [np.arctan2(rays[:, 8 + k], rays[:, 10]) - np.arctan2(rays[:, 11 + k], rays[:, 13]) for k in range(2)]
    a2 = ang[0] ** 2 + ang[1] ** 2
    xyz, length, count = oracle.siddon_batch(grid, p1, p2, grid.nx + grid.ny + grid.nz + 8)
    img, weight = np.zeros(grid.nvox), np.zeros(grid.nvox)
    for it in range(passes):
        for i in range(n):
            v, l = xyz[i, :count[i]].astype(np.int64), length[i, :count[i]]
            inside = (v < [grid.nx, grid.ny, grid.nz]).all(1)
            v, l = v[inside], l[inside]
            if not len(l):
                continue
            j = v[:, 0] + grid.nx * (v[:, 1] + grid.ny * v[:, 2])
            if weighted:
                w, iv = l / grid.dz, 0.5 * a2[i] * (l / total[i]) ** 2
            else:
                w, iv = np.ones(len(l)), np.full(len(l), 0.5 * a2[i] / float(count[i]) ** 2)
            if it:
                iv = iv * (img[j] / img[j].sum())
            if energy:
                iv = iv * rays[i, 0] ** 2
            weight[j] += w
            img[j] += iv
    return np.where(weight < 1e-8, 0.0, img / np.where(weight < 1e-8, 1.0, weight))


# 6^3 voxels: image in shared memory; 30^3: in global memory
@pytest.mark.gpu
@pytest.mark.parametrize("n,n_muons", [(6, 500), (30, 1500)])
@pytest.mark.parametrize("weighted,energy", [(True, False), (False, True)])
@pytest.mark.parametrize("schedule", ["levels", "sequential"])
def test_slr_iter_leaves_them_out(gpu, oracle, n, n_muons, weighted, energy, schedule):
    wl = W.small(n_muons=n_muons, seed=91, n=n)
    rng = np.random.default_rng(n)
    rays = np.concatenate([wl.tracks(), face_rays(wl.grid, rng, 60, 0), face_rays(wl.grid, rng, 60, 1)])
    rays = np.ascontiguousarray(rays[rng.permutation(rays.shape[0])])
    cfg = wl.poca_config(length_weighted=weighted, has_energy=energy, slr_iter_schedule=schedule)
    cfg["num_iteration"] = 3
    with M.MutoSLRIter(cfg) as rec:
        got = rec.reconstruct(rays).reshape(-1, order="F")
    want = expected(oracle, wl.grid, rays, 3, weighted, energy)
    assert np.linalg.norm(got - want) <= 1e-12 * np.linalg.norm(want)
    assert np.array_equal(got > 0, want > 0)


@pytest.mark.gpu
def test_only_lines_outside_the_image(gpu):
    wl = W.small(n=6)
    rays = face_rays(wl.grid, np.random.default_rng(3), 50, 0)
    cfg = wl.poca_config()
    cfg["num_iteration"] = 3
    with M.MutoSLRIter(cfg) as rec:
        assert not rec.reconstruct(rays).any()
