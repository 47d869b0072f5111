"""The walk of a track's two halves in one run of steps against the oracle, bit for
bit: halves that miss the grid, that are a point, of very different lengths in one
warp, with a negative or a far crossing (left to the plain form), tracks that turn
on a voxel's border; the lists of both forms, and PoCA's image with and without
length weights.

Tolerance: the lists are the oracle's bits.  PoCA's image is a quotient of sums of
at most some thousand FP64 terms in another order: 1e-12.
"""
import numpy as np
import pytest

import muontomography_gb300 as M
from muontomography_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def turned(wl, seed):
    """Tracks of the workload with their outgoing lines moved: the halves meet anywhere."""
    rng = np.random.default_rng(seed)
    g, rays = wl.grid, wl.tracks()
    n = rays.shape[0]
    lo = np.array([g.x_min, g.y_min, g.z_min])
    ext = np.array([g.nx * g.dx, g.ny * g.dy, g.nz * g.dz])
    at = lo + ext * rng.uniform(-0.3, 1.3, (n, 3))  # the point both lines go through
    k = n // 4
    at[:k] = lo + np.array([g.dx, g.dy, g.dz]) * np.round((at[:k] - lo) / np.array([g.dx, g.dy, g.dz]))
    at[k:2 * k, 2] = lo[2] + ext[2] * rng.choice([0.0, 1.0, 1e-9, 1.0 - 1e-9], k)
    for p, d, z in ((2, 8, lo[2] + ext[2]), (5, 11, lo[2])):
        v = rng.normal(size=(n, 3)) * [0.4, 0.4, 0.0] + [0.0, 0.0, 1.0]
        v /= np.linalg.norm(v, axis=1, keepdims=True)
        rays[:, d:d + 3] = v
        rays[:, p:p + 3] = at + v * ((z - at[:, 2:]) / v[:, 2:])
    return rays


@pytest.mark.parametrize("n,n_muons", [(1, 300), (5, 3000), (40, 3001), (90, 700)])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_lists_of_turned_tracks(gpu, oracle, n, n_muons, precision):
    wl = W.small(n_muons=n_muons, seed=91, n=n)
    rays = turned(wl, n)
    cfg = wl.em_config(precision=precision, update_with_mean=True)
    r = oracle.Mlsd(wl.grid, cfg, rays, np.full(wl.grid.nvox, 1e-7)).export()
    with M.MutoMLSD(cfg) as rec:
        rec.load_tracks(rays)
        rec.prepare()
        g = rec.export_paths()
    assert np.array_equal(g["off"], r["off"]) and np.array_equal(g["idx"], r["idx"])
    kind = np.float64 if precision == "fp64" else np.float32
    for key in ("len", "tail"):
        assert np.array_equal(g[key], r[key].astype(kind).astype(np.float64)), key


@pytest.mark.parametrize("n", [1, 6, 40])
@pytest.mark.parametrize("over", [{}, {"length_weighted": False}, {"straight_line": True}])
def test_poca_of_turned_tracks(gpu, oracle, n, over):
    wl = W.small(n_muons=4003, seed=92, n=n)
    rays = turned(wl, 3 + n)
    cfg = wl.poca_config(**over)
    with M.MutoPoCA(cfg) as rec:
        img = rec.reconstruct(rays).reshape(-1, order="F")
    want = oracle.poca(wl.grid, cfg, rays)
    want = np.asarray(want[0] if isinstance(want, tuple) else want).reshape(-1)
    assert np.linalg.norm(img - want) <= 1e-12 * max(np.linalg.norm(want), 1e-300)
