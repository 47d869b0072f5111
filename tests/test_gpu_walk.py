"""The FP64 walk's quick forms against the oracle, bit for bit: quotients by
corrected products, steps compared as integers (with a first crossing of -0.0: a
track that starts on the grid's top plane), the mixed form's tails summed by a
scan; and the forms they leave to the plain ones: coordinates beyond 1e100, walks
with a negative crossing.
"""
import numpy as np
import pytest

import muontomography_gb300 as M
from muontomography_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def same(oracle, grid, p1, p2, cap=512):
    p1, p2 = np.ascontiguousarray(p1, float), np.ascontiguousarray(p2, float)
    gx, gl, gc = M.siddon_batch(grid, p1, p2, cap)
    ox, ol, oc = oracle.siddon_batch(grid, p1, p2, cap)
    assert np.array_equal(gc, oc) and np.array_equal(gx, ox)
    assert np.array_equal(gl.view(np.uint64), ol.view(np.uint64))
    return oc


@pytest.mark.parametrize("mm", [10.0, 1.0 / 3.0, 17.3])
def test_walk_edges_bit_exact(gpu, oracle, mm):
    rng = np.random.default_rng(71)
    g = M.Grid(31, 17, 23, -15.5 * mm, 2.0, -3.7 * mm, mm, mm * 1.1, mm * 0.9)
    lo = np.array([g.x_min, g.y_min, g.z_min])
    ext = np.array([g.nx * g.dx, g.ny * g.dy, g.nz * g.dz])
    a, b = lo + ext * rng.uniform(-0.2, 1.2, (4000, 3)), lo + ext * rng.uniform(-0.2, 1.2, (4000, 3))
    a[:1000, 2] = lo[2] + g.nz * g.dz  # on the top plane, either way round
    b[500:1000, 2] = lo[2]
    a[1000:1500] = lo + ext * rng.integers(0, 2, (500, 3))  # at corners
    a[1500:2000] = lo + np.array([g.dx, g.dy, g.dz]) * rng.integers(0, 17, (500, 3))  # on lattice points
    b[1750:2000] = lo + np.array([g.dx, g.dy, g.dz]) * rng.integers(0, 17, (250, 3))
    b[2000:2300, :2] = a[2000:2300, :2]  # along an axis
    b[2300:2400] = a[2300:2400] + 1e-7 * rng.standard_normal((100, 3))  # shorter than the step tolerance
    assert (same(oracle, g, a, b) > 0).sum() > 1000


def test_walk_far_coordinates_bit_exact(gpu, oracle):
    g = M.Grid(10, 10, 10, 0.0, 0.0, 0.0, 10.0, 10.0, 10.0)
    p1 = np.array([[50.0, 50.0, 120.0], [50.0, 50.0, 1e101], [1e120, 50.0, 50.0], [5.0, 5.0, 99.0]])
    p2 = np.array([[51.0, 49.0, -20.0], [50.0, 50.0, -1e101], [-1e120, 50.0, 50.0], [1e101, 6.0, 1.0]])
    same(oracle, g, p1, p2, cap=64)


@pytest.mark.parametrize("n,n_muons", [(3, 200), (33, 4001), (90, 1203)])
@pytest.mark.parametrize("straight", [False, True])
def test_mixed_lists_bit_exact(gpu, oracle, n, n_muons, straight):
    # paths of 1 pair, around 32 (one scan) and of several scans
    wl = W.small(n_muons=n_muons, seed=73, n=n)
    rays = wl.tracks()
    cfg = wl.em_config(precision="mixed", straight_line=straight, update_with_mean=True)
    r = oracle.Mlsd(wl.grid, cfg, rays, np.full(wl.grid.nvox, 1e-7)).export()
    with M.MutoMLSD(cfg) as rec:
        rec.load_tracks(rays)
        rec.prepare()
        g = rec.export_paths()
    assert np.array_equal(g["off"], r["off"]) and np.array_equal(g["idx"], r["idx"])
    for key in ("len", "tail"):
        assert np.array_equal(g[key], r[key].astype(np.float32).astype(np.float64)), key
