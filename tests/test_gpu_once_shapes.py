"""The mixed form's one-pass mean kernel on short paths (4 and 8 lanes a muon, where there
are muons enough to fill the GPU) and in two passes (grids whose lambda and sums outgrow
L2): images against the FP64 oracle or form, and the sums of g_ij where one layer holds
most of every muon's sum lambda L.  Paths within the held pairs (32 and 64) and beyond.

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


# (voxels, mm, tracks, lanes a muon: 16 where there are few muons or few voxels)
SHORT = [(70, 66, 8, 20.0, 60_011, 4), (70, 66, 1, 200.0, 90_001, 4), (200, 170, 1, 20.0, 200_003, 16),
         (97, 101, 12, 15.0, 50_001, 8), (40, 41, 20, 20.0, 40_009, 8), (25, 24, 12, 20.0, 60_007, 8),
         (64, 60, 19, 20.0, 40_003, 8), (70, 66, 8, 20.0, 9_001, 16), (12, 12, 12, 50.0, 60_000, 16)]


@pytest.mark.parametrize("nx,ny,nz,mm,n_muons,group", SHORT)
def test_short_paths_match_oracle(gpu, oracle, nx, ny, nz, mm, n_muons, group):
    wl = scan(nx, ny, nz, mm, n_muons, 83)
    rays = wl.tracks()
    cfg = wl.em_config(update_with_mean=True, precision="mixed", compute_cost=True)
    ref = oracle.Mlsd(wl.grid, cfg, rays, np.full(wl.grid.nvox, 1e-7))
    ref.iterate(3)
    with M.MutoMLSD(cfg) as rec:
        img = rec.reconstruct(rays).reshape(-1, order="F")
        st = rec.status()
    assert st["muon_pass"] == 3 and st["muon_group"] == group
    assert st["n_singular"] == ref.counts()["n_singular"]
    assert rel_l2(img, ref.image()) < 2e-5
    assert abs(st["cost"] - ref.costs()[-1]) <= 1e-5 * abs(ref.costs()[-1])


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


@pytest.mark.parametrize("nx,ny,nz,mm,n_muons,group", [s for s in SHORT if s[5] < 16 and s[2] > 1])
def test_one_heavy_layer(gpu, nx, ny, nz, mm, n_muons, group):
    wl = scan(nx, ny, nz, mm, n_muons, 84)
    rays = wl.tracks()
    x = heavy_layer(wl, 0.9)
    v64, g64, _ = g_sums(wl, rays, x, "fp64")
    v, g, st = g_sums(wl, rays, x, "mixed")
    assert st["muon_group"] == group
    assert rel_l2(g, g64) < 1e-4 and abs(v - v64) <= 1e-4 * abs(v64)


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
