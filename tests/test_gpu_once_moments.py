"""The mixed form's one-pass mean kernel where one voxel holds most of a muon's sum
lambda L, as in sparse scans: Sigma is then nearly the matrix of one place on the
path, and the sums over a path's places have to be taken about that place for the
inverse to keep 32 bits.  And its rare branch, a determinant between the singular
threshold and twice it, whose terms come from the FP64 algebra, beside muons on
either side in the same warps.  Paths within the held pairs and beyond them, 16 and
32 lanes a muon.  Compared: the sums of g_ij per voxel (the gradient over lambda) of
the mixed form with the FP64 form's.

Tolerance: the places come in as 32-bit tails of up to 700 mm and the displacements as
32-bit values of that size times the angle: 2^-24 * 700 mm = 4e-5 mm, against a
spread of the path's places (the square root of Sigma11 / Sigma00 about their centre)
of 2 mm and more.  That is 2e-5 of an inverse's entry, twice it in the squared
forms, and as much again for the sums' own roundings: 1e-4.  (With sums taken about
the path's end the roundings count (500 mm / 2 .. 7 mm)^2 fold: 1e-3 and more.)
"""
import numpy as np
import pytest

import muontomography_gb300 as M
from muontomography_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def g_sums(wl, rays, x, precision, **over):
    cfg = wl.em_config(update_with_mean=True, precision=precision, num_iteration=0, **over)
    with M.MutoMLSD(cfg) as rec:
        rec.load_tracks(rays)
        rec.prepare()
        value, grad = rec.nll_grad(x)
        st = rec.status()
    assert precision == "fp64" or st["muon_pass"] == 3
    return value, grad / np.exp(x), st


def rel_l2(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


def layer_of(wl, height):
    n = wl.grid.nx
    return np.arange(wl.grid.nvox) // (n * n) == int(height * n)


@pytest.mark.parametrize("n,n_muons,group", [(24, 2003, 16), (48, 2001, 16), (64, 2002, 16), (140, 1001, 32), (200, 801, 32)])
@pytest.mark.parametrize("height", [0.95, 0.5, 0.08])
def test_one_heavy_layer(gpu, n, n_muons, group, height):
    wl = W.small(n_muons=n_muons, seed=71, n=n)
    rays = wl.tracks()
    x = np.full(wl.grid.nvox, np.log(1.0e-7))
    x[layer_of(wl, height)] = np.log(0.05)
    v64, g64, _ = g_sums(wl, rays, x, "fp64")
    v, g, st = g_sums(wl, rays, x, "mixed")
    assert st["muon_group"] == group
    assert rel_l2(g, g64) < 1e-4
    assert abs(v - v64) <= 1e-4 * abs(v64)


@pytest.mark.parametrize("n,n_muons", [(24, 2003), (64, 2002), (140, 1001), (200, 801)])
def test_determinants_next_to_the_threshold(gpu, oracle, n, n_muons):
    wl = W.small(n_muons=n_muons, seed=71, n=n)
    rays = wl.tracks()
    over = {"has_energy": False, "error_xy": 0.0}
    # lambda of one layer so that a steep muon's determinant, (lambda L^2)^2 / 12, lies
    # between 1e-12 and 2e-12
    lam = np.full(wl.grid.nvox, 1.0e-18)
    lam[layer_of(wl, 0.5)] = np.sqrt(1.45e-12 * 12) / (1.08 * 600.0 / n) ** 2
    e = oracle.Mlsd(wl.grid, wl.em_config(update_with_mean=True, **over), rays, lam).export()
    off, L = e["off"].astype(np.int64), e["len"]
    U, l = e["tail"] + L / 2, lam[e["idx"]]
    s = [np.add.reduceat(np.append(l * w, 0.0), off[:-1]) * (np.diff(off) > 0) for w in (L, L * U, L * (U * U + L * L / 12))]
    det = s[0] * s[2] - s[1] ** 2
    assert np.abs(det / 1e-12 - 1).min() > 1e-3  # no muon whose side rounding could choose
    shares = [(det < 1e-12).mean(), ((det > 1e-12) & (det < 2e-12)).mean(), (det > 2e-12).mean()]
    assert min(shares) > 0.03, shares
    x = np.log(lam)
    v64, g64, s64 = g_sums(wl, rays, x, "fp64", **over)
    v, g, st = g_sums(wl, rays, x, "mixed", **over)
    assert rel_l2(g, g64) < 1e-4
    assert abs(v - v64) <= 1e-4 * abs(v64)
