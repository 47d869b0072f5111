"""The mixed form's one-pass mean kernel (what fused_variant "auto" runs there):
16 lanes per muon up to a mean path of 160 pairs, 32 beyond, 8 pairs held per
lane.  Paths around the held ones and beyond them, muon counts that leave a
group, a warp or a block partly empty, and the cost of a pass against the FP64
oracle.

Tolerance: a pair's term and its sums are formed with about ten FP32 roundings
(6e-8 each); the sums over at most 2 000 pairs of a voxel and 600 of a muon add
terms of both signs, so a few hundred ulp (2e-5) after three iterations.
"""
import numpy as np
import pytest

import muontomography_gb300 as M
from muontomography_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def rel_l2(a, b):
    return float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300))


# (voxels a side, muons, lanes per muon): mean paths of 15 to 95 pairs (within the
# 128 held by 16 lanes, long ones beyond them), 170 to 250 (around the 256 of 32 lanes)
# and 300 (beyond); no kept muon, and counts that are not multiples of 2 or 8
@pytest.mark.parametrize("n,n_muons,group", [(12, 3, 16), (12, 37, 16), (12, 6001, 16), (24, 2003, 16), (48, 2001, 16),
                                             (64, 2002, 16), (110, 1203, 32), (140, 1001, 32), (170, 901, 32), (200, 801, 32)])
@pytest.mark.parametrize("cost", [False, True])
def test_one_pass_matches_oracle(gpu, oracle, n, n_muons, group, cost):
    wl = W.small(n_muons=n_muons, seed=53, n=n)
    rays = wl.tracks()
    cfg = wl.em_config(update_with_mean=True, mean_percentile=100, precision="mixed", num_iteration=3, compute_cost=cost)
    ref = oracle.Mlsd(wl.grid, cfg, rays, np.full(wl.grid.nvox, 1e-7))
    ref.iterate(3)
    with M.MutoMLSD(cfg) as rec:
        img = rec.reconstruct(rays).reshape(-1, order="F")
        st = rec.status()
    assert st["muon_pass"] == 3 and st["muon_group"] == group and st["n_singular"] == ref.counts()["n_singular"]
    assert rel_l2(img, ref.image()) < 2e-5
    if cost and st["n_scat_in_grid"]:  # (the mean over no muons is 0 / 0 in the oracle)
        assert abs(st["cost"] - ref.costs()[-1]) <= 1e-5 * abs(ref.costs()[-1])


def test_one_pass_without_muons(gpu):
    wl = W.small(n_muons=200, seed=54)
    rays = wl.tracks()
    rays[:, 2:4] += 1.0e5  # every line outside the grid
    rays[:, 5:7] += 1.0e5
    with M.MutoMLSD(wl.em_config(update_with_mean=True, precision="mixed", num_iteration=2)) as rec:
        img = rec.reconstruct(rays)
        assert rec.status()["n_scat_in_grid"] == 0 and not img.any()
