"""The FP64 form's passes over the muon-major lists: muons by decreasing path
length, W01 and W11 kept per pair, 4 lanes a muon up to a mean path of 80 pairs
and 8 beyond.  Against the FP64 oracle and through the path export, whose tails
are summed again from the lengths.

Tolerance: both sides are FP64 and differ in the order of their sums and in how
W11 is formed (a few ulp, 1e-15 relative, of terms that cancel by less than 1e3,
over three iterations): 1e-11.
"""
import numpy as np
import pytest

import muontomography_gb300 as M
from muontomography_gb300 import workloads as W

pytestmark = pytest.mark.gpu


# mean paths below and above 80 pairs; muon counts that leave a group, a warp or a
# block partly empty
@pytest.mark.parametrize("n,n_muons,group", [(12, 37, 4), (12, 6001, 4), (24, 2003, 4), (80, 1502, 8), (200, 401, 8)])
@pytest.mark.parametrize("update", ["mean", "median"])
def test_fp64_passes_match_oracle(gpu, oracle, n, n_muons, group, update):
    wl = W.small(n_muons=n_muons, seed=59, n=n)
    rays = wl.tracks()
    cfg = wl.em_config(update_with_mean=update == "mean", mean_percentile=100, precision="fp64", num_iteration=3,
                       compute_cost=True)
    ref = oracle.Mlsd(wl.grid, cfg, rays, np.full(wl.grid.nvox, 1e-7))
    ref.iterate(3)
    with M.MutoMLSD(cfg) as rec:
        img = rec.reconstruct(rays).reshape(-1, order="F")
        st, g = rec.status(), rec.export_paths()
    want = ref.image()
    assert st["muon_pass"] == (5 if update == "mean" else 2)
    if update == "median":
        assert st["muon_group"] == group
    assert np.linalg.norm(img - want) <= 1e-11 * np.linalg.norm(want)
    assert abs(st["cost"] - ref.costs()[-1]) <= 1e-11 * abs(ref.costs()[-1])
    r = ref.export()
    assert np.array_equal(g["off"], r["off"]) and np.array_equal(g["idx"], r["idx"])
    assert np.array_equal(g["len"].view(np.uint64), r["len"].view(np.uint64))
    assert np.array_equal(g["tail"].view(np.uint64), r["tail"].view(np.uint64))
