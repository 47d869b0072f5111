"""The mixed form's cost, four muons a thread with one logarithm, against the FP64
form's at the same image: muon counts around a thread's, a warp's and a block's
share (1 024 muons), and determinants small and large (with and without hit error).

Tolerance: a muon's sums carry about ten FP32 roundings, so its log det and its
quadratic form are 1e-6 off at most; the total adds terms of one size.
"""
import numpy as np
import pytest

import muontomography_gb300 as M
from muontomography_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_muons", [1, 2, 31, 33, 255, 257, 1023, 1024, 1025, 1500, 5003, 70_001])
@pytest.mark.parametrize("over", [{}, {"error_xy": 3.0}, {"error_xy": 0.0}])
def test_mixed_cost_matches_fp64(gpu, n_muons, over):
    wl = W.small(n_muons=n_muons, seed=61, n=6)
    rays = wl.tracks()
    f = {}
    for prec in ("fp64", "mixed"):
        with M.MutoMLSD(wl.em_config(precision=prec, num_iteration=0, update_with_mean=True, **over)) as rec:
            rec.load_tracks(rays)
            rec.prepare()
            x = np.full(wl.grid.nvox, np.log(1.3e-6))
            f[prec] = rec.nll(x), rec.status()["n_scat_in_grid"]
    assert f["mixed"][1] == f["fp64"][1]
    if f["fp64"][1]:
        assert abs(f["mixed"][0] - f["fp64"][0]) <= 1e-6 * max(abs(f["fp64"][0]), f["fp64"][1])
