"""The warp-batched muon pass with few muons: batches of 1 to 32 muons a warp and blocks of
32 to 256 threads (on 152 SMs the batch halves at 1 216, 2 432, .. 19 456 muons), in the
forms that run it: FP64 mean, medians in both precisions.  Kept muons 0.42 of the tracks.

Tolerances: as in test_gpu_parity.py, 1e-10 in FP64 and 1e-4 for mixed medians.
"""
import numpy as np
import pytest

import muontomography_gb300 as M
from muontomography_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_muons", [3, 20, 75, 80, 701, 1_430, 2_870, 2_920, 5_750, 11_590, 23_100, 46_400])
@pytest.mark.parametrize("precision,mean,tol", [("fp64", True, 1e-10), ("fp64", False, 1e-10), ("mixed", False, 1e-4)])
def test_every_batch_size_matches_oracle(gpu, oracle, n_muons, precision, mean, tol):
    wl = W.small(n_muons=n_muons, seed=91)
    rays = wl.tracks()
    cfg = wl.em_config(update_with_mean=mean, precision=precision, num_iteration=2, compute_cost=True)
    ref = oracle.Mlsd(wl.grid, cfg, rays, np.full(wl.grid.nvox, 1e-7))
    ref.iterate(2)
    want = ref.image()
    with M.MutoMLSD(cfg) as rec:
        img = rec.reconstruct(rays).reshape(-1, order="F")
        st = rec.status()
    assert st["n_scat_in_grid"] == ref.counts()["n_scat_in_grid"]
    assert np.linalg.norm(img - want) <= tol * np.linalg.norm(want)
    if st["n_scat_in_grid"]:
        assert abs(st["cost"] - ref.costs()[-1]) <= tol * abs(ref.costs()[-1])
