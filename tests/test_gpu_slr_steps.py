"""SLRIter's later passes in steps of at most 24 muons, 16 lanes a muon and a
thread a pair of 384: levels of several steps, muons of more than the 32 pairs held
per lane group and steps of more pairs than threads, the image in shared and in
global memory.

Tolerance: 1e-12, the bar of the other SLRIter tests: the FP64 sums and reciprocals
differ from the oracle's by a few ulp, of values that stay positive.
"""
import numpy as np
import pytest

import muontomography_gb300 as M
from muontomography_gb300 import workloads as W

pytestmark = pytest.mark.gpu


# 22^3 voxels: 2 V doubles still fit shared memory (those of 24^3, 221 KB, not on every part);
# 30^3 do not; 48^3: paths of 48 voxels and more, wide first levels
@pytest.mark.parametrize("n,n_muons", [(3, 301), (16, 25), (22, 3001), (30, 2003), (48, 4001)])
@pytest.mark.parametrize("lw,energy", [(True, True), (False, False)])
def test_slr_steps_match_oracle(gpu, oracle, n, n_muons, lw, energy):
    wl = W.small(n_muons=n_muons, seed=67, n=n)
    rays = wl.tracks()
    cfg = wl.poca_config(length_weighted=lw, has_energy=energy)
    cfg["num_iteration"] = 3
    ref = oracle.slr(wl.grid, cfg, rays, iterative=True)
    with M.MutoSLRIter(cfg) as rec:
        img = rec.reconstruct(rays).reshape(-1, order="F")
        assert rec.status()["slr_levels"] >= 1
    assert np.linalg.norm(img - ref) <= 1e-12 * np.linalg.norm(ref)
    assert np.array_equal(img > 0, ref > 0)
