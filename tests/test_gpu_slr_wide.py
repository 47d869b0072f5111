"""SLRIter's later passes with the image in global memory: steps of at most 64 muons on
1 024 threads.  The smallest grid that leaves shared memory, levels of several steps
with short paths on a flat grid, levels of a few muons, and long paths of which a step
holds many times the block's threads.

Tolerance: 1e-12, the bar of the other SLRIter tests: the FP64 sums and reciprocals
differ from the oracle's by a few ulp, of values that stay positive.
"""
import numpy as np
import pytest

import muontomography_gb300 as M
from muontomography_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def workload(nx, ny, nz, n_muons):
    g = M.Grid(nx, ny, nz, -300.0, -300.0, -300.0, 600.0 / nx, 600.0 / ny, 600.0 / nz)
    return W.Workload("slr", g, W.small().blocks, n_muons, 101, True, 5)


@pytest.mark.parametrize("nx,ny,nz,n_muons", [(25, 25, 25, 3001), (70, 61, 4, 20_011), (3, 3, 1700, 403),
                                              (110, 110, 110, 700), (40, 40, 40, 64)])
@pytest.mark.parametrize("lw,energy", [(True, True), (False, False)])
def test_wide_steps_match_oracle(gpu, oracle, nx, ny, nz, n_muons, lw, energy):
    wl = workload(nx, ny, nz, n_muons)
    rays = wl.tracks()
    cfg = wl.poca_config(length_weighted=lw, has_energy=energy)
    cfg["num_iteration"] = 3
    ref = oracle.slr(wl.grid, cfg, rays, iterative=True)
    with M.MutoSLRIter(cfg) as rec:
        img = rec.reconstruct(rays).reshape(-1, order="F")
    assert np.linalg.norm(img - ref) <= 1e-12 * np.linalg.norm(ref)
    assert np.array_equal(img > 0, ref > 0)
