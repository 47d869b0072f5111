"""The MAP step against the FP64 oracle over its forms: powers 2, 1 and between
(each its own kernel), 6 and 26 neighbours, with and without the object prior, and
a Newton cap below the one at which the FP32 start is used.

Tolerance: 1e-9, the bar of the other MAP tests: the two sides round differently
by a few ulp a step, which p = 1 amplifies.
"""
import numpy as np
import pytest

import muontomography_gb300 as M
from muontomography_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("p", [2.0, 1.0, 1.5])
@pytest.mark.parametrize("every,objects", [(False, False), (True, False), (True, True)])
@pytest.mark.parametrize("beta,cap", [(0.01, 200), (3.0, 200), (0.01, 99)])
def test_map_step_matches_oracle(gpu, oracle, p, every, objects, beta, cap):
    wl = W.small(n_muons=5003, seed=61, n=11)
    rays = wl.tracks()
    cfg = wl.em_config(precision="fp64", num_iteration=3, newton_max_iter=cap)
    cfg.update(beta=beta, p=p, delta=0.1, all_neighbours=every, add_object_prior=objects)
    ref = oracle.Mlsd(wl.grid, cfg, rays, np.full(wl.grid.nvox, 1e-7), method="map")
    ref.iterate(3)
    with M.MutoMAP(cfg) as rec:
        img = rec.reconstruct(rays).reshape(-1, order="F")
        assert rec.status()["n_nonconverged"] == 0
    want = ref.image()
    assert np.linalg.norm(img - want) <= 1e-9 * np.linalg.norm(want)
