"""The mixed form's lists from the walked slots, two pairs a store, two or four
lengths a lane in the scan of the tails (by the mean path's bound), in one chunk and
in chunks of odd sizes.

Tolerance: the lists are the oracle's FP64 ones rounded to FP32, bit for bit.
"""
import numpy as np
import pytest

import muontomography_gb300 as M
from muontomography_gb300 import workloads as W

pytestmark = pytest.mark.gpu


# mean paths of 1 to 40 pairs (two a lane: tiles of 64), around the rule's 112, and
# beyond it (four a lane: tiles of 128; paths of two to four tiles)
@pytest.mark.parametrize("n,n_muons", [(1, 40), (8, 901), (24, 900), (48, 601), (64, 600), (100, 500), (170, 301)])
@pytest.mark.parametrize("chunk", [0, 1501, 4096])
def test_lists_are_the_rounded_oracle_lists(gpu, oracle, n, n_muons, chunk):
    wl = W.small(n_muons=n_muons, seed=97, n=n)
    rays = wl.tracks()
    cfg = wl.em_config(precision="mixed", update_with_mean=True)
    r = oracle.Mlsd(wl.grid, cfg, rays, np.full(wl.grid.nvox, 1e-7)).export()
    with M.MutoMLSD(dict(cfg, **({"setup_chunk_pairs": chunk} if chunk else {}))) as rec:
        rec.load_tracks(rays)
        rec.prepare()
        g = rec.export_paths()
    assert np.array_equal(g["off"], r["off"]) and np.array_equal(g["idx"], r["idx"])
    for key in ("len", "tail"):
        assert np.array_equal(g[key], r[key].astype(np.float32).astype(np.float64)), key
