"""Grids of up to four layers: bricks half as high.  Memory against twice the layers', the
exported paths (bricked and back) bit for bit the oracle's, and images.

Tolerance: 1e-10 in FP64, as in test_gpu_parity.py.
"""
import numpy as np
import pytest

import muontomography_gb300 as M
from muontomography_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def scan(nx, ny, nz, n_muons=3_000):
    g = M.Grid(nx, ny, nz, -300.0, -300.0, -300.0, 600.0 / nx, 600.0 / ny, 600.0 / nz)
    return W.Workload("scan", g, [M.Block((-100.0, -100.0, -100.0), (100.0, 100.0, 100.0), M.X0_MM["iron"])], n_muons, 97, True, 3)


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
def test_no_memory_for_absent_layers(gpu, precision):
    held = {}
    for nz in (4, 8):
        wl = scan(512, 512, nz, 2)
        with M.MutoMLSD(wl.em_config(update_with_mean=True, precision=precision)) as rec:
            rec.load_tracks(wl.tracks())
            rec.prepare()
            held[nz] = rec.status()["device_bytes"]
    assert held[4] < 0.55 * held[8]


@pytest.mark.parametrize("nx,ny,nz", [(7, 5, 1), (4, 4, 2), (9, 6, 3), (10, 13, 4), (9, 6, 5), (8, 8, 8)])
def test_paths_and_images(gpu, oracle, nx, ny, nz):
    wl = scan(nx, ny, nz)
    rays = wl.tracks()
    cfg = wl.em_config(update_with_mean=True, precision="fp64")
    ref = oracle.Mlsd(wl.grid, cfg, rays, np.full(wl.grid.nvox, 1e-7))
    want = ref.export()
    with M.MutoMLSD(cfg) as rec:
        rec.load_tracks(rays)
        rec.prepare()
        got = rec.export_paths()
        rec.iterate(3)
        img = rec.image().reshape(-1, order="F")
    assert np.array_equal(got["idx"], want["idx"]) and np.array_equal(got["len"], want["len"])
    ref.iterate(3)
    assert np.linalg.norm(img - ref.image()) <= 1e-10 * np.linalg.norm(ref.image())
