"""Tracks loaded from device memory right behind the work that writes them: the load is
ordered after everything queued on the default stream, for a handle and for every scan
of a batch.  The buffer holds other tracks until that work has run, so a load that
does not wait gives another image.

Tolerance: the FP64 form differs between runs by the order of its sums alone (1e-12).
"""
import numpy as np
import pytest
import torch

import muontomography_gb300 as M
from muontomography_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def queue_work():
    """Some 0.2 s of kernels on the default stream."""
    a = torch.full((4096, 4096), 1e-4, device="cuda")
    for _ in range(100):
        a = a @ a
    return a


def rel_l2(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


@pytest.mark.parametrize("stream", ["default", "side"])
def test_load_waits_for_the_default_stream(gpu, stream):
    wl = W.small(n_muons=20_000, seed=81)
    rays, other = wl.tracks(), W.small(n_muons=20_000, seed=82).tracks()
    cfg = wl.em_config(precision="fp64", num_iteration=3)
    with M.MutoMLSD(cfg) as rec:
        want = rec.reconstruct(rays)
    new, buf = torch.from_numpy(rays).cuda(), torch.from_numpy(other).cuda()
    with M.MutoMLSD(cfg) as rec:
        rec.load_tracks(None, buf.data_ptr(), buf.shape[0])  # (so that the load below finds its memory)
        torch.cuda.synchronize()
        if stream == "side":  # one that the default stream waits for
            side = torch.cuda.Stream()
            with torch.cuda.stream(side):
                queue_work()
                buf.copy_(new)
            torch.cuda.default_stream().wait_stream(side)
        else:
            queue_work()
            buf.copy_(new)
        rec.load_tracks(None, buf.data_ptr(), buf.shape[0])
        buf.zero_()  # the copy is complete when the load returns
        rec.prepare()
        rec.iterate(3)
        got = rec.image()
    assert rel_l2(got, want) < 1e-12


def test_batch_loads_wait_for_the_default_stream(gpu):
    wls = [W.small(n_muons=8000 + 3000 * k, seed=84 + k, n=8 + k) for k in range(3)]
    cfg = wls[0].em_config(precision="fp64", num_iteration=3)
    cfg.pop("grid")
    tracks = [wl.tracks() for wl in wls]
    grids = [wl.grid for wl in wls]
    with M.Batch(cfg, grids) as b:
        want = b.reconstruct_all(tracks)
    new = [torch.from_numpy(t).cuda() for t in tracks]
    buf = [torch.from_numpy(np.ascontiguousarray(t[::-1] * np.where(np.arange(14) < 2, 1.5, 1.0))).cuda() for t in tracks]
    with M.Batch(cfg, grids) as b:
        for k, t in enumerate(buf):
            b.load_scan(k, on_device_ptr=t.data_ptr(), n=t.shape[0])
        for k, t in enumerate(buf):
            torch.cuda.synchronize()
            queue_work()
            t.copy_(new[k])
            b.load_scan(k, on_device_ptr=t.data_ptr(), n=t.shape[0])
        b.prepare()
        b.iterate(3)
        got = [b.scan_image(k) for k in range(3)]
    for g, w in zip(got, want):
        assert rel_l2(g, w) < 1e-12
