"""A handle's set-up on its own stream: allocations in stream order, streams from a
pool shared by handles, a batch's scans spread over them, constant starts and
images converted on the device.

Tolerances: the FP64 form differs between runs by the order of its sums alone
(1e-12); the mixed form's likewise in FP32 (1e-6); an image that is set and read
back is rounded once at most, to the form's storage type (exact).
"""
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest

import muontomography_gb300 as M
from muontomography_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def rel_l2(a, b):
    a, b = np.asarray(a, np.float64).ravel(), np.asarray(b, np.float64).ravel()
    return float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300))


@pytest.mark.parametrize("update", [{}, {"update_with_mean": True}])
def test_many_handles_of_many_threads(gpu, update):
    # 12 threads (the pool keeps 8 sets of streams), six handles each one after the
    # other and two at once
    wls = [W.small(n_muons=1500 + 700 * k, seed=300 + k, n=5 + k) for k in range(12)]
    cfgs = [wl.em_config(precision="fp64", num_iteration=3, **update) for wl in wls]
    tracks = [wl.tracks() for wl in wls]

    def one(k):
        with M.MutoMLSD(cfgs[k]) as rec:
            return rec.reconstruct(tracks[k])

    def many(k):
        out = []
        for _ in range(3):
            with M.MutoMLSD(cfgs[k]) as a, M.MutoMLSD(cfgs[k]) as b:
                out += [a.reconstruct(tracks[k]), b.reconstruct(tracks[k])]
        return out

    want = [one(k) for k in range(12)]
    with ThreadPoolExecutor(12) as pool:
        got = list(pool.map(many, range(12)))
    for k in range(12):
        for img in got[k]:
            assert rel_l2(img, want[k]) < 1e-12


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-12), ("mixed", 1e-6)])
@pytest.mark.parametrize("update", [{}, {"update_with_mean": True}])
def test_batch_in_one_chunk_and_in_many(gpu, precision, tol, update):
    # scans of very different sizes, the second and the last without kept muons
    wls = [W.small(n_muons=m, seed=330 + k, n=n)
           for k, (m, n) in enumerate([(3000, 9), (10, 4), (40, 12), (9000, 7), (1, 6), (700, 20), (25, 5)])]
    tracks = [wl.tracks() for wl in wls]
    for k in (1, 6):  # every line outside the grid
        tracks[k][:, 2:4] += 1.0e5
        tracks[k][:, 5:7] += 1.0e5
    cfg = wls[0].em_config(precision=precision, num_iteration=3, initialize_method=2, **update)
    cfg.pop("grid")
    out = {}
    for chunk in (0, 500):  # 0: sized by the memory left, one chunk here
        with M.Batch(dict(cfg, **({"setup_chunk_pairs": chunk} if chunk else {})), [wl.grid for wl in wls]) as b:
            out[chunk] = b.reconstruct_all(tracks), [b.scan_info(k) for k in range(len(wls))]
    assert out[0][1] == out[500][1] and [out[0][1][k][0] for k in (1, 6)] == [0, 0]
    for k, wl in enumerate(wls):
        with M.MutoMLSD(dict(cfg, grid=wl.grid.json())) as rec:
            one = rec.reconstruct(tracks[k])
            st = rec.status()
        assert out[0][1][k] == (st["n_scat_in_grid"], st["n_pairs"])
        for chunk in out:
            assert rel_l2(out[chunk][0][k], one) < tol


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("n", [1, 3, 17, 64])
def test_starts_and_images_are_the_values_given(gpu, precision, n):
    wl = W.small(n_muons=300, seed=360, n=n)
    store = np.float64 if precision == "fp64" else np.float32
    cfg = wl.em_config(precision=precision, num_iteration=0, initialize_method=2, initialize_value=3.3e-7)
    with M.MutoMLSD(cfg) as rec:
        rec.load_tracks(wl.tracks())
        rec.prepare()
        assert np.array_equal(rec.image(), np.full((n, n, n), store(3.3e-7), np.float64))
        img = np.random.default_rng(n).uniform(1e-9, 1e-6, (n, n, n))
        rec.set_image(img)
        assert np.array_equal(rec.image(), img.astype(store).astype(np.float64))
