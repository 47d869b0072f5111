"""The prior of the MAP objective and its gradient against a scatter over all stencil
terms in numpy, on grids whose edges clamp in every combination (sides of one and
two voxels among them), for the three forms of the power.

The prior is the objective of a MAP handle minus that of an MLSD handle on the same
tracks, FP64 form.  Tolerance: both likelihood parts are sums in FP64 whose order
changes between runs (a few 1e-16 of their size), the prior's sums have at most
V * 27 terms of a few roundings each: 1e-12 of the larger of prior and likelihood.
"""
import itertools

import numpy as np
import pytest

import muontomography_gb300 as M
from muontomography_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def scatter_prior(lam, mult, n, beta, p, delta, all_nb, obj):
    nx, ny, nz = n
    l = lam.reshape(n, order="F") * 1e7
    dl = np.zeros(n)
    value = 0.0
    idx = np.indices(n)
    for off in itertools.product((-1, 0, 1), repeat=3):
        kind = sum(o != 0 for o in off)
        if kind == 0 or (kind > 1 and not all_nb):
            continue
        w = 1.0 / np.sqrt(float(kind))
        m = tuple(np.clip(idx[k] + off[k], 0, n[k] - 1) for k in range(3))
        t = l - l[m]
        u = t * t + delta * delta
        value += 2 * beta * w * np.sum(u ** (p / 2))
        s = 2 * beta * w * p * t * u ** ((p - 2) / 2)
        dl += s
        np.add.at(dl, m, -s)
    if obj:
        u = l * l + delta * delta
        value += 2 * beta * np.sum(u ** (p / 2))
        dl += 2 * beta * p * l * u ** ((p - 2) / 2)
    return value, np.where(mult > 0, l.ravel(order="F") * dl.ravel(order="F"), 0.0)


@pytest.mark.parametrize("n", [(1, 1, 1), (2, 1, 3), (1, 5, 2), (7, 3, 6), (33, 9, 5), (96, 70, 11), (101, 97, 67)])
@pytest.mark.parametrize("p,all_nb,obj", [(2.0, True, True), (2.0, False, False), (1.0, True, False),
                                          (1.0, False, True), (1.4, True, True)])
def test_prior_matches_the_scatter(gpu, n, p, all_nb, obj):
    g = M.Grid(*n, *(-50.0 * k for k in n), 100.0, 100.0, 100.0)
    wl = W.Workload("p", g, [], 400, 7, True, 0)
    rays = wl.tracks()
    beta, delta = 0.3, 0.2
    cfg = wl.em_config(precision="fp64", num_iteration=0)
    with M.MutoMAP(dict(cfg, beta=beta, p=p, delta=delta, all_neighbours=all_nb, add_object_prior=obj)) as a, \
            M.MutoMLSD(cfg) as b:
        for rec in (a, b):
            rec.load_tracks(rays)
            rec.prepare()
        mult = a.multiplicity()
        x = np.log(1e-7 * np.random.default_rng(11).uniform(0.3, 6.0, g.nvox))
        fa, ga = a.nll_grad(x)
        fb, gb = b.nll_grad(x)
        only = a.nll(x)
    value, grad = scatter_prior(np.where(mult > 0, np.exp(x), 0.0), mult, n, beta, p, delta, all_nb, obj)
    assert abs((fa - fb) - value) <= 1e-12 * max(abs(value), abs(fb), abs(fa))
    assert abs(only - fa) <= 1e-12 * max(abs(fa), abs(fb), abs(value))
    scale = max(np.abs(grad).max(), np.abs(gb).max())
    assert np.abs((ga - gb) - grad).max() <= 1e-12 * scale
