"""The line fit's two ways to the principal axis (powers of the scatter matrix where
one eigenvalue stands out, rotations otherwise) against rotations in long double:
eigenvalue ratios from 0 across 0.09, where the powers stop, to 1; steep and almost
horizontal lines; two hits; hits in one point; scales of 1e-6 and 1e6; both record
types.

Tolerance: either way rounds the scatter matrix and the axis a few dozen times at
2^-53 of the largest eigenvalue, which turns the axis by at most that over the
relative gap 1 - ratio: 1e-14 / (1 - ratio); cases with a gap below 1e-3 have no
axis to compare.
"""
import numpy as np
import pytest

import muontomography_gb300 as M

pytestmark = pytest.mark.gpu


def axes(p):
    """Principal axes of the hits p (records, hits, 3), d_z >= 0, and the ratios of the
    two largest eigenvalues: rotations in long double (numpy's SVD is 1e-14 off)."""
    c = p.astype(np.longdouble)
    c = c - c.sum(axis=1, keepdims=True) / p.shape[1]
    a = np.einsum("nip,niq->pqn", c, c)
    v = np.zeros_like(a)
    for k in range(3):
        v[k, k] = 1
    for _ in range(15):
        for i, j in ((0, 1), (0, 2), (1, 2)):
            on = a[i, j] != 0
            with np.errstate(all="ignore"):
                th = (a[j, j] - a[i, i]) / (2 * np.where(on, a[i, j], 1))
                t = np.where(on, np.where(th >= 0, 1, -1) / (np.abs(th) + np.sqrt(th * th + 1)), 0)
            cs = 1 / np.sqrt(t * t + 1)
            sn = t * cs
            a[:, i], a[:, j] = cs * a[:, i] - sn * a[:, j], sn * a[:, i] + cs * a[:, j]
            a[i], a[j] = cs * a[i] - sn * a[j], sn * a[i] + cs * a[j]
            a[i, j] = a[j, i] = 0
            v[:, i], v[:, j] = cs * v[:, i] - sn * v[:, j], sn * v[:, i] + cs * v[:, j]
    lam = np.stack([a[k, k] for k in range(3)])
    order = np.argsort(lam, axis=0)
    d = np.take_along_axis(v, order[2][None, None], axis=1)[:, 0].T
    big, mid = (np.take_along_axis(lam, order[q][None], axis=0)[0] for q in (2, 1))
    return np.where(d[:, 2:] < 0, -d, d).astype(np.float64), (mid / np.where(big > 0, big, 1)).astype(np.float64)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("half", [2, 3, 4, 7])
@pytest.mark.parametrize("noise", [0.0, 1.0, 60.0, 150.0, 300.0, 900.0])
@pytest.mark.parametrize("slope", [0.0, 0.6, 3.0, 1e3, 1e8])
def test_axis_matches_rotations(gpu, dtype, half, noise, slope):
    rng = np.random.default_rng(17)
    n, nz = 300, 2 * half
    z = 500.0 * np.arange(nz)[::-1] - 100.0 * half
    phi = rng.uniform(0, 2 * np.pi, (n, 1))
    xy = [slope * f(phi) * z + rng.uniform(-1000, 1000, (n, 1)) + noise * rng.normal(size=(n, nz))
          for f in (np.cos, np.sin)]
    scale = [1e-6, 1.0, 1e6][(half + int(noise)) % 3]
    rec = np.empty((n, 2 * nz + 2))
    rec[:, 0] = rec[:, -1] = 3000.0
    rec[:, 1:-1:2], rec[:, 2:-1:2] = xy[0] * scale, xy[1] * scale
    rec = rec.astype(dtype)
    out = M.fit_tracks(rec, z * scale, n_middle=half)
    assert out.shape[0] == n
    for lo, cols in ((0, slice(8, 11)), (half, slice(11, 14))):
        pts = np.stack([rec[:, 1:-1:2], rec[:, 2:-1:2], np.broadcast_to(z * scale, (n, nz))], axis=2)
        want, ratio = axes(pts.astype(np.float64)[:, lo:lo + half])
        got = out[:, cols]
        flat = np.abs(want[:, 2]) < 1e-6  # (the sign is not settled)
        diff = np.abs(got - want).max(axis=1)
        diff = np.where(flat, np.minimum(diff, np.abs(got + want).max(axis=1)), diff)
        ok = 1.0 - ratio >= 1e-3
        assert np.all(diff[ok] <= 1e-14 / (1.0 - ratio[ok]))


def test_hits_in_one_point_and_bad_records(gpu):
    z = np.array([5.0, 5.0, 1.0, 1.0])  # both halves without extent
    rec = np.array([[1, 2, 3, 2, 3, 2, 3, 2, 3, 1], [1, np.nan, 3, 2, 3, 2, 3, 2, 3, 1]], np.float64)
    out = M.fit_tracks(rec, z, n_middle=2)
    assert out.shape[0] == 1 and np.isfinite(out[0, [0, 1]]).all()
