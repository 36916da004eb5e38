"""Roots, reciprocals and reflectors of the FP64 column chain (tri_col.cuh) over the exponent range, against extended
precision and CUDA's own functions."""
import ctypes as C

import numpy as np
import pytest

from nrltb import abi

pytestmark = pytest.mark.gpu
L = np.longdouble
U = 2.0 ** -53


def _scalars(ctx, x, y, z):
    given = np.ascontiguousarray([x, y, z], float)
    out = np.empty((11, len(x)))
    rc = ctx.lib.nrltb_bench_fp64_scalars(ctx.h, len(x), C.c_void_p(given.ctypes.data), C.c_void_p(out.ctypes.data))
    assert rc == abi.NRLTB_OK
    return out


def _values(rng, count, low, high):
    return np.ldexp(rng.uniform(1.0, 2.0, count), rng.integers(low, high, count))


@pytest.mark.parametrize("low,high", [(-1074, -1000), (-1001, -990), (-600, 600), (-1, 2), (990, 1002), (1000, 1024)])
def test_roots_and_reciprocals(ctx, low, high):
    """Root and reciprocal end with one rounding of a corrected value, 2^-53 (1 + 2^-20) relative; the reciprocal root
    with that of the sum and half of that of its residual, 2^-52.  Outside 2^-1000 .. 2^1000 all three are CUDA's.
    (2^-1074: subnormals' own spacing on top.)"""
    rng = np.random.default_rng(low + 2000)
    x = _values(rng, 20000, low, high)
    s, r, q, cs, cr, cq = _scalars(ctx, x, 0 * x, 0 * x)[:6]
    with np.errstate(over="ignore", divide="ignore"):
        for got, cuda, want, bound in ((s, cs, np.sqrt(x.astype(L)), 1.000001 * U), (r, cr, 1 / np.sqrt(x.astype(L)), 2 * U),
                                       (q, cq, 1 / x.astype(L), 1.000001 * U)):
            outside = (x < 2.0 ** -1000) | (x >= 2.0 ** 1001)
            assert np.array_equal(got[outside], cuda[outside])
            ok = ~outside
            assert (np.abs(got[ok].astype(L) - want[ok]) <= bound * np.abs(want[ok]) + 2.0 ** -1074).all()


def test_special_values_are_cudas(ctx):
    x = np.array([0.0, np.inf, np.nan, 5e-324, 1.0, 4.0, 2.0 ** -1022, np.finfo(float).max, -3.0])
    out = _scalars(ctx, x, 0 * x, 0 * x)
    assert np.array_equal(out[0][:8], out[3][:8], equal_nan=True)
    assert np.array_equal(out[1][:8], out[4][:8], equal_nan=True)
    assert np.array_equal(out[2][[0, 1, 2, 3, 4, 5, 6, 7]], out[5][:8], equal_nan=True)
    assert abs(out[2][8] + 1 / 3) <= U   # the reciprocal keeps a sign


@pytest.mark.parametrize("centre,spread", [(c, s) for c in (-470, -100, 0, 100, 470) for s in (1, 30, 200)
                                           if abs(c) + s < 510])   # (squares in FP64's range)
def test_reflectors(ctx, spread, centre):
    """beta, tau and scale within the roundings of their formulas (a sum of three squares, a root, a reciprocal root,
    a sum, a sum of two squares and a reciprocal, their products): 2, 8 and 12 units; and H = 1 - tau v v^H unitary
    with H^H (al, x) = (beta, 0) within 16."""
    rng = np.random.default_rng(centre + 1000 + spread)
    n = 20000
    sign = rng.choice([-1.0, 1.0], (2, n))
    ar, ai, x = (_values(rng, n, centre - spread, centre + spread) for _ in range(3))
    ar, ai = ar * sign[0], ai * sign[1]
    xn2 = x * x
    ai[::7] = 0.0
    xn2[3::11] = 0.0
    tr, ti, sr, si, beta = (v.astype(L) for v in _scalars(ctx, ar, ai, xn2)[6:])
    a, b, q = ar.astype(L), ai.astype(L), xn2.astype(L)
    none = (q == 0) & (b == 0)
    assert (tr[none] == 0).all() and (beta[none] == a[none]).all()
    a, b, q, tr, ti, sr, si, beta = (v[~none] for v in (a, b, q, tr, ti, sr, si, beta))
    want = -np.copysign(np.sqrt(a * a + b * b + q), a)
    assert (np.abs(beta - want) <= 2 * U * np.abs(want)).all()
    assert (np.hypot(tr - (want - a) / want, ti + b / want) <= 8 * U * np.hypot((want - a) / want, b / want)).all()
    den = (a - want) ** 2 + b * b
    size = 1 / np.sqrt(den)
    assert (np.hypot(sr - (a - want) / den, si + b / den) <= 12 * U * size).all()
    # tau + conj tau = |tau|^2 |v|^2, v = (1, scale x)
    v2 = 1 + (sr * sr + si * si) * q
    t2 = tr * tr + ti * ti
    assert (np.abs(t2 * v2 - 2 * tr) <= 16 * U * np.maximum(2 * tr, t2 * v2)).all()
