"""The pair kernels' FP64 reciprocal, logarithm, angle and inverse powers against extended precision.

Bounds, in units in the last place of the exact value: a reciprocal's iteration leaves e^3 = 2^-60
and one rounding, 0.6; the logarithm's leading sum is exact and its polynomial and last sum round once each, 1; the
angle's quotient, polynomial and two sums, 2; x^(-3/2) rounds the guess's cube and the last
fused step, 1.5; x^(-5/2) one product more, 2.5. Outside their ranges the functions hand over to
the library's: division (0.5), log and atan2 (2), and products of rsqrt (2 ulp, three or
five times, with two or three roundings: 8 and 13).
"""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
LD = np.longdouble


def _call(fn, x, y=None):
    from mbem_gb300 import _native as nat
    from mbem_gb300._device import ptr, stream_handle
    xd = torch.from_numpy(np.ascontiguousarray(x)).cuda()
    yd = torch.from_numpy(np.ascontiguousarray(y)).cuda() if y is not None else None
    out = torch.full_like(xd, 7.0)
    nat.call("mbem_dp_math_probe", fn, ptr(xd), ptr(yd), xd.numel(), ptr(out), stream_handle())
    return out.cpu().numpy()


def _ulps(got, ref):
    """|got - ref| in ulps of ref (longdouble); results that round to infinity or zero have to be that."""
    with np.errstate(all="ignore"):
        r64 = ref.astype(np.float64)
        unit = np.maximum(np.spacing(np.abs(np.where(np.isfinite(r64), r64, 1.0))), 5e-324).astype(LD)
        err = np.abs((got.astype(LD) - ref) / unit).astype(float)
    same = (got == r64) | (np.isnan(got) & np.isnan(r64))
    return np.where(same, np.minimum(np.nan_to_num(err, nan=0.0, posinf=0.0), 0.5), np.nan_to_num(err, nan=np.inf))


def _all_exponents(rng, n):
    return rng.choice([-1.0, 1.0], n) * np.ldexp(rng.uniform(0.5, 1.0, n), rng.integers(-1073, 1025, n).astype(np.int32))


def _around(values):
    v = np.asarray(values, np.float64)
    with np.errstate(over="ignore"):
        return np.concatenate([v, np.nextafter(v, np.inf), np.nextafter(v, -np.inf)])


SPECIAL = np.array([0.0, -0.0, 5e-324, -5e-324, 1e-310, -1e-310, 2.2250738585072014e-308, 1.7976931348623157e308, np.inf,
                    -np.inf, np.nan, 1.0, -1.0])


def _guards(lo, hi):
    """Both sides of an exponent guard [lo, hi)."""
    return _around([2.0 ** (lo - 1023), 2.0 ** (hi - 1023) if hi < 2047 else np.finfo(float).max])


def test_reciprocal(gpu):
    rng = np.random.default_rng(0)
    x = np.concatenate([SPECIAL, _guards(64, 1984), rng.uniform(0.5, 2.0, 200_000), _all_exponents(rng, 200_000)])
    with np.errstate(all="ignore"):
        ref = LD(1) / x.astype(LD)
    e = _ulps(_call(0, x), ref)
    assert e.max() <= 0.6, (e.max(), x[e.argmax()])


def test_logarithm(gpu):
    rng = np.random.default_rng(1)
    seams = np.concatenate([(1 + np.arange(129) / 128) * s for s in (0.5, 1.0, 2.0)])     # the table's intervals
    x = np.concatenate([SPECIAL, _guards(1, 2047), _around(seams), _around([1.4140625, 0.70703125]),
                        1.0 + rng.choice([-1, 1], 100_000) * 10.0 ** rng.uniform(-16, -1.5, 100_000),
                        rng.uniform(0.5, 2.0, 200_000), _all_exponents(rng, 200_000)])
    with np.errstate(all="ignore"):
        ref = np.log(x.astype(LD))
    e = _ulps(_call(1, x), ref)
    inside = x >= 2.0 ** -1022
    assert e[inside].max() <= 1.0, (e[inside].max(), x[inside][e[inside].argmax()])
    assert e.max() <= 2.0, (e.max(), x[e.argmax()])


def test_angle(gpu):
    rng = np.random.default_rng(2)
    n = 200_000
    q = np.concatenate([_around((np.arange(65) + h) / 64) for h in (-0.5, 0.0, 0.5)])     # the table's points and seams
    q = np.tile(np.abs(q), 8)
    k = np.arange(q.size) // (q.size // 8)
    sx, sy = np.where(k & 1, -1.0, 1.0), np.where(k & 2, -1.0, 1.0)
    a, b = sx * np.where(k & 4, q, 1.0), sy * np.where(k & 4, 1.0, q)
    g = np.concatenate([_guards(64, 1984), 2.0 ** np.arange(-25.0, 25.0), SPECIAL])
    gx, gy = (v.ravel() for v in np.meshgrid(np.concatenate([g, -g]), np.concatenate([g, -g])))
    th = rng.uniform(-np.pi, np.pi, n)
    x = np.concatenate([a, gx, np.cos(th), _all_exponents(rng, n), rng.normal(size=n)])
    y = np.concatenate([b, gy, np.sin(th), _all_exponents(rng, n), rng.normal(size=n) * 10.0 ** rng.uniform(-12, 0, n)])
    got = _call(2, x, y)
    ref = np.arctan2(y.astype(LD), x.astype(LD))
    e = _ulps(got, ref)
    assert e.max() <= 2.0, (e.max(), y[e.argmax()], x[e.argmax()])
    zero = ref == 0
    assert np.array_equal(np.signbit(got[zero]), np.signbit(y[zero]))


@pytest.mark.parametrize("m,inside,outside", [(3, 1.5, 8.0), (5, 2.5, 13.0)])
def test_inverse_powers(gpu, m, inside, outside):
    rng = np.random.default_rng(m)
    x = np.concatenate([SPECIAL, _guards(640, 1408), rng.uniform(0.25, 4.0, 200_000), np.abs(_all_exponents(rng, 200_000))])
    with np.errstate(all="ignore"):
        v = x.astype(LD)
        ref = (1 / np.sqrt(v)) ** m              # -0: minus infinity, as the reciprocal root
    e = _ulps(_call(3 if m == 3 else 4, x), ref)
    mid = (x >= 2.0 ** -383) & (x < 2.0 ** 385)
    assert e[mid].max() <= inside, (e[mid].max(), x[mid][e[mid].argmax()])
    out = x[~mid]
    assert e[~mid].max() <= outside, (e[~mid].max(), out[e[~mid].argmax()])
