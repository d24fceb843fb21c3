"""The scalar arithmetic that the factorizations use in place of the compiler's FP64
quotient, reciprocal square root and square root."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _run(sylver, op, a, b=None):
    a = np.ascontiguousarray(a, dtype=np.float64)
    b = a if b is None else np.ascontiguousarray(b, dtype=np.float64)
    out = np.empty_like(a)
    rc = sylver.load().sylver_gb300_pivot_math(op, a.size, a.ctypes.data, b.ctypes.data,
                                               out.ctypes.data)
    assert rc == 0
    return out


def _mantissas(rng, n):
    """Mantissas in [1, 2): random, few bits set at either end, and next to the powers."""
    m = rng.integers(0, 1 << 52, n, dtype=np.int64)
    k = n // 8
    m[:k] = rng.integers(0, 16, k)                          # just above 1
    m[k:2 * k] = (1 << 52) - 1 - rng.integers(0, 16, k)     # just below 2
    m[2 * k:3 * k] = rng.integers(0, 1 << 26, k) << 26      # short: quotients and ties
    m[3 * k:4 * k] = 1 << rng.integers(0, 52, k)
    return m


def _assemble(exp, mant, sign=0):
    return ((sign << 63) | (exp << 52) | mant).astype(np.int64).view(np.float64)


def test_quotient_is_ieee(sylver, gpu):
    rng = np.random.default_rng(1)
    n = 1 << 22
    a = _assemble(rng.integers(900, 1150, n), _mantissas(rng, n), rng.integers(0, 2, n))
    b = _assemble(rng.integers(900, 1150, n), rng.permutation(_mantissas(rng, n)),
                  rng.integers(0, 2, n))
    # quotients next to 1, and exactly halfway between two doubles: (odd / 2^53) b has 54
    # bits for a b of one bit; a = q b rounded for the others lands beside a tie
    b[: n // 8] = a[: n // 8] * (1 + rng.integers(-8, 9, n // 8) * 2.0 ** -52)
    q = 1 + rng.integers(0, 1 << 27, n // 8) * 2.0 ** -27
    a[n // 8: n // 4] = b[n // 8: n // 4] * q
    assert np.array_equal(_run(sylver, 0, a, b).view(np.int64), (a / b).view(np.int64))


def test_quotient_at_the_limits(sylver, gpu):
    """All pairs of operands at the ends of the exponent range (subnormal and infinite
    quotients, where the division itself takes over), zeros, infinities and NaN."""
    rng = np.random.default_rng(2)
    exps = np.array([0, 1, 2, 3, 52, 53, 54, 510, 1021, 1022, 1023, 1024, 1025, 1535, 1536, 1992,
                     2043, 2044, 2045, 2046])
    m = _mantissas(rng, 16 * exps.size).reshape(exps.size, 16)
    v = _assemble(np.repeat(exps, 16), m.ravel())
    v = np.concatenate([v, -v[::5], [0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324]])
    a, b = (x.ravel() for x in np.meshgrid(v, v))
    with np.errstate(all="ignore"):
        ref = a / b
    got = _run(sylver, 0, a, b)
    nan = np.isnan(ref)
    assert np.array_equal(np.isnan(got), nan)
    assert np.array_equal(got[~nan].view(np.int64), ref[~nan].view(np.int64))


def _ulps(got, ref):
    """Error in units of the last place of got (ref: long double)."""
    return float((np.abs(got.astype(np.longdouble) - ref) / np.spacing(got)).max())


def test_fp64_roots(sylver, gpu):
    rng = np.random.default_rng(3)
    n = 1 << 20
    d = _assemble(rng.integers(1, 2047, n), _mantissas(rng, n))
    d[: 1 << 17] = np.ldexp(1.0 + rng.integers(-64, 65, 1 << 17) * 2.0 ** -52,
                            2 * rng.integers(-500, 500, 1 << 17))  # around powers of four
    s = np.sqrt(d.astype(np.longdouble))
    # 2^-57.8 of the value before the rounding: half an ulp and 2^(53 - 57.8)
    assert _ulps(_run(sylver, 1, d), 1 / s) <= 0.5 + 2.0 ** -4.8
    big = d >= 2.0 ** -960  # the remainder d - s^2 has all its bits
    assert _ulps(_run(sylver, 2, d)[big], s[big]) <= 0.51
    assert _ulps(_run(sylver, 2, d), s) <= 2.0
    sub = _assemble(np.zeros(4096, np.int64), np.maximum(_mantissas(rng, 4096), 1))
    assert _ulps(_run(sylver, 1, sub), 1 / np.sqrt(sub.astype(np.longdouble))) <= 1.5
    assert _ulps(_run(sylver, 2, sub), np.sqrt(sub.astype(np.longdouble))) <= 2.0
    assert _run(sylver, 1, [np.inf])[0] == 0.0 and _run(sylver, 2, [np.inf])[0] == np.inf


def test_fp32_roots(sylver, gpu):
    rng = np.random.default_rng(4)
    bits = np.concatenate([rng.integers(1 << 23, 0xff << 23, 1 << 21),
                           np.arange(127 << 23, (127 << 23) + (1 << 20)),
                           np.arange((129 << 23) - (1 << 20), 129 << 23)]).astype(np.uint32)
    d = bits.view(np.float32)
    s = np.sqrt(d.astype(np.longdouble))
    got = _run(sylver, 3, d.astype(np.float64)).astype(np.float32)
    assert _ulps(got, 1 / s) <= 0.5001
    got = _run(sylver, 4, d.astype(np.float64)).astype(np.float32)
    big = d >= 2.0 ** -100
    assert _ulps(got[big], s[big]) <= 0.51
    assert _ulps(got, s) <= 2.0
    assert _run(sylver, 3, [np.inf])[0] == 0.0 and _run(sylver, 4, [np.inf])[0] == np.inf
