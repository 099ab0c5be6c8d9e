"""The product build's reciprocal, reciprocal square root, square root and
quotient (physics.cuh) against 80-bit arithmetic and against CUDA's own
operators (the parity build's), over the exponent range and at its ends.

Bounds, in units in the last place of the result.  rcp, sqrt and div end in one
rounding of a value whose own error is of second order: 0.5 and less than 0.01.
rsqrt corrects with e = 1 - fl(a y) y, whose rounding is 2^-53 of 1 and enters
with the factor 1/2: up to 0.5 more.  CUDA's division and square root are
correctly rounded, so the first three differ from them by one ulp at most; its
1 / sqrt(a) has two roundings (1 ulp), so rsqrt by two."""
import numpy as np
import pytest

from echo_gpu.lib import unit_recip

pytestmark = pytest.mark.gpu

RCP, RSQRT, SQRT, DIV, RCP_N, RSQRT_N, SQRT_N = range(7)
BOUND = {RCP: 0.51, RSQRT: 1.01, SQRT: 0.51, DIV: 0.51, RCP_N: 0.51, RSQRT_N: 1.01, SQRT_N: 0.51}
N = 1 << 20


def _log(rng, lo, hi, n=N):
    """Random mantissas with exponents spread over 2^lo .. 2^hi."""
    return np.ldexp(rng.uniform(1.0, 2.0, n), rng.integers(lo, hi, n))


def _operands(op):
    rng = np.random.default_rng(17 + op)
    sign = rng.choice([-1.0, 1.0], N)
    b = np.ones(N)
    if op in (RCP, RCP_N):
        # everything; determinants of both signs are among it
        a = _log(rng, -1021, 1021) * sign
        # denominators of the WENO weights, from 1e-42 up
        a[: N // 4] = 10.0 ** rng.uniform(-42, 60, N // 4)
        # 1 - v^2 and 1 - x: multiples of 2^-53
        a[N // 4: N // 2] = np.ldexp(rng.integers(1, 1 << 53, N // 4).astype(np.float64), -53)
        a[N // 2: N // 2 + 4096] = np.ldexp(np.arange(1, 4097, dtype=np.float64), -53)
    elif op in (RSQRT, RSQRT_N):
        a = _log(rng, -1021, 1023)
        a[: N // 2] = np.ldexp(rng.integers(1, 1 << 53, N // 2).astype(np.float64), -53)
        a[N // 2: N // 2 + 4096] = np.ldexp(np.arange(1, 4097, dtype=np.float64), -53)
    elif op in (SQRT, SQRT_N):
        a = _log(rng, -963, 1023)  # 2^-963 = 1.3e-290
        a[: N // 2] = rng.uniform(0.0, 1.0, N // 2)
        a[0] = 1e-290
    else:
        a = _log(rng, -400, 400) * sign
        b = _log(rng, -400, 400) * rng.choice([-1.0, 1.0], N)
        # speeds: sums and 1 - v^2 a^2 of order one
        a[: N // 2] = rng.uniform(1e-6, 2.0, N // 2)
        b[: N // 2] = rng.uniform(0.0, 2.0, N // 2)
        b[: N // 4] = 1.0
    return a, b


def _true(op, a, b):
    x, y = a.astype(np.longdouble), b.astype(np.longdouble)
    if op == DIV:
        return y / x
    if op in (SQRT, SQRT_N):
        return np.sqrt(x)
    return 1 / (x if op in (RCP, RCP_N) else np.sqrt(x))


@pytest.mark.parametrize("op", list(BOUND))
def test_within_the_stated_ulps(op):
    assert np.finfo(np.longdouble).nmant >= 63
    a, b = _operands(op)
    got, cuda, ref = unit_recip(op, a, b), unit_recip(op, a, b, exact=True), _true(op, a, b)
    ulp = np.spacing(np.abs(ref).astype(np.float64)).astype(np.longdouble)
    err = np.abs(got.astype(np.longdouble) - ref) / ulp
    apart = np.abs(got - cuda) / ulp.astype(np.float64)
    print(op, f"{float(err.max()):.4f} ulp, {float(apart.max()):.1f} from CUDA's")
    assert np.isfinite(got).all()
    assert err.max() <= BOUND[op] and apart.max() <= (2 if op in (RSQRT, RSQRT_N) else 1)


def _same(x, y):
    return np.array_equal(np.isnan(x), np.isnan(y)) and np.array_equal(x[~np.isnan(x)], y[~np.isnan(y)])


def test_ends_are_the_operators_own():
    """0, infinity, NaN (and negative square roots) as CUDA's operators."""
    a = np.array([0.0, -0.0, np.inf, -np.inf, np.nan])
    got, cuda = unit_recip(RCP, a), unit_recip(RCP, a, exact=True)
    assert _same(got, cuda) and np.array_equal(np.signbit(got[:4]), np.signbit(cuda[:4]))
    s = np.array([0.0, np.inf, np.nan, -1.0, -np.inf])
    assert _same(unit_recip(RSQRT, s), unit_recip(RSQRT, s, exact=True))
    assert _same(unit_recip(SQRT, s), unit_recip(SQRT, s, exact=True))


def test_subnormals_count_as_zero():
    a = np.array([5e-324, 2.0**-1023, 1.9 * 2.0**-1023, -2.0**-1040])
    assert np.array_equal(unit_recip(RCP, a), np.copysign(np.inf, a))
    big = np.array([1.5 * 2.0**1022, 2.0**1023, np.finfo(float).max, -np.finfo(float).max])
    assert np.array_equal(unit_recip(RCP, big), np.zeros(4))
    assert np.array_equal(unit_recip(RSQRT, a[:3]), np.full(3, np.inf))
    for op in (SQRT, SQRT_N):
        assert np.array_equal(unit_recip(op, np.array([0.0, 5e-324, 2.0**-1023, 1e-300, 9e-291])), np.zeros(5))
