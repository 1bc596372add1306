"""The kernels' own FP64 quotient, square root and reciprocals against IEEE's,
value by value.  The exact load build's bits rest on the quotient, which is to
be a / b for all operands; the square root is corrected to IEEE's rounding; a
reciprocal from the hardware's 20-bit seed by one third-order step is within 2
ulp (the seed's error cubed is below 2^-59, the step's own roundings add to 1)."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

QUOTIENT, SQRT, RSQRT, PIVOT = range(4)
INF, NAN, TINY, LEAST, MOST = np.inf, np.nan, np.finfo(float).tiny, 5e-324, np.finfo(float).max
EDGES = np.array([0.0, LEAST, 1e-310, TINY / 2, TINY, 2 * TINY, 1e-292, 1e-300, 1e-200, 1e-17, 1.0, 1.5, 2.0, 3.0,
                  np.nextafter(2.0, 0.0), np.nextafter(1.0, 2.0), 1e17, 1e200, 1e292, 1e300, 2.0**1022, 2.0**1023,
                  MOST / 3, MOST, INF, NAN])


def _run(lib, op, a, b):
    b = np.ascontiguousarray(b)
    a = np.ascontiguousarray(np.broadcast_to(a, b.shape))
    out = np.empty_like(b)
    p = [x.ctypes.data_as(C.c_void_p) for x in (a, b, out)]
    assert lib.xg_probe_arithmetic(op, b.size, *p) == 0
    return out


def _same_bits(got, want):
    nan = np.isnan(want)
    return np.array_equal(np.isnan(got), nan) and np.array_equal(got[~nan].view(np.int64), want[~nan].view(np.int64))


def _mantissas(rng, n):
    """Significands in [1, 2), a third of them next to either end."""
    m = rng.uniform(1.0, 2.0, n)
    k = rng.integers(0, 3, n)
    ulps = rng.integers(0, 64, n) * 2.0**-52
    return np.where(k == 0, 1.0 + ulps, np.where(k == 1, 2.0 - 2.0**-52 - ulps, m))


def test_quotients_of_edge_operands(engine_lib):
    e = np.r_[EDGES, -EDGES]
    a, b = (x.ravel() for x in np.meshgrid(e, e))
    with np.errstate(all="ignore"):
        assert _same_bits(_run(engine_lib, QUOTIENT, a, b), a / b)


@pytest.mark.parametrize("low,high", [(-40, 40), (-1074, 1023), (-1074, -950), (950, 1023)])
def test_quotients_of_random_operands(low, high, engine_lib):
    """Over the exponents that device values have, over all of them, and where
    quotients, remainders or reciprocals leave the normal numbers."""
    rng = np.random.default_rng(low + 5000)
    n = 4_000_000
    a, b = (np.ldexp(_mantissas(rng, n) * rng.choice([-1.0, 1.0], n), rng.integers(low, high + 1, n).astype(np.int32))
            for _ in range(2))
    with np.errstate(all="ignore"):
        assert _same_bits(_run(engine_lib, QUOTIENT, a, b), a / b)


def test_square_roots(engine_lib):
    rng = np.random.default_rng(1)
    n = 4_000_000
    b = np.r_[EDGES, -EDGES, np.ldexp(_mantissas(rng, n), rng.integers(-1074, 1024, n).astype(np.int32))]
    with np.errstate(all="ignore"):
        want = np.sqrt(b)
        assert _same_bits(_run(engine_lib, SQRT, 0.0, b), want)
        got, want = _run(engine_lib, RSQRT, 0.0, b), 1.0 / want
    ok = np.isfinite(want)
    assert _same_bits(got[~ok], want[~ok])
    assert np.all(np.abs(got[ok] - want[ok]) <= 2 * np.spacing(np.abs(want[ok])))


def test_pivot_reciprocals(engine_lib):
    rng = np.random.default_rng(2)
    n = 4_000_000
    b = np.r_[EDGES, -EDGES, np.ldexp(_mantissas(rng, n) * rng.choice([-1.0, 1.0], n),
                                      rng.integers(-1074, 1024, n).astype(np.int32))]
    got = _run(engine_lib, PIVOT, 0.0, b)
    with np.errstate(all="ignore"):
        want = 1.0 / b
    ok = np.isfinite(want)
    assert _same_bits(got[~ok], want[~ok])
    assert np.all(np.abs(got[ok] - want[ok]) <= 2 * np.spacing(np.abs(want[ok])))
