"""The plain bond order's FP64 reciprocal, inverse root, root and exponential
(csrc/md_exact64.cuh) against extended precision, in units in the last place.
Bars: half a unit for the last rounding and 0.02 for what comes before it (the
residual of a seed of 22 bits is cubed, below 2^-63; the exponential's sum before
its last addition is below 2^-7, rounded to 2^-60)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LD = np.longdouble


def _ulp(got, ref):
    return (np.abs(got.astype(LD) - ref) / np.spacing(np.abs(ref).astype(np.float64)).astype(LD)).max()


def test_reciprocal_roots_and_exponential(eng):
    rng = np.random.default_rng(5)
    n = 1 << 18
    # mantissas over and at the ends of the binade, exponents of both parities
    m = 1.0 + rng.random(n)
    m[:4096] = 1.0 + np.arange(4096) * 2.0 ** -52
    m[4096:8192] = 2.0 - np.arange(1, 4097) * 2.0 ** -52
    x = np.ldexp(m, rng.integers(-60, 60, n))
    y = rng.uniform(-160.0, 160.0, n)
    y[: n // 4] = rng.uniform(-6.0, 6.0, n // 4)
    # the ends of the table's intervals, the smallest arguments, zero
    k = np.arange(-4096, 4096) * (np.log(2.0) / 64)
    y[n // 4: n // 4 + 8192] = k
    y[n // 2: n // 2 + 8192] = k + np.log(2.0) / 128
    y[-2000:] = rng.uniform(-1.0, 1.0, 2000) * 10.0 ** rng.uniform(-300, -1, 2000)
    y[-1] = 0.0
    rcp, rsq, root, ex = eng.fp64_selftest(x, y)
    xl = x.astype(LD)
    assert _ulp(rcp, 1 / xl) < 0.52
    assert _ulp(rsq, 1 / np.sqrt(xl)) < 0.52
    assert _ulp(root, np.sqrt(xl)) < 0.52
    assert _ulp(ex, np.exp(y.astype(LD))) < 0.52
    assert ex[-1] == 1.0


def test_exponential_beyond_its_range(eng):
    # held at e^700 and e^-700; not a number stays one; the inverse root of 0
    y = np.array([699.9, 701.0, 1e9, np.inf, -699.9, -701.0, -1e9, -np.inf, np.nan])
    x = np.ones(len(y))
    x[0] = 0.0
    _, rsq, _, ex = eng.fp64_selftest(x, y)
    lim = np.exp(LD(700))
    assert abs(ex[0] / np.exp(LD(699.9)) - 1) < 1e-15 and abs(ex[4] * np.exp(LD(699.9)) - 1) < 1e-15
    assert (np.abs(ex[1:4] / lim - 1) < 0.02).all() and (np.abs(ex[5:8] * lim - 1) < 0.02).all()
    assert np.isnan(ex[8]) and np.isinf(rsq[0])
