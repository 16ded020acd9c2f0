"""The kernels' own reciprocal, square root, polynomials of the logarithmic mean and
FP32 quotient against values of 80 bits or 40 digits, over the ranges that their
comments state."""
import numpy as np
import pytest

from test_log_means import device_math

pytestmark = pytest.mark.gpu

RCP, SQRT, MEAN_F, MEAN_GH, MEAN_F_WIDE, DIV32 = 1, 2, 3, 4, 5, 6


def ulps(got, want):
    """Distance in units of the result's last place; ``want`` in 80 bits."""
    return np.abs(got.astype(np.longdouble) - want) / np.spacing(np.abs(got)).astype(np.longdouble)


def samples(lo, hi, n=200000, seed=5):
    rng = np.random.default_rng(seed)
    x = np.ldexp(rng.uniform(1, 2, n), rng.integers(lo, hi, n))
    edge = np.concatenate([np.ldexp(1 + k * np.finfo(float).eps, e) for k in (0, 1, 2, 3, 2 ** 51, 2 ** 52 - 2, 2 ** 52 - 1)
                           for e in (np.arange(lo, hi),)])
    return np.concatenate([x, edge])


@pytest.mark.skipif(np.finfo(np.longdouble).nmant < 63, reason="needs 80-bit long doubles")
def test_reciprocal_and_square_root():
    # the seed's error cubed is under 2^-60, the last operation rounds once: 0.51 ulp
    x = samples(-1021, 1021)
    for v in (x, -x):
        assert ulps(device_math(RCP, v, v), 1 / v.astype(np.longdouble)).max() <= 0.51
    x = samples(-968, 1023)
    assert ulps(device_math(SQRT, x, x), np.sqrt(x.astype(np.longdouble))).max() <= 0.51
    # below, the residual of the last correction underflows: half a place more at most
    x = samples(-1022, -968)
    assert ulps(device_math(SQRT, x, x), np.sqrt(x.astype(np.longdouble))).max() <= 1.0
    x = np.array([0.0, -0.0, -1.0, -1e-300, np.nan])
    assert np.array_equal(device_math(SQRT, x, x), [0.0, 0.0, np.nan, np.nan, np.nan], equal_nan=True)


@pytest.mark.parametrize("fn,top,half", [(MEAN_F, 0.00826, False), (MEAN_GH, 0.00826, True), (MEAN_F_WIDE, 0.25, False)])
def test_mean_polynomials(fn, top, half):
    """F(u) = atanh(sqrt u) / sqrt u, or 1 / (2 F), to the end of its range: the last
    operation rounds once, the sum before it enters times u <= 1/4, the polynomial
    leaves 3e-17: 0.8 ulp."""
    mp = pytest.importorskip("mpmath")
    u = np.concatenate([[0.0, 1e-300, 1e-20, 1e-9, top], np.random.default_rng(3).uniform(0, top, 3000)])
    got = device_math(fn, u, u)
    with mp.workdps(40):
        F = [mp.mpf(1) if v == 0 else mp.atanh(mp.sqrt(mp.mpf(v))) / mp.sqrt(mp.mpf(v)) for v in u]
        want = [1 / (2 * f) if half else f for f in F]
        err = max(float(abs(mp.mpf(g) - w)) / np.spacing(g) for g, w in zip(got, want))
    assert err <= 0.8, err


def test_fp32_quotient():
    """The corrected quotient rounds as the division does; where the reciprocal is not
    the nearest one, it may be the neighbour, seldom."""
    rng = np.random.default_rng(6)
    n = 400000
    x = (rng.uniform(-1, 1, n) * np.exp2(rng.integers(-20, 20, n))).astype(np.float32)
    y = (rng.uniform(0.5, 1, n) * np.exp2(rng.integers(-20, 20, n))).astype(np.float32)
    got, want = device_math(DIV32, x.astype(float), y.astype(float)).astype(np.float32), x / y
    assert np.all(np.abs(got - want) <= np.spacing(np.abs(want)))
    assert np.mean(got != want) <= 1e-3
