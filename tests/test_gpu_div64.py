"""The FP64 kernels' integer division and square root (sflow_div64.cuh) on the
device, whose first estimates are the device's own approximations: the bits of
the host's IEEE operations on the operand families of test_div64.py (random
patterns, quotients times the divisor and squares +-2 ulp, divisors of nearly
all ones, small integers, special values and the ends of the range)."""
import numpy as np
import pytest

from imex_sflow2d_dev_gb300 import lib as L

pytestmark = pytest.mark.gpu

SPECIAL = np.array([0.0, -0.0, 1.0, -1.0, np.inf, -np.inf, np.nan, 2.0 ** -1074, -2.0 ** -1030, 2.0 ** -1022,
                    np.finfo(float).max, 2.0 ** -430, 2.0 ** 430, 2.0 ** 423, 2.0 ** -423, 1.5, 3.0, 10.0, 0.1])


def _ulps(a, rng):
    return (a.view(np.int64) + rng.integers(-2, 3, a.size)).view(np.float64)


def _pairs(n, seed):
    rng = np.random.default_rng(seed)
    unit = lambda: rng.uniform(1.0, 2.0, n)
    bits = lambda: rng.integers(-2 ** 63, 2 ** 63 - 1, n, dtype=np.int64).view(np.float64)
    d = unit()
    sa, sd = np.meshgrid(SPECIAL, SPECIAL)
    m = unit()
    sq = m * m * np.where(rng.integers(0, 2, n) == 1, 2.0, 1.0)
    a = [bits(), unit(), _ulps(unit() * d, rng), unit(), rng.integers(-50000, 50000, n).astype(float), _ulps(sq, rng),
         SPECIAL[rng.integers(0, SPECIAL.size, n)], sa.ravel()]
    b = [bits(), unit(), d, 2.0 - rng.integers(1, 65, n) * 2.0 ** -52, rng.integers(1, 1001, n).astype(float), unit(),
         unit(), sd.ravel()]
    return np.concatenate(a), np.concatenate(b)


def _differ(x, y):
    return ((x.view(np.int64) != y.view(np.int64)) & ~(np.isnan(x) & np.isnan(y))).sum()


@pytest.mark.parametrize("seed", [31, 32])
def test_device_bits_are_the_ieee_ones(seed):
    a, b = _pairs(400000, seed)
    with np.errstate(all="ignore"):
        assert _differ(L.eval_math("div", a, b), a / b) == 0
        assert _differ(L.eval_math("sqrt", a), np.sqrt(a)) == 0
        assert _differ(L.eval_math("sqrt", b), np.sqrt(b)) == 0
