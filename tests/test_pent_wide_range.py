"""Pivots, divisors and right-hand sides over the whole range of doubles: quotients and reciprocals bit for bit those of
IEEE division, on both sides of the exponents where the kernels change to the operator (GPU)."""
import numpy as np
import pytest

import custen_gb300 as cs
from custen_gb300.buffers import DeviceBuffer
from tests.test_pent_rows_in_flight import check

pytestmark = pytest.mark.gpu


def powers(rng, shape, lo, hi):
    """Random significands and signs; exponents from lo to hi, the bounds of the kernels' ranges among them."""
    e = rng.integers(lo, hi + 1, shape)
    edges = [k for k in (lo, -201, -200, -199, -61, -60, 59, 60, 199, 200, 201, hi) if lo <= k <= hi]
    e = np.where(rng.random(shape) < 0.3, rng.choice(edges, shape), e)
    return np.ldexp(rng.uniform(1, 2, shape), e) * rng.choice([-1.0, 1.0], shape)


@pytest.mark.parametrize("span", [100, 199, 480])
def test_quotients(gpu, span):
    m, batch = 16, 4096
    rng = np.random.default_rng(span)
    zero = np.zeros((m, batch))
    d, b = powers(rng, (m, batch), -span, span), powers(rng, (m, batch), -span, span)
    d[:, ::7] = np.ldexp(1.0, rng.integers(-span, span, d[:, ::7].shape)) * (1 - 2.0 ** -53)   # fractions of all ones
    b[:, ::5] = rng.choice([0.0, -0.0], b[:, ::5].shape)
    check([zero, zero, d, zero, zero, b], m, batch)       # the factorisation divides 0 by d, the solve b by d


@pytest.mark.parametrize("scale", [1e24, 1e-24, 1e55, 1e75])
def test_systems_of_any_scale(gpu, scale):
    from custen_gb300.inputs import pent_system
    m, batch = 24, 500
    sysm = [a * scale for a in pent_system(m, batch, 4)[:5]] + [pent_system(m, batch, 4)[5]]
    check(sysm, m, batch)


def test_reciprocals(gpu):
    rng = np.random.default_rng(7)
    x = rng.integers(0, 1 << 64, 1 << 20, dtype=np.uint64).view(np.float64)
    x[:1 << 18] = powers(rng, 1 << 18, -1022, 1023)
    e = rng.choice([-1022, -1001, -1000, -999, -200, -60, 0, 60, 200, 999, 1000, 1001, 1023], 1 << 17)
    x[1 << 18:(1 << 18) + (1 << 17)] = np.ldexp(rng.choice([1.0, 2 - 2.0 ** -52, 1 + 2.0 ** -52, 1.5], 1 << 17), e)
    x[:8] = [0.0, -0.0, np.inf, -np.inf, 5e-324, -5e-324, 2.2250738585072014e-308, 1.7976931348623157e308]
    buf = DeviceBuffer.from_array(x)
    cs.pent_invert_pivots(buf.ptr, 4, x.size // 4)
    cs._check(cs.lib().custen_device_synchronize())
    got = buf.download(x.shape, np.float64)
    with np.errstate(all="ignore"):
        want = 1.0 / x
    nan = np.isnan(want)
    assert np.array_equal(np.isnan(got), nan)
    assert got[~nan].tobytes() == want[~nan].tobytes()


@pytest.mark.parametrize("seed", [21, 22])
def test_operators(gpu, seed):
    assert cs.selftest_fp64(1 << 28, seed=seed) == [0] * 6
