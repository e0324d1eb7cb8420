"""The Cahn-Hilliard line solves at the sizes where their schedule changes (fewer, as many and more chunks per
chain than ring stages; one and two segments per line) and over parameters that change the reach of the periodic closure: against a Fourier
solution of the same scheme, which shares nothing with the factored sweeps (GPU)."""
import math

import numpy as np
import pytest

import custen_gb300 as cs

pytestmark = pytest.mark.gpu

REL_L2 = 1e-10   # the tolerance of the Cahn-Hilliard parity tests


def fourier_steps(c, steps, lx, gamma, dt_factor):
    n = c.shape[0]
    dx = lx / n
    dt = dt_factor * dx
    sl, snl = 2 * dt * gamma / (3 * dx ** 4), 2 * dt / (3 * dx * dx)
    w = 2 - 2 * np.cos(2 * np.pi * np.arange(n) / n)
    inv = 1 / ((1 + sl * w[:, None] ** 2) * (1 + sl * w[None, :n // 2 + 1] ** 2))

    def lap(a):
        return np.roll(a, 1, 0) + np.roll(a, -1, 0) + np.roll(a, 1, 1) + np.roll(a, -1, 1) - 4 * a

    old = c.copy()
    for _ in range(steps):
        bar = 2 * c - old
        rhs = lap(snl * (c ** 3 - c) - sl * lap(bar)) - (2.0 / 3.0) * (c - old)
        old, c = c, bar + np.fft.irfft2(np.fft.rfft2(rhs) * inv, s=(n, n))
    return c, old


@pytest.mark.parametrize("config", [8, 20, 21])
@pytest.mark.parametrize("n", [64, 96, 128, 160, 192, 288, 512, 544, 576, 1088])
def test_sizes(gpu, n, config):
    c0 = np.random.default_rng(n).uniform(-0.1, 0.1, (n, n))
    b = cs.CahnHilliardBatch([n])
    b.set_config(config)
    b.set_state(0, c0)
    b.step(6)
    cur, old = b.state(0)
    rcur, rold = fourier_steps(c0, 6, 2 * np.pi, 0.01, 0.1)
    assert np.linalg.norm(cur - rcur) <= REL_L2 * np.linalg.norm(rcur)
    assert np.linalg.norm(old - rold) <= REL_L2 * np.linalg.norm(rold)
    b.close()


# (n, lx, gamma, dt_factor): sigma_lin from 0 through 1e-4 (closure of a few entries) to 3e4 (of the whole line),
# and negative values, which take the general sweeps
@pytest.mark.parametrize("n,lx,gamma,dt_factor", [(128, 2 * np.pi, 0.0, 0.1), (128, 60.0, 0.01, 0.1),
                                                  (96, 2 * np.pi, 1e-5, 0.1), (128, 1.0, 0.01, 0.1),
                                                  (64, 0.3, 0.01, 0.1), (128, 2 * np.pi, -1e-4, 0.05), (384, 2 * np.pi, -4e-6, 0.05),
                                                  (1056, 2 * np.pi, -1e-7, 0.1),
                                                  (64, 2 * np.pi, -0.002, 0.05)])
def test_parameters(gpu, n, lx, gamma, dt_factor):
    c0 = np.random.default_rng(3).uniform(-0.1, 0.1, (n, n))
    b = cs.CahnHilliardBatch([n], lx=lx, gamma=gamma, dt_factor=dt_factor)
    b.set_state(0, c0)
    b.step(3)
    cur, _ = b.state(0)
    rcur, _ = fourier_steps(c0, 3, lx, gamma, dt_factor)
    assert np.linalg.norm(cur - rcur) <= REL_L2 * np.linalg.norm(rcur)
    b.close()


def test_mixed_signs_in_one_batch(gpu):
    """A negative side length gives a negative time step: that grid takes the general sweeps beside the others."""
    sizes, lx = [64, 96, 128], [2 * np.pi, -40.0, 2 * np.pi]
    c0 = [np.random.default_rng(k).uniform(-0.1, 0.1, (n, n)) for k, n in enumerate(sizes)]
    b = cs.CahnHilliardBatch(sizes, lx=lx)
    for k, c in enumerate(c0):
        b.set_state(k, c)
    b.step(3)
    for k, (n, c) in enumerate(zip(sizes, c0)):
        r, _ = fourier_steps(c, 3, lx[k], 0.01, 0.1)
        assert np.linalg.norm(b.state(k)[0] - r) <= REL_L2 * np.linalg.norm(r), n
    b.close()


@pytest.mark.parametrize("n", [64, 96, 736])
def test_mean_over_few_and_many_blocks(gpu, n):
    """The compensated sum over 2, 5 and 256 CTAs (the cap), twice on the same scratch: exact to rounding."""
    c = np.random.default_rng(n).uniform(-0.1, 0.1, (n, n))
    b = cs.CahnHilliardBatch([n])
    b.set_state(0, c)
    exact = math.fsum(c.ravel()) / (n * n)
    for _ in range(2):
        assert abs(b.mean(0) - exact) <= 4e-16 * np.abs(c).mean()
    b.close()
