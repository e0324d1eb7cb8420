"""The FP64 right-hand side in units of sigma_nl and 2/3 where those units are extreme (no time step, a tiny one, no
biharmonic), in one pass and in two with 8 and with 4 and 2 warps per CTA: against the scheme in Fourier space, and
the three against one another bit for bit (GPU)."""
import numpy as np
import pytest

import custen_gb300 as cs

pytestmark = pytest.mark.gpu

REL_L2 = 1e-10   # the tolerance of the Cahn-Hilliard parity tests


def fourier_step(c, old, gamma, dt_factor):
    n = c.shape[0]
    dx = 2 * np.pi / n
    dt = dt_factor * dx
    sl, snl = 2 * dt * gamma / (3 * dx ** 4), 2 * dt / (3 * dx * dx)
    w = 2 - 2 * np.cos(2 * np.pi * np.arange(n) / n)
    inv = 1 / ((1 + sl * w[:, None] ** 2) * (1 + sl * w[None, :n // 2 + 1] ** 2))
    lap = lambda a: np.roll(a, 1, 0) + np.roll(a, -1, 0) + np.roll(a, 1, 1) + np.roll(a, -1, 1) - 4 * a
    bar = 2 * c - old
    rhs = lap(snl * (c ** 3 - c) - sl * lap(bar)) - (2.0 / 3.0) * (c - old)
    return bar + np.fft.irfft2(np.fft.rfft2(rhs) * inv, s=(n, n))


@pytest.mark.parametrize("gamma,dt_factor", [(0.01, 0.0), (0.01, 1e-12), (0.0, 0.05), (0.01, 0.1)])
@pytest.mark.parametrize("n", [64, 96, 160])
def test_units(gpu, n, gamma, dt_factor):
    old, cur = np.random.default_rng(n).uniform(-0.1, 0.1, (2, n, n))
    fields = []
    for config in (3, 7, 8):
        b = cs.CahnHilliardBatch([n], gamma=gamma, dt_factor=dt_factor)
        b.set_config(config)
        b.set_state(0, cur, old)
        b.step(3)
        fields.append(b.state(0)[0])
        b.close()
    for _ in range(3):
        old, cur = cur, fourier_step(cur, old, gamma, dt_factor)
    assert np.linalg.norm(fields[0] - cur) <= REL_L2 * np.linalg.norm(cur)
    assert np.array_equal(fields[0], fields[1]) and np.array_equal(fields[0], fields[2])
