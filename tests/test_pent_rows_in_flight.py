"""Batched pentadiagonal kernels with every number of rows in flight, shorter and longer than the system, below
and above the batch size where the default changes (8 x 152 warps of 32 systems): bit-identical to the oracle;
zero right-hand sides, power-of-two and out-of-range pivots (GPU)."""
import numpy as np
import pytest

import custen_gb300 as cs
import oracle
from custen_gb300.buffers import DeviceBuffer
from custen_gb300.inputs import pent_system

pytestmark = pytest.mark.gpu


def check(sysm, m, batch):
    bufs = [DeviceBuffer.from_array(a) for a in sysm]
    cs.pent_factor_batch(*[b.ptr for b in bufs[:5]], m, batch)
    cs.pent_solve_batch(*[b.ptr for b in bufs], m, batch)
    cs._check(cs.lib().custen_device_synchronize())
    got = [b.download((m, batch), np.float64) for b in bufs]
    f = oracle.pent_factor(*sysm[:5])
    for g, r in zip(got, [*f, oracle.pent_solve(f, sysm[5])]):
        assert g.tobytes() == r.tobytes()


@pytest.mark.parametrize("rows", [2, 4, 8])
@pytest.mark.parametrize("m,batch", [(4, 33), (7, 64), (8, 31), (9, 1), (40, 97)])
def test_rows_in_flight(gpu, rows, m, batch):
    for which in range(3):
        cs._pent_check(cs.lib().custen_pent_set_depth(which, rows))
    try:
        check(pent_system(m, batch, m + rows), m, batch)
    finally:
        for which in range(3):   # the depths the rule would take for these batches
            cs._pent_check(cs.lib().custen_pent_set_depth(which, 4))


@pytest.mark.parametrize("batch", [38912, 38913])
def test_both_sides_of_the_default(gpu, batch):
    check(pent_system(6, batch, 5), 6, batch)


def test_unusual_pivots_and_right_hand_sides(gpu):
    m, batch = 12, 96
    ds, dl, d, du, dw, b = pent_system(m, batch, 9)
    for a in (ds, dl, du, dw):
        a[:, :48] = 0.0                                     # diagonal systems: the pivots are d itself
    d[:, :48] = np.ldexp(np.where(np.arange(48) % 2, 1.0, -1.0), np.arange(48) * 8 - 180)[None, :]
    d[:, 24:48] *= np.nextafter(1.0, 0.0)
    b[:, ::3] = 0.0
    b[:, 1:48:5] *= 1e-290
    b[3, 60] = -0.0
    check([ds, dl, d, du, dw, b], m, batch)
