"""The Cahn-Hilliard sweeps' shared-memory rings when a copy never arrives (simulated: a byte count that nothing delivers,
no copy in flight): the waits give up, the copy warp starts no further copy, the flag is raised and the solver still
computes afterwards (GPU)."""
import numpy as np
import pytest

import custen_gb300 as cs

pytestmark = pytest.mark.gpu


def result():
    b = cs.CahnHilliardBatch([64, 96])
    for k, n in enumerate((64, 96)):
        b.set_state(k, np.random.default_rng(n).uniform(-0.1, 0.1, (n, n)))
    b.step(4)
    out = [b.state(k)[0].tobytes() for k in range(2)]
    b.close()
    return out


# chunks, the lost one, and the copies the chain's warp starts and stores back until then: the first four are started
# at once, then one for each chunk stored; the last four of the forward pass stay in the ring
@pytest.mark.parametrize("nchunk,lost,started,stored", [(12, 0, 4, 0), (12, 3, 7, 3), (12, 10, 12, 8), (4, 2, 4, 0), (2, 1, 2, 0)])
def test_lost_copy(gpu, nchunk, lost, started, stored):
    want = result()
    cs.device_error(clear=True)
    flags, counts = cs.selftest_ring_expiry(nchunk, lost)
    assert flags & 1 and cs.device_error(clear=True) & 1
    assert counts[:2] == [started, stored]
    assert result() == want and cs.device_error() == 0


@pytest.mark.parametrize("nchunk", [1, 4, 5, 12])
def test_nothing_lost(gpu, nchunk):
    cs.device_error(clear=True)
    again = max(nchunk - 4, 0)
    assert cs.selftest_ring_expiry(nchunk, -1) == (0, [nchunk + again, again + nchunk] * 2)
