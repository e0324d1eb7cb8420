"""The y sweep with the closure in it, whose two chains hand over their end values through the shared memory that held
the closure amplitudes, against the one without it: the same bits, for chains of one chunk (64 points), two and three,
and more chunks than ring stages, with few and many thread blocks on an SM (GPU)."""
import numpy as np
import pytest

import custen_gb300 as cs

pytestmark = pytest.mark.gpu

FUSED, APART = 7, 18   # two passes of 8 warps, the closure in the y sweep and in a kernel of its own


@pytest.mark.parametrize("n,count", [(64, 1), (64, 300), (96, 150), (128, 100), (160, 60), (288, 20)])
def test_same_bits(gpu, n, count):
    rng = np.random.default_rng(n)
    c0 = [rng.uniform(-0.1, 0.1, (n, n)) for _ in range(min(count, 4))]
    fields = []
    for config in (FUSED, APART):
        b = cs.CahnHilliardBatch([n] * count)
        b.set_config(config)
        for k in range(count):
            b.set_state(k, c0[k % 4 % len(c0)])
        b.step(30)
        fields.append([b.state(k)[0] for k in range(count)])
        b.close()
    for k in range(count):
        assert fields[0][k].tobytes() == fields[1][k].tobytes(), k
        assert fields[0][k].tobytes() == fields[0][k % 4 % len(c0)].tobytes(), k   # equal grids stay equal
    assert cs.device_error() == 0
