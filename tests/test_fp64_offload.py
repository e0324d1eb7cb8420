"""Conversions, divisions, sums and products that spare the FP64 pipe (csrc/fp64_offload.cuh): the same bits as the hardware's
on random, tie-constructed, near-midpoint and special operands (GPU)."""
import pytest

import custen_gb300 as cs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("seed", [1, 2, 3])
def test_same_bits_as_the_operators(gpu, seed):
    assert cs.selftest_fp64(1 << 28, seed=seed) == [0] * 6
