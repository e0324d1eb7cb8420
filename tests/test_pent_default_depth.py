"""The rows in flight of the batched pentadiagonal kernels go back to the rule by the batch size (set to 0), and the rule's
two sides (8 x 152 warps of 32 systems) are bit-identical to the oracle."""
import pytest

import custen_gb300 as cs
from custen_gb300.inputs import pent_system
from tests.test_pent_rows_in_flight import check


def set_depth(rows):
    return [cs.lib().custen_pent_set_depth(which, rows) for which in range(3)]


def test_accepted_depths(built):
    try:
        for rows in (2, 4, 8, 0):
            assert set_depth(rows) == [0] * 3
            for which in range(3):
                assert rows == 0 or cs.lib().custen_pent_depth(which, 1000) == rows
        for rows in (-1, 1, 3, 16):
            assert set_depth(rows) == [2] * 3
        assert cs.lib().custen_pent_set_depth(3, 0) == 2 and cs.lib().custen_pent_depth(3, 10) == 0
        assert cs.lib().custen_pent_depth(0, 0) == 0
    finally:
        set_depth(0)


@pytest.mark.gpu
@pytest.mark.parametrize("batch,rows", [(1, 8), (38912, 8), (38913, 4)])
def test_rule(gpu, batch, rows):
    set_depth(2)
    set_depth(0)
    assert [cs.lib().custen_pent_depth(which, batch) for which in range(3)] == [rows] * 3
    check(pent_system(6, batch, 5), 6, batch)
