"""WENO advection at the sizes where its tile height changes (fields of 512 and 4096 tiles of 64 x 32 points),
with partial tiles in both directions (GPU)."""
import pytest

from tests.test_weno import assert_close, run_weno

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,tiles", [(511, 2015, 1), (511, 2047, 1), (513, 1825, 1), (4033, 2047, 1), (4097, 2011, 1), (4100, 2049, 3)])
def test_tile_heights_match_oracle(gpu, nx, ny, tiles):
    got, ref = run_weno(nx, ny, tiles, seed=nx + ny, rough=True)
    assert_close(got, ref)
