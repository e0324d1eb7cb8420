"""The WENO handle names the tile it launches, on both sides of each size where the height changes, before and after a
Compute, and for fields whose tiles are launched one by one (GPU)."""
import numpy as np
import pytest

import custen_gb300 as cs
from custen_gb300.buffers import DeviceBuffer

pytestmark = pytest.mark.gpu


def names(nx, ny, tiles, managed=False):
    f, u, v = (DeviceBuffer.from_array(np.ones((ny, nx)), managed) for _ in range(3))
    out = DeviceBuffer.from_array(np.zeros((ny, nx)), managed)
    h = cs.WenoAdvection(nx, ny, out.ptr, f.ptr, u.ptr, v.ptr, dx=0.1, dy=0.1, num_tiles=tiles)
    before = h.config()
    h.compute(cs.DEVICE)
    cs._check(cs.lib().custen_device_synchronize())
    after = h.config()
    h.destroy()
    return before, after


@pytest.mark.parametrize("nx,ny,rows", [(64, 64, 8), (511, 2015, 8), (511, 2047, 16), (4097, 2011, 16), (4033, 2047, 32)])
def test_whole_field(gpu, nx, ny, rows):
    assert names(nx, ny, 1) == ("weno_tw64_th%d" % rows,) * 2


def test_tiles_launched_apart(gpu):
    assert names(512, 2048, 4, managed=True) == ("weno_tw64_th16", "weno_tw64_th8")
    assert names(512, 2048, 4) == ("weno_tw64_th16",) * 2
