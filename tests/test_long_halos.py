"""Halos longer than a tile: the windows of tiles behind the first tile row or column leave the field too. Every
configuration and the untuned default, whole and partial tiles, halos on one side, and tiles launched one by one (managed
and pinned memory) against the oracle, bit for bit (GPU)."""
import numpy as np
import pytest

import custen_gb300 as cs
from tests.test_ragged_tiles import same

pytestmark = pytest.mark.gpu

CONFIGS = [None, 0, 1, 2, 3, 4, 5]
SIZES = [(256, 256), (264, 250)]   # whole tiles of every configuration; partial last ones


def x_window(L, R):
    return L + R + 1, L, R, 1, 0, 0


def y_window(T, B):
    return 1, 0, 0, T + B + 1, T, B


def all_configs(variant, nx, ny, geom, dtype, fun=-1):
    for config in CONFIGS:
        before = cs.kernel_launches_tma()
        same(variant, nx, ny, 1, geom, fun_id=fun, dtype=dtype, config=config)
        if config == 5:   # its ring fits shared memory with every window here
            assert cs.kernel_launches_tma() > before, "the TMA-staged kernel did not run"
    assert cs.device_error() == 0


@pytest.mark.parametrize("dtype", [np.float64, np.float32], ids=["f64", "f32"])
@pytest.mark.parametrize("nx,ny", SIZES)
@pytest.mark.parametrize("T,B", [(17, 17), (20, 20), (33, 33), (40, 40), (40, 0), (0, 40)])
def test_rows(gpu, T, B, nx, ny, dtype):
    all_configs(cs.YP, nx, ny, y_window(T, B), dtype)


@pytest.mark.parametrize("dtype", [np.float64, np.float32], ids=["f64", "f32"])
@pytest.mark.parametrize("nx,ny", SIZES)
@pytest.mark.parametrize("L,R", [(33, 33), (40, 40), (70, 70), (40, 0), (0, 40)])
def test_columns(gpu, L, R, nx, ny, dtype):
    all_configs(cs.XP, nx, ny, x_window(L, R), dtype)


@pytest.mark.parametrize("dtype", [np.float64, np.float32], ids=["f64", "f32"])
@pytest.mark.parametrize("nx,ny", SIZES)
@pytest.mark.parametrize("geom", [(35, 17, 17, 35, 17, 17), (45, 40, 4, 37, 18, 18)])
@pytest.mark.parametrize("variant,fun", [(cs.XYP, -1), (cs.XYPFUN, 4), (cs.XYPFUN, 5)])
def test_both(gpu, variant, fun, geom, nx, ny, dtype):
    all_configs(variant, nx, ny, geom, dtype, fun)


@pytest.mark.parametrize("mem", ["managed", "pinned"])
@pytest.mark.parametrize("variant", [cs.YP, cs.YNP])
def test_tiles_launched_apart(gpu, variant, mem):
    for config in CONFIGS:
        same(variant, 256, 256, 2, y_window(40, 40), mem=mem, config=config)


@pytest.mark.parametrize("geom,config", [(x_window(2, 2), 1), (x_window(16, 16), 1), (x_window(40, 40), 5),
                                         (y_window(40, 40), 1), (y_window(100, 100), 5)])
def test_default_configuration(gpu, geom, config, tmp_path):
    """A field that takes the half-wide tile with short windows, whose ring two CTAs of an SM have to share."""
    from custen_gb300.buffers import DeviceBuffer
    H, L, R, V, T, B = geom
    nx, ny = 1536, 1280
    cs.set_tune_cache(tmp_path / "none.json")
    try:
        inp, out, w = DeviceBuffer(nx * ny * 8), DeviceBuffer(nx * ny * 8), DeviceBuffer.from_array(np.ones(H * V))
        cs._check(cs.lib().custen_memset(inp.ptr, 0, nx * ny * 8))
        names = []
        for pin in (None, config):
            h = cs.Stencil(cs.XP if H > 1 else cs.YP, nx, ny, out.ptr, inp.ptr, w.ptr, H=H, L=L, R=R, V=V, T=T, B=B)
            if pin is not None:
                h.set_config(pin)
            h.compute()
            cs._check(cs.lib().custen_device_synchronize())
            names.append(h.config())
            h.destroy()
        assert names[0] == names[1]
    finally:
        cs.set_tune_cache(None)
