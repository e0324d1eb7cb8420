"""Exact-zero weights over fields with infinities and NaN: dropped (the value under them does not matter) in FP64, in FP32
where rows are unaligned or a tile is partial, and in windows without a loop of their own; kept, as the reference keeps
them, in FP32 fields of whole 128 x 32 tiles. Every configuration, and the untuned default (GPU)."""
import numpy as np
import pytest

import custen_gb300 as cs
from custen_gb300.buffers import DeviceBuffer
from custen_gb300.inputs import field

pytestmark = pytest.mark.gpu

CROSS = [0, 1, 0, 2, -3, 2, 0, 1, 0]
BIHARMONIC = [0, 0, -1, 0, 0, 0, -2, 8, -2, 0, -1, 8, -20, 8, -1, 0, -2, 8, -2, 0, 0, 0, -1, 0, 0]
WINDOWS = {"X3": (cs.XP, 3, 1, [1, 0, -1], 1), "X5": (cs.XP, 5, 2, [1, 0, 0, -2, 3], 1), "X9": (cs.XP, 9, 4, [1, 0, 2, 0, 0, 3, 0, 0, 1], 1),
           "Y3": (cs.YP, 1, 0, [1, 0, -1], 3), "Y5": (cs.YP, 1, 0, [0, 1, 0, -2, 0], 5), "Y9": (cs.YP, 1, 0, [1, 0, 2, 0, 0, 3, 0, 0, 0], 9),
           "XY3": (cs.XYP, 3, 1, CROSS, 3), "XY5": (cs.XYP, 5, 2, BIHARMONIC, 5), "XY3x5": (cs.XYP, 3, 1, [0, 1, 0] * 5, 5)}


@pytest.mark.parametrize("dtype", [np.float64, np.float32], ids=["f64", "f32"])
@pytest.mark.parametrize("window", list(WINDOWS))
@pytest.mark.parametrize("nx,ny", [(256, 64), (192, 64), (256, 48), (132, 70), (131, 67)])
def test_infinities_under_zero_weights(gpu, nx, ny, window, dtype):
    v, H, L, w, V = WINDOWS[window]
    w = np.asarray(w, dtype)
    T = V // 2
    kept = dtype == np.float32 and nx % 128 == 0 and ny % 32 == 0 and window != "XY3x5"
    rng = np.random.default_rng(nx + ny)
    f = field(nx, ny, 1, dtype)
    bad = rng.random((ny, nx)) < 0.01
    g = np.where(bad, rng.choice(np.array([np.inf, -np.inf, np.nan], dtype), (ny, nx)), f)
    hit = np.zeros((ny, nx), bool)   # points whose chain holds one of them
    for k, wk in enumerate(w):
        if wk != 0 or kept:
            hit |= np.roll(bad, (T - k // H, L - k % H), (0, 1))
    code = cs.F64 if dtype == np.float64 else cs.F32
    out, wt = DeviceBuffer(f.nbytes), DeviceBuffer.from_array(w)
    for config in (None, 0, 1, 2, 3, 4, 5):
        got = []
        for a in (g, np.where(bad, dtype(0), f)):
            inp = DeviceBuffer.from_array(a)
            h = cs.Stencil(v, nx, ny, out.ptr, inp.ptr, wt.ptr, H=H, L=L, R=L, V=V, T=T, B=T, dtype=code, ncoef=w.size)
            if config is not None:
                h.set_config(config)
            h.compute()
            cs._check(cs.lib().custen_device_synchronize())
            got.append(out.download((ny, nx), dtype))
            h.destroy()
        assert np.array_equal(~np.isfinite(got[0]), hit), config
        assert got[0][~hit].tobytes() == got[1][~hit].tobytes(), config
