"""Stencil fields that no tile divides, bit for bit against the oracle (GPU): partial last tile columns and rows of the
TMA-staged kernels (aligned rows), last columns narrower than the halo, and the cp.async-staged kernels (unaligned
rows, windows beyond 256 rows) with three, two and one ring stages; several tiles per CTA; the sizes where the default
configuration changes."""
import numpy as np
import pytest

import custen_gb300 as cs
from tests.test_stencil_parity import run_both

pytestmark = pytest.mark.gpu

X5, X9, X4 = (5, 2, 2, 1, 0, 0), (9, 4, 4, 1, 0, 0), (4, 2, 1, 1, 0, 0)
Y5, Y9 = (1, 0, 0, 5, 2, 2), (1, 0, 0, 9, 4, 4)
XY3, XY5, XYA = (3, 1, 1, 3, 1, 1), (5, 2, 2, 5, 2, 2), (5, 3, 1, 4, 1, 2)
PERIODIC = [(cs.XP, X5, -1), (cs.XP, X9, -1), (cs.XP, X4, -1), (cs.YP, Y5, -1), (cs.YP, Y9, -1), (cs.XYP, XY3, -1),
            (cs.XYP, XY5, -1), (cs.XYP, XYA, -1), (cs.XPFUN, X5, 1), (cs.YPFUN, Y9, 2), (cs.XYPFUN, XY3, 4),
            (cs.XYPFUN, XY3, 5)]
NONPERIODIC = [(cs.XNP, X5), (cs.YNP, Y5), (cs.XYNP, XY3), (cs.XYNP, XY5)]


def block_of(n, halo):
    """A block size of the reference's contract: divides n at least twice and holds a halo."""
    return next(d for d in range(max(halo, 2), n) if n % d == 0 and n // d >= 2)


def same(variant, nx, ny, tiles, geom, **kw):
    H, L, R, V, T, B = geom
    got, ref, st, pre = run_both(variant, nx, ny, tiles, block_of(nx, max(L, R)), block_of(ny // tiles, max(T, B)), geom, **kw)
    known = st != 2   # points the reference leaves undefined
    assert np.array_equal(got[known], ref[known]), np.argwhere((got != ref) & known)[:4].tolist()


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("variant,geom,fun", PERIODIC)
@pytest.mark.parametrize("nx,ny", [(66, 33), (132, 30), (196, 70), (65, 34), (99, 65), (135, 18)])
def test_periodic(gpu, variant, geom, fun, nx, ny, dtype):
    for config in (0, 3, 5):
        same(variant, nx, ny, 1, geom, fun_id=fun, dtype=dtype, config=config)


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("variant,geom", NONPERIODIC)
@pytest.mark.parametrize("nx,ny,tiles", [(68, 36, 1), (132, 72, 2), (196, 24, 1)])
def test_nonperiodic(gpu, variant, geom, nx, ny, tiles, dtype):
    for config in (0, 1, 5):
        same(variant, nx, ny, tiles, geom, dtype=dtype, config=config)


@pytest.mark.parametrize("nx,ny,extent", [(65, 200, 30), (64, 300, 120), (33, 260, 120), (66, 150, 60)])
def test_tall_windows(gpu, nx, ny, extent):
    """Two and one ring stages, and windows of more rows than a tensor box takes."""
    same(cs.YP, nx, ny, 1, (1, 0, 0, 2 * extent + 1, extent, extent), config=0)


@pytest.mark.parametrize("variant,geom,fun", PERIODIC[:8:3] + PERIODIC[8:])
def test_many_tiles_per_cta(gpu, variant, geom, fun):
    cs.set_max_ctas(2)
    try:
        for nx, ny in ((226, 135), (225, 135)):
            same(variant, nx, ny, 1, geom, fun_id=fun, config=1)
    finally:
        cs.set_max_ctas(0)


@pytest.mark.parametrize("nx,ny,dtype,config", [(1250, 1199, np.float64, 5), (1250, 1200, np.float64, 1),
                                                (4000, 3000, np.float64, 0), (2000, 1499, np.float32, 5),
                                                (2000, 1500, np.float32, 1), (5000, 4000, np.float32, 0)])
def test_default_configuration_by_size(gpu, nx, ny, dtype, config, tmp_path):
    from custen_gb300.buffers import DeviceBuffer
    cs.set_tune_cache(tmp_path / "none.json")
    try:
        code = cs.F64 if dtype == np.float64 else cs.F32
        item = np.dtype(dtype).itemsize
        inp, out = DeviceBuffer(nx * ny * item), DeviceBuffer(nx * ny * item)
        w = DeviceBuffer.from_array(np.ones(5, dtype))
        cs._check(cs.lib().custen_memset(inp.ptr, 0, nx * ny * item))
        s = cs.Stencil(cs.XP, nx, ny, out.ptr, inp.ptr, w.ptr, H=5, L=2, R=2, dtype=code)
        s.compute()
        cs._check(cs.lib().custen_device_synchronize())
        t = cs.Stencil(cs.XP, nx, ny, out.ptr, inp.ptr, w.ptr, H=5, L=2, R=2, dtype=code)
        t.set_config(config)
        assert s.config() == t.config()
        s.destroy()
        t.destroy()
    finally:
        cs.set_tune_cache(None)
