"""Computes queued one behind the other without a synchronisation, each reading through its halo rows what the one
before wrote (the buffers swapped in between, as a time loop does): on the handle's own stream, on a caller's stream and
as a captured graph, with one and several tiles per thread block, bit for bit against the oracle (GPU)."""
import numpy as np
import pytest

import custen_gb300 as cs
import oracle
from custen_gb300.inputs import field

pytestmark = pytest.mark.gpu

STEPS = 24
W = np.array([0.05, 0.2, 0.4, 0.3, 0.05])   # sums to one: the field stays in range


def want(nx, ny, variant, dtype):
    a = field(nx, ny, 4, dtype)
    for _ in range(STEPS):
        ref = a.copy()
        w = (W if variant == cs.YP else np.outer(W, W).ravel()).astype(dtype)
        geom = dict(H=1, L=0, R=0, V=5, T=2, B=2) if variant == cs.YP else dict(H=5, L=2, R=2, V=5, T=2, B=2)
        oracle.stencil(variant, ref, a, w, num_tiles=1, block_x=nx if variant == cs.YP else nx // 2, block_y=ny // 2, **geom)
        a = ref
    return a, w, geom


@pytest.mark.parametrize("how", ["own", "stream", "graph"])
@pytest.mark.parametrize("max_ctas", [0, 3])
@pytest.mark.parametrize("variant,nx,ny,dtype", [(cs.YP, 64, 16, np.float64), (cs.YP, 512, 300, np.float64),
                                                 (cs.XYP, 256, 128, np.float64), (cs.XYP, 640, 100, np.float32),
                                                 (cs.YP, 65, 48, np.float64)])
def test_time_loop(gpu, variant, nx, ny, dtype, max_ctas, how):
    import torch
    ref, w, geom = want(nx, ny, variant, dtype)
    bufs = [torch.tensor(field(nx, ny, 4, dtype), device="cuda"), torch.zeros((ny, nx), device="cuda", dtype=torch.float64 if dtype == np.float64 else torch.float32)]
    wt = torch.tensor(w, device="cuda")
    cs.set_max_ctas(max_ctas)
    try:
        h = cs.Stencil(variant, nx, ny, bufs[1], bufs[0], wt, dtype=cs.F64 if dtype == np.float64 else cs.F32, ncoef=len(w), **geom)
        s = torch.cuda.Stream()
        torch.cuda.synchronize()

        def loop(**kw):
            for k in range(STEPS):
                h.compute(**kw)
                h.swap(bufs[(k + 1) % 2].data_ptr())

        if how == "own":
            loop()
        elif how == "stream":
            with torch.cuda.stream(s):
                loop(stream=s)
        else:
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g, stream=s):
                loop(stream=s)
            g.replay()
        torch.cuda.synchronize()
        h.destroy()
    finally:
        cs.set_max_ctas(0)
    assert bufs[0].cpu().numpy().tobytes() == ref.tobytes()   # an even number of steps
