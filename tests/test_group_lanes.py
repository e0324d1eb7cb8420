"""custen_compute_group's sharing of streams: groups smaller than, as large as and larger than the number of shared
streams, with members in device, managed and pinned host memory among them; each output equals the oracle's bit for bit
and the group keeps its place between the work before and after it on the caller's stream (GPU)."""
import numpy as np
import pytest

import custen_gb300 as cs
import oracle
from custen_gb300.buffers import DeviceBuffer
from custen_gb300.inputs import field, sentinel, sweep_operators

pytestmark = pytest.mark.gpu

N = 256


@pytest.mark.parametrize("kinds", ["d", "dd", "ddd", "dddd", "dpdddddm", "mpdddd", "ddpmddd", "pppppp", "mmmmmm"])
def test_members_in_any_memory(gpu, kinds):
    import torch
    dev = torch.device("cuda", 0)
    src, pre = field(N, N, 1), sentinel(N, N)
    d_src = torch.tensor(src, device=dev)
    d_in = torch.zeros((N, N), device=dev, dtype=torch.float64)
    hs, outs, keep = [], [], [d_src, d_in]
    ops = [sweep_operators(N)[k] for k in range(len(kinds))]
    for kind, (nm, v, H, L, R, V, T, B, w, fun, _) in zip(kinds, ops):
        if kind == "d":
            inp, out = d_in, torch.tensor(pre, device=dev)
            read = lambda t=out: t.cpu().numpy()
            ptrs = inp, out
        elif kind == "p":
            inp, out = torch.tensor(src).pin_memory(), torch.tensor(pre).pin_memory()
            read = lambda t=out: t.numpy()
            ptrs = inp, out
        else:
            inp, out = DeviceBuffer.from_array(src, managed=True), DeviceBuffer.from_array(pre, managed=True)
            read = lambda t=out: np.array(t.view((N, N), np.float64))
            ptrs = inp.ptr, out.ptr
        wt = (DeviceBuffer.from_array(np.asarray(w), managed=True) if kind == "m"
              else torch.tensor(w, device=dev, dtype=torch.float64))
        keep += [inp, out, wt]
        outs.append(read)
        hs.append(cs.Stencil(v, N, N, ptrs[1], ptrs[0], wt.ptr if kind == "m" else wt, H=H, L=L, R=R, V=V, T=T, B=B, num_tiles=2, ncoef=len(w),
                             func=cs.builtin_function(fun) if fun >= 0 else None))
    torch.cuda.synchronize(dev)
    s = torch.cuda.Stream(dev)
    with torch.cuda.stream(s):
        torch.cuda._sleep(2_000_000)
        d_in.copy_(d_src)                       # the group follows this
        cs.compute_group(hs, cs.DEVICE, s)
        d_in.zero_()                            # and precedes this
    s.synchronize()
    for kind, read, (nm, v, H, L, R, V, T, B, w, fun, _) in zip(kinds, outs, ops):
        ref = sentinel(N, N)
        oracle.stencil(v, ref, src, np.asarray(w), num_tiles=2, block_x=32, block_y=8, H=H, L=L, R=R, V=V, T=T, B=B,
                       fun_id=fun)
        assert read().tobytes() == ref.tobytes(), (kind, nm)
    for h in hs:
        h.destroy()
    assert cs.device_error() == 0


def test_a_handles_own_stream_stays_ordered(gpu):
    """Computes on a handle's own stream, then a group in which it shares another handle's stream, then its own again,
    without a synchronisation: each reads what the one before wrote (the buffers are swapped between them)."""
    import torch
    dev = torch.device("cuda", 0)
    big = 2048
    small = torch.tensor(field(N, N, 1), device=dev)
    a0 = field(big, big, 2)
    a, b = torch.tensor(a0, device=dev), torch.zeros((big, big), device=dev, dtype=torch.float64)
    nm, v, H, L, R, V, T, B, w, fun, _ = sweep_operators(N)[0]
    wt = torch.tensor(w, device=dev, dtype=torch.float64)
    outs = [torch.empty_like(small) for _ in range(3)]
    kw = dict(H=H, L=L, R=R, V=V, T=T, B=B, ncoef=len(w))
    hs = [cs.Stencil(v, N, N, o, small, wt, **kw) for o in outs]
    h = cs.Stencil(v, big, big, b, a, wt, **kw)
    s = torch.cuda.Stream(dev)
    torch.cuda.synchronize(dev)
    for _ in range(15):
        h.compute()                              # a -> b
    h.swap(b.data_ptr())
    cs.compute_group(hs + [h], cs.DEVICE, s)     # b -> a
    h.swap(a.data_ptr())
    h.compute()                                  # a -> b
    h.swap(b.data_ptr())
    cs.compute_group([h] + hs, cs.DEVICE, s)     # b -> a, on its own stream again
    h.swap(a.data_ptr())
    cs.compute_group(hs[::-1] + [h], cs.DEVICE, s)   # a -> b, on another handle's stream
    torch.cuda.synchronize(dev)
    want = a0
    for _ in range(5):
        ref = np.zeros((big, big))
        oracle.stencil(v, ref, want, np.asarray(w), num_tiles=1, block_x=32, block_y=8, H=H, L=L, R=R, V=V, T=T, B=B)
        want = ref
    assert b.cpu().numpy().tobytes() == want.tobytes()
    for k in hs + [h]:
        k.destroy()
