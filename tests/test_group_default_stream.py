"""custen_compute_group on the legacy default stream, which every work on the handles' streams waits for and which waits
for it in turn: right whatever memory the members lie in, and members with host copies still overlap (GPU)."""
import time

import numpy as np
import pytest

import custen_gb300 as cs
import oracle
from custen_gb300.inputs import field, sentinel, sweep_operators

pytestmark = pytest.mark.gpu


def members(kinds, n):
    import torch
    src, pre, hs, outs = field(n, n, 1), sentinel(n, n), [], []
    for kind, (nm, v, H, L, R, V, T, B, w, fun, _) in zip(kinds, sweep_operators(n)):
        place = (lambda a: torch.tensor(a).pin_memory()) if kind == "p" else (lambda a: torch.tensor(a, device="cuda"))
        inp, out, wt = place(src), place(pre), torch.tensor(w, device="cuda", dtype=torch.float64)
        hs.append(cs.Stencil(v, n, n, out, inp, wt, H=H, L=L, R=R, V=V, T=T, B=B, ncoef=len(w),
                             func=cs.builtin_function(fun) if fun >= 0 else None))
        outs.append((inp, out, wt))
    torch.cuda.synchronize()
    return hs, outs


@pytest.mark.parametrize("kinds", ["pppddd", "dpdpdpdd", "pppppp", "ddddd", "pd", "dp"])
def test_results(gpu, kinds):
    import torch
    n = 256
    hs, outs = members(kinds, n)
    for _ in range(3):
        cs.compute_group(hs)
    torch.cuda.synchronize()
    src = field(n, n, 1)
    for (inp, out, wt), (nm, v, H, L, R, V, T, B, w, fun, _) in zip(outs, sweep_operators(n)):
        ref = sentinel(n, n)
        oracle.stencil(v, ref, src, np.asarray(w), num_tiles=1, block_x=32, block_y=8, H=H, L=L, R=R, V=V, T=T, B=B,
                       fun_id=fun)
        assert out.cpu().numpy().tobytes() == ref.tobytes(), nm
    for h in hs:
        h.destroy()


def test_host_members_overlap(gpu):
    """Six pinned members move as many bytes in as out: one behind the other each direction waits for the other
    (measured 1.7 times the group's time), so four fifths of that bounds a group whose members overlap."""
    import torch
    hs, keep = members("pppppp", 2048)

    def best(run):
        t = []
        for _ in range(8):
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            run()
            torch.cuda.synchronize()
            t.append(time.perf_counter() - t0)
        return min(t)

    one = torch.cuda.Stream()
    apart = best(lambda: [h.compute(stream=one) for h in hs])
    assert best(lambda: cs.compute_group(hs)) < 0.8 * apart
    for h in hs:
        h.destroy()
