"""Performance cases of the framework, through its public Python entry points.

Each case is a dict of plain values; `kind` selects the path:

  ops    one Compute of each operator of a set over one device-resident field (a time step's derivatives)
  weno   one Compute of the WENO5 advection operator
  host   one Compute of each operator of a set over pinned host fields, streamed in numTiles tiles (HOST offload)
  ch     `steps` steps of a batch of Cahn-Hilliard grids, then every grid's two fields read into device arrays
  serve  a Cahn-Hilliard server run of a list of requests, results read back
  pent   factorisation and solve of batched pentadiagonal systems whose coefficients change every step
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

import custen_gb300 as cs
from custen_gb300 import inputs

GAMMA, DT_FACTOR = 0.01, 0.1


def listed():
    return [
        # a 256^2 model problem's twelve derivatives: every launch is a few microseconds, so launches count
        {"name": "ops_256", "kind": "ops", "set": "sweep", "nx": 256, "ny": 256, "dtype": "f64", "group": False, "tiles": 1},
        # the benchmark's smallest size, as one grouped call: one tile wave per operator
        {"name": "ops_1024_group", "kind": "ops", "set": "sweep", "nx": 1024, "ny": 1024, "dtype": "f64", "group": True, "tiles": 1},
        # a production field (0.5 GB, larger than L2), one grouped call per step as in the benchmark
        {"name": "ops_8192_group", "kind": "ops", "set": "sweep", "nx": 8192, "ny": 8192, "dtype": "f64", "group": True, "tiles": 1},
        # the precision variant, bound by HBM, in four tiles as a program written for streaming leaves it
        {"name": "ops_f32_4096", "kind": "ops", "set": "sweep", "nx": 4096, "ny": 4096, "dtype": "f32", "group": False, "tiles": 4},
        # the wider windows and user functions of the examples on a field whose sides fit no tile
        {"name": "ops_wide_1999x1501", "kind": "ops", "set": "wide", "nx": 1999, "ny": 1501, "dtype": "f64", "group": False, "tiles": 1},
        # level-set advection on a medium field
        {"name": "weno_2048", "kind": "weno", "nx": 2048, "ny": 2048, "tiles": 1},
        # the reference's way of working: fields in host memory, larger than a user wants to keep on the device
        {"name": "host_4096_tiles4", "kind": "host", "set": "short", "nx": 4096, "ny": 4096, "tiles": 4},
        # one simulation alone, as the reference's program runs it
        {"name": "ch_alone_512", "kind": "ch", "sizes": "512", "steps": 40, "dtype": "f64"},
        # a parameter study of uneven grids, the batch the solver was built for
        {"name": "ch_batch_96", "kind": "ch", "sizes": "64x20,128x19,256x20,512x18,1024x19", "steps": 20, "dtype": "f64"},
        # the FP32-stencil variant on a small study
        {"name": "ch_batch_24_f32", "kind": "ch", "sizes": "96x6,160x6,256x6,384x6", "steps": 40, "dtype": "f32"},
        # a served queue of requests of different sizes and lengths, all waiting when the server starts
        {"name": "serve_24", "kind": "serve", "requests": 24, "lo": 64, "hi": 512, "steps_lo": 20, "steps_hi": 80},
        # implicit solves of many lines whose coefficients depend on the solution, so they are factorised every step
        {"name": "pent_131072x256", "kind": "pent", "m": 256, "batch": 131072, "inverted": False},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["ops", "ops", "ops", "weno", "host", "ch", "ch", "ch", "serve", "pent", "pent"])
    if kind == "ops":
        s = rng.choice(["sweep", "sweep", "wide"])
        nx, ny = _log(rng, 200, 6000), _log(rng, 200, 6000)
        if s == "sweep":   # the non-periodic operators take whole 8 x 8 blocks
            nx, ny = nx // 8 * 8, ny // 8 * 8
        return {"kind": "ops", "set": s, "nx": nx, "ny": ny, "dtype": rng.choice(["f64", "f64", "f32"]),
                "group": rng.random() < 0.4, "tiles": 1}
    if kind == "weno":
        return {"kind": "weno", "nx": _log(rng, 150, 4000), "ny": _log(rng, 150, 4000), "tiles": 1}
    if kind == "host":
        return {"kind": "host", "set": "short", "nx": _log(rng, 1024, 4096) // 8 * 8, "ny": _log(rng, 1024, 4096) // 32 * 32, "tiles": 4}
    if kind == "ch":
        count = _log(rng, 1, 40)
        steps = _log(rng, 4, 40)
        top = rng.choice([256, 512, 1024, 2048]) if count <= 4 else rng.choice([256, 512, 1024])
        ns = [32 * max(2, round(_log(rng, 64, top) / 32)) for _ in range(count)]
        steps = min(steps, max(1, 400_000_000 // sum(n * n for n in ns)))
        return {"kind": "ch", "sizes": ",".join("%dx1" % n for n in sorted(ns)), "steps": steps, "dtype": rng.choice(["f64", "f64", "f32"])}
    if kind == "serve":
        lo = rng.choice([64, 128])
        a = _log(rng, 4, 40)
        return {"kind": "serve", "requests": _log(rng, 2, 24), "lo": lo, "hi": rng.choice([256, 512]), "steps_lo": a, "steps_hi": 2 * a}
    m = _log(rng, 16, 1024)
    return {"kind": "pent", "m": m, "batch": _log(rng, 500, 32_000_000 // m), "inverted": rng.random() < 0.4}


# ---- operators --------------------------------------------------------------------------------------------

def _operators(case):
    """(variant, H, L, R, V, T, B, weights, function id) of the case's operator set; weights for spacing 2 pi / nx."""
    n = case["nx"]
    h = 2 * math.pi / n
    sweep = [o[1:10] for o in inputs.sweep_operators(n)]
    if case["set"] == "sweep":
        return sweep
    if case["set"] == "short":   # d2/dx2, d2/dy2 and the cross derivative, each without and with boundaries
        return [sweep[k] for k in (0, 1, 4, 5, 8, 9)]
    w9 = [w / (5040 * h * h) for w in (-9, 128, -1008, 8064, -14350, 8064, -1008, 128, -9)]   # 8th-order d2
    bih = [w / h ** 4 for w in (0, 0, -1, 0, 0, 0, -2, 8, -2, 0, -1, 8, -20, 8, -1, 0, -2, 8, -2, 0, 0, 0, -1, 0, 0)]
    k = np.random.default_rng(7).uniform(0.1, 1.0, 9).tolist()   # a dense 3 x 3 filter
    up = [w / (6 * h) for w in (1, -6, 3, 2)]                     # third-order upwind-biased d/dx, uneven halo
    return [(cs.XP, 9, 4, 4, 1, 0, 0, w9, -1), (cs.YP, 1, 0, 0, 9, 4, 4, w9, -1),
            (cs.XYP, 5, 2, 2, 5, 2, 2, bih, -1), (cs.XYP, 3, 1, 1, 3, 1, 1, k, -1),
            (cs.XP, 4, 2, 1, 1, 0, 0, up, -1), (cs.XPFUN, 3, 1, 1, 1, 0, 0, [1 / (h * h)], 0),
            (cs.YPFUN, 1, 0, 0, 9, 4, 4, w9, 2), (cs.XYPFUN, 3, 1, 1, 3, 1, 1, k, 4),
            (cs.XYPFUN, 3, 1, 1, 3, 1, 1, sweep[10][7], 5)]


def _field(nx, ny, seed):
    """sin(3x)cos(5y) + U(-1e-3, 1e-3), the benchmark's field."""
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    x = torch.arange(nx, device="cuda", dtype=torch.float64) * (2 * math.pi / nx)
    y = torch.arange(ny, device="cuda", dtype=torch.float64) * (2 * math.pi / ny)
    f = torch.rand(ny, nx, device="cuda", dtype=torch.float64, generator=g).mul_(2e-3).sub_(1e-3)
    return f.add_(torch.sin(3 * x)[None, :] * torch.cos(5 * y)[:, None])


def _prepare_ops(case, seed):
    host = case["kind"] == "host"
    nx, ny = case["nx"], case["ny"]
    dt, code = (torch.float32, cs.F32) if case.get("dtype") == "f32" else (torch.float64, cs.F64)
    inp = _field(nx, ny, seed).to(dt)
    if host:
        inp = torch.empty(ny, nx, dtype=dt, pin_memory=True).copy_(inp)
    outs, ws, handles = [], [], []
    for v, H, L, R, V, T, B, w, fid in _operators(case):
        out = torch.zeros(ny, nx, dtype=dt, pin_memory=True) if host else torch.zeros(ny, nx, dtype=dt, device="cuda")
        wt = torch.tensor(w, dtype=dt)
        wt = wt.pin_memory() if host else wt.cuda()
        func = cs.builtin_function(fid, code) if fid >= 0 else None
        block = 8 if nx % 8 == 0 and ny % 8 == 0 else 1
        handles.append(cs.Stencil(v, nx, ny, out, inp, wt, H=H, L=L, R=R, V=V, T=T, B=B, num_tiles=case["tiles"],
                                  block_x=block, block_y=block, dtype=code, ncoef=len(w), func=func))
        outs.append(out)
        ws.append(wt)
    return {"case": case, "inp": inp, "outs": outs, "weights": ws, "handles": handles}


def _run_ops(state):
    s = torch.cuda.current_stream()
    if state["case"].get("group"):
        cs.compute_group(state["handles"], stream=s)
    elif state["case"]["kind"] == "host":
        for h in state["handles"]:
            h.compute(cs.HOST)
        torch.cuda.synchronize()   # the fields are read on the host
    else:
        for h in state["handles"]:
            h.compute(stream=s)
    return state["outs"]


def _exact_ops(case, seed):
    dt = torch.float32 if case.get("dtype") == "f32" else torch.float64
    f = _field(case["nx"], case["ny"], seed).to(dt).double()
    nx, ny = case["nx"], case["ny"]
    res = []
    for v, H, L, R, V, T, B, w, fid in _operators(case):
        w = torch.tensor(w, dtype=dt).double().tolist()
        if fid == 0:
            w = [w[0], -2 * w[0], w[0]]
        src = f * f * f - f if fid in (1, 3, 5) else f
        out = torch.zeros_like(src)
        for j in range(V):
            for i in range(H):
                if w[j * H + i] != 0.0:
                    out.add_(torch.roll(src, (T - j, L - i), (0, 1)), alpha=w[j * H + i])
        if v in (cs.XNP, cs.XNPFUN, cs.XYNP, cs.XYNPFUN):   # columns and rows the operator does not write stay zero
            out[:, :L] = 0
            out[:, nx - R:] = 0
        if v in (cs.YNP, cs.YNPFUN, cs.XYNP, cs.XYNPFUN):
            out[:T] = 0
            out[ny - B:] = 0
        res.append(out)
    return res


# ---- WENO advection ---------------------------------------------------------------------------------------

def _weno_inputs(case, seed):
    nx, ny = case["nx"], case["ny"]
    g = torch.Generator(device="cuda").manual_seed(1000 + int(seed))
    u, v = (torch.rand(ny, nx, device="cuda", dtype=torch.float64, generator=g).mul_(2).sub_(1) for _ in range(2))
    u[torch.rand(ny, nx, device="cuda", generator=g) < 0.05] = 0.0   # still fluid: exact zeros
    v[torch.rand(ny, nx, device="cuda", generator=g) < 0.05] = 0.0
    return _field(nx, ny, seed), u, v, 2 * math.pi / nx, 2 * math.pi / ny


def _prepare_weno(case, seed):
    f, u, v, dx, dy = _weno_inputs(case, seed)
    out = torch.zeros_like(f)
    h = cs.WenoAdvection(case["nx"], case["ny"], out, f, u, v, dx=dx, dy=dy, num_tiles=case["tiles"])
    return {"case": case, "fields": (f, u, v), "outs": [out], "handles": [h]}


def _weno5(a, b, c, d, e):
    s1 = 13 / 12 * (a - 2 * b + c) ** 2 + 0.25 * (a - 4 * b + 3 * c) ** 2
    s2 = 13 / 12 * (b - 2 * c + d) ** 2 + 0.25 * (b - d) ** 2
    s3 = 13 / 12 * (c - 2 * d + e) ** 2 + 0.25 * (3 * c - 4 * d + e) ** 2
    g1, g2, g3 = 0.1 / (s1 + 1e-6) ** 2, 0.6 / (s2 + 1e-6) ** 2, 0.3 / (s3 + 1e-6) ** 2
    q1, q2, q3 = a / 3 - 7 / 6 * b + 11 / 6 * c, -b / 6 + 5 / 6 * c + d / 3, c / 3 + 5 / 6 * d - e / 6
    return (g1 * q1 + g2 * q2 + g3 * q3) / (g1 + g2 + g3)


def _exact_weno(case, seed):
    f, u, v, dx, dy = _weno_inputs(case, seed)
    out = torch.zeros_like(f)
    for vel, dim, h in ((u, 1, dx), (v, 0, dy)):
        D = (f - torch.roll(f, 1, dim)) / h
        at = lambda k: torch.roll(D, -k, dim)   # noqa: E731
        out += vel * torch.where(vel > 0, _weno5(at(-2), at(-1), D, at(1), at(2)), _weno5(at(3), at(2), at(1), D, at(-1)))
    return [out]


# ---- Cahn-Hilliard ----------------------------------------------------------------------------------------

def _sizes(case):
    out = []
    for part in case["sizes"].split(","):
        n, _, k = part.partition("x")
        out += [int(n)] * int(k or 1)
    return out


def _start_field(n, seed):
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    return torch.rand(n, n, device="cuda", dtype=torch.float64, generator=g).mul_(0.2).sub_(0.1)


def _prepare_ch(case, seed):
    sizes = _sizes(case)
    batch = cs.CahnHilliardBatch(sizes, gamma=GAMMA, dt_factor=DT_FACTOR, rhs_dtype=cs.F32 if case["dtype"] == "f32" else cs.F64)
    total = sum(n * n for n in sizes)
    cur, old = (torch.empty(total, dtype=torch.float64, device="cuda") for _ in range(2))
    for k, n in enumerate(sizes):
        c0 = _start_field(n, 10_000 * seed + k)
        torch.cuda.synchronize()
        cs._ch_check(cs.lib().custen_ch_batch_set_state(batch.h, k, c0.data_ptr(), None))   # device fields
    return {"case": case, "batch": batch, "sizes": sizes, "cur": cur, "old": old}


def _run_ch(state):
    batch, cur, old = state["batch"], state["cur"], state["old"]
    batch.step(state["case"]["steps"])
    off = 0
    for k, n in enumerate(state["sizes"]):
        cs._ch_check(cs.lib().custen_ch_batch_get_state(batch.h, k, cur.data_ptr() + 8 * off, old.data_ptr() + 8 * off))
        off += n * n
    return {"c": cur, "c_old": old}


def _ch_exact_steps(c, steps):
    n = c.shape[0]
    dx = 2 * math.pi / n
    dt = DT_FACTOR * dx
    sl, snl = 2 * dt * GAMMA / (3 * dx ** 4), 2 * dt / (3 * dx * dx)
    w = 2 - 2 * torch.cos(2 * math.pi * torch.arange(n, device=c.device, dtype=torch.float64) / n)
    inv = 1 / ((1 + sl * w[:, None] ** 2) * (1 + sl * w[None, : n // 2 + 1] ** 2))

    def lap(a):
        return torch.roll(a, 1, 0) + torch.roll(a, -1, 0) + torch.roll(a, 1, 1) + torch.roll(a, -1, 1) - 4 * a

    old = c.clone()
    for _ in range(steps):
        bar = 2 * c - old
        rhs = lap(snl * (c * c * c - c) - sl * lap(bar)) - (2.0 / 3.0) * (c - old)
        old, c = c, bar + torch.fft.irfft2(torch.fft.rfft2(rhs) * inv, s=(n, n))
    return c, old


def _exact_ch(case, seed):
    got = [_ch_exact_steps(_start_field(n, 10_000 * seed + k), case["steps"]) for k, n in enumerate(_sizes(case))]
    return {"c": torch.cat([a.reshape(-1) for a, _ in got]), "c_old": torch.cat([b.reshape(-1) for _, b in got])}


def _requests(case, seed):
    """(size, steps) of each request: sizes and lengths as a mixed queue has them, the same for every seed."""
    rng = np.random.default_rng(11 + case["requests"])
    ns = [int(n) // 32 * 32 for n in np.exp(rng.uniform(np.log(case["lo"]), np.log(case["hi"] + 1), case["requests"]))]
    return list(zip(ns, [int(s) for s in rng.integers(case["steps_lo"], case["steps_hi"] + 1, case["requests"])]))


def _prepare_serve(case, seed):
    reqs = _requests(case, seed)
    return {"case": case, "reqs": reqs, "c0": [_start_field(n, 10_000 * seed + k).cpu().numpy() for k, (n, _) in enumerate(reqs)]}


def _run_serve(state):
    srv = cs.CahnHilliardServer(hbm_budget_bytes=20e9, gamma=GAMMA, dt_factor=DT_FACTOR)
    ids = [srv.submit(n, steps, arrival=0.0, c0=c0) for (n, steps), c0 in zip(state["reqs"], state["c0"])]
    srv.run()
    res = [srv.result(r)["field"] for r in ids]
    srv.close()
    return res


def _exact_serve(case, seed):
    return [_ch_exact_steps(_start_field(n, 10_000 * seed + k), steps)[0].cpu().numpy() for k, (n, steps) in enumerate(_requests(case, seed))]


# ---- batched pentadiagonal systems ------------------------------------------------------------------------

def _pent_system(case, seed):
    """Diagonally dominant systems in cuPentBatch's interleaved layout (inputs.pent_system, made on the GPU)."""
    m, batch = case["m"], case["batch"]
    g = torch.Generator(device="cuda").manual_seed(2000 + int(seed))
    ds, dl, du, dw, d, b = (torch.rand(m, batch, device="cuda", dtype=torch.float64, generator=g) for _ in range(6))
    for a in (ds, dl, du, dw, b):
        a.mul_(2).sub_(1)
    d.mul_(3).add_(5)
    d *= torch.where(torch.rand(m, batch, device="cuda", generator=g) < 0.5, 1.0, -1.0)
    ds[:2] = 0
    dl[:1] = 0
    du[m - 1:] = 0
    dw[m - 2:] = 0
    return [ds, dl, d, du, dw, b]


def _prepare_pent(case, seed):
    src = _pent_system(case, seed)
    return {"case": case, "src": src, "work": [torch.empty_like(a) for a in src]}


def _run_pent(state):
    case, work = state["case"], state["work"]
    for w, a in zip(work, state["src"]):   # this step's coefficients and right-hand sides
        w.copy_(a)
    s = torch.cuda.current_stream()
    cs.pent_factor_batch(*work[:5], case["m"], case["batch"], stream=s)
    if case["inverted"]:
        cs.pent_invert_pivots(work[2], case["m"], case["batch"], stream=s)
    cs.pent_solve_batch(*work, case["m"], case["batch"], stream=s, inverted_pivots=case["inverted"])
    return work


def _exact_pent(case, seed):
    ds, dl, d, du, dw, b = _pent_system(case, seed)
    m = case["m"]
    for i in range(m):
        if i >= 2:
            dl[i] -= ds[i] * du[i - 2]
            d[i] -= ds[i] * dw[i - 2]
        if i >= 1:
            d[i] -= dl[i] * du[i - 1]
            du[i] -= dl[i] * dw[i - 1]
        if i < m - 1:
            du[i] /= d[i]
        if i < m - 2:
            dw[i] /= d[i]
    for i in range(m):
        if i >= 2:
            b[i] -= ds[i] * b[i - 2]
        if i >= 1:
            b[i] -= dl[i] * b[i - 1]
        b[i] /= d[i]
    for i in range(m - 2, -1, -1):
        b[i] -= du[i] * b[i + 1]
        if i < m - 2:
            b[i] -= dw[i] * b[i + 2]
    return [ds, dl, 1 / d if case["inverted"] else d, du, dw, b]


# ---- interface --------------------------------------------------------------------------------------------

_PREPARE = {"ops": _prepare_ops, "host": _prepare_ops, "weno": _prepare_weno, "ch": _prepare_ch, "serve": _prepare_serve,
            "pent": _prepare_pent}
_EXACT = {"ops": _exact_ops, "host": _exact_ops, "weno": _exact_weno, "ch": _exact_ch, "serve": _exact_serve,
          "pent": _exact_pent}


def prepare(case, seed):
    return _PREPARE[case["kind"]](case, int(seed))


def run(state):
    kind = state["case"]["kind"]
    if kind in ("ops", "host"):
        return _run_ops(state)
    if kind == "weno":
        state["handles"][0].compute(stream=torch.cuda.current_stream())
        return state["outs"]
    return {"ch": _run_ch, "serve": _run_serve, "pent": _run_pent}[kind](state)


def exact(case, seed):
    return _EXACT[case["kind"]](case, int(seed))


def work(case):
    kind = case["kind"]
    if kind in ("ops", "host"):
        pts, size = case["nx"] * case["ny"], 4 if case.get("dtype") == "f32" else 8
        ops = _operators(case)
        cube = sum(3 for o in ops if o[8] in (1, 3, 5))
        return {"bytes": pts * size * (1 + len(ops)), "flops": pts * (cube + sum(2 * sum(x != 0.0 for x in o[7]) for o in ops))}
    if kind == "weno":
        pts = case["nx"] * case["ny"]
        return {"bytes": 32 * pts, "flops": 200 * pts}
    if kind in ("ch", "serve"):
        if kind == "ch":
            todo = [(n, case["steps"]) for n in _sizes(case)]
        else:
            todo = _requests(case, 0)
        # per pass: the two fields in, the two fields out; per point and step the explicit stencils, two
        # five-operation line solves and the update
        return {"bytes": sum(32 * n * n for n, _ in todo), "flops": sum(50 * n * n * s for n, s in todo)}
    return {"bytes": 8 * case["m"] * case["batch"] * 12, "flops": 23 * case["m"] * case["batch"]}
