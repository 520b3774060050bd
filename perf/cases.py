"""The work a user has this framework do, as cases that can be timed and checked.

A case is a dict of plain values.  `prepare` makes what a program holds before the call
(static data set up once, initial states made from the seed), `run` is one pass through
the public entry points, `exact` the same results from plain torch in 64 bits.

Kinds
    forecast   the plain drop-in form: initial state in, `steps` RK4 steps, final state
               out; "loop" is "step" (swe_cuda_step) or "substep" (the reference's time
               loop, one swe_cuda_rk_substep per stage); "watch" adds the mass / energy
               watchdog at the end
    rhs        one right-hand side through the parity entry point, arrays in the
               reference's default (tiled) layout
    noalloc    steps on the caller's own device arrays
    ensemble   the batched form: states of all members in, `steps` steps, states out
    serve      a batch of forecast requests over two resident grids
    generate   stencils and weights of a node set
    order      the bandwidth-reducing node order of a stencil graph
"""
import functools
import math
import os
import random
import sys
import types

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "rbf-fd-swe_b200"))

from swe_b200 import capi, gen, layout, swe_input  # noqa: E402

STATIC = ("x", "y", "z", "f", "ghm", "p_u", "p_v", "p_w", "gradghm", "Dx", "Dy", "Dz", "L")
TILE = 32                      # SIMD_LENGTH of the tiled layout
L2_BYTES = 126 << 20           # static data above this is read again in every stage


def listed():
    return [
        # a few steps of the shipped N=2562 input's grid: launches and latency
        {"name": "forecast_n2562_short", "kind": "forecast", "n": 2562, "nnbr": 31, "dtype": "fp64", "steps": 10,
         "loop": "step", "watch": False},
        # the reference's own time loop (one call per RK stage) on a grid of odd size and narrower stencils
        {"name": "forecast_n9731_substeps", "kind": "forecast", "n": 9731, "nnbr": 28, "dtype": "fp64", "steps": 50,
         "loop": "substep", "watch": False},
        # the headline grid between two outputs, with the watchdog
        {"name": "forecast_n40962", "kind": "forecast", "n": 40962, "nnbr": 31, "dtype": "fp64", "steps": 100,
         "loop": "step", "watch": True},
        # single precision, the reference's FP32 build
        {"name": "forecast_n163842_fp32", "kind": "forecast", "n": 163842, "nnbr": 31, "dtype": "fp32", "steps": 40,
         "loop": "step", "watch": False},
        # the largest configured grid
        {"name": "forecast_n655362", "kind": "forecast", "n": 655362, "nnbr": 31, "dtype": "fp64", "steps": 20,
         "loop": "step", "watch": False},
        # a parity check of one right-hand side from the reference's default layout
        {"name": "rhs_n40962", "kind": "rhs", "n": 40962, "nnbr": 31, "dtype": "fp64"},
        # a caller that owns all device memory
        {"name": "noalloc_n10242", "kind": "noalloc", "n": 10242, "nnbr": 31, "dtype": "fp64", "steps": 20},
        # 64 members of a 60 km grid in the default precision
        {"name": "ensemble_n163842_m64", "kind": "ensemble", "n": 163842, "nnbr": 31, "members": 64,
         "precision": "tf32x3", "steps": 20},
        # 32 members of the headline grid in split FP16
        {"name": "ensemble_n40962_m32_fp16", "kind": "ensemble", "n": 40962, "nnbr": 31, "members": 32,
         "precision": "fp16x3", "steps": 50},
        # a burst of forecast requests over two grids
        {"name": "serve_n40962", "kind": "serve", "n": 40962, "nnbr": 31, "requests": 12, "members": 8, "steps": 50},
        # stencils and weights of a new node set
        {"name": "generate_n163842", "kind": "generate", "n": 163842, "nnbr": 31},
        # node order of a new stencil graph
        {"name": "order_n655362", "kind": "order", "n": 655362, "nnbr": 31},
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["forecast"] * 5 + ["rhs", "noalloc", "ensemble", "ensemble", "serve", "generate", "order"])
    nnbr = rng.choice([31, 31, 31, 25, 28, 32])
    c = {"kind": kind, "nnbr": nnbr}
    if kind == "forecast":
        c["n"] = size(1000, 655362)
        c["dtype"] = rng.choice(["fp64", "fp64", "fp32"])
        c["steps"] = max(1, min(size(5, 200), 13_000_000 // c["n"]))
        c["loop"] = rng.choice(["step", "step", "substep"])
        c["watch"] = rng.random() < 0.3
    elif kind == "rhs":
        c["n"] = size(1000, 655362)
        c["dtype"] = rng.choice(["fp64", "fp32"])
    elif kind == "noalloc":
        c["dtype"] = rng.choice(["fp64", "fp32"])
        c["n"] = size(1000, 43690 if c["dtype"] == "fp64" else 87381)
        c["steps"] = size(1, 50)
    elif kind == "ensemble":
        c["n"] = size(2562, 163842)
        c["members"] = rng.choice([32, 64])
        c["precision"] = rng.choice(["tf32x3", "fp16x3", "bf16x3"])
        c["steps"] = max(1, min(size(5, 100), 3_200_000 // c["n"]))
    elif kind == "serve":
        c["n"] = size(5000, 40962)
        c["requests"], c["members"], c["steps"] = rng.randint(2, 16), rng.randint(1, 8), rng.randint(10, 40)
    elif kind == "generate":
        c["n"] = size(1000, 163842)
    else:
        c["n"] = size(1000, 655362)
    return c


# ---- inputs ---------------------------------------------------------------------------------


def _bisected(n):
    return any(n == 10 * 4 ** level + 2 for level in range(12))


def _nodes(n):
    """Quasi-uniform unit vectors: the bisected icosahedron where n is one of its sizes, else a spiral."""
    if _bisected(n):
        return gen.icosahedral_nodes(gen.level_of(n))
    t = np.arange(n) + 0.5
    z = 1.0 - 2.0 * t / n
    a = math.pi * (1.0 + math.sqrt(5.0)) * t
    r = np.sqrt(1.0 - z * z)
    return np.stack([r * np.cos(a), r * np.sin(a), z], 1)


@functools.lru_cache(maxsize=2)
def _model(n, nnbr):
    """The grid in reverse Cuthill-McKee order, from the package's host and torch path.  The
    hyperviscosity of the spiral's stencils allows a quarter of the bisected grids' time step."""
    X = _nodes(n)
    idx = gen.stencils(X, nnbr)
    Dx, Dy, Dz, L = gen.rbffd_weights(X, idx, device="cuda")
    H, ghm = gen.tc5_state(X, 0, noise=0.0)
    gradghm = np.stack([np.einsum("ij,ij->i", D, ghm[idx]) / gen.A_EARTH for D in (Dx, Dy, Dz)], 1)
    P = np.eye(3)[None] - X[:, :, None] * X[:, None, :]
    d = swe_input.SweInput(
        N=n, Nnbr=nnbr, a=gen.A_EARTH, gh0=gen.G * gen.H0, dt=min(900.0, 225.0 * math.sqrt(40962 / n)) * (1.0 if _bisected(n) else 0.25),
        gamma=-gen.GAMMA_COEF * float(n) ** -4,
        x=X[:, 0].copy(), y=X[:, 1].copy(), z=X[:, 2].copy(), f=2.0 * gen.OMEGA * X[:, 2], ghm=ghm,
        p_u=P[:, 0].copy(), p_v=P[:, 1].copy(), p_w=P[:, 2].copy(), gradghm=gradghm,
        Dx=Dx, Dy=Dy, Dz=Dz, L=L, idx1=(idx + 1).astype(np.int32), H_init=H, H_100=np.zeros_like(H))
    m = swe_input.to_model(d)
    return layout.reorder(m, layout.rcm_mapping(m))


def _members(m, count, seed, dtype=torch.float64):
    """[count, n, 4] states on the host (pinned): the zonal flow with 1e-3 noise on h."""
    g = torch.Generator("cuda").manual_seed(int(seed))
    H = torch.from_numpy(m.H_init).cuda().repeat(count, 1, 1)
    H[:, :, 3] *= 1.0 + gen.NOISE * torch.randn((count, m.N), generator=g, device="cuda", dtype=torch.float64)
    return H.to(dtype).cpu().pin_memory()


def _jittered(n, seed):
    """Device [n, 3] unit vectors: the node set moved by a few per cent of its spacing."""
    g = torch.Generator("cuda").manual_seed(int(seed))
    X = torch.from_numpy(_nodes(n)).cuda()
    X = X + 0.04 * math.sqrt(4 * math.pi / n) * torch.randn((n, 3), generator=g, device="cuda", dtype=torch.float64)
    return (X / X.norm(dim=1, keepdim=True)).contiguous()


def _mix(case):
    """(grid 0 / 1, members, steps) of each request of a serve case."""
    r = random.Random(case["n"])
    return [(r.randrange(2), r.randint(1, case["members"]), r.randint((case["steps"] + 4) // 5, case["steps"]))
            for _ in range(case["requests"])]


def _tiled(a, n, w):
    """[n, w] node-major -> the reference's tiled order (SVM_LIN_ID, DM_LIN_ID, VECT_LIN_ID without CFDL / with SFDL)."""
    return np.ascontiguousarray(a.reshape(n // TILE, TILE, w).transpose(0, 2, 1)).reshape(-1)


# ---- the handles a program keeps; the library has one of each form per process -----------------

_live = {"key": None, "drop": None, "handle": None}


def _handle(key, make, drop):
    if _live["key"] != key:
        if _live["drop"]:
            _live["drop"](_live["handle"])
            _live.update(key=None, drop=None)
        torch.cuda.synchronize()
        _live["handle"] = make()
        _live.update(key=key, drop=drop)
    return _live["handle"]


def _plain(case, tiled=False):
    m = _model(case["n"], case["nnbr"])

    def make():
        p = capi.Plain()
        if not tiled:
            p.init_model(m, case["dtype"])
            return p
        mp = layout.pad(m, TILE)
        t = np.float64 if case["dtype"] == "fp64" else np.float32
        arrs = {}
        for k in STATIC:
            a = np.ascontiguousarray(getattr(mp, k), dtype=t)
            arrs[k] = a if a.ndim == 1 else _tiled(a, mp.N, a.shape[1])
        arrs["idx"] = _tiled(np.ascontiguousarray(mp.idx, dtype=np.int32), mp.N, mp.Nnbr)
        p.init(np.dtype(t).itemsize, capi.SWE_LAYOUT_SFDL, TILE, mp.N, mp.N, 0, mp.Nnbr, mp.Nnbr,
               float(mp.gh0), float(mp.dt), arrs)
        return p

    return m, _handle(("plain", case["n"], case["nnbr"], case["dtype"], tiled), make, lambda p: p.finalize())


def _ensemble(case):
    m = _model(case["n"], case["nnbr"])

    def make():
        e = capi.Ensemble()
        e.init(m, case["members"])
        e.set_precision(case["precision"])
        return e

    key = ("ensemble", case["n"], case["nnbr"], case["members"], case["precision"])
    return m, _handle(key, make, lambda e: e.finalize())


def _server(case):
    models = [_model(n, case["nnbr"]) for n in (case["n"], case["n"] // 4)]

    def make():
        s = capi.Server(6e9, max_requests=64)
        return s, [s.add_grid(m) for m in models]

    return models, _handle(("serve", case["n"], case["nnbr"]), make, lambda h: h[0].stop())


def _dtype(case):
    return torch.float64 if case["dtype"] == "fp64" else torch.float32


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind == "forecast":
        m, s["plain"] = _plain(case)
        s["H0"] = _members(m, 1, seed, _dtype(case))[0]
        s["H"] = torch.empty_like(s["H0"]).pin_memory()
    elif kind == "rhs":
        m, s["plain"] = _plain(case, tiled=True)
        K = _members(m, 1, seed)[0].numpy()
        pad = -case["n"] % TILE
        K = np.concatenate([K, np.repeat(K[-1:], pad, 0)]).astype(np.float64 if case["dtype"] == "fp64" else np.float32)
        s["K"] = _tiled(K, len(K), 4)
    elif kind == "noalloc":
        m = _model(case["n"], case["nnbr"])
        s["gh0"], s["dt"] = float(m.gh0), float(m.dt)
        s["idx"] = torch.from_numpy(m.idx).cuda()
        s["static"] = {k: torch.from_numpy(np.ascontiguousarray(getattr(m, k))).to("cuda", _dtype(case)) for k in STATIC}
        s["H0"] = _members(m, 1, seed, _dtype(case))[0].cuda()
        s["H"] = torch.empty_like(s["H0"])
        fn = capi.load().swe_cuda_step_noalloc
        c = capi.ctypes
        fn.argtypes = [c.c_int, c.c_int, c.c_int, c.c_double, c.c_double] + [c.c_void_p] * 15 + [c.c_int, c.c_void_p]
    elif kind == "ensemble":
        m, s["ens"] = _ensemble(case)
        s["H0"] = _members(m, case["members"], seed)
        s["H"] = torch.empty_like(s["H0"]).pin_memory()
    elif kind == "serve":
        models, (s["server"], s["grids"]) = _server(case)
        s["requests"] = [(g, _members(models[g], mb, seed * 1000 + r).numpy(), st)
                         for r, (g, mb, st) in enumerate(_mix(case))]
    elif kind == "generate":
        s["X"] = _jittered(case["n"], seed)
    else:
        idx = gen.stencils_gpu(_jittered(case["n"], seed).cpu().numpy(), case["nnbr"])
        s["graph"] = types.SimpleNamespace(N=case["n"], Nnbr=case["nnbr"], idx=idx)
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "forecast":
        p = s["plain"]
        p.set_state_ptr(s["H0"].data_ptr())
        if case["loop"] == "step":
            p.step(case["steps"])
        else:
            for _ in range(case["steps"]):
                for k in range(4):
                    p.rk_substep(k)
        out = {}
        if case["watch"]:
            out["invariants"] = p.invariants()
        p.get_state_ptr(s["H"].data_ptr())
        return {"H": s["H"], **out}
    if kind == "rhs":
        return s["plain"].eval_rhs(s["K"])
    if kind == "noalloc":
        s["H"].copy_(s["H0"])
        st = s["static"]
        capi.check("swe_cuda_step_noalloc", capi.load().swe_cuda_step_noalloc(
            s["H"].element_size(), case["n"], case["nnbr"], s["gh0"], s["dt"], s["idx"].data_ptr(),
            *[st[k].data_ptr() for k in ("Dx", "Dy", "Dz", "L", "x", "y", "z", "f", "ghm", "p_u", "p_v", "p_w", "gradghm")],
            s["H"].data_ptr(), case["steps"], torch.cuda.current_stream().cuda_stream))
        return s["H"]
    if kind == "ensemble":
        e = s["ens"]
        e.set_state_ptr(s["H0"].data_ptr())
        e.step(case["steps"])
        e.get_state_ptr(s["H"].data_ptr())
        return s["H"]
    if kind == "serve":
        srv = s["server"]
        ids = [srv.submit(s["grids"][g], H0, st) for g, H0, st in s["requests"]]
        srv.wait(ids)
        return [srv.fetch(r) for r in ids]
    if kind == "generate":
        lib, n, k = capi.load(), case["n"], case["nnbr"]
        idx = torch.empty((n, k), dtype=torch.int32, device="cuda")
        D = torch.empty((4, n, k), dtype=torch.float64, device="cuda")
        capi.check("swe_gen_stencils", lib.swe_gen_stencils(n, k, s["X"].data_ptr(), idx.data_ptr()))
        capi.check("swe_gen_weights", lib.swe_gen_weights(n, k, s["X"].data_ptr(), idx.data_ptr(), D.data_ptr()))
        return {"idx": idx, "Dx": D[0], "Dy": D[1], "Dz": D[2], "L": D[3]}
    return layout.rcm_mapping(s["graph"], device=True)


# ---- what a pass cannot do without -----------------------------------------------------------


def _stage_work(n, nnbr, fsize, members=1):
    """(static bytes, state bytes, flops) of one RK stage: 16 stencil sums and the pointwise part per node and member;
    stencil weights, indices and 17 pointwise values read once; K in and K, D, H in and out as the stages have it."""
    static = n * (nnbr * (4 * fsize + 4) + 17 * fsize)
    state = n * members * 18 * fsize
    return static, state, n * members * (32 * nnbr + 110)


def _steps_work(n, nnbr, fsize, steps, members=1):
    static, state, flops = _stage_work(n, nnbr, fsize, members)
    if static + state <= L2_BYTES:        # stays on the chip: initial state in, final state out
        return {"bytes": static + 8 * n * members * fsize, "flops": 4 * steps * flops}
    return {"bytes": 4 * steps * (static + state), "flops": 4 * steps * flops}


def work(case):
    n, k, kind = case["n"], case["nnbr"], case["kind"]
    fsize = 4 if case.get("dtype") == "fp32" else 8
    if kind in ("forecast", "noalloc"):
        return _steps_work(n, k, fsize, case["steps"])
    if kind == "rhs":
        static, _, flops = _stage_work(n, k, fsize)
        return {"bytes": static + 8 * n * fsize, "flops": flops}
    if kind == "ensemble":                # FP32 states
        return _steps_work(n, k, 4, case["steps"], case["members"])
    if kind == "serve":
        ws = [_steps_work(n if g == 0 else n // 4, k, 8, st, mb) for g, mb, st in _mix(case)]
        return {x: sum(w[x] for w in ws) for x in ("bytes", "flops")}
    if kind == "generate":                # two dense solves a node: LU and the right-hand sides
        ns = k + 15
        return {"bytes": n * (24 + 4 * k + 32 * k), "flops": n * (2 * (2 * ns ** 3 / 3) + 4 * 2 * ns * ns)}
    return {"bytes": n * (4 * k + 4), "flops": 0}


# ---- the same results in 64 bits ---------------------------------------------------------------


def _static64(m, dtype=np.float64):
    f = {k: torch.from_numpy(np.ascontiguousarray(getattr(m, k)).astype(dtype)).cuda().double() for k in STATIC}
    f["W"] = torch.stack([f["Dx"], f["Dy"], f["Dz"], f["L"]], 1)          # [n, 4, nnbr]
    f["idx"] = torch.from_numpy(m.idx).cuda().long()
    f["gh0"], f["dt"] = float(dtype(m.gh0)), float(dtype(m.dt))
    return f


def _rhs64(f, K):
    """K, F: [n, B, 4]."""
    n, B, _ = K.shape
    G = K.reshape(n, 4 * B)[f["idx"]]                                      # [n, nnbr, 4 B]
    S = torch.bmm(f["W"], G).reshape(n, 4, B, 4)
    dx, dy, dz, hyp = S.unbind(1)                                          # [n, B, 4]
    u, v, w, h = (K[..., i] for i in range(4))
    x, y, z, cor, ghm = (f[k][:, None] for k in ("x", "y", "z", "f", "ghm"))
    adv = [u * dx[..., i] + v * dy[..., i] + w * dz[..., i] for i in range(3)]
    ru = -(adv[0] + cor * (y * w - z * v) + dx[..., 3])
    rv = -(adv[1] + cor * (z * u - x * w) + dy[..., 3])
    rw = -(adv[2] + cor * (x * v - y * u) + dz[..., 3])
    out = []
    for i, p in enumerate(("p_u", "p_v", "p_w")):
        P = f[p][:, None, :]
        out.append(P[..., 0] * ru + P[..., 1] * rv + P[..., 2] * rw + hyp[..., i])
    g = f["gradghm"][:, None, :]
    out.append(-(u * (dx[..., 3] - g[..., 0]) + v * (dy[..., 3] - g[..., 1]) + w * (dz[..., 3] - g[..., 2])
                 + (h + f["gh0"] - ghm) * (dx[..., 0] + dy[..., 1] + dz[..., 2])) + hyp[..., 3])
    return torch.stack(out, -1)


def _forecast64(f, H, steps, block=8):
    """H: [B, n, 4] on the host -> the states after `steps` RK4 steps."""
    done = []
    for b in range(0, H.shape[0], block):
        Y = H[b:b + block].cuda().double().transpose(0, 1).contiguous()    # [n, B, 4]
        for _ in range(steps):
            k1 = _rhs64(f, Y)
            k2 = _rhs64(f, Y + 0.5 * f["dt"] * k1)
            k3 = _rhs64(f, Y + 0.5 * f["dt"] * k2)
            k4 = _rhs64(f, Y + f["dt"] * k3)
            Y = Y + (f["dt"] / 6.0) * (k1 + 2.0 * k2 + 2.0 * k3 + k4)
        done.append(Y.transpose(0, 1).contiguous())
    return torch.cat(done)


def _invariants64(m, H):
    phi = H[:, 3] + float(m.gh0)
    thick = phi - torch.from_numpy(np.ascontiguousarray(m.ghm)).cuda()
    area = 4.0 * math.pi / m.N
    e = 0.5 * thick * (H[:, :3] ** 2).sum(1) + 0.5 * phi ** 2
    return np.array([float(thick.sum()) * area, float(e.sum()) * area])


def _knn64(X, k, chunk=1024):
    rows = []
    for s in range(0, len(X), chunk):
        d = sum((X[s:s + chunk, None, c] - X[None, :, c]) ** 2 for c in range(3))
        rows.append(d.topk(k, dim=1, largest=False, sorted=True).indices)
    return torch.cat(rows)


def exact(case, seed):
    kind = case["kind"]
    if kind == "order":
        return None
    if kind == "generate":
        X = _jittered(case["n"], seed)
        idx = _knn64(X, case["nnbr"]).cpu().numpy()
        D = _weights64(X.cpu().numpy(), idx)
        return {"idx": None, "Dx": D[0], "Dy": D[1], "Dz": D[2], "L": D[3]}
    if kind == "serve":
        models = [_model(n, case["nnbr"]) for n in (case["n"], case["n"] // 4)]
        f = [_static64(m) for m in models]
        return [_forecast64(f[g], _members(models[g], mb, seed * 1000 + r), st).cpu().numpy()
                for r, (g, mb, st) in enumerate(_mix(case))]
    m = _model(case["n"], case["nnbr"])
    np_t = np.float32 if case.get("dtype") == "fp32" else np.float64
    f = _static64(m, np_t)
    if kind == "ensemble":
        return _forecast64(f, _members(m, case["members"], seed), case["steps"]).cpu()
    H0 = _members(m, 1, seed, _dtype(case))
    if kind == "rhs":
        F = _rhs64(f, H0.cuda().double().transpose(0, 1).contiguous())[:, 0].cpu().numpy()
        pad = -case["n"] % TILE
        return _tiled(np.concatenate([F, np.repeat(F[-1:], pad, 0)]), case["n"] + pad, 4)
    H = _forecast64(f, H0, case["steps"])[0]
    if kind == "noalloc":
        return H
    return {"H": H, **({"invariants": _invariants64(m, H)} if case["watch"] else {})}


def _weights64(X, idx, chunk=16384):
    """[4, n, k] unit-sphere weights by batched dense solves: r^7 with the 15 tangent-plane
    polynomials for the projected gradient, r^9 on tangent-plane distances for Delta^4."""
    X, idx = torch.from_numpy(X).cuda(), torch.from_numpy(idx).cuda().long()
    n, k = idx.shape
    out = torch.empty((4, n, k), dtype=torch.float64, device="cuda")
    for s in range(0, n, chunk):
        c, S = X[s:s + chunk], X[idx[s:s + chunk]]
        a = torch.zeros_like(c)
        polar = c[:, 2].abs() >= 0.9
        a[:, 2], a[polar, 2], a[polar, 0] = 1.0, 0.0, 1.0
        e1 = torch.linalg.cross(c, a)
        e1 = e1 / e1.norm(dim=1, keepdim=True)
        e2 = torch.linalg.cross(c, e1)
        d = S - c[:, None]
        rho = d.norm(dim=2).amax(1)
        xi, eta = ((d * e[:, None]).sum(2) / rho[:, None] for e in (e1, e2))
        P = torch.stack([xi ** (t - b) * eta ** b for t in range(5) for b in range(t + 1)], -1)
        zero = torch.zeros((len(c), 15, 15), dtype=P.dtype, device="cuda")

        def solve(phi, rhs, low):
            A = torch.cat([torch.cat([phi, P], 2), torch.cat([P.transpose(1, 2), zero], 2)], 1)
            return torch.linalg.solve(A, torch.cat([rhs, low], 1))[:, :k]

        r = (S[:, :, None] - S[:, None]).norm(dim=3) / rho[:, None, None]
        rc = d.norm(dim=2) / rho[:, None]
        proj = c[:, None] * (S * c[:, None]).sum(2, keepdim=True) - S
        low = torch.zeros((len(c), 15, 3), dtype=P.dtype, device="cuda")
        low[:, 1], low[:, 2] = e1 / rho[:, None], e2 / rho[:, None]
        w = solve(r ** 7, 7.0 * (rc ** 5)[..., None] * proj / (rho ** 2)[:, None, None], low)
        out[:3, s:s + chunk] = w.permute(2, 0, 1)
        r = torch.sqrt((xi[:, :, None] - xi[:, None]) ** 2 + (eta[:, :, None] - eta[:, None]) ** 2)
        rhs = float((9 * 7 * 5 * 3) ** 2) * torch.sqrt(xi ** 2 + eta ** 2) / (rho ** 8)[:, None]
        out[3, s:s + chunk] = solve(r ** 9, rhs[..., None], zero[:, :, :1])[..., 0]
    return out
