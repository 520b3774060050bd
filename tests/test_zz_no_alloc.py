"""swe_cuda_step_noalloc: RK4 steps for callers that cannot allocate device memory.

Callers whose device memory belongs to an outer framework's pool, or whose
loops may not pay an allocation's implicit device synchronisation, own every
buffer themselves and pass device pointers; the entry point keeps its K/D
registers in a static device array instead of calling cudaMalloc.  This test
owns its buffers through torch (the test is the caller), runs the entry point
twice in a row through the C ABI, and compares each result with the
allocating entry point (swe_cuda_init + swe_cuda_step) at the tolerance the
other plain-form tests use, in FP64 and FP32, on a small grid and on one that
fills most of the static array.  It lives in its own file so that it is collected
last.
"""
import ctypes
import os

import numpy as np
import pytest

from conftest import GOLDEN, scaled_err
from swe_b200 import capi, swe_input

pytestmark = pytest.mark.gpu

NSTEPS = 20
# FP64: the other plain-form tests' 1e-12 relative bar.  FP32: both paths round every
# operation to FP32 in different summation orders (this path sums slots in the 8-lane
# tree, the allocating one in the kernel its init timing picked), so they are held to
# each other within 1e-4 of each field's scale after 20 steps (u, v, w on the velocity
# scale max|(u, v, w)|, h on max|h|) and to the reference's FP32 verify tolerance,
# 4e-2 absolute (swe_config.h:80).
REL_BAR = {"fp64": 1e-12, "fp32": 1e-4}


def _bind():
    lib = capi.load()
    vp, i, d = ctypes.c_void_p, ctypes.c_int, ctypes.c_double
    lib.swe_cuda_step_noalloc.argtypes = [i, i, i, d, d] + [vp] * 15 + [i, vp]
    lib.swe_cuda_step_noalloc.restype = i
    return lib


def _model(which):
    if which == "n162":
        return swe_input.load_model(os.path.join(GOLDEN, "icos162_seed7.bin"))
    # N=40962 (level 6): 94% of the FP64 node limit, so K, K and D fill most of the array
    from swe_b200 import gen
    return swe_input.to_model(gen.generate(6, seed=1, device="cuda"))


def _reference_steps(m, prec):
    plain = capi.Plain()
    plain.init_model(m, prec)
    plain.set_state(m.H_init.astype(np.float64 if prec == "fp64" else np.float32))
    plain.step(NSTEPS)
    H = plain.get_state().reshape(-1, 4)
    plain.finalize()
    return H


@pytest.mark.parametrize("which", ["n162", "n40962"])
@pytest.mark.parametrize("prec", ["fp64", "fp32"])
def test_noalloc_matches_allocating_entry_point_twice(prec, which):
    import torch

    lib = _bind()
    m = _model(which)
    fsize = 8 if prec == "fp64" else 4
    assert m.N <= capi.NOALLOC_SCRATCH_BYTES // (12 * fsize)
    dt = np.float64 if prec == "fp64" else np.float32
    want = _reference_steps(m, prec)
    dev = torch.device("cuda", torch.cuda.current_device())
    t = {k: torch.from_numpy(np.ascontiguousarray(getattr(m, k), dtype=dt)).to(dev) for k in
         ("Dx", "Dy", "Dz", "L", "x", "y", "z", "f", "ghm", "p_u", "p_v", "p_w", "gradghm")}
    t["idx"] = torch.from_numpy(np.ascontiguousarray(m.idx, dtype=np.int32)).to(dev)
    stream = torch.cuda.current_stream(dev)
    for call in range(2):
        H = torch.from_numpy(np.ascontiguousarray(m.H_init, dtype=dt)).to(dev)
        st = lib.swe_cuda_step_noalloc(
            fsize, m.N, m.Nnbr, float(m.gh0), float(m.dt), t["idx"].data_ptr(),
            *[t[k].data_ptr() for k in ("Dx", "Dy", "Dz", "L", "x", "y", "z", "f", "ghm",
                                        "p_u", "p_v", "p_w", "gradghm")],
            H.data_ptr(), NSTEPS, stream.cuda_stream)
        assert st == 0, lib.swe_cuda_last_error()
        # nsteps = 0 waits for the stream and reports any out-of-range stencil index
        # the kernels met: none here
        st = lib.swe_cuda_step_noalloc(
            fsize, m.N, m.Nnbr, float(m.gh0), float(m.dt), t["idx"].data_ptr(),
            *[t[k].data_ptr() for k in ("Dx", "Dy", "Dz", "L", "x", "y", "z", "f", "ghm",
                                        "p_u", "p_v", "p_w", "gradghm")],
            H.data_ptr(), 0, stream.cuda_stream)
        assert st == 0, lib.swe_cuda_last_error()
        got = H.cpu().numpy().reshape(-1, 4)
        assert np.isfinite(got).all(), f"call {call}"
        err = scaled_err(got, want)
        print(f"{prec} {which} call {call}: rel err per field {err}")
        assert err.max() <= REL_BAR[prec], f"call {call}"
        if prec == "fp32":
            assert np.abs(got.astype(np.float64) - want).max() <= 4e-2


def test_noalloc_rejects_sizes_beyond_its_static_scratch():
    lib = _bind()
    limit = capi.NOALLOC_SCRATCH_BYTES // (12 * 8)
    dummy = ctypes.c_void_p(16)          # never dereferenced: the size check comes first
    st = lib.swe_cuda_step_noalloc(8, limit + 1, 31, 0.0, 1.0, *([dummy] * 15), 1, None)
    assert st == 1
    assert b"static scratch" in lib.swe_cuda_last_error()


def _spiral(n, nnbr):
    """A grid of any size: nodes on a spiral, stencils and weights from the library's generator."""
    from swe_b200 import gen
    t = np.arange(n) + 0.5
    z = 1.0 - 2.0 * t / n
    r = np.sqrt(1.0 - z * z)
    X = np.stack([r * np.cos(np.pi * (1 + 5 ** 0.5) * t), r * np.sin(np.pi * (1 + 5 ** 0.5) * t), z], 1)
    idx = gen.stencils_gpu(X, nnbr)
    Dx, Dy, Dz, L = gen.rbffd_weights_gpu(X, idx)
    H, ghm = gen.tc5_state(X, n)
    P = np.eye(3)[None] - X[:, :, None] * X[:, None, :]
    gg = np.stack([np.einsum("ij,ij->i", D, ghm[idx]) / gen.A_EARTH for D in (Dx, Dy, Dz)], 1)
    return swe_input.to_model(swe_input.SweInput(
        N=n, Nnbr=nnbr, a=gen.A_EARTH, gh0=gen.G * gen.H0, dt=100.0, gamma=-gen.GAMMA_COEF * float(n) ** -4,
        x=X[:, 0].copy(), y=X[:, 1].copy(), z=X[:, 2].copy(), f=2 * gen.OMEGA * X[:, 2], ghm=ghm, p_u=P[:, 0].copy(),
        p_v=P[:, 1].copy(), p_w=P[:, 2].copy(), gradghm=gg, Dx=Dx, Dy=Dy, Dz=Dz, L=L, idx1=idx + 1, H_init=H,
        H_100=np.zeros_like(H)))


def _call(m, prec, nsteps, H, stream, t):
    lib = _bind()
    st = lib.swe_cuda_step_noalloc(
        8 if prec == "fp64" else 4, m.N, m.Nnbr, float(m.gh0), float(m.dt), t["idx"].data_ptr(),
        *[t[k].data_ptr() for k in ("Dx", "Dy", "Dz", "L", "x", "y", "z", "f", "ghm", "p_u", "p_v", "p_w", "gradghm")],
        H.data_ptr(), nsteps, stream)
    assert st == 0, lib.swe_cuda_last_error()


def _device_arrays(m, prec):
    import torch
    dt = np.float64 if prec == "fp64" else np.float32
    t = {k: torch.from_numpy(np.ascontiguousarray(getattr(m, k), dtype=dt)).cuda() for k in
         ("Dx", "Dy", "Dz", "L", "x", "y", "z", "f", "ghm", "p_u", "p_v", "p_w", "gradghm")}
    t["idx"] = torch.from_numpy(np.ascontiguousarray(m.idx, dtype=np.int32)).cuda()
    return t


# (nodes, neighbours): below and above the resident kernel's first size, nodes per block at and
# around multiples of 8, its 512- and 640-thread shapes with 4 and 2 lanes a node, the largest
# grids its shared memory holds and the first ones past it
@pytest.mark.parametrize("prec,n,nnbr", [
    ("fp64", 4999, 31), ("fp64", 5921, 17), ("fp64", 11840, 31), ("fp64", 18944, 32), ("fp64", 18945, 31),
    ("fp64", 23681, 28), ("fp64", 27232, 31), ("fp64", 27233, 32), ("fp32", 10001, 31), ("fp32", 18945, 32),
    ("fp32", 37889, 25), ("fp32", 47360, 31), ("fp32", 47361, 31)])
def test_noalloc_sizes_match_oracle_steps(prec, n, nnbr):
    import oracle
    import torch

    m = _spiral(n, nnbr)
    t = _device_arrays(m, prec)
    dt = np.float64 if prec == "fp64" else np.float32
    buf = torch.empty(4 * n + 2, dtype=torch.float64 if prec == "fp64" else torch.float32, device="cuda")
    for off in ((0, 2) if prec == "fp64" else (0,)):          # FP64: H 32- and 16-byte aligned
        H = buf[off:off + 4 * n].view(n, 4)
        H.copy_(torch.from_numpy(m.H_init.astype(dt)))
        _call(m, prec, 3, H, torch.cuda.current_stream().cuda_stream, t)
        want = oracle.Port(m, prec).run(m.H_init.astype(dt), 3)
        assert scaled_err(H.cpu().numpy(), want).max() <= (1e-12 if prec == "fp64" else 1e-4)


@pytest.mark.parametrize("n", [2000, 10242])
def test_noalloc_calls_can_be_captured(n):
    """A call captured in a CUDA graph and replayed twice gives what two calls give (stage
    launches at the smaller size, the resident kernel at the larger)."""
    import torch

    m = _spiral(n, 31)
    t = _device_arrays(m, "fp64")
    H0 = torch.from_numpy(m.H_init).cuda()
    want = H0.clone()
    for _ in range(2):
        _call(m, "fp64", 3, want, torch.cuda.current_stream().cuda_stream, t)
    H = H0.clone()
    g = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(g):
        _call(m, "fp64", 3, H, torch.cuda.current_stream().cuda_stream, t)
    assert torch.equal(H, H0)
    g.replay()
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(H, want)
    del g


def test_noalloc_calls_from_two_threads_do_not_disturb_each_other():
    """Two threads issue calls of different sizes at once, as callers that order them on the GPU
    by events do.  Each thread captures and instantiates its calls, so that none runs: a launch
    whose shared memory the other thread lowered would be refused."""
    import threading
    import torch

    cu = ctypes.CDLL("libcuda.so.1")
    vp = ctypes.c_void_p
    models = [_spiral(n, 31) for n in (5000, 18000)]
    arrays = [_device_arrays(m, "fp64") for m in models]
    states = [torch.from_numpy(m.H_init).cuda() for m in models]
    for m, t, H in zip(models, arrays, states):                # first calls, outside capture
        _call(m, "fp64", 2, H, torch.cuda.current_stream().cuda_stream, t)
    torch.cuda.synchronize()
    errors = []

    def issue(m, t, H):
        try:
            torch.cuda.set_device(0)
            stream = torch.cuda.Stream()
            for _ in range(400):
                graph, executable = vp(), vp()
                assert cu.cuStreamBeginCapture_v2(vp(stream.cuda_stream), 1) == 0
                try:
                    _call(m, "fp64", 2, H, stream.cuda_stream, t)
                finally:
                    assert cu.cuStreamEndCapture(vp(stream.cuda_stream), ctypes.byref(graph)) == 0
                assert cu.cuGraphInstantiateWithFlags(ctypes.byref(executable), graph, ctypes.c_ulonglong(0)) == 0
                cu.cuGraphExecDestroy(executable)
                cu.cuGraphDestroy(graph)
        except Exception as e:                                  # noqa: BLE001 (reported by the main thread)
            errors.append(e)

    threads = [threading.Thread(target=issue, args=a) for a in zip(models, arrays, states)]
    for th in threads:
        th.start()
    for th in threads:
        th.join()
    assert not errors, errors[0]


@pytest.mark.parametrize("prec,n", [("fp64", 4999), ("fp64", 5000), ("fp64", 9999), ("fp64", 10000), ("fp32", 9999),
                                    ("fp32", 10000), ("fp32", 19999)])
def test_noalloc_steps_give_the_same_bits_in_one_call_or_several(prec, n):
    """Sizes on both sides of the line between stage launches and the resident kernel."""
    import torch

    m = _spiral(n, 31)
    t = _device_arrays(m, prec)
    H0 = torch.from_numpy(m.H_init).to(torch.float64 if prec == "fp64" else torch.float32).cuda()
    stream = torch.cuda.current_stream().cuda_stream
    states = []
    for calls in ((3,), (1, 1, 1), (2, 1)):
        H = H0.clone()
        for steps in calls:
            _call(m, prec, steps, H, stream, t)
        states.append(H)
    assert torch.equal(states[0], states[1])
    assert torch.equal(states[0], states[2])
