"""Whole steps of the plain form (swe_cuda_step) in the kernel swe_cuda_init chose, resident
or one launch per stage, on small and mid-sized grids of odd sizes: the bits of the same
number of swe_cuda_rk_substep rounds, and the oracle's states."""
import time

import numpy as np
import pytest

import oracle
from conftest import scaled_err
from swe_b200 import capi, layout
from test_zz_no_alloc import _spiral

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec,n,nnbr", [("fp64", 149, 31), ("fp64", 1193, 20), ("fp64", 9731, 28), ("fp64", 23681, 31),
                                         ("fp64", 31000, 25), ("fp64", 35009, 31), ("fp64", 42600, 32), ("fp32", 1185, 31), ("fp32", 20001, 32), ("fp32", 40001, 31)])
def test_steps_equal_substeps_bitwise_and_match_oracle(prec, n, nnbr):
    m = _spiral(n, nnbr)
    m = layout.reorder(m, layout.rcm_mapping(m))
    H0 = m.H_init.astype(np.float64 if prec == "fp64" else np.float32)
    p = capi.Plain()
    try:
        p.init_model(m, prec)
        got = {}
        for steps in (1, 30):                       # a single step and one of many
            p.set_state(H0)
            p.step(steps)
            got[steps] = p.get_state().reshape(-1, 4)
            p.set_state(H0)
            for _ in range(steps):
                for s in range(4):
                    p.rk_substep(s)
            assert np.array_equal(got[steps], p.get_state().reshape(-1, 4)), steps
    finally:
        p.finalize()
    want = oracle.Port(m, prec).run(H0, 30)
    assert scaled_err(got[30], want).max() <= (1e-12 if prec == "fp64" else 1e-4)


@pytest.mark.parametrize("n", [47361, 60001])
def test_fp32_rhs_of_one_lane_per_node_is_as_exact_as_the_restatement(n):
    """Above 47,360 nodes one lane sums a node's slots: in the caller's order, as the FP32
    restatement does, with fewer roundings (fused multiply-adds).  Other orders (ascending
    rows, or placed for shared lines) are 1.4 to 2 times further from 64 bits."""
    m = _spiral(n, 31)
    m = layout.reorder(m, layout.rcm_mapping(m))
    K = m.H_init.astype(np.float32)
    want = oracle.Port(m, "fp64").eval_rhs(K.astype(np.float64))
    p = capi.Plain()
    try:
        p.init_model(m, "fp32")
        p.select_kernel(capi.Plain.lane_shape(1, 4))
        err = np.linalg.norm(p.eval_rhs(K).reshape(-1, 4) - want)
    finally:
        p.finalize()
    assert err <= 1.25 * np.linalg.norm(oracle.Port(m, "fp32").eval_rhs(K) - want)


# lanes per node and whether the weights are streamed, at sizes around the splits' edges (148 SMs,
# 31 neighbours: 2 lanes hold 27,232 nodes in FP64 and stream to 42,624; nodes per block in
# multiples of 8, streamed of 32)
@pytest.mark.parametrize("prec,n,nnbr,lanes,streamed", [
    ("fp64", 149, 31, 4, False), ("fp64", 9731, 28, 4, False), ("fp64", 10242, 31, 2, False), ("fp64", 27232, 31, 2, False),
    ("fp64", 27233, 31, 2, True), ("fp64", 35009, 25, 2, True), ("fp64", 37889, 31, 2, True), ("fp64", 42624, 32, 2, True),
    ("fp32", 1185, 31, 2, False), ("fp32", 20001, 32, 4, False), ("fp32", 47360, 17, 2, False)])
def test_whole_steps_in_the_resident_kernel_equal_substeps(prec, n, nnbr, lanes, streamed):
    """The resident kernel, selected: a call is one launch (two where it streams) and gives the
    bits of the stage launches of as many substeps; stage launches when they are selected again."""
    m = _spiral(n, nnbr)
    m = layout.reorder(m, layout.rcm_mapping(m))
    H0 = m.H_init.astype(np.float64 if prec == "fp64" else np.float32)
    p = capi.Plain()
    try:
        p.init_model(m, prec)
        p.select_step_kernel(lanes)
        info = p.step_kernel_info()
        assert (info["lanes_per_node"], info["streamed"], info["min_steps"]) == (lanes, streamed, 1)
        for steps in (1, 7):
            p.set_state(H0)
            before = capi.kernel_launches()
            p.step(steps)
            assert capi.kernel_launches() - before == (2 if streamed else 1)
            got = p.get_state()
            p.set_state(H0)
            for _ in range(steps):
                for s in range(4):
                    p.rk_substep(s)
            assert np.array_equal(got, p.get_state()), steps
        p.select_step_kernel(0)
        assert p.step_kernel_info()["lanes_per_node"] == 0
        p.set_state(H0)
        before = capi.kernel_launches()
        p.step(7)
        assert capi.kernel_launches() - before == 28
        assert np.array_equal(got, p.get_state())
    finally:
        p.finalize()


@pytest.mark.parametrize("prec,n,lanes", [("fp64", 10242, 2), ("fp64", 10242, 4), ("fp64", 35009, 2), ("fp32", 20001, 4)])
def test_resident_rows_of_both_widths(prec, n, lanes):
    """swe_cuda_set_index_width holds for the resident kernel too (its 32-bit rows took no part
    before on grids whose rows fit 16 bits): the same bits."""
    m = _spiral(n, 31)
    m = layout.reorder(m, layout.rcm_mapping(m))
    H0 = m.H_init.astype(np.float64 if prec == "fp64" else np.float32)
    p = capi.Plain()
    try:
        p.init_model(m, prec)
        p.select_step_kernel(lanes)
        assert p.kernel_info()["index_offsets_16bit"]
        got = []
        for bits in (16, 32):
            p.set_index_width(bits)
            assert p.step_kernel_info()["lanes_per_node"] == lanes
            p.set_state(H0)
            p.step(7)
            got.append(p.get_state())
        assert np.array_equal(*got)
    finally:
        p.finalize()


@pytest.mark.parametrize("form", ["plain", "noalloc"])
def test_long_calls_run_in_launches_of_200_steps(form):
    """A call of 401 steps is three launches and gives the state of calls of 1, 200 and 200."""
    import torch
    from test_zz_no_alloc import _call, _device_arrays

    m = _spiral(5921, 31)
    m = layout.reorder(m, layout.rcm_mapping(m))
    p = capi.Plain()
    try:
        if form == "plain":
            p.init_model(m, "fp64")
            p.select_step_kernel(4)
            start, step, state = lambda: p.set_state(m.H_init), p.step, p.get_state
        else:
            t = _device_arrays(m, "fp64")
            H, stream = torch.from_numpy(m.H_init).cuda(), torch.cuda.current_stream().cuda_stream
            start = lambda: H.copy_(torch.from_numpy(m.H_init))  # noqa: E731
            step = lambda n: _call(m, "fp64", n, H, stream, t)  # noqa: E731
            state = lambda: H.cpu().numpy()  # noqa: E731
        got = []
        for calls, launches in (((401,), 3), ((1, 200, 200), 3), ((200, 201), 3)):
            start()
            before = capi.kernel_launches()
            for n in calls:
                step(n)
            assert capi.kernel_launches() - before == launches
            got.append(state())
        assert np.isfinite(got[0]).all()
        assert np.array_equal(got[0], got[1]) and np.array_equal(got[0], got[2])
    finally:
        if form == "plain":
            p.finalize()


def test_step_kernel_selection_refuses_what_does_not_fit():
    m = _spiral(25001, 31)
    p = capi.Plain()
    try:
        p.init_model(m, "fp64")
        p.select_step_kernel(2)
        for lanes in (1, 3, 4):                     # 4 lanes a node: more threads than a block has
            with pytest.raises(capi.SweError) as e:
                p.select_step_kernel(lanes)
            assert capi.STATUS[e.value.status] == "SWE_ERR_ARG"
            assert p.step_kernel_info()["lanes_per_node"] == 2
    finally:
        p.finalize()


def test_init_chooses_the_resident_kernel():
    """swe_cuda_init chooses by timing: 40,001 nodes in FP32, clearly faster resident (4.2 against 4.7 us
    a stage), in one of three tries."""
    m = _spiral(40001, 31)
    m = layout.reorder(m, layout.rcm_mapping(m))
    p = capi.Plain()
    try:
        for _ in range(3):
            p.init_model(m, "fp32")
            if p.step_kernel_info()["lanes_per_node"]:
                break
        info = p.step_kernel_info()
        assert info["lanes_per_node"]
        p.set_state(m.H_init.astype(np.float32))
        before = capi.kernel_launches()
        p.step(max(20, info["min_steps"]))
        assert capi.kernel_launches() - before == 1
    finally:
        p.finalize()


# blocks of a kernel that holds an SM each, seconds, whether the steps have to end before it does:
# some SMs held, all but one for a while (the other blocks join as it ends), and all of them
HELD = [(20, 0.25, True), (147, 0.02, False), (148, 0.02, False)]


def _beside(held, seconds, first, run, share=1.0):
    """run() on its stream while another's blocks hold `share` of an SM each; whether that one
    still ran at the end."""
    import torch
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    assert capi.load().swe_selftest_hold_sms(held, share, seconds, side.cuda_stream) == 0
    if first:
        time.sleep(0.02)                            # it has its SMs
    run()
    return not side.query()


@pytest.mark.parametrize("held,seconds,first", HELD)
# (every kernel there is: 2 and 4 lanes in blocks of up to 512 and 640 threads, and streamed)
@pytest.mark.parametrize("prec,n,lanes,steps", [
    ("fp64", 10242, 4, 40), ("fp64", 23001, 4, 10), ("fp64", 27232, 2, 10), ("fp64", 35009, 2, 10),
    ("fp32", 10242, 4, 40), ("fp32", 23001, 4, 10), ("fp32", 25001, 2, 20), ("fp32", 40001, 2, 20)])
def test_steps_run_beside_a_kernel_that_holds_sms(prec, n, lanes, steps, held, seconds, first):
    """Steps go on, on the SMs that another stream's kernel leaves, while it runs: the bits of the
    undisturbed steps."""
    m = _spiral(n, 31)
    m = layout.reorder(m, layout.rcm_mapping(m))
    H0 = m.H_init.astype(np.float64 if prec == "fp64" else np.float32)
    p = capi.Plain()
    try:
        p.init_model(m, prec)
        p.select_step_kernel(lanes)
        p.set_state(H0)
        p.step(steps)
        want = p.get_state()
        p.set_state(H0)
        p.sync()
        got = []
        running = _beside(held, seconds, first, lambda: (p.step(steps), got.append(p.get_state())))
        assert running or not first
        assert np.array_equal(got[0], want)
    finally:
        p.finalize()


@pytest.mark.parametrize("held,seconds,first", HELD)
@pytest.mark.parametrize("prec,n,steps,off", [
    ("fp64", 10242, 40, 2), ("fp64", 20001, 10, 0), ("fp64", 25001, 10, 2), ("fp32", 10242, 20, 0), ("fp32", 20001, 20, 0),
    ("fp32", 25001, 20, 0), ("fp32", 40001, 20, 0)])
def test_noalloc_steps_run_beside_a_kernel_that_holds_sms(prec, n, steps, off, held, seconds, first):
    import torch
    from test_zz_no_alloc import _call, _device_arrays

    m = _spiral(n, 31)
    t = _device_arrays(m, prec)
    buf = torch.empty(4 * n + 2, dtype=torch.float64 if prec == "fp64" else torch.float32, device="cuda")
    H = buf[off:off + 4 * n].view(n, 4)             # FP64: H 32- and 16-byte aligned
    H0 = torch.from_numpy(m.H_init).to(H)
    stream = torch.cuda.Stream()

    def run():
        _call(m, prec, steps, H, stream.cuda_stream, t)
        stream.synchronize()

    H.copy_(H0)
    torch.cuda.synchronize()
    run()
    want = H.clone()
    H.copy_(H0)
    running = _beside(held, seconds, first, run)
    assert running or not first
    assert torch.equal(H, want)
    _call(m, prec, 0, H, stream.cuda_stream, t)     # no wait ran out


@pytest.mark.parametrize("n", [20001, 42600, 47360])
def test_fp32_rhs_of_one_lane_is_as_exact_on_small_grids(n):
    """The slot order goes with the lanes that sum it, not with the grid's size alone.  One lane
    per node reads the caller's order, also where 2 and 4 lanes read placed slots: the
    restatement's sums with one rounding a term instead of two, so an error below the
    restatement's (as large as it with placed slots).  Each choice keeps its bits after the
    others."""
    m = _spiral(n, 31)
    m = layout.reorder(m, layout.rcm_mapping(m))
    K = m.H_init.astype(np.float32)
    want = oracle.Port(m, "fp64").eval_rhs(K.astype(np.float64))
    restated = np.linalg.norm(oracle.Port(m, "fp32").eval_rhs(K) - want)
    bar = {1: 0.95 * restated, 2: 1.25 * restated, 4: 1.25 * restated}
    p = capi.Plain()
    try:
        p.init_model(m, "fp32")
        first = {}
        for lanes in (1, 2, 4, 1, 4, 2):
            p.select_kernel(capi.Plain.lane_shape(lanes, 4))
            F = p.eval_rhs(K).reshape(-1, 4)
            assert np.linalg.norm(F - want) <= bar[lanes], lanes
            assert np.array_equal(F, first.setdefault(lanes, F)), lanes
    finally:
        p.finalize()


@pytest.mark.parametrize("form", ["plain", "noalloc"])
def test_stage_launches_run_beside_a_kernel_on_every_sm(form):
    """What a program selects whose own kernel sits on every SM and waits for the steps."""
    import torch
    from test_zz_no_alloc import _bind, _device_arrays

    m = _spiral(10242, 31)
    m = layout.reorder(m, layout.rcm_mapping(m))
    got = []
    if form == "plain":
        p = capi.Plain()
        p.init_model(m, "fp64")
        p.select_step_kernel(0)
        p.set_state(m.H_init)
        p.sync()
        run = lambda: (p.step(20), got.append(p.get_state().reshape(-1, 4)))  # noqa: E731
    else:
        lib = _bind()
        lib.swe_cuda_step_noalloc_stages.argtypes = lib.swe_cuda_step_noalloc.argtypes
        t = _device_arrays(m, "fp64")
        H = torch.from_numpy(m.H_init).cuda()
        out = torch.empty((m.N, 4), dtype=torch.float64, pin_memory=True)
        stream = torch.cuda.Stream()

        def step(steps):
            assert lib.swe_cuda_step_noalloc_stages(
                8, m.N, m.Nnbr, float(m.gh0), float(m.dt), t["idx"].data_ptr(),
                *[t[k].data_ptr() for k in ("Dx", "Dy", "Dz", "L", "x", "y", "z", "f", "ghm", "p_u", "p_v", "p_w",
                                            "gradghm")], H.data_ptr(), steps, stream.cuda_stream) == 0

        def run():
            before = capi.kernel_launches()
            step(20)
            assert capi.kernel_launches() - before == 80
            with torch.cuda.stream(stream):
                out.copy_(H, non_blocking=True)
            stream.synchronize()
            got.append(out.numpy())

        step(1)                                     # the first call loads the kernels
        H.copy_(torch.from_numpy(m.H_init))

    try:
        # (the no-allocation form's stage kernel takes 6 KB of shared memory a block: an SM split
        # for none has none to give)
        assert _beside(148, 0.25, True, run, share=0.0 if form == "plain" else 0.08)
    finally:
        if form == "plain":
            p.finalize()
    assert scaled_err(got[0], oracle.Port(m, "fp64").run(m.H_init, 20)).max() <= 1e-12
