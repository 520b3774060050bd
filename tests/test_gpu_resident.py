"""Whole steps of the plain form (swe_cuda_step) in the kernel swe_cuda_init chose, resident
or one launch per stage, on small and mid-sized grids of odd sizes: the bits of the same
number of swe_cuda_rk_substep rounds, and the oracle's states."""
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
    """The resident kernel, selected: a call is one launch and gives the bits of the stage
    launches of as many substeps; stage launches when they are selected again."""
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
            assert capi.kernel_launches() - before == 1
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
