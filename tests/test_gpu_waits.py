"""The bounded-wait path of the pipelined kernels, exercised without a fault:
a wait that nothing completes gives up after its limit, the kernel returns,
the host reads SWE_ERR_TIMEOUT and the same context keeps working."""
import ctypes

import numpy as np
import pytest

from conftest import generated_input, scaled_err
from swe_b200 import capi, swe_input

pytestmark = pytest.mark.gpu


def test_wait_that_never_completes_times_out_and_context_survives():
    lib = capi.load()
    waited = ctypes.c_double(0.0)
    st = lib.swe_selftest_wait_timeout(0.05, ctypes.byref(waited))
    assert st == 6, (st, lib.swe_cuda_last_error())         # SWE_ERR_TIMEOUT
    assert 0.05 <= waited.value < 1.0, waited.value
    # the context is intact: a normal run afterwards
    _, d = generated_input(4)
    m = swe_input.to_model(d)
    p = capi.Plain()
    p.init_model(m, "fp64")
    p.set_state(m.H_init)
    p.step(3)
    assert np.isfinite(p.get_state()).all()
    p.finalize()


def test_selftest_rejects_unbounded_limits():
    lib = capi.load()
    assert lib.swe_selftest_wait_timeout(0.0, None) == 1      # SWE_ERR_ARG
    assert lib.swe_selftest_wait_timeout(5.0, None) == 1


def test_step_wait_that_runs_out_is_reported_until_the_next_init():
    """A wait between the resident step kernel's blocks runs out: every call that answers
    from the state says so, whichever stage kernel is selected meanwhile, and a new init
    steps again."""
    from test_zz_no_alloc import _spiral
    lib = capi.load()
    m = _spiral(10242, 31)                                    # a size whose steps run resident
    p = capi.Plain()
    p.init_model(m, "fp64")
    p.set_state(m.H_init)
    p.step(10)
    want = p.get_state()
    assert lib.swe_selftest_step_wait(0.0) == 1               # SWE_ERR_ARG
    assert lib.swe_selftest_step_wait(5.0) == 1
    assert lib.swe_selftest_step_wait(0.05) == 0
    for call in (p.sync, p.get_state, p.invariants):
        with pytest.raises(capi.SweError, match="ran out"):
            call()
    p.select_kernel(5)
    for call in (p.get_state, p.invariants, p.sync):
        with pytest.raises(capi.SweError, match="ran out"):
            call()
    p.init_model(m, "fp64")
    p.set_state(m.H_init)
    p.step(10)
    # (the new init may choose other lanes per node: another order of the sums)
    assert scaled_err(p.get_state().reshape(-1, 4), want.reshape(-1, 4)).max() <= 1e-12
    p.invariants()
    p.finalize()
