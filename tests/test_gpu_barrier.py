"""A grid barrier of the late passes whose wait runs out (an injected arrival
that never comes, a bound of about half a millisecond): every block leaves, the
call fails with its own message, and the next call on the GPU is bit-exact."""

import pytest

from cusmic_b200 import _native
from tests import cabi
from tests.test_gpu_failures import SETTINGS, WAIT_CYCLES, expect_exact, inject, scene  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", ((64, 80), (256, 512), (1500, 2048)))
def test_barrier_wait_runs_out(cuda, oracle, inject, size):  # noqa: F811
    """Grids from the fewest blocks to one per SM."""
    frame = scene(5, *size)
    two = cabi.Frames([frame, scene(6)])
    opts = cabi.options(**SETTINGS)
    healthy = cabi.Plan(two, opts, _native.PLAN_GRAPH, scalars=False)
    inject(_native.FAULT_BARRIER_WAIT, WAIT_CYCLES)
    poisoned = cabi.Plan(two, opts, _native.PLAN_GRAPH, scalars=False)
    try:
        st, msg = cabi.run_batch(_native.lib(), cabi.Frames([frame]), opts)
        assert st == _native.CUSMIC_CUDA_ERROR and "grid barrier" in msg
        st, msg = cabi.run_ragged(two, opts, scalars=False)
        assert st == _native.CUSMIC_CUDA_ERROR and "grid barrier" in msg
        st, msg = poisoned.run()
        assert st == _native.CUSMIC_CUDA_ERROR and "grid barrier" in msg
        # One pass has no barrier; a plan made before keeps its bound.
        st, msg = cabi.run_batch(_native.lib(), cabi.Frames([frame]), 
                                 cabi.options(**SETTINGS, maxiter=1))
        assert st == 0, msg
        st, msg = healthy.run()
        assert st == 0, msg
        assert max(healthy.passes()) > 1
    finally:
        poisoned.close()
        healthy.close()
    assert _native.lib().cusmic_inject_fault(_native.FAULT_BARRIER_WAIT, 0) == 0
    expect_exact(oracle, frame, SETTINGS)
