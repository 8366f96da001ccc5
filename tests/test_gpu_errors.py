"""What a failed call leaves behind."""

import ctypes

import numpy as np
import pytest

from cusmic_b200 import _native
from tests import cabi
from tests.conftest import assert_bits_equal
from tests.test_gpu_failures import SETTINGS, expect_exact, scene

pytestmark = pytest.mark.gpu


def test_call_after_a_failed_reservation(cuda, oracle):
    """A batch whose work lists do not fit the GPU (65535 frames of one column:
    more than 200 GB reserved for 25 Mpixel) fails with CUSMIC_NO_MEMORY before
    anything runs, and the next call knows nothing of it."""
    nf, h = 65535, 384
    column = cuda.ones(h, dtype=cuda.float64, device="cuda")
    ims = (_native.Image * nf)()
    for i in range(nf):
        ims[i] = _native.Image(column.data_ptr(), column.data_ptr(), None, None, None, None, 1, h)
    clean = cuda.empty(nf * h, dtype=cuda.float64, device="cuda")
    mask = cuda.empty(nf * h, dtype=cuda.uint8, device="cuda")
    msg = ctypes.create_string_buffer(256)
    st = _native.lib().remove_cosmics_batch_device(
        ims, nf, ctypes.byref(cabi.options(**SETTINGS)), clean.data_ptr(), mask.data_ptr(), None, msg, 256)
    assert st == _native.CUSMIC_NO_MEMORY, msg.value
    expect_exact(oracle, scene(9), SETTINGS)


@pytest.mark.parametrize("flags", (0, _native.PLAN_GRAPH))
def test_failed_execution_runs_nothing(cuda, oracle, flags):
    """An execution that cannot reserve the memory for its status fails before
    anything is queued, so nothing still writes the buffers after it returned;
    the next one is that of a fresh plan."""
    frame = scene(12, 1500, 2048)
    fr = cabi.Frames([frame])
    plan = cabi.Plan(fr, cabi.options(**SETTINGS), flags)
    lib, msg = _native.lib(), ctypes.create_string_buffer(256)
    try:
        fr.clean.fill_(7.0)
        cuda.cuda.synchronize()
        assert lib.cusmic_inject_fault(_native.FAULT_NO_MEMORY, 1) == 0
        st = lib.cusmic_plan_execute(plan.handle, None, msg, 256)
        idle = cuda.cuda.default_stream().query()
        lib.cusmic_inject_fault(_native.FAULT_NO_MEMORY, 0)
        assert st == _native.CUSMIC_NO_MEMORY, msg.value
        assert idle and bool((fr.clean == 7.0).all())
        assert lib.cusmic_plan_wait(plan.handle, msg, 256) == _native.CUSMIC_INVALID
        st, text = plan.run()
        assert st == 0, text
        want_clean, want_mask, _ = cabi.oracle_frame(oracle, frame, **SETTINGS)
        clean, mask = fr.outputs()[0]
        np.testing.assert_array_equal(mask, want_mask)
        assert_bits_equal(clean, want_clean)
    finally:
        plan.close()
