"""Output masks that take the input masks' place: the input is read before the
buffer is written, by one-shot calls and plans, on both prepare paths."""

import ctypes

import numpy as np
import pytest

from cusmic_b200 import _native
from tests import cabi
from tests.conftest import assert_bits_equal
from tests.test_gpu_failures import SETTINGS

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("run", ("call", 0, _native.PLAN_GRAPH, "rebound"))
@pytest.mark.parametrize("width", (64, 61))
@pytest.mark.parametrize("shared", (False, True))
def test_mask_in_place(cuda, oracle, width, run, shared):
    """Width 64 takes the fused prepare, 61 the other; `shared`: every frame's
    input mask is the first one's."""
    rng = np.random.default_rng(width)
    h, nf = 90, 3
    mask = rng.random((nf, h, width)) < 0.1
    if shared:
        mask[:] = mask[0]
    frames = []
    for f in range(nf):
        data = 200 + rng.normal(0, 12, (h, width))
        hit = rng.random((h, width)) < 0.05
        data[hit] += rng.uniform(100, 4000, int(hit.sum()))
        frames.append(dict(data=data, error=np.full((h, width), 12.0), mask=mask[f]))
    fr = cabi.Frames(frames)
    apart = run == "rebound"  # a plan made for buffers of their own
    plan = None if run == "call" else \
        cabi.Plan(fr, cabi.options(**SETTINGS), _native.PLAN_GRAPH if apart else run, scalars=False)
    fr.mask.copy_(cuda.from_numpy(mask.astype(np.uint8)).reshape(-1))
    for f in range(nf):
        fr.ims[f].mask = fr.mask.data_ptr() + (0 if shared else f * h * width)
    try:
        if plan is None:
            st, msg = cabi.run_batch(_native.lib(), fr, cabi.options(**SETTINGS))
        else:
            err = ctypes.create_string_buffer(256)
            st = _native.lib().cusmic_plan_bind(plan.handle, fr.ims, fr.clean.data_ptr(), fr.mask.data_ptr(),
                                                err, 256)
            assert st == 0, err.value
            st, msg = plan.run()
        assert st == 0, msg
        for (clean, flags), frame in zip(fr.outputs(), frames):
            want_clean, want_mask, _ = cabi.oracle_frame(oracle, frame, **SETTINGS)
            assert want_mask.any()
            np.testing.assert_array_equal(flags, want_mask)
            assert_bits_equal(clean, want_clean)
    finally:
        if plan is not None:
            plan.close()
