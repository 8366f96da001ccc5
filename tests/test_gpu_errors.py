"""What a failed call leaves behind."""

import ctypes

import pytest

from cusmic_b200 import _native
from tests import cabi
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
