"""What remove_cosmics does for its calibration maps besides the checks' results."""

import pytest

pytestmark = pytest.mark.gpu


class Counting:
    """The native library with the calls of its entry points counted."""

    def __init__(self, lib):
        self.lib, self.calls = lib, {}

    def __getattr__(self, name):
        self.calls[name] = self.calls.get(name, 0) + 1
        return getattr(self.lib, name)


def test_failing_map_is_checked_once(cuda, monkeypatch):
    """A failing map is found by the call's own checks; they run apart from the
    call only when it failed before them."""
    from cusmic_b200 import _native, remove_cosmics
    lib = Counting(_native.lib())
    monkeypatch.setattr(_native, "lib", lambda: lib)
    data = cuda.full((40, 50), 10.0, dtype=cuda.float64, device="cuda")
    error = cuda.ones_like(data)
    error[7, 9] = 0.0
    with pytest.raises(ValueError, match="error must be positive"):
        remove_cosmics(data, 3, 5, 3, error=error)
    assert lib.calls["cusmic_checked_batch_device"] == 1 and "cusmic_check_maps" not in lib.calls
    lib.calls.clear()
    with pytest.raises(ValueError, match="error must be positive"):
        remove_cosmics(data, -1, 5, 3, error=error)  # rejected before anything runs
    assert lib.calls.get("cusmic_check_maps") == 1


@pytest.mark.parametrize("call", ("plain", "differentiable"))
def test_strided_map_is_copied_once(cuda, call):
    """The checks and the cleaning share the contiguous copy of a map that is a
    transposed view; the results are those of the copy itself."""
    from cusmic_b200 import remove_cosmics
    from cusmic_b200.autograd import remove_cosmics_differentiable
    run = remove_cosmics if call == "plain" else remove_cosmics_differentiable
    gen = cuda.Generator(device="cuda")
    gen.manual_seed(4)
    h, w = 1000, 1200
    data = 200 + 12 * cuda.randn((h, w), generator=gen, dtype=cuda.float64, device="cuda")
    data[cuda.rand((h, w), generator=gen, device="cuda") < 4e-3] += 900
    strided = (12 + cuda.rand((w, h), generator=gen, dtype=cuda.float64, device="cuda")).T

    def peak(error):
        cuda.cuda.synchronize()
        cuda.cuda.reset_peak_memory_stats()
        before = cuda.cuda.memory_allocated()
        out = run(data, 3, 5, 3, error=error)
        cuda.cuda.synchronize()
        return cuda.cuda.max_memory_allocated() - before, out
    peak(strided.contiguous())
    own, (clean, mask) = peak(strided.contiguous())
    copied, (clean2, mask2) = peak(strided)
    assert bool(mask.any()) and cuda.equal(mask, mask2) and cuda.equal(clean, clean2)
    # (A contiguous argument's own memory is not in its call's count.)
    assert copied - own <= 8 * h * w + (1 << 20)


def test_image_keeps_scalar_tensors(cuda):
    """A scalar calibration given as a tensor is the Image's, on the data's
    device, with its autograd graph."""
    from cusmic_b200.api import Cleaner, Image
    gain = cuda.tensor(2.0, dtype=cuda.float64, requires_grad=True)
    image = Image(cuda.full((8, 9), 10.0, dtype=cuda.float64), effective_gain=gain, readnoise=3.0)
    assert image.effective_gain.requires_grad and image.effective_gain.is_cuda
    image.effective_gain.backward()
    assert float(gain.grad) == 1.0
    assert image.readnoise.is_cuda and image.readnoise.dtype == cuda.float64
    clean, mask = Cleaner(3, 5, 3)(image)
    assert bool((clean == 10).all()) and not bool(mask.any())
