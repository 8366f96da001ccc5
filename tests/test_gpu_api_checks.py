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
