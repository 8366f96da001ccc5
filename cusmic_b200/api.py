"""Reference-shaped Python API: ``remove_cosmics``, ``Cleaner`` and ``Image``.

Mirrors rndsrc/cusmic ``mod/cusmic/api.py:20-63``, ``image.py:22-79`` and
``cleaner.py:26-118`` (same names, argument meaning, defaults, validation
messages and exception types), but the arrays are ``torch.Tensor`` on a CUDA
device (NumPy arrays and other ``__dlpack__`` objects are accepted and
uploaded) and the work is done by libcusmic_b200.so through its C ABI on the
input device's current stream.
"""

import ctypes
from dataclasses import dataclass
from math import isfinite, nan
from numbers import Integral, Real
from typing import Any

import numpy as np
import torch

from . import _native

Array = Any
MODES = ("mirror", "reflect", "nearest", "wrap", "constant")


def _as_tensor(value, device=None):
    """Tensor view of a tensor, a __dlpack__ object, a NumPy array or a scalar."""
    if isinstance(value, torch.Tensor):
        t = value
    elif hasattr(value, "__dlpack__") and not isinstance(value, np.ndarray):
        t = torch.from_dlpack(value)
    else:
        t = torch.as_tensor(value)
    if device is not None and t.device != device:
        t = t.to(device)
    return t


def _cuda_device(data):
    if data.is_cuda:
        return data.device
    return torch.device("cuda", torch.cuda.current_device())


@dataclass
class Image:
    """Float64 pixels with calibration validated on the input device.

    Maps match the data or one shared frame.  Gain, read noise and background
    may also be scalars.  An error map overrides gain and read noise.  See
    :func:`remove_cosmics` for units, exclusions and stream use.
    """

    data: Array
    error: Array | None = None
    mask: Array | None = None
    background: Array | float | None = None
    effective_gain: Array | float | None = None
    readnoise: Array | float | None = None

    def __post_init__(self):
        self.data, device = _checked_data(self.data)
        with torch.cuda.device(device):
            fields, checks = _calibration(self.data, device, self.error, self.background,
                                          self.effective_gain, self.readnoise, views=True)
            checks.run()
            for name, value in fields.items():
                setattr(self, name, value)
            self.mask = _checked_mask(self.mask, self.data, device)


def _checked_data(data):
    data = _as_tensor(data)
    if data.dtype != torch.float64:
        raise TypeError("data must contain float64 pixels")
    if data.dim() not in (2, 3) or not data.numel():
        raise ValueError("data must be a nonempty 2D frame or 3D stack")
    device = _cuda_device(data)
    return data if data.is_cuda else data.to(device), device


def _checked_mask(mask, data, device):
    if mask is None:
        return None
    mask = _as_tensor(mask, device).to(torch.bool)
    if tuple(mask.shape) not in (tuple(data.shape), tuple(data.shape[-2:])):
        raise ValueError("mask must match the data or one frame")
    return mask


class _Checks:
    """The content checks of an image's calibration, in the reference's order:
    scalars are decided here, maps on the device (cusmic_check_maps, or with
    the cleaning itself); the first that failed raises."""

    RULES = {"error": (1, "positive"), "effective_gain": (1, "positive"),
             "readnoise": (0, "nonnegative"), "background": (-1, None)}

    def __init__(self):
        self.items = []   # (name, index of its map or None, failed bits of a scalar)
        self.tensors = []  # the maps, contiguous
        self.failed = False  # report() raised

    def add(self, name, value):
        """Adds a check; returns the value as the check reads it (contiguous)."""
        minimum, _ = self.RULES[name]
        if isinstance(value, float):
            low = value <= 0 if minimum == 1 else value < 0 if minimum == 0 else False
            self.items.append((name, None, (not isfinite(value)) | low << 1))
        else:
            self.items.append((name, len(self.tensors), 0))
            value = value.detach().contiguous()
            self.tensors.append(value)
        return value

    def maps(self):
        """The maps as struct cusmic_map_check."""
        arr = (_native.MapCheck * max(1, len(self.tensors)))()
        names = [name for name, index, _ in self.items if index is not None]
        for i, (name, t) in enumerate(zip(names, self.tensors)):
            arr[i] = _native.MapCheck(t.data_ptr(), t.numel(), self.RULES[name][0])
        return arr, len(self.tensors)

    @property
    def scalar_failed(self):
        return any(bits for _, _, bits in self.items)

    def report(self, flags):
        for name, index, bits in self.items:
            if index is not None:
                bits = flags >> (2 * index) & 3
            self.failed = bits != 0
            if bits & 1:
                raise ValueError(f"{name} must be finite")
            if bits & 2:
                raise ValueError(f"{name} must be {self.RULES[name][1]}")

    def run(self):
        flags = ctypes.c_uint(0)
        if self.tensors:
            arr, n = self.maps()
            msg = ctypes.create_string_buffer(256)
            stream = torch.cuda.current_stream(self.tensors[0].device).cuda_stream
            _native.raise_for(_native.lib().cusmic_check_maps(arr, n, ctypes.byref(flags), stream,
                                                              msg, len(msg)), msg)
        self.report(flags.value)


def _calibration(data, device, error, background, effective_gain, readnoise, views=False):
    """The calibration that applies (an error map replaces gain and read
    noise) as float64 device maps or floats, and its content checks.  ``views``:
    everything as float64 device tensors, as given; else maps as the checks read
    them, so that a map that is not contiguous is copied once."""
    shape, frame = tuple(data.shape), tuple(data.shape[-2:])
    given = {"error": error} if error is not None else \
        {"effective_gain": effective_gain, "readnoise": readnoise}
    given["background"] = background
    fields, checks = {}, _Checks()
    for name, value in given.items():
        if value is None:
            continue
        value = _as_tensor(value)
        if value.dim() or value.is_cuda:
            value = _as_tensor(value, device)
        if value.dtype.is_complex or value.dtype == torch.bool or \
                not (value.dtype.is_floating_point or value.dtype in (
                    torch.int8, torch.int16, torch.int32, torch.int64, torch.uint8)):
            raise TypeError(f"{name} must be real numeric data")
        if tuple(value.shape) not in (shape, frame) and (name == "error" or value.dim() != 0):
            raise ValueError(f"{name} has an incompatible shape")
        value = value.to(torch.float64)
        checked = checks.add(name, value if value.dim() else float(value.detach()))
        fields[name] = value.to(device) if views else checked
    return fields, checks


@dataclass(frozen=True)
class Cleaner:
    """Reusable detection settings; call with an Image to get pixels and a mask."""

    contrast: float = 3
    cr_threshold: float = 5
    neighbor_threshold: float = 3
    maxiter: int = 4
    border_mode: str = "mirror"

    def __post_init__(self):
        for name in ("contrast", "cr_threshold", "neighbor_threshold"):
            value = getattr(self, name)
            if isinstance(value, bool) or not isinstance(value, Real) or not isfinite(value) \
                    or value < 0:
                raise ValueError(f"{name} must be finite and nonnegative")
        if isinstance(self.maxiter, bool) or not isinstance(self.maxiter, Integral) or \
                self.maxiter < 0:
            raise ValueError("maxiter must be a nonnegative integer")
        if not isinstance(self.border_mode, str) or self.border_mode not in MODES:
            raise ValueError(f"border_mode must be one of {', '.join(MODES)}")

    def options(self, gain=nan, readnoise=0.0, background=nan):
        o = _native.default_options()
        o.contrast = float(self.contrast)
        o.cr_threshold = float(self.cr_threshold)
        o.neighbor_threshold = float(self.neighbor_threshold)
        o.maxiter = int(self.maxiter)
        o.border = _native.BORDERS[self.border_mode]
        o.gain, o.readnoise, o.background = gain, readnoise, background
        return o

    def __call__(self, image: Image):
        """Return new (cleaned float64, mask bool) tensors on the input device."""
        if self.maxiter and image.error is None and (
                image.effective_gain is None or image.readnoise is None):
            raise ValueError("Provide error, or both effective_gain and readnoise")
        names = ("error",) if image.error is not None else ("effective_gain", "readnoise")
        fields = {}
        for name in (*names, "background"):
            value = getattr(image, name)
            if value is not None:
                fields[name] = float(value) if value.dim() == 0 else value
        return self._clean(image.data, fields, image.mask)

    def _clean(self, data, fields, mask, checks=None):
        """The cleaning of validated inputs; with ``checks``, their content
        checks run with it and raise first."""
        device = data.device
        stack = data if data.dim() == 3 else data.unsqueeze(0)
        stack = stack.contiguous()
        nf, h, w = stack.shape
        step = 8 * h * w
        keep = [stack]

        def maps(value, size=8):
            if value is None or isinstance(value, float):
                return [None] * nf
            v = value.contiguous()
            keep.append(v)
            at = v.data_ptr()
            return [at + i * size * h * w for i in range(nf)] if v.dim() == 3 else [at] * nf

        def scalar(name, default):
            value = fields.get(name)
            return value if isinstance(value, float) else default

        err, gain, rn, bg = (maps(fields.get(name)) for name in
                             ("error", "effective_gain", "readnoise", "background"))
        # A bool tensor's bytes are the mask bytes.
        msk = maps(None if mask is None else mask.contiguous().view(torch.uint8), 1)
        opts = self.options(gain=scalar("effective_gain", nan), readnoise=scalar("readnoise", 0.0),
                            background=scalar("background", nan))
        ims = (_native.Image * nf)()
        at = stack.data_ptr()
        for i in range(nf):
            ims[i] = _native.Image(at + i * step, err[i], gain[i], rn[i], bg[i], msk[i], w, h)
        clean = torch.empty((nf, h, w), dtype=torch.float64, device=device)
        flags = torch.empty((nf, h, w), dtype=torch.bool, device=device)
        msg = ctypes.create_string_buffer(512)
        with torch.cuda.device(device):
            stream = torch.cuda.current_stream(device).cuda_stream
            if checks is None:
                status = _native.lib().remove_cosmics_batch_device(
                    ims, nf, ctypes.byref(opts), clean.data_ptr(), flags.data_ptr(), stream, msg,
                    len(msg))
            else:
                failed = ctypes.c_uint(0)
                arr, n = checks.maps()
                status = _native.lib().cusmic_checked_batch_device(
                    ims, nf, ctypes.byref(opts), clean.data_ptr(), flags.data_ptr(), arr, n,
                    ctypes.byref(failed), stream, msg, len(msg))
                checks.report(failed.value)
        del keep
        _native.raise_for(status, msg)
        if data.dim() == 2:
            return clean[0], flags[0]
        return clean, flags


def remove_cosmics(
    data,
    contrast,
    cr_threshold,
    neighbor_threshold,
    error=None,
    mask=None,
    background=None,
    effective_gain=None,
    readnoise=None,
    maxiter=4,
    border_mode="mirror",
):
    """Return cleaned float64 pixels and a boolean cosmic-ray mask on the GPU.

    ``data`` is a nonempty float64 frame (height, width) or stack (frames,
    height, width): a CUDA tensor (used on its device) or a host array
    (uploaded to the current device).  Frames are cleaned independently and
    outputs do not alias inputs.

    Supply a finite, positive 1-sigma ``error`` map in image units, or both
    ``effective_gain`` (electrons per image unit, positive) and ``readnoise``
    (electrons, nonnegative).  Error overrides gain and read noise.  Maps may
    match data or one shared frame; gain and read noise also accept scalars.

    ``contrast`` rejects fine structure; ``cr_threshold`` and
    ``neighbor_threshold`` set detection and growth thresholds in sigma; all
    three must be finite and nonnegative.  ``mask`` excludes seed and donor
    pixels, but neighbouring detections may grow into masked pixels.
    Non-finite input pixels are preserved and never flagged.

    ``background`` is a finite scalar or map in image units, added before
    cleaning and subtracted afterwards.  ``maxiter`` is nonnegative; zero
    disables detection and needs no noise model but still applies the
    background arithmetic.  Border modes are mirror, reflect, nearest, wrap and
    constant (zero padding).

    Work runs on the input device's current stream; the call returns after it
    completes.  A replacement with no finite, unmasked donors raises ValueError.
    """
    # As Cleaner(...)(Image(...)), with the maps checked on the device by the
    # call that cleans them: one submission and one synchronisation.  Whatever
    # else fails, a failing map is reported first, as Image would.
    data, device = _checked_data(data)
    with torch.cuda.device(device):
        fields, checks = _calibration(data, device, error, background, effective_gain, readnoise)
        if checks.scalar_failed:
            checks.run()
        try:
            mask = _checked_mask(mask, data, device)
            cleaner = Cleaner(contrast, cr_threshold, neighbor_threshold, maxiter, border_mode)
            if maxiter and error is None and ("effective_gain" not in fields or
                                              "readnoise" not in fields):
                raise ValueError("Provide error, or both effective_gain and readnoise")
            return cleaner._clean(data, fields, mask, checks)
        except Exception:
            if not checks.failed:  # the call failed before, or apart from, its checks
                checks.run()
            raise
