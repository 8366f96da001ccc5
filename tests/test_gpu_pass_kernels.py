"""The kernels of a detection pass where their work splits: candidates within
two pixels of an edge (read from the first pass's sig_raw map) and the late
passes, which work on lists in one launch.  Masks and
pixels are those of the CPU oracle bit for bit."""

import numpy as np
import pytest

from tests import cabi
from tests.test_gpu_parity import (MODES, SETTINGS, assert_bits_equal, check_against_oracle,
                                   small_scene)

pytestmark = pytest.mark.gpu


def edge_scene(seed, h, w):
    """Hits on the frame's edges and corners and one pixel inside them."""
    data, _ = small_scene(seed, h, w, rays=max(1, h * w // 60))
    rng = np.random.default_rng(seed + 1000)
    for k in (0, 1, 2):
        for row in (k, h - 1 - k):
            if 0 <= row < h:
                hit = rng.random(w) < 0.2
                data[row, hit] += rng.uniform(300, 4000, int(hit.sum()))
        for col in (k, w - 1 - k):
            if 0 <= col < w:
                hit = rng.random(h) < 0.2
                data[hit, col] += rng.uniform(300, 4000, int(hit.sum()))
    return data


@pytest.mark.parametrize("mode", MODES)
@pytest.mark.parametrize("shape", ((1, 9), (2, 2), (3, 40), (5, 33), (64, 31), (97, 70)))
def test_model_candidates_on_edges(cuda, oracle, mode, shape):
    """Noise-model candidates whose window crosses an edge, every border mode,
    frames down to one row (the border maps fold the window onto itself)."""
    data = edge_scene(shape[0] * 101 + shape[1], *shape)
    frame = dict(data=data, gain=1.5, readnoise=3.0)
    check_against_oracle(oracle, [frame], dict(SETTINGS, border=mode, gain=1.5, readnoise=3.0))


def structured(seed, h, w, hits=60):
    """Clusters of hits and tracks whose growth takes several passes."""
    rng = np.random.default_rng(seed)
    data = 200 + rng.normal(0, 12, (h, w))
    for _ in range(max(1, h * w * hits // 10000)):
        y, x = rng.integers(0, h), rng.integers(0, w)
        n = int(rng.integers(1, 9))
        ang = rng.uniform(0, np.pi)
        a = rng.uniform(150, 3000)
        for t in range(n):
            yy, xx = int(y + t * np.sin(ang)), int(x + t * np.cos(ang))
            if 0 <= yy < h and 0 <= xx < w:
                data[yy, xx] += a * rng.uniform(0.15, 1)
    return data


@pytest.mark.parametrize("mode", MODES)
@pytest.mark.parametrize("shape", ((1, 1), (4, 6), (12, 13), (13, 45), (40, 32), (64, 97),
                                   (150, 260)))
@pytest.mark.parametrize("noise", ("error", "model"))
def test_late_passes(cuda, oracle, mode, shape, noise):
    """Eight passes on frames from one pixel to several blocks of the late
    launch, narrower than the 13 x 13 neighbourhood of a changed pixel too
    (wrap folds it onto itself), with holes and masked pixels."""
    h, w = shape
    data = structured(h * 31 + w, h, w)
    rng = np.random.default_rng(h + w)
    mask = rng.random((h, w)) < 0.02
    if h * w > 100:
        data[rng.random((h, w)) < 0.005] = np.nan
    frame = dict(data=data, mask=mask)
    kw = dict(contrast=1.5, cr_threshold=4.0, neighbor_threshold=1.0, border=mode, maxiter=8)
    if noise == "error":
        frame["error"] = np.full((h, w), 12.0)
    else:
        frame.update(gain=1.5, readnoise=3.0)
        kw.update(gain=1.5, readnoise=3.0)
    check_against_oracle(oracle, [frame], kw)


def test_late_passes_everything_listed(cuda, oracle):
    """Zero thresholds: every pixel is a candidate in every pass, so the work
    lists fill their buffers."""
    data = structured(5, 60, 75)
    for kw, frame in ((dict(), dict(data=data, error=np.full(data.shape, 12.0))),
                      (dict(gain=1.5, readnoise=3.0), dict(data=data, gain=1.5, readnoise=3.0))):
        check_against_oracle(oracle, [frame], dict(contrast=0.5, cr_threshold=0.0, maxiter=4,
                                                   neighbor_threshold=0.0, **kw))


def test_late_passes_ragged_mixed(cuda, oracle):
    """Frames of both noise kinds that stop after different numbers of passes,
    in one batch."""
    frames = []
    for i, (h, w) in enumerate(((40, 50), (7, 200), (130, 90), (64, 64), (3, 3))):
        data = structured(i, h, w, hits=(5, 60, 120, 0, 40)[i])
        if i % 2:
            frames.append(dict(data=data, error=np.full((h, w), 12.0)))
        else:
            frames.append(dict(data=data, gain=1.5, readnoise=3.0))
    check_against_oracle(oracle, frames, dict(contrast=1.5, cr_threshold=4.0, gain=1.5,
                                              readnoise=3.0, neighbor_threshold=1.0, maxiter=6),
                         ragged=True)


@pytest.mark.parametrize("contrast", (0.0, 1.0, 2.0, 3.0, 500.0))
@pytest.mark.parametrize("noise", ("error", "odd_errors", "model"))
def test_contrast_ties(cuda, oracle, contrast, noise):
    """Small integers under power-of-two noise: the contrast and significance
    tests meet their thresholds exactly at many pixels, so decisions by counts
    have to fall back to the medians; zero, tiny and non-finite error values,
    and contrasts from zero to one that nothing passes."""
    rng = np.random.default_rng(int(contrast) + len(noise))
    h, w = 120, 160
    data = rng.integers(0, 6, (h, w)) * 4.0 + 64
    hit = rng.random((h, w)) < 0.05
    data[hit] += rng.choice([16.0, 32.0, 48.0, 64.0, 256.0], int(hit.sum()))
    frame = dict(data=data)
    kw = dict(contrast=contrast, cr_threshold=4.0, neighbor_threshold=2.0, maxiter=3)
    if noise == "model":
        frame.update(gain=1.0, readnoise=0.0)
        kw.update(gain=1.0, readnoise=0.0)
    else:
        frame["error"] = np.full((h, w), 2.0)
        if noise == "odd_errors":
            odd = rng.random((h, w)) < 0.03
            frame["error"][odd] = rng.choice([0.0, 1e-200, np.inf, np.nan], int(odd.sum()))
    check_against_oracle(oracle, [frame], kw)


@pytest.mark.parametrize("kw,message", [
    (dict(error="zero"), "error must be positive"),
    (dict(error="nan"), "error must be finite"),
    (dict(error="nan", contrast=-1.0), "error must be finite"),
    (dict(error="zero", mask="shape"), "error must be positive"),
    (dict(error="zero", background="nan"), "error must be positive"),
    (dict(error="ones", background="nan"), "background must be finite"),
    (dict(effective_gain="zero", readnoise=-1.0), "effective_gain must be positive"),
    (dict(effective_gain="nan"), "effective_gain must be finite"),
    (dict(effective_gain="ones", readnoise="minus"), "readnoise must be nonnegative"),
    (dict(effective_gain=2.0, readnoise=-1.0, background="nan"), "readnoise must be nonnegative"),
    (dict(error="ones", contrast=-1.0), "contrast must be finite"),
    (dict(error="ones", mask="shape"), "mask must match"),
    (dict(effective_gain=2.0), "Provide error"),
])
@pytest.mark.parametrize("at", (0, 1, -1))
def test_map_checks_with_the_call(cuda, kw, message, at):
    """remove_cosmics checks its maps in the call that cleans them: the first
    failing one is reported first, before other faults of the call, as Image
    does; failing values at a map's ends, in a map of odd length."""
    from cusmic_b200 import remove_cosmics
    h, w = 7, 33
    bad = {"zero": 0.0, "nan": np.nan, "minus": -1.0, "ones": 1.0}

    def make(name, v):
        if name == "mask":
            return np.zeros((h, w + 1), bool)
        if not isinstance(v, str):
            return v
        # One value past the buffer's start: 8 but not 16-byte aligned.
        flat = cuda.ones(h * w + 1, dtype=cuda.float64, device="cuda")[1:]
        flat[at] = bad[v]
        return flat.view(h, w)
    args = dict(contrast=3.0, cr_threshold=5.0, neighbor_threshold=3.0)
    args.update({k: make(k, v) for k, v in kw.items()})
    with pytest.raises(ValueError, match=message):
        remove_cosmics(np.full((h, w), 10.0), **args)
    clean, mask = remove_cosmics(np.full((h, w), 10.0), 3, 5, 3, error=make("error", "ones"))
    assert mask.dtype == cuda.bool and not bool(mask.any()) and bool((clean == 10).all())


@pytest.mark.parametrize("kind", ("model", "model_background", "mask", "maps"))
@pytest.mark.parametrize("width", (1, 31, 33, 127, 128, 129, 255, 256, 511, 513, 1023, 1024, 1025,
                                   1151, 1536, 2177))
def test_prepare_rows(cuda, oracle, kind, width):
    """Rows around the sizes of a warp's groups and segments, per kind of
    frame: whole groups of donors, and groups with non-finite or masked pixels
    at their first and last columns.  Odd widths also put each row at another
    alignment."""
    h = 9
    rng = np.random.default_rng(width)
    data = structured(width, h, width)
    frame, kw = dict(data=data), {}
    edges = [x for x in (0, 31, 32, 127, 128, 255, 256, 511, 512, 1023, 1024, width - 1) if x < width]
    for y, bad in ((1, np.nan), (3, np.inf), (5, -np.inf)):
        data[y, edges[:: y + 1]] = bad
    if kind in ("mask", "maps"):
        frame["mask"] = np.zeros((h, width), dtype=bool)
        frame["mask"][[2, 3, 7], :] = rng.random((3, width)) < 0.03
        frame["mask"][4, edges] = True
        frame["mask"][8, :] = True
    if kind == "mask":
        frame["error"] = np.full((h, width), 12.0)
    else:
        frame.update(gain=1.5, readnoise=3.0)
        kw.update(gain=1.5, readnoise=3.0)
    if kind == "maps":
        frame["background"] = rng.normal(20, 2, (h, width))
    elif kind == "model_background":
        frame["background"] = 12.25
        kw["background"] = 12.25
    check_against_oracle(oracle, [frame], dict(SETTINGS, **kw))


@pytest.mark.parametrize("mode", ("reflect", "wrap"))
def test_long_late_lists(cuda, mode):
    """A batch above 8 Mpixel, whose first late pass classifies in parts,
    against the same frames one at a time (which the tests above compare with
    the oracle): noise models with and without maps, an error map and a frame
    with every pixel alike."""
    frames = []
    for i in range(10):
        h, w = 900 + 13 * i, 1000 - 7 * i
        data = structured(i, h, w, hits=40) if i != 4 else np.full((h, w), 50.0)
        frame = dict(data=data, gain=1.5, readnoise=3.0)
        if i % 3 == 1:
            frame["gain"] = np.random.default_rng(i).uniform(1.2, 1.8, (h, w))
        elif i % 3 == 2:
            frame = dict(data=data, error=np.full((h, w), 12.0))
        frames.append(frame)
    assert sum(f["data"].size for f in frames) > 8 << 20
    kw = dict(contrast=1.5, cr_threshold=4.0, neighbor_threshold=1.0, maxiter=4, gain=1.5,
              readnoise=3.0, border=mode)
    fr = cabi.Frames(frames)
    st, msg = cabi.run_ragged(fr, cabi.options(**kw))
    assert st == 0, msg
    for frame, (clean, mask) in zip(frames, fr.outputs()):
        one = cabi.Frames([frame])
        st, msg = cabi.run_ragged(one, cabi.options(**kw))
        assert st == 0, msg
        want_clean, want_mask = one.outputs()[0]
        np.testing.assert_array_equal(mask, want_mask)
        assert_bits_equal(clean, want_clean)


@pytest.mark.parametrize("offset", (0, 2, 4))
@pytest.mark.parametrize("width", (16, 112, 128, 144, 272, 528, 656))
@pytest.mark.parametrize("noise", ("error", "model"))
def test_dense_columns_and_alignment(cuda, oracle, noise, width, offset):
    """Widths at which some of the dense kernels' warps have no column of their
    512-column items, and output buffers at 16- and 32-byte boundaries (one
    store or two per lane); 37 rows leave items of 32 and 5."""
    h = 37
    data = structured(width, h, width, hits=80)
    rng = np.random.default_rng(width)
    data[rng.random((h, width)) < 0.01] = np.nan
    frame = dict(data=data, mask=rng.random((h, width)) < 0.01)
    kw = dict(SETTINGS)
    if noise == "error":
        frame["error"] = np.full((h, width), 12.0)
    else:
        frame.update(gain=1.5, readnoise=3.0)
        kw.update(gain=1.5, readnoise=3.0)
    fr = cabi.Frames([frame])
    whole = fr.clean.new_empty(fr.total + offset)
    fr.clean = whole[offset:]
    st, msg = cabi.run_ragged(fr, cabi.options(**kw))
    assert st == 0, msg
    settings = {k: v for k, v in kw.items() if k not in ("gain", "readnoise")}
    want_clean, want_mask, _ = cabi.oracle_frame(oracle, frame, **settings)
    clean, mask = fr.outputs()[0]
    np.testing.assert_array_equal(mask, want_mask)
    assert_bits_equal(clean, want_clean)


def test_large_map_lists(cuda):
    """A batch above 32 Mpixel lists the sig_raw map's pixels in items of eight
    rows; the same frames one at a time in items of four."""
    rng = np.random.default_rng(3)
    frames = []
    for i in range(9):
        h, w = 1999 + i, 2001 - i
        data = 200 + rng.normal(0, 12, (h, w))
        hit = rng.random((h, w)) < 2e-3
        data[hit] += rng.uniform(100, 4000, int(hit.sum()))
        frames.append(dict(data=data, gain=1.5, readnoise=3.0))
    assert sum(f["data"].size for f in frames) > 32 << 20
    opts = cabi.options(**SETTINGS, gain=1.5, readnoise=3.0)
    fr = cabi.Frames(frames)
    st, msg = cabi.run_ragged(fr, opts)
    assert st == 0, msg
    for frame, (clean, mask) in zip(frames, fr.outputs()):
        one = cabi.Frames([frame])
        st, msg = cabi.run_ragged(one, opts)
        assert st == 0, msg
        want_clean, want_mask = one.outputs()[0]
        assert want_mask.any()
        np.testing.assert_array_equal(mask, want_mask)
        assert_bits_equal(clean, want_clean)
