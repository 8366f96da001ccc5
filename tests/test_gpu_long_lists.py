"""Batches whose size takes the long-list kernels (above 8 Mpixel the first late
pass classifies in parts with block thresholds, above 32 Mpixel the sig_raw map's
pixels are listed in items of eight rows): small frames of many shapes beside one
large one, against the CPU oracle, in every border mode."""

import numpy as np
import pytest

from tests import cabi
from tests.conftest import assert_bits_equal
from tests.test_gpu_parity import MODES
from tests.test_gpu_pass_kernels import edge_scene, structured

pytestmark = pytest.mark.gpu

SHAPES = ((1, 9), (7, 200), (13, 45), (31, 33), (33, 31), (40, 32), (64, 97), (65, 161), (97, 70))


@pytest.mark.parametrize("side", (2900, 5800))
@pytest.mark.parametrize("mode", MODES)
def test_small_frames_in_a_large_batch(cuda, oracle, mode, side):
    assert side ** 2 > (8 << 20 if side < 4000 else 32 << 20)
    kw = dict(contrast=1.5, cr_threshold=4.0, neighbor_threshold=1.0, border=mode, maxiter=5)
    frames, want = [], []
    for i, (h, w) in enumerate(SHAPES):
        for kind in ("scalars", "maps", "background", "error"):
            rng = np.random.default_rng(1000 * i + len(kind))
            data = structured(i, h, w) if i % 2 else edge_scene(i, h, w)
            frame = dict(data=data, mask=rng.random((h, w)) < 0.02)
            if h * w > 100:
                data[rng.random((h, w)) < 0.005] = np.nan
            if kind == "error":
                frame["error"] = np.full((h, w), 12.0)
            else:
                frame.update(gain=1.5, readnoise=3.0)
            if kind == "maps":
                frame.update(gain=rng.uniform(1.2, 1.8, (h, w)), readnoise=rng.uniform(2, 4, (h, w)))
            elif kind == "background":
                frame["background"] = 12.25
            try:
                want.append(cabi.oracle_frame(oracle, frame, **kw))
            except oracle.OracleError:
                continue  # (constant: every pixel of the smallest frames is flagged)
            frames.append(frame)
    assert len(frames) > 30 and sum(int(m.sum()) for _, m, _ in want) > 100
    rng = np.random.default_rng(side)
    large = rng.normal(200, 12, (side, side))
    hit = rng.integers(0, side * side, side * side // 500)
    large.reshape(-1)[hit] += rng.uniform(100, 4000, hit.size)
    frames.append(dict(data=large, gain=1.5, readnoise=3.0))
    fr = cabi.Frames(frames)
    st, msg = cabi.run_ragged(fr, cabi.options(**kw))
    assert st == 0, msg
    *outputs, (_, large_mask) = fr.outputs()
    assert large_mask.any()
    for (clean, mask), (want_clean, want_mask, _) in zip(outputs, want):
        np.testing.assert_array_equal(mask, want_mask)
        assert_bits_equal(clean, want_clean)
