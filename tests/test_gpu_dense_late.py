"""Late passes that start from much of the frames: stage 1 takes the mask row by
row instead of each changed target's neighbourhood, and the replacement gives a
block's targets a thread each.  The same frames beside a large blank one take the
lists (the rule counts the batch's pixels).  Both against the CPU oracle."""

import numpy as np
import pytest

from tests import cabi
from tests.conftest import assert_bits_equal
from tests.test_gpu_parity import MODES
from tests.test_gpu_pass_kernels import structured

pytestmark = pytest.mark.gpu

SHAPES = ((1, 40), (4, 6), (12, 13), (13, 45), (31, 70), (64, 97), (45, 33), (150, 260), (210, 300))


@pytest.mark.parametrize("mode", MODES)
@pytest.mark.parametrize("noise", ("error", "model"))
def test_rows_and_lists(cuda, oracle, mode, noise):
    kw = dict(contrast=1.0, cr_threshold=1.5, neighbor_threshold=0.7, border=mode, maxiter=6)
    frames, want = [], []
    for i, (h, w) in enumerate(SHAPES):
        rng = np.random.default_rng(i)
        data = structured(40 + i, h, w, hits=250)
        if h * w > 100:
            data[rng.random((h, w)) < 0.01] = np.nan
        frame = dict(data=data, mask=rng.random((h, w)) < 0.1)
        frame.update(dict(error=np.full((h, w), 12.0)) if noise == "error" else
                     dict(gain=rng.uniform(1.2, 1.8, (h, w)), readnoise=3.0))
        try:
            want.append(cabi.oracle_frame(oracle, frame, **kw))
        except oracle.OracleError:
            continue  # every donor flagged
        frames.append(frame)
    assert len(frames) >= 6 and max(p for _, _, p in want) > 3
    # The rule's two sides: over a 64th of the pixels, and far below.
    flagged = sum(int(m.sum()) for _, m, _ in want)
    assert 64 * flagged > 4 * sum(f["data"].size for f in frames)
    blank = dict(data=np.full((2600, 2600), 100.0))
    blank.update(dict(error=np.full((2600, 2600), 12.0)) if noise == "error" else dict(gain=1.5, readnoise=3.0))
    assert 64 * 2 * flagged < blank["data"].size
    for batch in (frames, [*frames, blank]):
        fr = cabi.Frames(batch)
        st, msg = cabi.run_ragged(fr, cabi.options(**kw, gain=1.5))
        assert st == 0, msg
        for (clean, mask), (want_clean, want_mask, _) in zip(fr.outputs(), want):
            np.testing.assert_array_equal(mask, want_mask)
            assert_bits_equal(clean, want_clean)
