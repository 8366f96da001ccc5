"""The kernels of a detection pass where their work splits: candidates within
two pixels of an edge (read from the first pass's sig_raw map).  Masks and
pixels are those of the CPU oracle bit for bit."""

import numpy as np
import pytest

from tests.test_gpu_parity import MODES, SETTINGS, check_against_oracle, small_scene

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
