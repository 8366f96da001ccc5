"""Replacements whose nearest donor is far away: windows of more than 128 cells
are found from bit words and take their median from the window's rim, in the
hole fill, the first pass, the late passes and the backward.  Masks, pixels and
gradients are those of the CPU oracle."""

import numpy as np
import pytest

from tests.conftest import assert_bits_equal

pytestmark = pytest.mark.gpu


def check(torch, oracle, data, error, mask, hits, **settings):
    """Forward bits, mask and gradient of one error-map frame."""
    from cusmic_b200.plan import Batch, Plan
    up = lambda a: torch.from_numpy(a).cuda()
    batch = Batch.stack(up(data[None]), error=up(error), mask=up(mask))
    plan = Plan(batch, graph=False, keep=True, **settings)
    try:
        plan.execute()
        plan.wait()
        want_clean, want_mask, _ = oracle.clean_frame(data, error=error, mask=mask, **settings)
        np.testing.assert_array_equal(batch.mask_out[0].cpu().numpy().astype(bool), want_mask)
        assert_bits_equal(batch.clean[0].cpu().numpy(), want_clean)
        assert want_mask[tuple(np.transpose(hits))].all()
        g = np.random.default_rng(1).normal(size=(1, *data.shape))
        gx, _ = plan.backward(up(g))
        rgx, _, _ = oracle.backward(data, want_mask, g[0], mask=mask)
        # Atomic additions in any order: n terms of N(0, 1) differ by at most about
        # n x 2^-53 x their absolute sum, for the 80 targets that few donors can
        # share 80 x 1.1e-16 x 64 = 6e-13 on each side.
        np.testing.assert_allclose(gx[0].cpu().numpy(), rgx, rtol=1e-13, atol=1.2e-12)
    finally:
        plan.close()


@pytest.mark.parametrize("donors", ("rim", "few"))
@pytest.mark.parametrize("radius", (5, 6, 15, 16, 17, 31, 32, 33, 64, 101))
def test_far_donors(cuda, oracle, radius, donors):
    """Hits amid excluded squares of a radius, at the frame's corner, edge and
    middle, whose donors are the pixels past the square, or a few of them; a sky
    of small values with zeros of both signs, so that donors tie, and clusters of
    hits elsewhere, whose growth keeps the passes going."""
    rng = np.random.default_rng(radius)
    side = 2 * radius + 5
    h, w = 2 * side + 3, 2 * side + radius + 40
    data = rng.choice(np.array([-0.0, 0.0, 1.0, -1.0, 0.5]), size=(h, w))
    hits = [(0, 0), (h - 1, radius + 2), (side, side), (h - 1, w - 1)]
    mask = np.zeros((h, w), dtype=bool)
    for y, x in hits:
        mask[max(0, y - radius):y + radius + 1, max(0, x - radius):x + radius + 1] = True
    if donors == "few":
        mask |= rng.random((h, w)) < 0.99
    for k in range(8):  # clusters, unmasked
        y, x = int(rng.integers(0, 12)), int(rng.integers(w - 34, w - 6))
        mask[y:y + 4, x:x + 4] = False
        data[y:y + 3, x:x + 3] += rng.uniform(5, 600, (3, 3))
    data[side + 8, side:side + 2] = np.nan  # holes with far donors
    for y, x in hits:
        mask[y, x] = False
        data[y, x] += 5000.0
    check(cuda, oracle, data, np.full((h, w), 0.4), mask, hits, contrast=3.0, cr_threshold=5.0,
          neighbor_threshold=3.0, maxiter=4)


def test_donor_a_thousand_pixels_away(cuda, oracle):
    """A lone bright pixel in a masked amplifier, more than 1000 pixels from its
    nearest donor, and ordinary rays beside the amplifier: every pass replaces the
    pixel again."""
    rng = np.random.default_rng(11)
    h, w = 2110, 2300
    data = 100 + rng.normal(0, 3, (h, w))
    mask = np.zeros((h, w), dtype=bool)
    mask[:, :2105] = True
    ys, xs = rng.integers(0, h - 3, 400), rng.integers(2105, w - 3, 400)
    for y, x in zip(ys, xs):
        data[y:y + 3, x:x + 3] += rng.uniform(5, 3000, (3, 3))
    hit = (1055, 1055)
    mask[hit] = False
    data[hit] += 5000
    check(cuda, oracle, data, np.full((h, w), 3.0), mask, [hit], contrast=1.5, cr_threshold=4.0,
          neighbor_threshold=1.5, maxiter=4)
