"""Canny on caller-given derivatives of any size in both forms of the suppression:
four warps per tile up to 2,960 tiles of 32 x 32, one warp above, with partial
tiles on both borders, and gradients of a few units up to all of int16."""
import numpy as np
import pytest

import cctag_b200

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(1889, 1601), (1931, 1627), (2047, 1537)])  # 3,060, 3,111 and 3,136 tiles
@pytest.mark.parametrize("lim", [3, 200, 1500, 32767])
def test_one_warp_per_tile_matches_oracle(built_library, orc, w, h, lim):
    assert -(-w // 32) * -(-h // 32) > 2960
    check(orc, w, h, lim)


@pytest.mark.parametrize("lim", [3, 32767])
def test_four_warps_per_tile_match_oracle(built_library, orc, lim):
    assert -(-1887 // 32) * -(-1567 // 32) <= 2960
    check(orc, 1887, 1567, lim)


def check(orc, w, h, lim):
    rng = np.random.default_rng(w + lim)
    p = cctag_b200.default_params(3)
    p.edgeCapacityDivisor = 1  # noise: an edge point per few pixels
    # noise all over, and patches of one gradient with noise on top (long components across tiles)
    patch = rng.integers(-lim, lim + 1, (2, -(-h // 48), -(-w // 48))).repeat(48, 1).repeat(48, 2)[:, :h, :w]
    noise = rng.integers(-(lim // 8 + 1), lim // 8 + 2, (2, h, w))
    with cctag_b200.Detector(p, max_w=w, max_h=h) as det:
        for d in (rng.integers(-lim, lim + 1, (2, h, w)), patch + noise):
            dx, dy = (np.ascontiguousarray(a) for a in np.clip(d, -32768, 32767).astype(np.int16))
            np.testing.assert_array_equal(det.canny_from_derivatives(dx, dy), orc.thin(orc.canny(dx, dy)))
