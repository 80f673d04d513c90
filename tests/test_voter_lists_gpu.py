"""Voter lists, flow lengths and seeds on the GPU against the oracle where the
lists are long (concentric rings: one list per center region, above the sizes a
thread or a warp sorts) and at the ends of the votes a seed needs."""
import numpy as np
import pytest

import cctag_b200

pytestmark = pytest.mark.gpu


def rings(w, h, cx, cy, radii, noise, seed):
    """Concentric rings whose inner circle is a few pixels wide, so that many
    outer points vote for the same inner ones."""
    y, x = np.mgrid[0:h, 0:w].astype(np.float32)
    r = np.hypot(x - cx, y - cy)
    img = np.full((h, w), 220.0, np.float32)
    for k, q in enumerate(sorted(radii, reverse=True)):
        img = np.where(r < q, 30.0 if k % 2 == 0 else 220.0, img)
    rng = np.random.default_rng(seed)
    img = (img + np.roll(img, 1, 0) + np.roll(img, 1, 1) + np.roll(img, (1, 1), (0, 1))) / 4
    return np.clip(np.rint(img + noise * rng.standard_normal(img.shape)), 0, 255).astype(np.uint8)


@pytest.mark.parametrize("min_votes", [1, 3, 9, 70])
@pytest.mark.parametrize("radii,noise", [((5, 17, 29, 41, 53, 65), 1.0), ((12, 26, 40, 54, 68, 82), 4.0),
                                         ((30, 45, 60, 75, 90, 105), 0.0)])
def test_voter_lists_match_oracle(built_library, orc, min_votes, radii, noise):
    img = rings(401, 307, 200.3, 150.8, radii, noise, 5)
    p = cctag_b200.default_params(3)
    p.distSearch = 60
    p.minVotesToSelectCandidate = min_votes
    p.edgeCapacityDivisor = 1
    longest = 0
    with cctag_b200.Detector(p, max_w=401, max_h=307) as det:
        det.image_stage(img)
        for level, src in enumerate(orc.pyramid(img, 4)):
            dx, dy, e = orc.level(src)
            v = orc.vote(e, dx, dy, distSearch=60, minVotes=min_votes)
            g = det.votes(level)
            for k in ("chosen", "nvotes", "voff", "vlist"):
                np.testing.assert_array_equal(g[k], v[k], err_msg=f"level {level} {k}")
            np.testing.assert_array_equal(g["flow"].view(np.int32), v["flow"].view(np.int32))
            np.testing.assert_array_equal(det.seeds(level), v["seeds"])
            longest = max(longest, int(v["nvotes"].max(initial=0)))
    assert longest > 8


def test_flat_frame_has_empty_lists(built_library):
    with cctag_b200.Detector(max_w=64, max_h=64) as det:
        det.image_stage(np.full((64, 64), 9, np.uint8))
        assert len(det.votes(0)["vlist"]) == 0 and det.votes(0)["voff"].tolist() == [0]
