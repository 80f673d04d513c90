"""The seeds' processing order (placed by the voter that made each, then sorted
by votes) is the oracle's, from no seeds to many and at the fewest votes a seed
can need."""
import numpy as np
import pytest

import cctag_b200
from cctag_b200.synth import render_frame

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("min_votes", [0, 1, 2, 5, 1000])
@pytest.mark.parametrize("w,h,markers", [(64, 48, 0), (333, 259, 2), (640, 480, 6)])
def test_seed_order_matches_oracle(built_library, orc, w, h, markers, min_votes):
    img = render_frame(w, h, markers, (20, 40), 50, seed=9, noise_sigma=6.0, ss=2).image
    p = cctag_b200.default_params(3)
    p.minVotesToSelectCandidate = min_votes
    p.edgeCapacityDivisor = 1
    seeds = 0
    with cctag_b200.Detector(p, max_w=w, max_h=h) as det:
        det.detect(img)
        for level, src in enumerate(orc.pyramid(img, 4)):
            dx, dy, e = orc.level(src)
            v = orc.vote(e, dx, dy, minVotes=min_votes)
            np.testing.assert_array_equal(det.seeds(level), v["seeds"], err_msg=f"level {level}")
            seeds += len(v["seeds"])
    assert (seeds > 0) == (markers > 0 and min_votes < 1000)
