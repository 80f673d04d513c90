"""Edge linking from the seeds on the GPU against the oracle where its two
walks per seed meet (closed contours shorter than both), where the running mean
of the votes ends a walk, and at the ends of the convexity window's range; and
the outlier removal of candidates with few points, whose random draws need many
outputs (5 distinct residues of as few as 5)."""
import numpy as np
import pytest

import cctag_b200
from cctag_b200.synth import render_frame

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("vote_min,window", [(0.0, 20), (0.0, 1), (0.0, 2), (0.0, 64), (0.75, 20), (3.0, 20), (0.75, 64)])
def test_links_match_oracle(built_library, orc, vote_min, window):
    p = cctag_b200.default_params(3)
    p.averageVoteMin = vote_min
    p.windowSizeOnInnerEllipticSegment = window
    frames = [render_frame(640, 480, 6, (12, 30), 50, seed=40, noise_sigma=3.0).image,
              render_frame(500, 371, 4, (20, 60), 60, seed=41, noise_sigma=9.0).image]
    with cctag_b200.Detector(p, max_w=640, max_h=480) as det:
        for img in frames:
            det.detect(img)
            for level in range(4):
                got, want = det.level_loop_two(level), orc.loop_two(img, level, p)
                for g, w in zip(got[:3], want[:3]):
                    np.testing.assert_array_equal(g, w, err_msg=f"level {level}")
                assert all(np.array_equal(a, b) for a, b in zip(got[3], want[3])), level


@pytest.mark.parametrize("seed", range(4))
def test_outlier_removal_of_few_points(built_library, orc, seed):
    p = cctag_b200.default_params(3)
    p.minPointsSegmentCandidate = 5
    p.minVotesToSelectCandidate = 1
    p.maximumNbCandidatesLoopTwo = 200
    p.edgeCapacityDivisor = 1  # noise: an edge point per three pixels
    img = render_frame(320, 240, 2, (10, 25), 60, seed=60 + seed, noise_sigma=10.0).image
    with cctag_b200.Detector(p, max_w=320, max_h=240) as det:
        det.detect(img)
        sizes = []
        for level in range(4):
            got, want = det.level_loop_two(level), orc.loop_two(img, level, p)
            for g, w in zip(got[:3], want[:3]):
                np.testing.assert_array_equal(g, w, err_msg=f"level {level}")
            assert all(np.array_equal(a, b) for a, b in zip(got[3], want[3])), level
            sizes += got[1].tolist()
        assert min(s for s in sizes if s) < 10
