"""Cut selection of markers with many outer points: more than 2,048, which the
kernel sorts with several keys per thread, and more than its 4,096, which the host
sorts and subsamples.  The selected cut ends are the oracle's, bit for bit."""
import numpy as np
import pytest

import cctag_b200
from cctag_b200.synth import render_frame

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("side,radius,low,high", [(2100, 500, 2500, 4000), (4200, 1000, 5000, 9000)])
@pytest.mark.parametrize("outer,samples,refine", [(150, 100, 20), (256, 128, 64), (20, 33, 7)])
def test_selected_cuts_match_oracle_bits(built_library, orc, side, radius, low, high, outer, samples, refine):
    fr = render_frame(side, side, 1, (radius, radius), 20, seed=radius, noise_sigma=2.0, ss=1)
    p = cctag_b200.default_params(3)
    p.nSamplesOuterEllipse = outer
    p.sampleCutLength = samples
    p.numSamplesOuterEdgePointsRefinement = refine
    with cctag_b200.Detector(p, max_w=side, max_h=side) as det:
        det.detect(fr.image)
        tasks = det.last_tasks()
        edges = det.level_planes(0)[3]
    sel = orc.cut_selection(fr.image, p)
    want = [stops for st, stops in sel if st == 1]
    assert len(want) >= 1 and len(tasks) == len(want)
    # the edge points along the outer ellipse are the points that are sorted
    y, x = np.nonzero(edges)
    t = max(tasks, key=lambda t: t.a * t.b)
    c, s = np.cos(t.angle), np.sin(t.angle)
    u, v = c * (x - t.cx) + s * (y - t.cy), -s * (x - t.cx) + c * (y - t.cy)
    near = np.abs(np.hypot(u / t.a, v / t.b) - 1.0) * min(t.a, t.b) < 1.5
    assert low <= near.sum() <= high, near.sum()
    for t, w in zip(tasks, want):
        got = np.array([[t.stop[k][0], t.stop[k][1]] for k in range(t.ncuts)], np.float32).reshape(-1, 2)
        assert got.shape == w.shape and np.array_equal(got.view(np.uint32), w.view(np.uint32))
