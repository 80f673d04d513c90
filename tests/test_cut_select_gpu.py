"""Cut selection at the sizes where its phases change: keys sorted by one warp,
by one key per thread and by more, few and the most outer points, sample counts
with whole and partial shares of the four lanes.  The selected cut ends are the oracle's, bit for bit."""
import numpy as np
import pytest

import cctag_b200
from cctag_b200.synth import render_frame

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("side,radius", [(320, 24), (640, 100), (1000, 170), (1000, 225)])
@pytest.mark.parametrize("outer,samples,refine", [(150, 100, 20), (256, 128, 64), (5, 32, 2), (4, 33, 7), (251, 35, 3)])
def test_selected_cuts_match_oracle_bits(orc, side, radius, outer, samples, refine):
    fr = render_frame(side, side, 1, (radius, radius), 50, seed=radius, noise_sigma=3.0, ss=2)
    p = cctag_b200.default_params(3)
    p.nSamplesOuterEllipse = outer
    p.sampleCutLength = samples
    p.numSamplesOuterEdgePointsRefinement = refine
    with cctag_b200.Detector(p, max_w=side, max_h=side) as det:
        det.detect(fr.image)
        tasks = det.last_tasks()
    sel = orc.cut_selection(fr.image, p)
    assert len(sel) > 0
    want = [stops for st, stops in sel if st == 1]
    assert len(tasks) == len(want)
    for t, w in zip(tasks, want):
        got = np.array([[t.stop[k][0], t.stop[k][1]] for k in range(t.ncuts)], np.float32).reshape(-1, 2)
        assert got.shape == w.shape and np.array_equal(got.view(np.uint32), w.view(np.uint32))
