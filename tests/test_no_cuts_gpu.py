"""A detection whose parameters leave a marker no cut (a number of cuts of zero
or below): it is found with the status of no selected cuts and no id, whatever
the number."""
import numpy as np
import pytest

import cctag_b200
from cctag_b200 import capi
from cctag_b200.synth import render_frame

pytestmark = pytest.mark.gpu

NO_SELECTED_CUTS = -2


@pytest.mark.parametrize("mode", [capi.REFINE_GRID, capi.REFINE_GAUSS_NEWTON])
def test_markers_without_cuts(built_library, mode):
    img = render_frame(640, 480, 3, (25, 50), 40, seed=11, noise_sigma=3.0).image
    with cctag_b200.Detector(cctag_b200.default_params(3), max_w=640, max_h=480) as det:
        whole, _ = det.detect(img)
    assert len(whole) >= 2
    for cuts in (0, -1, -5, -12, -100, -(2**31)):
        p = cctag_b200.default_params(3)
        p.refineMode = mode
        p.numCutsInIdentStep = cuts
        with cctag_b200.Detector(p, max_w=640, max_h=480) as det:
            got, _ = det.detect(img)
        assert [m.status for m in got] == [NO_SELECTED_CUTS] * len(got) and len(got) >= len(whole), cuts
        assert all(m.id == -1 for m in got), cuts
