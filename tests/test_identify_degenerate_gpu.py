"""Candidates whose axes have no usable mean (no conditioner of their conic exists):
they diverge at their initial center, however many are identified together."""
import numpy as np
import pytest

import cctag_b200
from cctag_b200 import capi
from cctag_b200.synth import cut_task_from_marker, render_frame

pytestmark = pytest.mark.gpu

OPTI_HAS_DIVERGED = -3


@pytest.mark.parametrize("mode", [capi.REFINE_GRID, capi.REFINE_GAUSS_NEWTON])
@pytest.mark.parametrize("layout", [capi.IDENT_AUTO, capi.IDENT_BLOCK])
def test_axes_without_a_mean(built_library, mode, layout):
    import torch

    fr = render_frame(200, 200, 1, (40, 40), 30, seed=5, noise_sigma=3.0)
    dev = torch.from_numpy(fr.image).cuda()
    p = cctag_b200.default_params(3)
    p.identLayout = layout
    indefinite = (0.9235779, 1.1785244, -1.7037003, -0.49956608, -0.676365, 0.52758455, 0.37097597, 0.9026692, 0.95444864)
    with cctag_b200.Detector(p, max_w=640, max_h=480) as det:
        for a, b, q in ((1e30, 535.0, None), (3e38, 3e38, None), (40.0, -40.0, None), (1e30, 535.0, indefinite)):
            t = cut_task_from_marker(fr.markers[0], (0, 0, 200, 200), n_cuts=22, local=True)
            t.a, t.b = a, b
            for k, v in enumerate(q or ()):
                t.Q[k] = v
            for n in (1, 2, 17, 30, 60, 100, 200, 400):
                got = det.identify_tasks(dev.data_ptr(), 200, 200, 200, [t] * n, mode)
                assert {r.status for r in got} == {OPTI_HAS_DIVERGED}, (a, b, n)
                assert {(r.x, r.y) for r in got} == {(t.x0, t.y0)}, (a, b, n)
                assert len({bytes(r) for r in got}) == 1, (a, b, n)
