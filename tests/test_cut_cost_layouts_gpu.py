"""The cost kernel's two block sizes (a warp per cut while the tasks are no more
than the SMs, else four warps) give the same cost and adjoints, over few and many
cuts and samples.  They differ in how samples are grouped in the double sums
only, so a value may differ by one rounding to float, and by 1e-9 of the task's
largest adjoint where the sums cancel."""
import numpy as np
import pytest

import cctag_b200
from test_identify_layouts_gpu import crops, place  # noqa: F401  (a fixture)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("samples,cuts", [(100, 22), (32, 2), (33, 32), (64, 5), (127, 9), (128, 32)])
def test_block_sizes_agree(built_library, crops, samples, cuts):  # noqa: F811
    import torch

    p = cctag_b200.default_params(3)
    p.sampleCutLength = samples
    img, tasks = place(crops, cuts, 1021, 3)
    dev = torch.from_numpy(img).cuda()
    with cctag_b200.Detector(p, max_w=640, max_h=480) as det:
        def run(n):
            t = [tasks[i % len(tasks)] for i in range(n)]
            cen = np.array([[x.x0 + 0.3, x.y0 - 0.2] for x in t], np.float32)
            return det.cut_cost(dev.data_ptr(), img.shape[1], img.shape[0], img.shape[1], t, cen)

        few, many = run(len(tasks)), run(400)
    assert (few[0] < 1e30).sum() >= len(crops)
    at = np.arange(400) % len(tasks)
    for a, b in zip(few, many):
        a = a.reshape(len(tasks), -1)[at]
        b = b.reshape(400, -1)
        scale = np.abs(few[2]).max(1)[at][:, None]
        assert np.all(np.abs(a - b) <= 2.0**-23 * np.abs(a) + 1e-9 * scale)
