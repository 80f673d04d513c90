"""Candidates whose pixels do not fit in a block's shared memory, alone and among
smaller ones: they read the image, several chunks of a cut at once where a block
has a warp per trial, and a launch then gives less of its shared memory to the
others or none.  The results are the same bits as of each candidate by itself,
where all but the largest are staged."""
import numpy as np
import pytest

import cctag_b200
from cctag_b200 import capi
from cctag_b200.synth import render_frame
from test_identify_layouts_gpu import bits, place

pytestmark = pytest.mark.gpu

RADII = (12, 60, 140, 200, 300)


@pytest.fixture(scope="module")
def large_crops():
    return [render_frame(int(4.2 * r + 12), int(4.2 * r + 12), 1, (r, r), 50, seed=90 + i, noise_sigma=4.0, ss=2)
            for i, r in enumerate(RADII)]


@pytest.mark.parametrize("mode,grid", [(capi.REFINE_GRID, 5), (capi.REFINE_GRID, 3), (capi.REFINE_GAUSS_NEWTON, 5)])
@pytest.mark.parametrize("samples,cuts", [(100, 22), (32, 5), (33, 32), (65, 12), (128, 32)])
def test_shares_of_large_candidates(built_library, large_crops, mode, grid, samples, cuts):
    import torch

    p = cctag_b200.default_params(3)
    p.sampleCutLength = samples
    p.imagedCenterNGridSample = grid
    q = cctag_b200.default_params(3)
    q.sampleCutLength = samples
    q.imagedCenterNGridSample = grid
    q.identLayout = capi.IDENT_BLOCK
    img, tasks = place(large_crops, cuts, 1300, 3)
    dev = torch.from_numpy(img).cuda()
    with cctag_b200.Detector(p, max_w=640, max_h=480) as det, cctag_b200.Detector(q, max_w=640, max_h=480) as block:
        def run(d, which, n):
            t = [tasks[which[i % len(which)]] for i in range(n)]
            got = d.identify_tasks(dev.data_ptr(), img.shape[1], img.shape[0], img.shape[1], t, mode)
            return bits(got), [which[i % len(which)] for i in range(n)]

        one = [run(det, [i], 1)[0][0] for i in range(len(tasks))]
        every = list(range(len(tasks)))
        # all sizes (a third beyond a block's shared memory), the largest only, one
        # of them among many, and sizes up to a block's whole shared memory
        for which in (every, [4], [0, 1, 2] * 6 + [4], [3, 2, 1, 0]):
            for d, ns in ((det, (2, 17, 30, 60, 90, 120, 200, 400)), (block, (3, 160))):
                for n in ns:
                    got, src = run(d, which, n)
                    assert got == [one[i] for i in src], (which, n)
        assert [capi.IdentResult.from_buffer_copy(b).status for b in one].count(1) >= 1
