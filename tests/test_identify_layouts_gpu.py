"""The identification kernel's block layouts (clusters of 8, 4 and 2 blocks, one
block of 20, 12 or 4 warps per marker) and its two ways of reading pixels
(staged in shared memory, from the image) give the same bits: candidates of all
sizes, one whose rectangle cuts it off, rows on and off word boundaries, whole
and partial sample chunks, few and many cuts."""
import numpy as np
import pytest

import cctag_b200
from cctag_b200 import capi
from cctag_b200.synth import cut_task_from_marker, render_frame

pytestmark = pytest.mark.gpu

RADII = (9, 30, 75, 120, 150, 200)


@pytest.fixture(scope="module")
def crops():
    out = []
    for i, r in enumerate(RADII):
        side = int(4.2 * r + 12)
        out.append(render_frame(side, side, 1, (r, r), 50, seed=70 + i, noise_sigma=4.0, ss=2))
    return out


def place(crops, cuts, width, x_off):
    """The crops below one another in an image, x_off from its left edge, as
    local tasks; the last one again with a rectangle that cuts off its side."""
    rows = sum(c.image.shape[0] for c in crops)
    img = np.full((rows, width), 128, np.uint8)
    tasks, y = [], 0
    for c in crops:
        h, w = c.image.shape
        img[y:y + h, x_off:x_off + w] = c.image
        tasks.append(cut_task_from_marker(c.markers[0], (x_off, y, w, h), n_cuts=cuts, local=True))
        y += h
    h, w = crops[-1].image.shape
    m = crops[-1].markers[0]
    tasks.append(cut_task_from_marker(m, (x_off, y - h, int(m.center[0] + 0.8 * m.radius_px), h), n_cuts=cuts,
                                      local=True))
    return img, tasks


def bits(results):
    return [bytes(r) for r in results]


@pytest.mark.parametrize("mode", [capi.REFINE_GRID, capi.REFINE_GAUSS_NEWTON])
@pytest.mark.parametrize("samples,cuts", [(100, 22), (32, 5), (33, 32), (64, 22), (127, 9), (128, 32)])
def test_layouts_and_staging_give_the_same_bits(built_library, crops, mode, samples, cuts):
    import torch

    p = cctag_b200.default_params(3)
    p.sampleCutLength = samples
    q = cctag_b200.default_params(3)
    q.sampleCutLength = samples
    q.identLayout = capi.IDENT_BLOCK
    with cctag_b200.Detector(p, max_w=640, max_h=480) as det, cctag_b200.Detector(q, max_w=640, max_h=480) as block:
        def run(d, img, tasks, n):
            t = [tasks[i % len(tasks)] for i in range(n)]
            dev = torch.from_numpy(img).cuda()
            return bits(d.identify_tasks(dev.data_ptr(), img.shape[1], img.shape[0], img.shape[1], t, mode))

        img, tasks = place(crops, cuts, 1024, 0)
        one = [run(det, img, [t], 1)[0] for t in tasks]
        for n in (len(tasks), 30, 80, 120, 200, 400):
            got = run(det, img, tasks, n)
            assert got == [one[i % len(tasks)] for i in range(n)], n
        for n in (len(tasks), 200):
            assert run(block, img, tasks, n) == [one[i % len(tasks)] for i in range(n)], n
        for width, x_off in ((1024, 3), (1021, 0), (1022, 1)):  # rows off the word boundaries
            img2, tasks2 = place(crops, cuts, width, x_off)
            got = run(det, img2, tasks2, len(tasks))
            assert got == one, (width, x_off)
            got = run(det, img2, tasks2, 200)
            assert got == [one[i % len(tasks)] for i in range(200)], (width, x_off)
        statuses = [capi.IdentResult.from_buffer_copy(b).status for b in one]
        assert statuses.count(1) >= 1
