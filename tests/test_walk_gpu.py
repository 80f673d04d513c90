"""Gradient walks on the GPU against the oracle at the search distances where
their first three steps, the steps after them and their end meet, on images
whose edges lie along every border and on and off bitmap word boundaries."""
import numpy as np
import pytest

import cctag_b200

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dist", [0, 1, 2, 3, 4, 5, 6, 30, 200])
@pytest.mark.parametrize("w,h", [(40, 24), (97, 61), (320, 200)])
def test_walks_match_oracle(built_library, orc, w, h, dist):
    rng = np.random.default_rng(w)
    y, x = np.mgrid[0:h, 0:w]
    img = 60.0 + 120.0 * ((np.hypot(x - 0.4 * w, y - 0.6 * h) // 7) % 2) + 12.0 * rng.standard_normal((h, w))
    img = np.clip(np.rint(img), 0, 255).astype(np.uint8)
    p = cctag_b200.default_params(3)
    p.distSearch = dist
    p.edgeCapacityDivisor = 1
    links = 0
    with cctag_b200.Detector(p, max_w=w, max_h=h) as det:
        det.image_stage(img)
        for level, src in enumerate(orc.pyramid(img, 4)):
            dx, dy, e = orc.level(src)
            v = orc.vote(e, dx, dy, distSearch=dist)
            before, after = det.links(level)
            np.testing.assert_array_equal(before, v["before"], err_msg=f"level {level}")
            np.testing.assert_array_equal(after, v["after"], err_msg=f"level {level}")
            links += int((v["before"] >= 0).sum() + (v["after"] >= 0).sum())
    assert links > 0
