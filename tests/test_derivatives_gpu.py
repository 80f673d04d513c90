"""The separable derivatives against the reference's tap chains: images whose
sums lie on or near rounding boundaries (ramps, steps, repeated rows, extreme
contrast), sizes around the tiles, rows and buffers off the wide accesses."""
import ctypes as C

import numpy as np
import pytest

from cctag_b200 import capi

pytestmark = pytest.mark.gpu


def images(w, h):
    rng = np.random.default_rng(w * 1000 + h)
    y, x = np.mgrid[0:h, 0:w]
    yield "noise", rng.integers(0, 256, (h, w))
    yield "extremes", rng.integers(0, 2, (h, w)) * 255
    yield "columns", np.broadcast_to(rng.integers(0, 256, (1, w)), (h, w))  # every row alike: all unsure or none
    yield "rows", np.broadcast_to(rng.integers(0, 256, (h, 1)), (h, w))
    yield "ramp", (x + 2 * y) % 256
    yield "steps", (x // 5 * 37 + y // 7 * 11) % 256
    yield "smooth", 128 + 100 * np.sin(x / 9.0) * np.cos(y / 7.0)
    yield "white", np.full((h, w), 255)


def edges_noalloc(img, pad_in, pad_out):
    import torch

    lib = capi.load()
    h, w = img.shape
    gray = torch.zeros(h * w + 8, dtype=torch.uint8, device="cuda")
    gray[pad_in:pad_in + h * w] = torch.from_numpy(img.reshape(-1)).cuda()
    dx, dy = (torch.zeros(h * w + 8, dtype=torch.int16, device="cuda") for _ in range(2))
    e = torch.zeros(h * w + 8, dtype=torch.uint8, device="cuda")
    st = torch.full((1,), -1, dtype=torch.int32, device="cuda")
    s = torch.cuda.current_stream()
    r = lib.cctagb_edges_noalloc(gray.data_ptr() + pad_in, w, h, w, C.c_float(0.01), C.c_float(0.04),
                                 dx.data_ptr() + 2 * pad_out, dy.data_ptr() + 2 * pad_out, e.data_ptr() + pad_out,
                                 st.data_ptr(), s.cuda_stream)
    assert r == capi.OK
    s.synchronize()
    assert int(st.item()) == 0
    out = [t.cpu().numpy() for t in (dx, dy, e)]
    for t in out:  # nothing written around the planes
        assert not t[:pad_out].any() and not t[pad_out + h * w:].any()
    return [t[pad_out:pad_out + h * w].reshape(h, w) for t in out]


@pytest.mark.parametrize("w,h", [(1, 1), (3, 2), (31, 33), (32, 32), (127, 31), (128, 64), (129, 65), (260, 97),
                                 (641, 47), (64, 300)])
@pytest.mark.parametrize("pad_in,pad_out", [(0, 0), (1, 1), (2, 3)])
def test_edges_match_oracle(built_library, orc, w, h, pad_in, pad_out):
    for name, a in images(w, h):
        img = np.ascontiguousarray(a.astype(np.uint8))
        dx, dy, e = edges_noalloc(img, pad_in, pad_out)
        wdx, wdy, we = orc.level(img)
        np.testing.assert_array_equal(dx, wdx, err_msg=f"{name} dx")
        np.testing.assert_array_equal(dy, wdy, err_msg=f"{name} dy")
        np.testing.assert_array_equal(e, we, err_msg=f"{name} edges")


def test_given_derivatives_of_any_size(detector, orc):
    """Canny on caller-given derivatives, which may take all of int16."""
    rng = np.random.default_rng(3)
    for lim in (3, 200, 1500, 20000):
        dx, dy = (rng.integers(-lim, lim + 1, (77, 203)).astype(np.int16) for _ in range(2))
        np.testing.assert_array_equal(detector.canny_from_derivatives(dx, dy), orc.thin(orc.canny(dx, dy)))


def test_many_tiles_match_oracle(detector, orc):
    """A frame with more tiles than the four-warp form of the suppression takes
    (odd sides: partial tiles on both borders), by the image stage."""
    for seed, kind in enumerate(("noise", "steps", "smooth")):
        img = np.ascontiguousarray(dict(images(1931, 1627))[kind].astype(np.uint8))[:1627]
        img = (img // 4 + 90).astype(np.uint8) if kind == "noise" else img  # fewer edge points than the capacity
        detector.image_stage(img)
        for level, src in enumerate(orc.pyramid(img, 4)):
            dx, dy, e = orc.level(src)
            _, gdx, gdy, ge = detector.level_planes(level)
            np.testing.assert_array_equal(gdx, dx, err_msg=f"{kind} {level}")
            np.testing.assert_array_equal(gdy, dy, err_msg=f"{kind} {level}")
            np.testing.assert_array_equal(ge, e, err_msg=f"{kind} {level}")
