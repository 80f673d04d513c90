"""Timed cases of the library: the calls a user's program makes, through the C ABI
(``include/cctag_b200.h``, bound by ``cctag_b200.capi``).

Five kinds of call cover the library's use:

``edges``   cctagb_edges_noalloc: derivatives and edge map of one gray image in device memory, on the
            caller's stream (a program that wants edges only and owns every buffer).
``detect``  cctagb_detect / cctagb_detect_device: all markers of one frame (a single camera, where
            latency counts), the frame in pinned host memory or already on the device.
``batch``   cctagb_detect_batch: all markers of several frames per call (a rig of cameras, or a
            recorded sequence), of one size or of mixed sizes.
``refine``  cctagb_identify_tasks: center refinement and ID reading of given candidates, many per call,
            by the shrinking grid or by Gauss-Newton.
``cost``    cctagb_cut_cost: the cut-consistency cost of given candidates and its gradients in the
            center and in the homography (an outer optimiser's forward and backward pass).

Frames and crops are rendered on the GPU from the seed: ring markers of the 3-crown bank under random
homographies, noise, motion blur, an illumination gradient, and for the clutter frames a band-limited
texture, ellipses and line segments.
"""
import ctypes as C
import math

import numpy as np
import torch

from cctag_b200 import capi
from cctag_b200.bank import THREE_CROWNS
from cctag_b200.synth import CAMERA_SIZES, marker_homography

EDGE_PIXELS = 1 << 20                    # pixel limit of cctagb_edges_noalloc
MARKER_CAP = 128                         # room for markers per frame
BEGIN = 0.25                             # where a 3-crown cut's samples begin, in outer radii
WHITE, BLACK = 235.0, 20.0


# ------------------------------------------------------------------ the cases --
def listed():
    return [
        # A small sensor's image, edges only: launch latency.
        dict(name="edges_640x480", kind="edges", w=640, h=480, markers=3, rmin=20.0, rmax=90.0, noise=4.0),
        # A cropped window of odd size near the call's pixel limit.
        dict(name="edges_1153x907", kind="edges", w=1153, h=907, markers=6, rmin=20.0, rmax=120.0, noise=6.0),
        # The smallest detection: one marker in a 320x240 frame from host memory (robot or drone preview).
        _detect("detect_320x240_host", 320, 240, 1, 40.0, 60.0, noise=3.0, tilt=30.0, host=True),
        # A 720p camera frame with a few large markers, already on the device (a decoder's output).
        _detect("detect_1280x720", 1280, 720, 4, 40.0, 120.0, noise=4.0, tilt=45.0),
        # A 1080p camera frame from host memory, 12 markers of all sizes, noise, motion blur, uneven light.
        _detect("detect_1920x1080_host", 1920, 1080, 12, 20.0, 200.0, noise=8.0, motion=3.0, gradient=40.0, host=True),
        # A frame whose sides divide by nothing (a cropped region of interest): the general pyramid.
        _detect("detect_1621x913", 1621, 913, 8, 20.0, 150.0, noise=6.0),
        # A 4K frame of a cluttered scene: over a million edge points.
        _detect("detect_3840x2160_clutter", 3840, 2160, 30, 15.0, 300.0, noise=6.0, clutter=True),
        # Sixteen 1080p frames per call, on the device (throughput of a recorded sequence).
        _batch("batch_16x1080p", 16, 1920, 1080, 12, 20.0, 200.0, noise=8.0, motion=3.0, gradient=40.0, wave=16,
               slots=16),
        # A rig of sixteen cameras, 640x480 to 3840x2160, 0 to 20 markers each, from host memory.
        _batch("batch_16_cameras_host", 16, 0, 0, 20, 15.0, 200.0, noise=6.0, wave=4, slots=8, host=True),
        # Candidates of many frames refined in one call, by the reference's grid ...
        dict(name="refine_grid_1024", kind="refine", n=1024, cuts=22, samples=100, mode="grid", local=True),
        # ... and by Gauss-Newton.
        dict(name="refine_gn_4096", kind="refine", n=4096, cuts=22, samples=100, mode="gn", local=True),
        # One evaluation of an outer optimiser over the same number of candidates.
        dict(name="cost_4096", kind="cost", n=4096, cuts=22, samples=100, local=True),
    ]


def _detect(name, w, h, markers, rmin, rmax, noise, tilt=60.0, motion=0.0, gradient=0.0, clutter=False, host=False):
    return dict(name=name, kind="detect", w=w, h=h, markers=markers, rmin=rmin, rmax=rmax, noise=noise, tilt=tilt,
                motion=motion, gradient=gradient, clutter=clutter, host=host)


def _batch(name, frames, w, h, markers, rmin, rmax, noise, wave, slots, tilt=60.0, motion=0.0, gradient=0.0,
           host=False):
    """w = h = 0: the frames cycle through CAMERA_SIZES, with marker counts spread over 0..markers."""
    return dict(name=name, kind="batch", frames=frames, w=w, h=h, markers=markers, rmin=rmin, rmax=rmax, noise=noise,
                tilt=tilt, motion=motion, gradient=gradient, clutter=False, host=host, wave=wave, slots=slots)


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["edges", "detect", "detect", "batch", "refine", "refine", "cost"])
    if kind == "edges":
        w = _log_int(rng, 160, 2400)
        h = _log_int(rng, 120, min(EDGE_PIXELS // w, 1600))
        return dict(kind=kind, w=w, h=h, markers=rng.randint(0, 6), rmin=15.0, rmax=min(w, h) / 5.0 + 16.0,
                    noise=round(rng.uniform(2.0, 9.0), 2))
    if kind in ("detect", "batch"):
        frames = rng.randint(2, 16) if kind == "batch" else 1
        w = _log_int(rng, 320, 3840 if frames == 1 else min(3840, int(6000 / math.sqrt(frames))))
        h = max(240, int(w * rng.choice([9 / 16, 3 / 4, 1.0, 0.61])))
        if w * h > 3840 * 2160:
            h = 3840 * 2160 // w
        if rng.random() < 0.5:  # the sizes cameras give
            w, h = w // 8 * 8, h // 8 * 8
        side = min(w, h)
        c = dict(kind=kind, w=w, h=h, markers=rng.randint(1, 20), rmin=15.0, rmax=round(max(20.0, side / 5.0), 1),
                 noise=round(rng.uniform(2.0, 8.0), 2), tilt=round(rng.uniform(30.0, 60.0), 1),
                 motion=rng.choice([0.0, 0.0, 2.0, 4.0]), gradient=rng.choice([0.0, 40.0]),
                 clutter=frames == 1 and rng.random() < 0.25, host=rng.random() < 0.5)
        if kind == "batch":
            c.update(frames=frames, wave=rng.choice([1, 2, 4, 8, 16]), slots=rng.choice([4, 8, 16]))
        return c
    mode = rng.choice(["grid", "gn"]) if kind == "refine" else None
    n = _log_int(rng, 1, 1024 if mode == "grid" else 4096)
    # image coordinates for the candidates of one frame, crop coordinates for those of many
    c = dict(kind=kind, n=n, cuts=rng.randint(12, 22), samples=rng.randint(64, 100), local=n > 24)
    return dict(c, mode=mode) if mode else c


# ------------------------------------------------------------------ rendering --
def _phi(t):
    return 0.5 * (1.0 + torch.erf(t * (1.0 / math.sqrt(2.0))))


def _marker_layers(Hi, radii, X, Y, sigma=1.0, margin=1.3):
    """Coverage and value of markers seen through a Gaussian blur of `sigma` px: each ring edge is a step in
    the plane radius rho, blurred along its gradient.  Hi: [..., 3, 3]; radii: [..., 5], descending."""
    a = [Hi[..., i // 3, i % 3].float() for i in range(9)]
    u, v, w = a[0] * X + a[1] * Y + a[2], a[3] * X + a[4] * Y + a[5], a[6] * X + a[7] * Y + a[8]
    p, q = u / w, v / w
    rho = torch.sqrt(p * p + q * q).clamp_min(1e-6)
    gx = (p * (a[0] - p * a[6]) + q * (a[3] - q * a[6])) / (rho * w)
    gy = (p * (a[1] - p * a[7]) + q * (a[4] - q * a[7])) / (rho * w)
    s = 1.0 / (sigma * torch.sqrt(gx * gx + gy * gy).clamp_min(1e-6))
    cov = _phi((margin - rho) * s)
    val = torch.full_like(rho, WHITE)
    step = BLACK - WHITE
    for k in range(6):
        r = 1.0 if k == 0 else radii[..., k - 1]
        val = val + step * _phi((r - rho) * s)
        step = -step
    return cov, val


def _radii(ids, dev):
    rows = np.sort(1.0 / np.asarray(THREE_CROWNS, np.float64)[ids], axis=-1)[..., ::-1]
    return torch.from_numpy(np.ascontiguousarray(rows).astype(np.float32)).to(dev)


def _taps(img, taps):
    """Sum of shifted copies of img, edges repeated: taps = [(dy, dx, weight)]."""
    r = max(max(abs(y), abs(x)) for y, x, _ in taps)
    h, w = img.shape
    yi = torch.arange(-r, h + r, device=img.device).clamp(0, h - 1)
    xi = torch.arange(-r, w + r, device=img.device).clamp(0, w - 1)
    pad = img[yi][:, xi]
    out = torch.zeros_like(img)
    for y, x, k in taps:
        out += k * pad[r + y:r + y + h, r + x:r + x + w]
    return out


def _gauss(img, sigma):
    r = int(math.ceil(3 * sigma))
    k = np.exp(-0.5 * (np.arange(-r, r + 1) / sigma) ** 2)
    k /= k.sum()
    return _taps(_taps(img, [(0, i, float(k[r + i])) for i in range(-r, r + 1)]),
                 [(i, 0, float(k[r + i])) for i in range(-r, r + 1)])


def _motion_taps(length, angle):
    acc = {}
    n = 2 * int(math.ceil(length)) + 1
    for t in np.linspace(-length / 2, length / 2, n):
        dx, dy = t * math.cos(angle), t * math.sin(angle)
        ix, iy = math.floor(dx), math.floor(dy)
        fx, fy = dx - ix, dy - iy
        for y, x, k in ((iy, ix, (1 - fx) * (1 - fy)), (iy, ix + 1, fx * (1 - fy)), (iy + 1, ix, (1 - fx) * fy),
                        (iy + 1, ix + 1, fx * fy)):
            acc[y, x] = acc.get((y, x), 0.0) + k / n
    return [(y, x, k) for (y, x), k in sorted(acc.items()) if k > 1e-6]


def _box(cx, cy, ext, w, h, dev):
    x0, x1 = max(int(cx - ext), 0), min(int(cx + ext) + 1, w - 1)
    y0, y1 = max(int(cy - ext), 0), min(int(cy + ext) + 1, h - 1)
    if x1 <= x0 or y1 <= y0:
        return None
    X = torch.arange(x0, x1 + 1, device=dev, dtype=torch.float32)[None, :]
    Y = torch.arange(y0, y1 + 1, device=dev, dtype=torch.float32)[:, None]
    return slice(y0, y1 + 1), slice(x0, x1 + 1), X, Y


def _clutter(canvas, rng, gen):
    """A textured background, single and double ellipses, line segments (30 markers' worth of 4K clutter,
    in proportion for smaller frames)."""
    h, w = canvas.shape
    dev = canvas.device
    t = _gauss(torch.randn(h, w, generator=gen, device=dev), 2.0)
    canvas += 6.0 / (1.0 / (2.0 * 2.0 * math.sqrt(math.pi))) * t
    share = w * h / (3840 * 2160)
    for _ in range(int(200 * share)):
        cx, cy, a = rng.uniform(0, w), rng.uniform(0, h), rng.uniform(8, 120)
        b, ang, val, width = a * rng.uniform(0.3, 1.0), rng.uniform(0, math.pi), rng.uniform(0, 255), rng.uniform(1.5, 6)
        box = _box(cx, cy, a + 8, w, h, dev)
        rings = 1 + int(rng.uniform() < 0.5)
        if box is None:
            continue
        ys, xs, X, Y = box
        c, s = math.cos(ang), math.sin(ang)
        U, V = c * (X - cx) + s * (Y - cy), -s * (X - cx) + c * (Y - cy)
        for k in range(rings):
            sc = 1.0 - 0.35 * k
            d = (torch.sqrt((U / (a * sc)) ** 2 + (V / (b * sc)) ** 2) - 1.0).abs() * (b * sc)
            canvas[ys, xs] += (width / 2 - d + 0.5).clamp(0, 1) * (val - canvas[ys, xs])
    for _ in range(int(300 * share)):
        x0, y0, length = rng.uniform(0, w), rng.uniform(0, h), rng.uniform(20, 300)
        ang, width, val = rng.uniform(0, 2 * math.pi), rng.uniform(1, 4), rng.uniform(0, 255)
        dx, dy = length * math.cos(ang), length * math.sin(ang)
        box = _box(x0 + dx / 2, y0 + dy / 2, length / 2 + 4, w, h, dev)
        if box is None:
            continue
        ys, xs, X, Y = box
        t = (((X - x0) * dx + (Y - y0) * dy) / (length * length)).clamp(0, 1)
        d = torch.hypot(X - (x0 + t * dx), Y - (y0 + t * dy))
        canvas[ys, xs] += (width / 2 - d + 0.5).clamp(0, 1) * (val - canvas[ys, xs])


def _frame(case, w, h, markers, seed):
    """One gray frame (uint8, on the GPU) of the case."""
    dev = torch.device("cuda")
    rng = np.random.default_rng(seed)
    gen = torch.Generator(device=dev).manual_seed(seed)
    canvas = torch.full((h, w), 128.0, device=dev)
    if case.get("clutter"):
        _clutter(canvas, rng, gen)
        canvas = _gauss(canvas, 1.0)
    placed, tries = [], 0
    rmax = min(case["rmax"], min(w, h) / 4.0)
    while len(placed) < markers and tries < 200 * max(1, markers):
        tries += 1
        r = rng.uniform(min(case["rmin"], rmax), rmax)
        ext = 2.08 * r + 4
        if 2 * ext >= min(w, h):
            continue
        cx, cy = rng.uniform(ext, w - ext), rng.uniform(ext, h - ext)
        if any((cx - x) ** 2 + (cy - y) ** 2 < (ext + e) ** 2 for x, y, e in placed):
            continue
        placed.append((cx, cy, ext))
        H = marker_homography(rng, cx, cy, r, case.get("tilt", 60.0), 1.2 * max(w, h))
        ys, xs, X, Y = _box(cx, cy, ext, w, h, dev)
        cov, val = _marker_layers(torch.from_numpy(np.linalg.inv(H)).to(dev),
                                  _radii(int(rng.integers(len(THREE_CROWNS))), dev), X, Y)
        canvas[ys, xs] += cov * (val - canvas[ys, xs])
    if case.get("motion"):
        canvas = _taps(canvas, _motion_taps(case["motion"], rng.uniform(0, math.pi)))
    if case.get("gradient"):
        ang = rng.uniform(0, 2 * math.pi)
        X = torch.arange(w, device=dev, dtype=torch.float32)[None, :] - w / 2
        Y = torch.arange(h, device=dev, dtype=torch.float32)[:, None] - h / 2
        c, s = math.cos(ang), math.sin(ang)
        canvas += case["gradient"] / (abs(c) * w / 2 + abs(s) * h / 2) * (c * X + s * Y)
    canvas += case["noise"] * torch.randn(h, w, generator=gen, device=dev)
    return canvas.round_().clamp_(0, 255).to(torch.uint8)


# ---------------------------------------------------------------- the library --
class _Handle:
    """A detection handle of the C ABI, destroyed with its owner."""

    def __init__(self, max_w, max_h, max_batch=1, **params):
        self.lib = capi.load()
        p = capi.default_params(3)
        for k, v in params.items():
            setattr(p, k, v)
        self.h = C.c_void_p()
        st = self.lib.cctagb_create(C.byref(p), max_w, max_h, max_batch, C.byref(self.h))
        if st != capi.OK:
            raise capi.CCTagError(st, "cctagb_create")

    def check(self, st):
        if st != capi.OK:
            raise capi.CCTagError(st, self.lib.cctagb_last_error_string(self.h).decode())

    def __del__(self):
        if getattr(self, "h", None):
            self.lib.cctagb_destroy(self.h)
            self.h = None


MARKER = np.dtype(capi.Marker)
TASK = np.dtype(capi.CutTask)
RESULT = np.dtype(capi.IdentResult)


def _marker_arrays(markers):
    """The fields of a marker array (structured; zeros past the markers found) as plain arrays."""
    o = markers["outer"]
    return {"id": markers["id"], "status": markers["status"], "level": markers["pyramidLevel"],
            "center": np.stack([markers["x"], markers["y"]], -1),
            "ellipse": np.stack([o[k] for k in ("cx", "cy", "a", "b", "angle")], -1), "conic": o["m"],
            "homography": markers["homography"], "quality": markers["quality"], "scale": markers["scale"]}


# ------------------------------------------------------------ candidate crops --
def _candidates(case, seed):
    """A device image holding n marker crops (outer radius 8-150 px, tilt up to 70 degrees, noise 2-12) and
    their cut tasks: true outer ellipse, cut ends spread evenly on it, started at the ellipse center."""
    n, cuts = case["n"], case["cuts"]
    dev = torch.device("cuda")
    rng = np.random.default_rng(seed)
    gen = torch.Generator(device=dev).manual_seed(seed)
    r = np.sort(rng.uniform(8.0, 150.0, n))[::-1]
    if n < 64:  # few: their sizes as of a real frame's markers
        r = np.sort(rng.uniform(15.0, 120.0, n))[::-1]
    side = np.ceil(4.2 * r + 12).astype(np.int64)
    H = np.empty((n, 3, 3))
    for i in range(n):
        mid = side[i] / 2
        H[i] = marker_homography(rng, mid + rng.uniform(-1, 1), mid + rng.uniform(-1, 1), r[i], 70.0, 1.2 * side[i])
    radii = _radii(rng.integers(0, len(THREE_CROWNS), n), dev)
    noise = torch.from_numpy(rng.uniform(2.0, 12.0, n).astype(np.float32)).to(dev)
    Hi = torch.from_numpy(np.linalg.inv(H)).to(dev)
    width = int(max(4096, side[0]))
    strips, roi, y0 = [], np.zeros((n, 4), np.int32), 0
    i = 0
    while i < n:  # a strip of the atlas: crops of one (rounded up) size side by side
        s = int(side[i])
        m = min(width // s, n - i)
        X = torch.arange(s, device=dev, dtype=torch.float32)[None, None, :]
        Y = torch.arange(s, device=dev, dtype=torch.float32)[None, :, None]
        cov, val = _marker_layers(Hi[i:i + m, None, None], radii[i:i + m, None, None], X, Y)
        crop = 128.0 + cov * (val - 128.0)
        crop += noise[i:i + m, None, None] * torch.randn(m, s, s, generator=gen, device=dev)
        strip = torch.full((s, width), 128, device=dev, dtype=torch.uint8)
        strip[:, :m * s] = crop.round_().clamp_(0, 255).to(torch.uint8).permute(1, 0, 2).reshape(s, m * s)
        strips.append(strip)
        roi[i:i + m, 0], roi[i:i + m, 1] = np.arange(m) * s, y0
        roi[i:i + m, 2] = roi[i:i + m, 3] = side[i:i + m]
        y0 += s
        i += m
    image = torch.cat(strips)
    # the outer ellipse: the image of the unit circle
    off = np.zeros((n, 2)) if case["local"] else roi[:, :2].astype(np.float64)
    T = np.tile(np.eye(3), (n, 1, 1))
    T[:, 0, 2], T[:, 1, 2] = -off[:, 0], -off[:, 1]
    P = np.linalg.inv(H) @ T
    Q = P.transpose(0, 2, 1) @ np.diag([1.0, 1.0, -1.0]) @ P
    Q /= np.abs(Q).max(axis=(1, 2), keepdims=True)
    A, b = Q[:, :2, :2], Q[:, :2, 2]
    c = -np.linalg.solve(A, b[..., None])[..., 0]
    k = Q[:, 2, 2] + (b * c).sum(-1)
    ev, V = np.linalg.eigh(A / -k[:, None, None])
    ax, ang = 1.0 / np.sqrt(ev), np.arctan2(V[:, 1, 0], V[:, 0, 0])
    th = 2 * math.pi * np.arange(cuts)[None, :] / cuts
    ca, sa = np.cos(ang)[:, None], np.sin(ang)[:, None]
    ex, ey = ax[:, :1] * np.cos(th), ax[:, 1:] * np.sin(th)
    t = np.zeros(n, TASK)
    t["Q"] = Q.reshape(n, 9)
    t["cx"], t["cy"], t["a"], t["b"], t["angle"] = c[:, 0], c[:, 1], ax[:, 0], ax[:, 1], ang
    t["x0"], t["y0"] = c[:, 0], c[:, 1]
    t["ncuts"] = cuts
    t["stop"][:, :cuts, 0] = c[:, :1] + ex * ca - ey * sa
    t["stop"][:, :cuts, 1] = c[:, 1:] + ex * sa + ey * ca
    t["roi"] = roi
    t["local"] = int(case["local"])
    # centers an optimiser would ask for: off the start by up to a pixel
    centers = (np.stack([t["x0"], t["y0"]], -1) + rng.uniform(-1, 1, (n, 2))).astype(np.float32)
    order = rng.permutation(n)
    return image, np.ascontiguousarray(t[order]), np.ascontiguousarray(centers[order])


# --------------------------------------------------------------- prepare, run --
def _sizes(case):
    """(w, h, markers) of each frame of a batch."""
    n = case["frames"]
    if case["w"]:
        return [(case["w"], case["h"], case["markers"])] * n
    return [CAMERA_SIZES[i % len(CAMERA_SIZES)] + (case["markers"] * (n - 1 - i) // max(1, n - 1),) for i in range(n)]


def prepare(case, seed):
    kind = case["kind"]
    if kind == "edges":
        w, h = case["w"], case["h"]
        gray = _frame(case, w, h, case["markers"], seed)
        return {"kind": kind, "lib": capi.load(), "w": w, "h": h, "gray": gray,
                "dx": torch.empty((h, w), dtype=torch.int16, device="cuda"),
                "dy": torch.empty((h, w), dtype=torch.int16, device="cuda"),
                "edges": torch.empty((h, w), dtype=torch.uint8, device="cuda"),
                "status": torch.zeros(1, dtype=torch.int32, device="cuda")}
    if kind == "detect":
        w, h = case["w"], case["h"]
        gray = _frame(case, w, h, case["markers"], seed)
        out = np.zeros(MARKER_CAP, MARKER)
        return {"kind": kind, "handle": _Handle(w, h), "w": w, "h": h, "host": case["host"],
                "gray": gray.cpu().pin_memory() if case["host"] else gray, "out": out, "found": C.c_int()}
    if kind == "batch":
        sizes = _sizes(case)
        handle = _Handle(max(s[0] for s in sizes), max(s[1] for s in sizes), case["slots"],
                         batchWaveFrames=case["wave"], hostThreads=8)
        grays, outs = [], np.zeros((len(sizes), MARKER_CAP), MARKER)
        frames = (capi.Frame * len(sizes))()
        for i, (w, h, markers) in enumerate(sizes):
            g = _frame(case, w, h, markers, seed * 100 + i)
            g = g.cpu().pin_memory() if case["host"] else g
            f = frames[i]
            f.gray, f.w, f.h, f.pitch, f.frame_id, f.is_device = g.data_ptr(), w, h, w, i, int(not case["host"])
            f.out, f.cap = C.cast(capi.ptr(outs[i]), C.POINTER(capi.Marker)), MARKER_CAP
            grays.append(g)
        torch.cuda.synchronize()
        return {"kind": kind, "handle": handle, "gray": grays, "out": outs, "frames": frames}
    image, tasks, centers = _candidates(case, seed)
    torch.cuda.synchronize()
    n = case["n"]
    s = {"kind": kind, "handle": _Handle(640, 480, sampleCutLength=case["samples"]), "image": image, "tasks": tasks,
         "n": n}
    if kind == "refine":
        s["mode"] = capi.REFINE_GRID if case["mode"] == "grid" else capi.REFINE_GAUSS_NEWTON
        s["out"] = np.zeros(n, RESULT)
    else:
        s.update(centers=centers, cost=np.zeros(n, np.float32), d_center=np.zeros((n, 2), np.float32),
                 d_h=np.zeros((n, 9), np.float32))
    return s


def run(state):
    kind = state["kind"]
    if kind == "edges":
        w, h = state["w"], state["h"]
        st = state["lib"].cctagb_edges_noalloc(
            state["gray"].data_ptr(), w, h, w, 0.01, 0.04, state["dx"].data_ptr(), state["dy"].data_ptr(),
            state["edges"].data_ptr(), state["status"].data_ptr(), torch.cuda.current_stream().cuda_stream)
        if st != capi.OK:
            raise capi.CCTagError(st, "cctagb_edges_noalloc")
        return state["dx"], state["dy"], state["edges"], state["status"]
    handle = state["handle"]
    lib, h = handle.lib, handle.h
    if kind == "detect":
        call = lib.cctagb_detect if state["host"] else lib.cctagb_detect_device
        handle.check(call(h, state["gray"].data_ptr(), state["w"], state["h"], state["w"], 0, capi.ptr(state["out"]),
                          MARKER_CAP, C.byref(state["found"]), None))
        return {"found": state["found"].value, **_marker_arrays(state["out"])}
    if kind == "batch":
        frames = state["frames"]
        handle.check(lib.cctagb_detect_batch(h, frames, len(frames)))
        return {"found": np.array([f.n_out for f in frames]), **_marker_arrays(state["out"])}
    image, tasks, n = state["image"], state["tasks"], state["n"]
    if kind == "refine":
        out = state["out"]
        handle.check(lib.cctagb_identify_tasks(h, image.data_ptr(), image.shape[1], image.shape[0], image.shape[1],
                                               capi.ptr(tasks), n, state["mode"], capi.ptr(out)))
        return {"status": out["status"], "id": out["id"], "center": np.stack([out["x"], out["y"]], -1), "H": out["H"],
                "residual": out["residual"], "score": out["score"], "nvalid": out["nvalid"],
                "iterations": out["iterations"]}
    handle.check(lib.cctagb_cut_cost(h, image.data_ptr(), image.shape[1], image.shape[0], image.shape[1],
                                     capi.ptr(tasks), n, capi.ptr(state["centers"]), capi.ptr(state["cost"]),
                                     capi.ptr(state["d_center"]), capi.ptr(state["d_h"])))
    return {"cost": state["cost"], "d_center": state["d_center"], "d_h": state["d_h"]}


# ----------------------------------------------------------------------- work --
def work(case):
    """Bytes: the frame or the samples' pixels read once, results written once.  Operations: the derivative
    filter of every level as a separable one (34 per pixel) for images; 33 per bilinear sample of a
    refinement's cuts (its homography point, the read, the cost sums), three times that with gradients."""
    kind = case["kind"]
    if kind == "edges":
        px = case["w"] * case["h"]
        return {"bytes": 6 * px + 4, "flops": 34 * px}
    if kind in ("detect", "batch"):
        px = sum(w * h for w, h, _ in _sizes(case)) if kind == "batch" else case["w"] * case["h"]
        return {"bytes": px + case["markers"] * MARKER.itemsize, "flops": 34 * px * 85 // 64}
    n, cuts, samples = case["n"], case["cuts"], case["samples"]
    one = n * cuts * samples
    if kind == "cost":
        return {"bytes": 4 * one + n * (TASK.itemsize + 14 * 4), "flops": 99 * one}
    # the grid: 25 trial centers in each of about ten rounds; Gauss-Newton: 9 trials, then about 7 evaluations
    flops = 25 * 10 * 33 * one if case["mode"] == "grid" else (9 * 33 + 7 * 99) * one
    return {"bytes": 4 * one + n * (TASK.itemsize + RESULT.itemsize), "flops": flops}


# ---------------------------------------------------------------------- exact --
def _canonic(Q):
    """Rotation and center of the conics Q [n, 3, 3]: the canonical conic's diagonal, the map to its axes and
    back (the fit's own axis convention, which fixes the homography's axes)."""
    th = 0.5 * torch.atan2(2 * Q[:, 0, 1], Q[:, 0, 0] - Q[:, 1, 1])
    c, s = torch.cos(th), torch.sin(th)
    center = -torch.linalg.solve(Q[:, :2, :2], Q[:, :2, 2:])[..., 0]
    z, o = torch.zeros_like(c), torch.ones_like(c)
    Td = torch.stack([c, -s, center[:, 0], s, c, center[:, 1], z, z, o], -1).reshape(-1, 3, 3)
    D = torch.diagonal(Td.transpose(1, 2) @ Q @ Td, dim1=1, dim2=2)
    return D, torch.linalg.inv(Td), Td


def _homography(canonic, p):
    """Plane -> image homographies sending the unit circle to the conic and the origin to p [n, t, 2]."""
    D, Tp, Td = canonic
    a, b, k = (D[:, i, None] for i in range(3))
    x = (Tp[:, None, 0, 0] * p[..., 0] + Tp[:, None, 0, 1] * p[..., 1] + Tp[:, None, 0, 2])
    y = (Tp[:, None, 1, 0] * p[..., 0] + Tp[:, None, 1, 1] * p[..., 1] + Tp[:, None, 1, 2])
    d0, d1, d2 = torch.sqrt(b * k / a * (a * x * x + b * y * y + k)), k.expand_as(x), torch.sqrt(-b * (a * x * x + k))
    one = torch.ones_like(x)
    h = torch.stack([k * one * d0, b * x * y * d1, -k * x * d2, 0 * one, (-a * x * x - k) * d1, -k * y * d2,
                     -a * x * d0, b * y * d1, -k * one * d2], -1).reshape(*x.shape, 3, 3)
    return Td[:, None] @ h


def _signals(image, roi, H, stop, samples):
    """Bilinear samples (halved) along the cuts: H [n, t, 3, 3], stop [n, c, 2] -> [n, t, c, samples]."""
    one = torch.ones_like(stop[..., :1])
    z = torch.einsum("ntij,ncj->ntci", torch.linalg.inv(H), torch.cat([stop, one], -1))
    end = z[..., :2] / z[..., 2:]
    f = BEGIN + (1 - BEGIN) * torch.arange(samples, device=H.device, dtype=torch.float64) / (samples - 1)
    x, y = end[..., 0, None] * f, end[..., 1, None] * f
    h = [H[..., i // 3, i % 3][..., None, None] for i in range(9)]
    w = h[6] * x + h[7] * y + h[8]
    x, y = (h[0] * x + h[1] * y + h[2]) / w, (h[3] * x + h[4] * y + h[5]) / w
    shape = (-1, 1, 1, 1)
    ix = torch.minimum(x.detach().floor().long().clamp_min(0), roi[:, 2].reshape(shape) - 2)
    iy = torch.minimum(y.detach().floor().long().clamp_min(0), roi[:, 3].reshape(shape) - 2)
    fx, fy = x - ix, y - iy
    at = (iy + roi[:, 1].reshape(shape)) * image.shape[1] + ix + roi[:, 0].reshape(shape)
    px = image.reshape(-1)
    p0, p1, p2, p3 = (px[at + d].double() for d in (0, 1, image.shape[1], image.shape[1] + 1))
    return 0.5 * ((p0 * (1 - fx) + p1 * fx) * (1 - fy) + (p2 * (1 - fx) + p3 * fx) * fy)


def _cost(s):
    """Mean over the pairs of cuts of their squared distance: s [..., c, samples]."""
    c = s.shape[-2]
    d = s - s.mean(-2, keepdim=True)
    return 2.0 / (c - 1) * (d * d).sum((-1, -2))


def exact(case, seed):
    """Candidates' costs, gradients and grid-refined centers in 64 bits.  Detections and edges return decisions
    and rounded integers, and Gauss-Newton stops wherever its step falls below its threshold: no such value."""
    if case["kind"] == "cost" or (case["kind"] == "refine" and case["mode"] == "grid"):
        image, tasks, centers = _candidates(case, seed)
    else:
        return None
    parts = [_exact_some(case, image, tasks[i:i + 64], centers[i:i + 64]) for i in range(0, len(tasks), 64)]
    return {k: None if parts[0][k] is None else torch.cat([p[k] for p in parts]) for k in parts[0]}


def _exact_some(case, image, t, centers):
    def up(a, kind=torch.float64):
        return torch.from_numpy(np.array(a)).to("cuda", kind)

    n, cuts, samples = len(t), case["cuts"], case["samples"]
    roi, stop, Q = up(t["roi"], torch.int64), up(t["stop"][:, :cuts]), up(t["Q"]).reshape(n, 3, 3)
    if not case["local"]:  # to the crop's own coordinates
        off = roi[:, :2].double()
        T = torch.eye(3, device="cuda", dtype=torch.float64).repeat(n, 1, 1)
        T[:, 0, 2], T[:, 1, 2] = off[:, 0], off[:, 1]
        Q, stop = T.transpose(1, 2) @ Q @ T, stop - off[:, None]
    else:
        off = torch.zeros(n, 2, device="cuda", dtype=torch.float64)
    if case["kind"] == "cost":
        p = (up(centers) - off).requires_grad_()
        # in the caller's coordinates, which the gradient in H is asked in
        T = torch.eye(3, device="cuda", dtype=torch.float64).repeat(n, 1, 1)
        T[:, 0, 2], T[:, 1, 2] = off[:, 0], off[:, 1]
        H = T @ _homography(_canonic(Q), p[:, None])[:, 0]
        cost = _cost(_signals(image, roi, (torch.linalg.inv(T) @ H)[:, None], stop, samples))[:, 0]
        d_center, d_h = torch.autograd.grad(cost.sum(), [p, H])
        return {"cost": cost.detach(), "d_center": d_center, "d_h": d_h.reshape(n, 9)}
    canonic = _canonic(Q)
    center = up(np.stack([t["x0"], t["y0"]], -1)) - off
    size = torch.maximum(up(t["a"]), up(t["b"])) * 0.2
    g = torch.arange(5, device="cuda", dtype=torch.float64) / 4 - 0.5
    grid = torch.stack([g.repeat_interleave(5), g.repeat(5)], -1)
    best = torch.zeros(n, device="cuda", dtype=torch.float64)
    while True:
        go = size > 0.02
        if not go.any():
            break
        trial = center[:, None] + size[:, None, None] * grid
        cost = torch.cat([_cost(_signals(image, roi, _homography(canonic, q), stop, samples))
                          for q in trial.split(5, 1)], 1)
        low, at = cost.min(1)
        best = torch.where(go, low, best)
        center = torch.where(go[:, None], trial[torch.arange(n, device="cuda"), at], center)
        size = torch.where(go, size / 2, size)
    H = _homography(canonic, center[:, None])
    s = _signals(image, roi, H, stop, samples)[:, 0].sort(1).values
    bar = 0.5 * (s[:, (cuts - 1) // 2] + s[:, cuts // 2])
    residual = torch.sqrt(best) / (bar.max(1).values - bar.min(1).values)
    T = torch.eye(3, device="cuda", dtype=torch.float64).repeat(n, 1, 1)
    T[:, 0, 2], T[:, 1, 2] = off[:, 0], off[:, 1]
    return {"status": None, "id": None, "center": center + off, "H": (T @ H[:, 0]).reshape(n, 9), "residual": residual,
            "score": None, "nvalid": None, "iterations": None}
