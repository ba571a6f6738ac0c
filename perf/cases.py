"""Workloads for timing the framework through its public entry points.

Two families, as a program meets them:

* OpenVX graphs: the program creates images over its own device memory (a decoder's or a
  network's buffers; one case works from page-locked host memory, as a camera loop does),
  builds and verifies a graph once, and calls vxProcessGraph per batch of frames, then reads
  the arrays and distributions on the host.  Image outputs stay in the program's buffers.
* Differentiable warps on torch tensors: a registration step (warp + L2 loss + gradients in one
  call) and the autograd functions, forward and backward.

`listed()` has the fixed cases, `draw(rng)` gives more of the same ranges.  `prepare` makes the
inputs from a seed and builds the graph, `run` is one pass, `work` the bytes and operations that
a pass cannot do without, `exact` the float results in 64 bits.
"""
from __future__ import annotations

import ctypes as C
import math
import random

import numpy as np
import torch

from mivisionx_b200 import diffwarp
from mivisionx_b200 import vx as V

VGA, HD, FHD, UHD = (640, 480), (1280, 720), (1920, 1080), (3840, 2160)


# ---------------------------------------------------------------- the cases
def listed():
    return [
        # one small frame through the edge-mask chain: what a call costs when the work is tiny
        dict(name="chain_vga_1", kind="chain", w=640, h=480, n=1, shift=0, thr=128),
        # the same chain over a batch of video frames
        dict(name="chain_1080p_64", kind="chain", w=1920, h=1080, n=64, shift=0, thr=128),
        # a camera loop: one 720p frame from page-locked host memory, edges back to the host, corners
        dict(name="features_camera_720p", kind="features", w=1280, h=720, n=1, host=True, gradient=3, l2=False, block=3),
        # offline feature extraction: edges and corners of a batch of 4K frames
        dict(name="features_4k_16", kind="features", w=3840, h=2160, n=16, host=False, gradient=3, l2=False, block=3),
        # wider windows, as noisy footage needs them, at an odd size
        dict(name="features_wide_1917x1077_4", kind="features", w=1917, h=1077, n=4, host=False, gradient=5, l2=True, block=5),
        # one pair of a tracker that follows 1000 points
        dict(name="flow_720p_1", kind="flow", w=1280, h=720, n=1, uneven=False, levels=5, window=9, points=1000),
        # many streams of different sizes, 2000 points each, in one graph
        dict(name="flow_uneven_64", kind="flow", w=3840, h=2160, n=64, uneven=True, levels=5, window=9, points=2000),
        # encoder front end: RGB frames to NV12 and IYUV, half-size previews, stabilised by a warp
        dict(name="colour_4k_8", kind="colour", w=3840, h=2160, n=8),
        # motion masks of consecutive surveillance frames
        dict(name="motion_4k_16", kind="motion", w=3840, h=2160, n=16, thr=24),
        # image registration: one optimiser step's loss and gradients for a batch
        dict(name="align_affine_1024_32", kind="align", w=1024, h=1024, n=32, warp="affine"),
        # a learned warp inside a torch model: forward and backward, at an odd size
        dict(name="warpgrad_field_511x767_6", kind="warpgrad", w=511, h=767, n=6, warp="field"),
        # lens correction followed by the usual measurements of the corrected frames
        dict(name="measure_1080p_4", kind="measure", w=1920, h=1080, n=4, taps=5),
    ]


def _log(rng: random.Random, lo: float, hi: float) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _size(rng, n_most, px_most, even=False, lo=(200, 150), hi=(3840, 2160)):
    """(w, h, n): a frame size over the whole range, odd ones among them, and a batch of such
    frames with at most `px_most` pixels in all."""
    w, h = _log(rng, lo[0], hi[0]), _log(rng, lo[1], hi[1])
    if even:
        w, h = w & ~1, h & ~1
    return w, h, max(1, min(_log(rng, 1, n_most), int(px_most // (w * h))))


def draw(rng: random.Random):
    kind = rng.choice(["chain", "features", "flow", "colour", "motion", "align", "warpgrad", "measure"])
    mp = 1e6
    if kind == "chain":
        w, h, n = _size(rng, 64, 130 * mp)
        return dict(kind=kind, w=w, h=h, n=n, shift=rng.choice([0, 0, 1]), thr=rng.randint(40, 200))
    if kind == "features":
        gradient = rng.choice([3, 3, 3, 5, 7])
        w, h, n = _size(rng, 16, 130 * mp if gradient == 3 else 8 * mp)
        host = n <= 2 and rng.random() < 0.5
        return dict(kind=kind, w=w, h=h, n=n, host=host, gradient=gradient, l2=rng.random() < 0.5,
                    block=3 if gradient == 3 else rng.choice([3, 5]))
    if kind == "flow":
        w, h, n = _size(rng, 32, 60 * mp, lo=(320, 240))
        return dict(kind=kind, w=w, h=h, n=n, uneven=rng.random() < 0.5, levels=rng.choice([3, 4, 5]),
                    window=rng.choice([5, 7, 9, 9]), points=_log(rng, 100, 2000))
    if kind == "colour":
        w, h, n = _size(rng, 8, 66 * mp, even=True)
        return dict(kind=kind, w=w, h=h, n=n)
    if kind == "motion":
        w, h, n = _size(rng, 16, 130 * mp)
        return dict(kind=kind, w=w, h=h, n=n, thr=rng.randint(12, 40))
    if kind == "measure":
        w, h, n = _size(rng, 4, 8 * mp)
        return dict(kind=kind, w=w, h=h, n=n, taps=rng.choice([3, 5, 7]))
    w, h, n = _size(rng, 32, 32 * mp, lo=(64, 64), hi=(1600, 1600))
    if kind == "align":
        return dict(kind=kind, w=w, h=h, n=n, warp=rng.choice(["affine", "perspective"]))
    return dict(kind=kind, w=w, h=h, n=n, warp=rng.choice(["field", "affine", "perspective"]))


# ---------------------------------------------------------------- inputs, made on the GPU
def _gen(seed: int) -> torch.Generator:
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _u8(t: torch.Tensor) -> torch.Tensor:
    return t.round_().clamp_(0, 255).to(torch.uint8)


def _scene(rng, gen, w, h, sigma=8.0, top=200.0) -> torch.Tensor:
    """Float scene: a horizontal gradient, rectangles of 16 to 400 px, Gaussian noise."""
    img = torch.linspace(0.0, top, w, device="cuda").repeat(h, 1)
    for _ in range(max(8, round(200 * w * h / (3840 * 2160)))):
        rw, rh = rng.randint(16, 400), rng.randint(16, 400)
        x, y = rng.randrange(max(1, w - rw)), rng.randrange(max(1, h - rh))
        img[y:y + rh, x:x + rw] = float(rng.randrange(256))
    return img.add_(torch.randn(h, w, device="cuda", generator=gen), alpha=sigma)


def _shifted(img: torch.Tensor, dx: float, dy: float) -> torch.Tensor:
    """img translated by (dx, dy), bilinear, edges clamped."""
    h, w = img.shape
    xs = (torch.arange(w, device="cuda", dtype=torch.float32) - dx).clamp_(0, w - 1)
    ys = (torch.arange(h, device="cuda", dtype=torch.float32) - dy).clamp_(0, h - 1)
    x0, y0 = xs.floor().long().clamp_(max=w - 2), ys.floor().long().clamp_(max=h - 2)
    fx, fy = xs - x0, (ys - y0)[:, None]
    top, bot = img[y0], img[y0 + 1]
    r = lambda a: a[:, x0] * (1 - fx) + a[:, x0 + 1] * fx
    return r(top) * (1 - fy) + r(bot) * fy


def _motion_pair(rng, gen, w, h):
    a = torch.linspace(0.0, 160.0, w, device="cuda").repeat(h, 1)
    b = a.clone()
    for _ in range(max(6, round(150 * w * h / (3840 * 2160)))):
        rw, rh, level = rng.randint(16, 256), rng.randint(16, 256), float(rng.randrange(256))
        x, y = rng.randrange(max(1, w - rw)), rng.randrange(max(1, h - rh))
        a[y:y + rh, x:x + rw] = level
        x, y = max(0, x + rng.randint(-12, 12)), max(0, y + rng.randint(-12, 12))
        b[y:y + rh, x:x + rw] = level
    return [_u8(t.add_(torch.randn(h, w, device="cuda", generator=gen), alpha=3.0)) for t in (a, b)]


def _rgb(rng, gen, w, h):
    """(h, w, 3): per channel a sum of 8 random 2-D sinusoids plus uniform noise of 10 levels."""
    xs, ys = (torch.arange(k, device="cuda", dtype=torch.float32) for k in (w, h))
    out = torch.empty(h, w, 3, dtype=torch.uint8, device="cuda")
    for ch in range(3):
        acc = torch.zeros(h, w, device="cuda")
        for _ in range(8):
            fx, fy, ph, amp = (rng.random() - 0.5) * 0.02, (rng.random() - 0.5) * 0.02, rng.random() * 2 * math.pi, 0.5 + rng.random()
            acc += amp * torch.sin((fx * xs)[None, :] + (fy * ys + ph)[:, None])
        acc = (acc - acc.min()) / (acc.max() - acc.min()) * 255.0
        out[..., ch] = _u8(acc + torch.rand(h, w, device="cuda", generator=gen) * 20.0 - 10.0)
    return out


def _smooth(gen, n, h, w):
    """(n, h, w) float32 in [0, 1): uniform noise smoothed by a Gaussian of sigma 2."""
    k = torch.exp(-0.5 * (torch.arange(-8, 9, device="cuda", dtype=torch.float32) / 2.0) ** 2)
    k = k / k.sum()
    u = torch.nn.functional.pad(torch.rand(n, 1, h, w, device="cuda", generator=gen), (8, 8, 8, 8), mode="reflect")
    v = sum(k[j] * u[..., j:j + w] for j in range(17))
    return sum(k[j] * v[..., j:j + h, :] for j in range(17))[:, 0].contiguous()


# ---------------------------------------------------------------- OpenVX graphs
_api = None


def _vx() -> V.OpenVX:
    global _api
    if _api is None:
        _api = V.OpenVX()
    return _api


class _Planes:
    """n planes of (h, w * bpp) bytes in one buffer of the program, laid out as the framework
    takes device memory: bases aligned to 256 bytes, row pitches to 64."""

    def __init__(self, n, w, h, bpp=1, host=False):
        self.w, self.h, self.bpp = w, h, bpp
        self.pitch = -(-w * bpp // 64) * 64
        self.host = host
        rows = -(-h // 4) * 4
        self.t = torch.zeros(n, rows, self.pitch, dtype=torch.uint8, **({"pin_memory": True} if host else {"device": "cuda"}))

    def view(self, i=None, rect=None, dtype=None):
        """The pixels of plane i (of all planes), or of its rectangle."""
        t = self.t if dtype is None else self.t.view(dtype)
        k = self.bpp if dtype is None else 1
        x0, y0, x1, y1 = rect or (0, 0, self.w, self.h)
        t = t[:, y0:y1, x0 * k:x1 * k]
        return t if i is None else t[i]


class _State:
    """A verified graph, its buffers, and what one pass gives back."""

    def __init__(self):
        self.api = _vx()
        self.ctx = self.api.obj(self.api.vxCreateContext(), "context")
        self.graph = self.api.obj(self.api.vxCreateGraph(self.ctx), "graph")
        self.images, self.arrays, self.hists, self.keep = [], [], [], []

    def image(self, planes, i, fmt, w, h):
        """Image i over the program's buffers `planes` (one per plane of the format)."""
        addrs = (V.vx_imagepatch_addressing_t * len(planes))()
        for a, p in zip(addrs, planes):
            a.dim_x, a.dim_y, a.stride_x, a.stride_y = p.w, p.h, p.bpp, p.pitch
            a.scale_x = a.scale_y = 1024
            a.step_x = a.step_y = 1
        addrs[0].dim_x, addrs[0].dim_y = w, h
        ptrs = (C.c_void_p * len(planes))(*[p.t[i].data_ptr() for p in planes])
        kind = V.VX_MEMORY_TYPE_HOST if planes[0].host else V.VX_MEMORY_TYPE_HIP
        self.keep += planes
        return self.api.obj(self.api.vxCreateImageFromHandle(self.ctx, fmt, addrs, ptrs, kind), "image")

    def u8(self, planes, i):
        return self.image([planes], i, V.VX_DF_IMAGE_U8, planes.w, planes.h)

    def virtual(self, w, h, fmt=V.VX_DF_IMAGE_U8):
        return self.api.vxCreateVirtualImage(self.graph, w, h, fmt)

    def node(self, n):
        return self.api.obj(n, "node")

    def corners(self, capacity):
        arr = self.api.obj(self.api.vxCreateArray(self.ctx, V.VX_TYPE_KEYPOINT, capacity), "array")
        self.arrays.append(arr)
        self.capacity = capacity
        return arr

    def verify(self):
        self.api.ok(self.api.vxVerifyGraph(self.graph), "vxVerifyGraph")
        if self.arrays:     # the program's lists: as many keypoints as were found, zeros after them
            self.points = np.zeros((len(self.arrays), self.capacity, 7), np.int32)
            self.found = np.zeros(len(self.arrays), np.int64)

    def gives(self, planes, image, dtype=None):
        """`planes` come back, inside the rectangle that the framework declares valid."""
        r = self.api.valid_region(image)
        v = planes.view(rect=r, dtype=dtype)
        self.images.append(v.numpy() if planes.host else v)

    def run(self):
        a = self.api
        a.ok(a.vxProcessGraph(self.graph), "vxProcessGraph")
        out = list(self.images)
        for i, k in enumerate(self.arrays):
            n = C.c_size_t(0)
            a.ok(a.vxQueryArray(k, V.VX_ARRAY_NUMITEMS, C.byref(n), C.sizeof(n)), "vxQueryArray")
            n, at = n.value, self.points[i]
            if n:
                a.ok(a.vxCopyArrayRange(k, 0, n, 28, at.ctypes.data, V.VX_READ_ONLY, V.VX_MEMORY_TYPE_HOST), "vxCopyArrayRange")
            at[n:self.found[i]] = 0
            self.found[i] = n
        if self.arrays:
            out += [self.points, self.found]
        for d in self.hists:
            h = np.zeros(256, np.int32)
            a.ok(a.vxCopyDistribution(d, h.ctypes.data, V.VX_READ_ONLY, V.VX_MEMORY_TYPE_HOST), "vxCopyDistribution")
            out.append(h)
        return out

    def __del__(self):
        if getattr(self, "ctx", None):
            self.api.vxReleaseContext(C.byref(C.c_void_p(self.ctx)))
            self.ctx = None


def _chain(s, c, rng, gen):
    a, w, h, n = s.api, c["w"], c["h"], c["n"]
    src, dst = _Planes(n, w, h), _Planes(n, w, h)
    src.view().copy_(torch.randint(0, 256, (n, h, w), dtype=torch.uint8, device="cuda", generator=gen))
    shift, thr = a.scalar(s.ctx, V.VX_TYPE_INT32, c["shift"]), a.threshold_binary(s.ctx, c["thr"])
    for i in range(n):
        v = [s.virtual(w, h, f) for f in (V.VX_DF_IMAGE_U8, V.VX_DF_IMAGE_S16, V.VX_DF_IMAGE_S16, V.VX_DF_IMAGE_S16, V.VX_DF_IMAGE_U8)]
        out = s.u8(dst, i)
        s.node(a.vxGaussian3x3Node(s.graph, s.u8(src, i), v[0]))
        s.node(a.vxSobel3x3Node(s.graph, v[0], v[1], v[2]))
        s.node(a.vxMagnitudeNode(s.graph, v[1], v[2], v[3]))
        s.node(a.vxConvertDepthNode(s.graph, v[3], v[4], V.VX_CONVERT_POLICY_SATURATE, shift))
        s.node(a.vxThresholdNode(s.graph, v[4], thr, out))
    s.verify()
    s.gives(dst, out)


def _features(s, c, rng, gen):
    a, w, h, n = s.api, c["w"], c["h"], c["n"]
    src, dst = _Planes(n, w, h, host=c["host"]), _Planes(n, w, h, host=c["host"])
    hyst = a.threshold_range(s.ctx, 80, 100)
    strength, dist, k = (a.scalar(s.ctx, V.VX_TYPE_FLOAT32, f) for f in (1e-3, 5.0, 0.04))
    norm = V.VX_NORM_L2 if c["l2"] else V.VX_NORM_L1
    for i in range(n):
        src.view(i).copy_(_u8(_scene(rng, gen, w, h)))
        img, edge = s.u8(src, i), s.u8(dst, i)
        s.node(a.vxCannyEdgeDetectorNode(s.graph, img, hyst, c["gradient"], norm, edge))
        s.node(a.vxHarrisCornersNode(s.graph, img, strength, dist, k, c["gradient"], c["block"],
                                     s.corners(max(1024, w * h // 256)), a.scalar(s.ctx, V.VX_TYPE_SIZE, 0)))
    s.verify()
    s.gives(dst, edge)


def _flow(s, c, rng, gen):
    a = s.api
    eps, its, est = (a.scalar(s.ctx, t, v) for t, v in ((V.VX_TYPE_FLOAT32, 0.01), (V.VX_TYPE_UINT32, 20), (V.VX_TYPE_BOOL, 0)))
    for w, h in _flow_sizes(c):
        p = _Planes(2, w, h)
        first = _scene(rng, gen, w, h)
        moved = _shifted(_u8(first.clone()).float(), rng.uniform(-8, 8), rng.uniform(-8, 8))
        p.view(0).copy_(_u8(first))
        p.view(1).copy_(_u8(moved.add_(torch.randn(h, w, device="cuda", generator=gen), alpha=2.0)))
        pyr = [a.obj(a.vxCreateVirtualPyramid(s.graph, c["levels"], V.VX_SCALE_PYRAMID_HALF, w, h, V.VX_DF_IMAGE_U8)) for _ in range(2)]
        kp = np.zeros(c["points"], V.KEYPOINT_DTYPE)
        kp["x"] = [rng.randrange(w) for _ in range(c["points"])]
        kp["y"] = [rng.randrange(h) for _ in range(c["points"])]
        kp["tracking_status"] = 1
        old = a.obj(a.vxCreateArray(s.ctx, V.VX_TYPE_KEYPOINT, c["points"]))
        a.array_set(old, kp)
        for i in range(2):
            s.node(a.vxGaussianPyramidNode(s.graph, s.u8(p, i), pyr[i]))
        s.node(a.vxOpticalFlowPyrLKNode(s.graph, pyr[0], pyr[1], old, old, s.corners(c["points"]), V.VX_TERM_CRITERIA_BOTH,
                                        eps, its, est, c["window"]))
    s.verify()


def _flow_sizes(c):
    """The sizes of a flow case's pairs: all alike, or a fixed mix of video sizes up to the
    case's own, the same for every seed."""
    if not c["uneven"]:
        return [(c["w"], c["h"])] * c["n"]
    rng = random.Random(4)
    some = [(c["w"], c["h"])] + [k for k in (VGA, HD, FHD) if k[0] * k[1] < c["w"] * c["h"]]
    return [rng.choice(some) for _ in range(c["n"])]


def _colour(s, c, rng, gen):
    a, w, h, n = s.api, c["w"], c["h"], c["n"]
    rgb = _Planes(n, w, h, 3)
    nv12 = [_Planes(n, w, h), _Planes(n, w // 2, h // 2, 2)]
    iyuv = [_Planes(n, w, h), _Planes(n, w // 2, h // 2), _Planes(n, w // 2, h // 2)]
    half = [_Planes(n, w // 2, h // 2) for _ in range(4)]
    for i in range(n):
        rgb.view(i).copy_(_rgb(rng, gen, w, h).view(h, w * 3))
        src = s.image([rgb], i, V.VX_DF_IMAGE_RGB, w, h)
        o_nv12, o_iyuv = s.image(nv12, i, V.VX_DF_IMAGE_NV12, w, h), s.image(iyuv, i, V.VX_DF_IMAGE_IYUV, w, h)
        small = [s.u8(p, i) for p in half]
        y = s.virtual(w, h)
        th, sc = math.radians(rng.uniform(-15, 15)), rng.uniform(0.8, 1.2)
        p, q, cx, cy = sc * math.cos(th), sc * math.sin(th), w / 4, h / 4
        m = a.matrix_f32(s.ctx, np.array([[p, q], [-q, p], [cx - p * cx + q * cy + rng.uniform(-50, 50),
                                                           cy - q * cx - p * cy + rng.uniform(-50, 50)]], np.float32))
        s.node(a.vxColorConvertNode(s.graph, src, o_nv12))
        s.node(a.vxColorConvertNode(s.graph, src, o_iyuv))
        s.node(a.vxChannelExtractNode(s.graph, o_nv12, V.VX_CHANNEL_Y, y))
        s.node(a.vxScaleImageNode(s.graph, y, small[0], V.VX_INTERPOLATION_BILINEAR))
        s.node(a.vxScaleImageNode(s.graph, y, small[1], V.VX_INTERPOLATION_AREA))
        for k, mode in ((2, V.VX_INTERPOLATION_NEAREST_NEIGHBOR), (3, V.VX_INTERPOLATION_BILINEAR)):
            nd = s.node(a.vxWarpAffineNode(s.graph, small[0], m, mode, small[k]))
            a.set_border(nd, V.VX_BORDER_CONSTANT, 0)
    s.verify()
    s.images += [p.view() for p in nv12 + iyuv + half]


def _motion(s, c, rng, gen):
    a, w, h, n = s.api, c["w"], c["h"], c["n"]
    prev, cur, dst = (_Planes(n, w, h) for _ in range(3))
    thr = a.threshold_binary(s.ctx, c["thr"])
    for i in range(n):
        for p, t in zip((prev, cur), _motion_pair(rng, gen, w, h)):
            p.view(i).copy_(t)
        v, out = [s.virtual(w, h) for _ in range(5)], s.u8(dst, i)
        s.node(a.vxAbsDiffNode(s.graph, s.u8(cur, i), s.u8(prev, i), v[0]))
        s.node(a.vxGaussian3x3Node(s.graph, v[0], v[1]))
        s.node(a.vxThresholdNode(s.graph, v[1], thr, v[2]))
        s.node(a.vxDilate3x3Node(s.graph, v[2], v[3]))
        s.node(a.vxErode3x3Node(s.graph, v[3], v[4]))
        s.node(a.vxMedian3x3Node(s.graph, v[4], out))
    s.verify()
    s.gives(dst, out)


def _measure(s, c, rng, gen):
    """Lens correction by a remap table, then of each corrected frame: a custom convolution to
    16 bits, corners by FAST, a histogram, an integral image."""
    a, w, h, n = s.api, c["w"], c["h"], c["n"]
    src, flat, conv, integral = _Planes(n, w, h), _Planes(n, w, h), _Planes(n, w, h, 2), _Planes(n, w, h, 4)
    ys, xs = torch.meshgrid(torch.arange(h, dtype=torch.float32), torch.arange(w, dtype=torch.float32), indexing="ij")
    u, v = (xs - w / 2) / w, (ys - h / 2) / w
    k = 1.0 + rng.uniform(0.02, 0.08) * (u * u + v * v)
    table = torch.stack([u * k * w + w / 2, v * k * w + h / 2], -1).contiguous()
    remap = a.obj(a.vxCreateRemap(s.ctx, w, h, w, h), "remap")
    rect = V.vx_rectangle_t(0, 0, w, h)
    a.ok(a.vxCopyRemapPatch(remap, C.byref(rect), w * 8, table.data_ptr(), V.VX_TYPE_COORDINATES2DF, V.VX_WRITE_ONLY,
                            V.VX_MEMORY_TYPE_HOST), "vxCopyRemapPatch")
    taps = np.array([[rng.randint(-8, 8) for _ in range(c["taps"])] for _ in range(c["taps"])], np.int16)
    cv = a.convolution(s.ctx, taps, 16)
    thr = a.scalar(s.ctx, V.VX_TYPE_FLOAT32, 20.0)
    for i in range(n):
        src.view(i).copy_(_u8(_scene(rng, gen, w, h)))
        f = s.u8(flat, i)
        nd = s.node(a.vxRemapNode(s.graph, s.u8(src, i), remap, V.VX_INTERPOLATION_BILINEAR, f))
        a.set_border(nd, V.VX_BORDER_CONSTANT, 0)
        o_conv = s.image([conv], i, V.VX_DF_IMAGE_S16, w, h)
        s.node(a.vxConvolveNode(s.graph, f, cv, o_conv))
        s.node(a.vxFastCornersNode(s.graph, f, thr, 1, s.corners(max(1024, w * h // 64)), a.scalar(s.ctx, V.VX_TYPE_SIZE, 0)))
        d = a.obj(a.vxCreateDistribution(s.ctx, 256, 0, 256), "distribution")
        s.node(a.vxHistogramNode(s.graph, f, d))
        s.hists.append(d)
        o_int = s.image([integral], i, V.VX_DF_IMAGE_U32, w, h)
        s.node(a.vxIntegralImageNode(s.graph, f, o_int))
    s.verify()
    s.gives(flat, f)
    s.gives(conv, o_conv, dtype=torch.int16)
    s.gives(integral, o_int, dtype=torch.int32)


_GRAPHS = {"chain": _chain, "features": _features, "flow": _flow, "colour": _colour, "motion": _motion, "measure": _measure}


# ---------------------------------------------------------------- differentiable warps
def _theta(rng, w, h, warp, spread=1.0):
    """Map output -> source: rotation within 10 degrees, scale 0.9 to 1.1, shift within 20 px
    about the centre (and a slight tilt), times `spread`."""
    cx, cy = (w - 1) / 2, (h - 1) / 2
    th, sc = math.radians(rng.uniform(-10, 10) * spread), 1.0 + rng.uniform(-0.1, 0.1) * spread
    a, d = sc * math.cos(th), sc * math.sin(th)
    x, y = cx - a * cx + d * cy + rng.uniform(-20, 20) * spread, cy - d * cx - a * cy + rng.uniform(-20, 20) * spread
    if warp == "affine":
        return [a, d, -d, a, x, y]
    g, k = rng.uniform(-0.05, 0.05) / w, rng.uniform(-0.05, 0.05) / h
    return [a, d, g, -d, a, k, x, y, 1.0 - g * cx - k * cy]


def _warp_inputs(c, seed):
    rng, gen = random.Random(seed), _gen(seed)
    n, w, h = c["n"], c["w"], c["h"]
    src = _smooth(gen, n, h, w)
    if c["warp"] == "field":       # a smooth displacement of up to 4 px
        ys, xs = torch.meshgrid(torch.arange(h, device="cuda") / h, torch.arange(w, device="cuda") / w, indexing="ij")
        f = [rng.random() for _ in range(8 * n)]
        p = torch.stack([torch.stack([torch.sin(6.28 * (3 * f[8 * i] * xs + f[8 * i + 1])) * torch.cos(6.28 * (3 * f[8 * i + 2] * ys + f[8 * i + 3])),
                                      torch.cos(6.28 * (3 * f[8 * i + 4] * xs + f[8 * i + 5])) * torch.sin(6.28 * (3 * f[8 * i + 6] * ys + f[8 * i + 7]))], -1)
                         for i in range(n)]).mul_(4.0).contiguous()
    else:
        p = torch.tensor([_theta(rng, w, h, c["warp"]) for _ in range(n)], dtype=torch.float32, device="cuda")
    return src, p, rng, gen


_WARP = {"affine": diffwarp.warp_affine, "perspective": diffwarp.warp_perspective, "field": diffwarp.remap}
_STEP = {"affine": diffwarp.warp_affine_l2_step, "perspective": diffwarp.warp_perspective_l2_step}


def _align_inputs(c, seed):
    """Images, the estimate, and the target: the images seen through a map near the estimate."""
    src, theta, rng, gen = _warp_inputs(c, seed)
    near = torch.tensor([_theta(rng, c["w"], c["h"], c["warp"], spread=0.15) for _ in range(c["n"])], device="cuda")
    base = torch.tensor(_theta(random.Random(0), c["w"], c["h"], c["warp"], spread=0.0), device="cuda")
    goal = theta + (near - base)
    target = torch.stack([_sample64(src[i].double(), *_positions64(goal[i].double(), c))["value"].float() for i in range(c["n"])])
    return src, theta, target


def _grad_inputs(c, seed):
    src, p, _, gen = _warp_inputs(c, seed)
    gout = torch.randn(src.shape, device="cuda", generator=gen)
    return src.requires_grad_(), p.requires_grad_(), gout


# ---------------------------------------------------------------- entry points
def prepare(case, seed):
    if case["kind"] == "align":
        return ("align", _STEP[case["warp"]], _align_inputs(case, seed))
    if case["kind"] == "warpgrad":
        return ("warpgrad", _WARP[case["warp"]], _grad_inputs(case, seed))
    s = _State()
    _GRAPHS[case["kind"]](s, case, random.Random(seed), _gen(seed))
    torch.cuda.synchronize()
    return s


def run(state):
    if isinstance(state, _State):
        return state.run()
    kind, f, (src, p, other) = state
    if kind == "align":
        loss, gsrc, gtheta = f(src, p, other)
        return {"loss": loss, "gsrc": gsrc, "gtheta": gtheta}
    out = f(src, p)
    gsrc, gp = torch.autograd.grad(out, (src, p), other)
    return {"out": out, "gsrc": gsrc, "gp": gp}


def work(case):
    """Inputs read once, outputs written once; operations per pixel of the arithmetic itself."""
    w, h, n, kind = case["w"], case["h"], case["n"], case["kind"]
    px = w * h * n
    if kind == "chain":          # U8 in, U8 out; 3x3 smoothing, two gradients, magnitude
        return {"bytes": 2 * px, "flops": 35 * px}
    if kind == "features":       # U8 in, U8 edges out, up to w h / 256 corners of 28 bytes
        return {"bytes": 2 * px + 28 * px // 256, "flops": (30 + 25 * case["block"]) * px}
    if kind == "flow":           # both frames in, the points in and out
        px = 2 * sum(a * b for a, b in _flow_sizes(case))
        pts = n * case["points"]
        return {"bytes": px + 2 * 28 * pts, "flops": 20 * px // 3 + pts * case["levels"] * 6 * 20 * case["window"] ** 2}
    if kind == "colour":         # RGB in; NV12, IYUV and four half-size planes out
        return {"bytes": 7 * px, "flops": 30 * px}
    if kind == "motion":         # two frames in, one mask out
        return {"bytes": 3 * px, "flops": 60 * px}
    if kind == "measure":        # U8 and the table in; U8, S16 and U32 out
        return {"bytes": 8 * px + 8 * w * h, "flops": (2 * case["taps"] ** 2 + 40) * px}
    if kind == "align":          # source and target in, source gradient out
        return {"bytes": 12 * px, "flops": 60 * px}
    # out, gradient of out, source (forward and backward), source gradient; the field's both
    return {"bytes": (20 + (24 if case["warp"] == "field" else 0)) * px, "flops": 70 * px}


# ---------------------------------------------------------------- 64-bit results of the warps
def _positions64(p, c):
    """Source position of every output pixel, and z of a perspective map."""
    h, w = c["h"], c["w"]
    y, x = torch.meshgrid(torch.arange(h, device="cuda", dtype=torch.float64), torch.arange(w, device="cuda", dtype=torch.float64), indexing="ij")
    if c["warp"] == "field":
        return x + p[..., 0], y + p[..., 1]
    if c["warp"] == "affine":
        return p[0] * x + p[2] * y + p[4], p[1] * x + p[3] * y + p[5]
    z = p[2] * x + p[5] * y + p[8]
    return (p[0] * x + p[3] * y + p[6]) / z, (p[1] * x + p[4] * y + p[7]) / z


def _sample64(img, xs, ys):
    """Bilinear samples with a zero border, their derivatives, the taps and their weights."""
    h, w = img.shape
    x0, y0 = xs.floor(), ys.floor()
    fx, fy = xs - x0, ys - y0
    x0, y0 = x0.clamp(-2, w).long(), y0.clamp(-2, h).long()
    taps = []
    for dy in (0, 1):
        for dx in (0, 1):
            x, y = x0 + dx, y0 + dy
            ok = (x >= 0) & (x < w) & (y >= 0) & (y < h)
            at = y.clamp(0, h - 1) * w + x.clamp(0, w - 1)
            taps.append((torch.where(ok, img.reshape(-1)[at], 0.0), at, ok, (fx if dx else 1 - fx) * (fy if dy else 1 - fy)))
    p00, p01, p10, p11 = (t[0] for t in taps)
    return {"value": (p00 * (1 - fx) + p01 * fx) * (1 - fy) + (p10 * (1 - fx) + p11 * fx) * fy, "taps": taps,
            "dx": (1 - fy) * (p01 - p00) + fy * (p11 - p10), "dy": (1 - fx) * (p10 - p00) + fx * (p11 - p01)}


def _adjoint64(img, p, s, g, xs, ys, c):
    """Gradients with respect to the source and the parameters for the output gradient g."""
    gsrc = torch.zeros(img.numel(), dtype=torch.float64, device="cuda")
    for _, at, ok, weight in s["taps"]:
        gsrc.index_add_(0, at.reshape(-1), torch.where(ok, g * weight, 0.0).reshape(-1))
    gx, gy = g * s["dx"], g * s["dy"]
    if c["warp"] == "field":
        return gsrc.view_as(img), torch.stack([gx, gy], -1)
    y, x = torch.meshgrid(torch.arange(c["h"], device="cuda", dtype=torch.float64), torch.arange(c["w"], device="cuda", dtype=torch.float64), indexing="ij")
    if c["warp"] == "affine":
        terms = [gx * x, gy * x, gx * y, gy * y, gx, gy]
    else:
        z = p[2] * x + p[5] * y + p[8]
        gx, gy = gx / z, gy / z
        q = -(gx * xs + gy * ys)
        terms = [k * f for f in (x, y, torch.ones_like(x)) for k in (gx, gy, q)]
    return gsrc.view_as(img), torch.stack([t.sum() for t in terms])


def exact(case, seed):
    if case["kind"] == "align":
        src, theta, target = _align_inputs(case, seed)
        loss, gsrc, gtheta = [], [], []
        for i in range(case["n"]):
            img, p = src[i].double(), theta[i].double()
            xs, ys = _positions64(p, case)
            s = _sample64(img, xs, ys)
            r = s["value"] - target[i].double()
            a, b = _adjoint64(img, p, s, 2 * r, xs, ys, case)
            loss.append((r * r).sum()); gsrc.append(a); gtheta.append(b)
        return {"loss": torch.stack(loss), "gsrc": torch.stack(gsrc), "gtheta": torch.stack(gtheta)}
    if case["kind"] == "warpgrad":
        src, p, gout = _grad_inputs(case, seed)
        out, gsrc, gp = [], [], []
        for i in range(case["n"]):
            img, q = src[i].detach().double(), p[i].detach().double()
            xs, ys = _positions64(q, case)
            s = _sample64(img, xs, ys)
            a, b = _adjoint64(img, q, s, gout[i].double(), xs, ys, case)
            out.append(s["value"]); gsrc.append(a); gp.append(b)
        return {"out": torch.stack(out), "gsrc": torch.stack(gsrc), "gp": torch.stack(gp)}
    return None
