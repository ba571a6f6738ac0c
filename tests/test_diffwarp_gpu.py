"""GPU differentiable warps (mivisionx_b200.diffwarp, CUDA kernels of include/agocuda.h)
against the FP64 CPU reference (oracle/diffwarp_f64.py, itself checked against central
differences in test_diffwarp_ref.py).

Tolerances: forward within 2e-5 absolute (values in [0, 1], float32 arithmetic);
theta gradients within 1e-4 relative; source and field gradients within 1e-4 of the
largest gradient magnitude; losses within 1e-5 relative."""
import numpy as np
import pytest

from oracle import diffwarp_f64 as D
from mivisionx_b200 import workloads as WL

pytestmark = pytest.mark.gpu


def setup(n, size, seed=5):
    import torch
    imgs = WL.cfg5_images(n, seed=seed, size=size)
    gt, init = WL.cfg5_params(n, seed=seed, size=size)
    tgts = np.stack([D.warp_affine(imgs[i].astype(np.float64), gt[i]) for i in range(n)]).astype(np.float32)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    return imgs, init, tgts, dev(imgs), dev(init.astype(np.float32)), dev(tgts)


def fp64(imgs, theta, tgts, i):
    img = imgs[i].astype(np.float64)
    th = theta[i].astype(np.float32).astype(np.float64)       # the GPU sees float32 theta
    out = D.warp_affine(img, th)
    gsrc, gth = D.warp_affine_adjoint(img, th, 2 * (out - tgts[i].astype(np.float64)))
    return out, D.l2_loss(out, tgts[i].astype(np.float64)), gsrc, gth


def close_grad(got, want, what):
    scale = np.abs(want).max()
    err = np.abs(got - want).max()
    assert err <= 1e-4 * scale, f"{what}: max error {err} vs scale {scale}"


@pytest.mark.parametrize("size", [128, 1024])
def test_l2_step_matches_fp64(cuda, size):
    from mivisionx_b200 import diffwarp
    n = 4
    imgs, theta, tgts, d_img, d_th, d_tgt = setup(n, size)
    loss, gsrc, gth = diffwarp.warp_affine_l2_step(d_img, d_th, d_tgt)
    loss, gsrc, gth = loss.cpu().numpy(), gsrc.cpu().numpy(), gth.cpu().numpy()
    for i in range(n):
        _, l, gs, gt = fp64(imgs, theta, tgts, i)
        assert abs(loss[i] - l) <= 1e-5 * l, (i, loss[i], l)
        np.testing.assert_allclose(gth[i], gt, rtol=1e-4, err_msg=f"image {i}")
        close_grad(gsrc[i], gs, f"gsrc image {i}")


def test_autograd_matches_fp64(cuda):
    import torch

    from mivisionx_b200 import diffwarp
    n, size = 3, 256
    imgs, theta, tgts, d_img, d_th, d_tgt = setup(n, size, seed=11)
    src = d_img.clone().requires_grad_(True)
    th = d_th.clone().requires_grad_(True)
    out = diffwarp.warp_affine(src, th)
    loss = ((out - d_tgt) ** 2).sum()
    loss.backward()
    for i in range(n):
        o, _, gs, gt = fp64(imgs, theta, tgts, i)
        assert np.abs(out[i].detach().cpu().numpy() - o).max() <= 2e-5
        np.testing.assert_allclose(th.grad[i].cpu().numpy().astype(np.float64), gt, rtol=1e-4)
        close_grad(src.grad[i].cpu().numpy(), gs, f"gsrc image {i}")
    # the fused step gives the same gradients as forward + autograd backward
    l2, gs2, gt2 = diffwarp.warp_affine_l2_step(d_img, d_th, d_tgt)
    np.testing.assert_allclose(gt2.cpu().numpy(), th.grad.cpu().numpy().astype(np.float64), rtol=1e-4)
    assert abs(float(l2.sum()) - loss.item()) <= 1e-5 * loss.item()
    assert torch.allclose(gs2, src.grad, rtol=0, atol=1e-4 * float(gs2.abs().max()))


def test_remap_forward_and_adjoint_match_fp64(cuda):
    import torch

    from mivisionx_b200 import diffwarp
    size = 256
    img = WL.cfg5_images(2, seed=21, size=size)
    fields = np.stack([WL.cfg5_field(seed=s, size=size) for s in (1, 2)])
    tgt = np.stack([D.remap(img[i].astype(np.float64), WL.cfg5_field(seed=7 + i, size=size).astype(np.float64))
                    for i in range(2)]).astype(np.float32)
    src = torch.from_numpy(img).cuda().requires_grad_(True)
    fld = torch.from_numpy(fields).cuda().requires_grad_(True)
    out = diffwarp.remap(src, fld)
    ((out - torch.from_numpy(tgt).cuda()) ** 2).sum().backward()
    for i in range(2):
        o = D.remap(img[i].astype(np.float64), fields[i].astype(np.float64))
        assert np.abs(out[i].detach().cpu().numpy() - o).max() <= 2e-5
        gs, gf = D.remap_adjoint(img[i].astype(np.float64), fields[i].astype(np.float64), 2 * (o - tgt[i]))
        close_grad(src.grad[i].cpu().numpy(), gs, "gsrc")
        close_grad(fld.grad[i].cpu().numpy(), gf, "gfield")


def test_border_value_and_far_outside_positions(cuda):
    import torch

    from mivisionx_b200 import diffwarp
    img = WL.cfg5_images(1, seed=3, size=64)
    # shift far outside, a NaN-free but huge scale, and a half-outside shift
    thetas = np.array([[1, 0, 0, 1, 5000.0, -7000.0], [1e6, 0, 0, 1e6, 0, 0], [1, 0, 0, 1, 40.5, -20.25]], np.float32)
    src = torch.from_numpy(np.repeat(img, 3, 0)).cuda()
    out = diffwarp.warp_affine(src, torch.from_numpy(thetas).cuda(), border=0.25).cpu().numpy()
    for i in range(3):
        want = D.warp_affine(img[0].astype(np.float64), thetas[i].astype(np.float64), border=0.25)
        assert np.abs(out[i] - want).max() <= 2e-5, i


def _persp_setup(n, size, seed=6):
    import torch
    imgs = WL.cfg5_images(n, seed=seed, size=size)
    gt, init = WL.cfg5_perspective_params(n, seed=seed, size=size)
    tgts = np.stack([D.warp_perspective(imgs[i].astype(np.float64), gt[i]) for i in range(n)]).astype(np.float32)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    return imgs, init, tgts, dev(imgs), dev(init.astype(np.float32)), dev(tgts)


def _persp_fp64(imgs, theta, tgts, i):
    img = imgs[i].astype(np.float64)
    th = theta[i].astype(np.float32).astype(np.float64)
    out = D.warp_perspective(img, th)
    gsrc, gth = D.warp_perspective_adjoint(img, th, 2 * (out - tgts[i].astype(np.float64)))
    return out, D.l2_loss(out, tgts[i].astype(np.float64)), gsrc, gth


@pytest.mark.parametrize("size", [128, 1024])
def test_perspective_l2_step_matches_fp64(cuda, size):
    from mivisionx_b200 import diffwarp
    n = 4
    imgs, theta, tgts, d_img, d_th, d_tgt = _persp_setup(n, size)
    loss, gsrc, gth = diffwarp.warp_perspective_l2_step(d_img, d_th, d_tgt)
    loss, gsrc, gth = loss.cpu().numpy(), gsrc.cpu().numpy(), gth.cpu().numpy()
    for i in range(n):
        _, l, gs, gt = _persp_fp64(imgs, theta, tgts, i)
        assert abs(loss[i] - l) <= 1e-5 * l, (i, loss[i], l)
        np.testing.assert_allclose(gth[i], gt, rtol=1e-4, err_msg=f"image {i}")
        close_grad(gsrc[i], gs, f"gsrc image {i}")


def test_perspective_autograd_matches_fp64(cuda):
    from mivisionx_b200 import diffwarp
    n, size = 3, 256
    imgs, theta, tgts, d_img, d_th, d_tgt = _persp_setup(n, size, seed=12)
    src = d_img.clone().requires_grad_(True)
    th = d_th.clone().requires_grad_(True)
    out = diffwarp.warp_perspective(src, th)
    loss = ((out - d_tgt) ** 2).sum()
    loss.backward()
    for i in range(n):
        o, _, gs, gt = _persp_fp64(imgs, theta, tgts, i)
        assert np.abs(out[i].detach().cpu().numpy() - o).max() <= 2e-5
        np.testing.assert_allclose(th.grad[i].cpu().numpy().astype(np.float64), gt, rtol=1e-4)
        close_grad(src.grad[i].cpu().numpy(), gs, f"gsrc image {i}")


def test_perspective_degenerate_rows(cuda):
    """z = 0 on a line through the image and z < 0 beyond it: samples there read the border,
    contribute no theta gradient, and nothing becomes NaN."""
    import torch

    from mivisionx_b200 import diffwarp
    size = 64
    img = WL.cfg5_images(1, seed=4, size=size)
    th = np.array([[1, 0, 1.0 / 32, 0, 1, 0, 0, 0, -1.0]], np.float32)   # z = x/32 - 1: zero at x = 32
    src = torch.from_numpy(img).cuda().requires_grad_(True)
    tht = torch.from_numpy(th).cuda().requires_grad_(True)
    out = diffwarp.warp_perspective(src, tht, border=0.5)
    out.sum().backward()
    o = out.detach().cpu().numpy()[0]
    assert np.isfinite(o).all() and np.all(o[:, 32] == 0.5)
    assert torch.isfinite(tht.grad).all() and torch.isfinite(src.grad).all()


# maps whose neighbouring samples share taps (unit scale), skip columns (2.5), sit on one cell (0.2),
# run backwards or leave the source
STRIP_MAPS = ["shift", "wide", "tight", "mirror", "off"]


def _strip_map(kind, H, W):
    return {"shift": [1, 0, 0, 1, 0.3, -0.4], "wide": [2.5, 0.1, -0.1, 2.5, -3.2, 1.1], "tight": [0.2, 0, 0, 0.2, 1.1, 0.6],
            "mirror": [-1, 0, 0, -1, W - 1.25, H - 1.75], "off": [1, 0, 0, 1, W - 2.5, -H + 1.5]}[kind]


# sizes around the 32 columns of a warp's strip; batches this small have strips of one row
@pytest.mark.parametrize("kind", STRIP_MAPS)
@pytest.mark.parametrize("H,W", [(1, 1), (1, 40), (2, 33), (17, 31), (67, 130)])
def test_adjoint_at_strip_edges(cuda, H, W, kind):
    import torch

    from mivisionx_b200 import diffwarp
    rng = np.random.default_rng(H * 1000 + W)
    n = 3
    img = rng.random((n, H, W)).astype(np.float32)
    tgt = rng.random((n, H, W)).astype(np.float32)
    base = _strip_map(kind, H, W)
    theta = np.array([base, base, [1.01, 0.02, -0.02, 0.99, 0.1, 0.2]], np.float32)
    d = [torch.from_numpy(a).cuda() for a in (img, theta, tgt)]
    loss, gsrc, gth = diffwarp.warp_affine_l2_step(*d)
    field = torch.from_numpy(rng.uniform(-3, 3, (n, H, W, 2)).astype(np.float32)).cuda().requires_grad_(True)
    src = d[0].clone().requires_grad_(True)
    (diffwarp.remap(src, field) * d[2]).sum().backward()
    for i in range(n):
        _, l, gs, gt = fp64(img, theta, tgt, i)
        assert abs(float(loss[i]) - l) <= 1e-5 * max(l, 1e-6)
        # float residuals and derivatives (1e-6 of a term), each term at most the size of the sum's scale
        scale = 4 * H * W * max(H, W)
        assert np.abs(gth[i].cpu().numpy() - gt).max() <= 1e-6 * scale
        assert np.abs(gsrc[i].cpu().numpy() - gs).max() <= 1e-5 * max(np.abs(gs).max(), 1.0)
        f = field[i].detach().cpu().numpy().astype(np.float64)
        gs, gf = D.remap_adjoint(img[i].astype(np.float64), f, tgt[i].astype(np.float64))
        assert np.abs(src.grad[i].cpu().numpy() - gs).max() <= 1e-5 * max(np.abs(gs).max(), 1.0)
        assert np.abs(field.grad[i].cpu().numpy() - gf).max() <= 1e-5 * max(np.abs(gf).max(), 1.0)


# strips of several rows, where the lower contributions of a row join the upper ones of the next.  A
# strip has the most rows (up to 32) that leave 32 warps for every SM: the batch sets them.  The rows
# of each size end in a part strip.
@pytest.mark.parametrize("kind", STRIP_MAPS)
@pytest.mark.parametrize("rows", [8, 32])
@pytest.mark.parametrize("H,W", [(67, 130), (40, 33)])
def test_adjoint_in_strips_of_many_rows(cuda, H, W, rows, kind):
    import torch

    from mivisionx_b200 import diffwarp
    warps = 32 * torch.cuda.get_device_properties(0).multi_processor_count
    strips = lambda r: -(-W // 32) * -(-H // r)
    n = -(-warps // strips(rows))
    assert rows == 32 or n * strips(2 * rows) < warps
    rng = np.random.default_rng(H + rows)
    img, tgt = rng.random((n, H, W)).astype(np.float32), rng.random((n, H, W)).astype(np.float32)
    theta = np.array([_strip_map(kind, H, W)] * n, np.float32)
    d = [torch.from_numpy(a).cuda() for a in (img, theta, tgt)]
    loss, gsrc, gth = diffwarp.warp_affine_l2_step(*d)
    src, th = d[0].clone().requires_grad_(True), d[1].clone().requires_grad_(True)
    (diffwarp.warp_affine(src, th) * d[2]).sum().backward()
    ys, xs = np.meshgrid(np.arange(H), np.arange(W), indexing="ij")
    m = theta[0]
    at = np.stack([m[0] * xs + m[2] * ys + m[4] - xs, m[1] * xs + m[3] * ys + m[5] - ys], -1).astype(np.float32)
    field = torch.from_numpy(np.broadcast_to(at, (n, H, W, 2)).copy()).cuda().requires_grad_(True)
    fsrc = d[0].clone().requires_grad_(True)
    (diffwarp.remap(fsrc, field) * d[2]).sum().backward()
    scale = 4 * H * W * max(H, W)          # as above: 1e-6 of each term, terms at most the size of the sum's scale
    near = lambda a, b: np.abs(a - b).max() <= 1e-5 * max(np.abs(b).max(), 1.0)
    for i in (0, n // 2, n - 1):
        _, l, gs, gt = fp64(img, theta, tgt, i)
        assert abs(float(loss[i]) - l) <= 1e-5 * max(l, 1e-6)
        assert np.abs(gth[i].cpu().numpy() - gt).max() <= 1e-6 * scale
        assert near(gsrc[i].cpu().numpy(), gs)
        gs, gt = D.warp_affine_adjoint(img[i].astype(np.float64), theta[i].astype(np.float64), tgt[i].astype(np.float64))
        assert near(src.grad[i].cpu().numpy(), gs)
        assert np.abs(th.grad[i].cpu().numpy() - gt).max() <= 1e-6 * scale
        gs, gf = D.remap_adjoint(img[i].astype(np.float64), at.astype(np.float64), tgt[i].astype(np.float64))
        assert near(fsrc.grad[i].cpu().numpy(), gs)
        assert near(field.grad[i].cpu().numpy(), gf)


def test_source_beyond_int_indexes(cuda):
    """A source whose element indexes pass 2^31 (two rows 2^30 elements apart)."""
    import ctypes as CT
    import torch

    from devbuf import stream_ptr
    from mivisionx_b200 import diffwarp
    W, H, stride = 40, 2, 1 << 30
    rng = np.random.default_rng(3)
    img, g = rng.random((H, W)).astype(np.float32), rng.random((H, W)).astype(np.float32)
    big = torch.empty(stride + W, dtype=torch.float32, device="cuda")
    rows = torch.as_strided(big, (H, W), (stride, 1))
    rows.copy_(torch.from_numpy(img))
    theta = np.array([1.02, 0.01, -0.01, 0.97, 0.3, 0.2], np.float32)
    th, gout = torch.from_numpy(theta).cuda(), torch.from_numpy(g).cuda()
    out, gth = torch.zeros(H, W, device="cuda"), torch.zeros(6, dtype=torch.float64, device="cuda")
    L = diffwarp._L()
    assert L.agocuda_WarpAffine_F32_Bilinear_Constant_batch(stream_ptr(), 1, W, H, out.data_ptr(), H * W, W, W, H, big.data_ptr(),
                                                            0, stride, th.data_ptr(), 0.0) == 0
    gbig = torch.empty(stride + W, dtype=torch.float32, device="cuda")
    grows = torch.as_strided(gbig, (H, W), (stride, 1))
    grows.zero_()
    assert L.agocuda_WarpAffine_F32_Bilinear_Constant_adjoint_batch(
        stream_ptr(), 1, W, H, gout.data_ptr(), H * W, W, W, H, big.data_ptr(), 0, stride, th.data_ptr(), 0.0, gbig.data_ptr(),
        gth.data_ptr()) == 0
    t64 = theta.astype(np.float64)
    assert np.abs(out.cpu().numpy() - D.warp_affine(img.astype(np.float64), t64)).max() <= 2e-5
    gs, gt = D.warp_affine_adjoint(img.astype(np.float64), t64, g.astype(np.float64))
    close_grad(grows.cpu().numpy(), gs, "gsrc")
    assert np.abs(gth.cpu().numpy() - gt).max() <= 1e-6 * 4 * H * W * W
