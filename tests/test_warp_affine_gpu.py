"""GPU parity of the U8 WarpAffine kernels against the oracle at the edges of their short path
(four pixels that all read inside the source): ends that touch the last column or row, flips,
integer and fractional shifts, positions outside, a valid rectangle, other source sizes."""
import ctypes as C

import numpy as np
import pytest

import oracle_chains as OC

pytestmark = pytest.mark.gpu

u32, vp, u8 = C.c_uint32, C.c_void_p, C.c_uint8
ARGS = [u32, u32, vp, u32, u32, u32, vp, u32, vp, u8]


def matrices(W, H, sW, sH):
    return {"identity": (1, 0, 0, 1, 0, 0), "shift": (1, 0, 0, 1, 3, 2), "half": (1, 0, 0, 1, 0.5, 0.25),
            "negative": (1, 0, 0, 1, -0.5, -1e-7), "flip": (-1, 0, 0, -1, sW - 1, sH - 1),
            "flip_in": (-1, 0, 0, -1, sW - 1.5, sH - 1.5), "fit": ((sW - 1) / W, 0, 0, (sH - 1) / H, 0, 0),
            "fill": (sW / W, 0, 0, sH / H, 0, 0), "rotate": (0.98, 0.11, -0.12, 0.97, 4.3, -2.6),
            "shear": (0.5, 0.25, 0.125, 0.5, -0.0, 1.0), "outside": (1, 0, 0, 1, 2.0 * sW, 0), "zero": (0, 0, 0, 0, sW - 1, sH - 1)}


@pytest.mark.parametrize("W,H,sW,sH", [(64, 48, 64, 48), (62, 21, 61, 23), (5, 3, 16, 9), (200, 40, 131, 77), (1920, 24, 1920, 24)])
@pytest.mark.parametrize("interp", ["Nearest", "Bilinear"])
def test_warp_affine_matches_oracle(cuda, rng, W, H, sW, sH, interp):
    import oracle as O
    from devbuf import DevImg, stream_ptr
    from mivisionx_b200 import native

    img = rng.integers(0, 256, (sH, sW), dtype=np.uint8)
    src, dsrc = OC.ago_img(sH, sW), DevImg(sH, sW).upload(img)
    src.set(img)
    gpu = getattr(native.agocuda(), f"agocuda_WarpAffine_U8_U8_{interp}_Constant")
    ora = getattr(O.oracle_lib(), f"oracle_WarpAffine_U8_U8_{interp}_Constant")
    near = interp == "Nearest"
    gpu.argtypes, ora.argtypes = [vp] + ARGS + ([vp] if near else []), ARGS + ([u32] * 4 if near else [])
    for name, m in matrices(W, H, sW, sH).items():
        m = np.array(m, np.float32)
        for border, rect in ((0, (0, 0, sW, sH)), (77, (1, 2, sW - 1, sH - 1))):
            ref, out = OC.ago_img(H, W), DevImg(H, W)
            r = np.array(rect, np.uint32)
            ora(W, H, ref.ptr, ref.stride, sW, sH, src.ptr, src.stride, m.ctypes.data, border, *(rect if near else ()))
            assert gpu(stream_ptr(), W, H, out.ptr, out.stride, sW, sH, dsrc.ptr, dsrc.stride, m.ctypes.data, border,
                       *([r.ctypes.data] if near else [])) == 0
            got, want = out.download(), ref.get()
            if not near:            # a footprint that passes the last row reads past the reference's buffer
                x, y = np.arange(W, dtype=np.float32)[None, :], np.arange(H, dtype=np.float32)[:, None]
                xs, ys = m[0] * x + (y * m[2] + m[4]), m[1] * x + (y * m[3] + m[5])
                past = (xs >= 0) & (xs < sW) & (ys < sH) & (np.trunc(ys) >= sH - 1)
                got, want = np.where(past, 0, got), np.where(past, 0, want)
            np.testing.assert_array_equal(got, want, err_msg=f"{name} border {border}")
