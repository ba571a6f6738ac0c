"""The half-lane Sobel / threshold arithmetic of the TMA-staged configuration-1 kernel
(k_fused_c1_tma, mivisionx_b200/csrc/filters.cu), restated step by step in numpy: every half
step has to be exact (its float64 value is a float16), every fused multiply-add of halves into
fp32 too, and the sign of the result has to be the oracle chain's answer."""
import numpy as np
import pytest

import oracle_chains as OC

f16, f32 = np.float16, np.float32


def _h(v64):
    r = v64.astype(f16)
    assert np.all(r.astype(np.float64) == v64), "a half step of the kernel would round"
    return r


def _sq(a, c):
    r64 = a.astype(np.float64) ** 2 + c.astype(np.float64)
    r = r64.astype(f32)
    assert np.all(r.astype(np.float64) == r64), "a fused multiply-add of the kernel would round"
    return r


def _w(a):
    return a.astype(np.float64)


def fused_c1_half(img, shift, thr):
    H, W = img.shape
    pp = np.pad(img.astype(np.int64), ((0, 0), (1, 1)))
    h = pp[:, :-2] + 2 * pp[:, 1:-1] + pp[:, 2:]                 # horizontal [1 2 1] (16-bit lanes)
    g = (h[:-2] + 2 * h[1:-1] + h[2:]) >> 4                      # Gaussian of rows 1 .. H-2
    t = (np.uint16(0x6400) | g.astype(np.uint16)).view(f16)
    assert np.all(_w(t) == 1024 + g)
    d = _h(_w(t[:, 2:]) - _w(t[:, :-2]))
    D = _h(_w(d[:-1]) + _w(d[1:]))
    gx = _h(_w(D[:-1]) + _w(D[1:]))
    e = _h(_w(t[2:]) - _w(t[:-2]))
    gy = _h(_w(_h(2 * _w(e[:, 1:-1]) + _w(e[:, :-2]))) + _w(e[:, 2:]))
    M = ((thr & 255) + 1) << shift
    never = (thr & 255) == 255 or M > 2048
    tr, tt = (-8388608.0, -8388608.0) if never else (0.5 - (M * M - M + 1), 0.5 - M * M)
    assert float(f32(tr)) == tr and float(f32(tt)) == tt
    T = np.where(np.arange(1, W - 1) < W - W % 16, f32(tr), f32(tt)).astype(f32)[None, :]
    r = _sq(gx, _sq(gy, np.broadcast_to(T, gx.shape)))
    assert not np.any(r == 0)
    out = np.zeros((H, W), np.uint8)
    out[2:H - 2, 1:W - 1] = np.where(np.signbit(r), 0, 255)
    return out


@pytest.mark.parametrize("W,H", [(64, 40), (37, 21), (130, 66)])
def test_half_chain_matches_oracle(rng, W, H):
    yy, xx = np.indices((H, W))
    for img in (rng.integers(0, 256, (H, W), dtype=np.uint8), (rng.integers(0, 2, (H, W)) * 255).astype(np.uint8),
                ((yy + xx) % 2 * 255).astype(np.uint8),          # checkerboard: largest |gx|, |gy|
                (xx % 2 * 255).astype(np.uint8), ((yy % 3 == 0) * 255).astype(np.uint8)):
        for shift in range(6):
            for thr in range(0, 256, 3):
                ref, (sx, sy, ex, ey) = OC.cfg1_chain(img, shift, thr)
                got = fused_c1_half(img, shift, thr)
                assert np.array_equal(got[sy:ey, sx:ex], ref[sy:ey, sx:ex]), (shift, thr)


def test_half_chain_every_threshold_and_shift(rng):
    for img in (rng.integers(0, 256, (20, 40), dtype=np.uint8), (rng.integers(0, 2, (20, 40)) * 255).astype(np.uint8)):
        for shift in range(6):
            for thr in range(256):
                ref, (sx, sy, ex, ey) = OC.cfg1_chain(img, shift, thr)
                got = fused_c1_half(img, shift, thr)
                assert np.array_equal(got[sy:ey, sx:ex], ref[sy:ey, sx:ex]), (shift, thr)
