// diffwarp.cu -- differentiable F32 warps on sm_100a: bilinear WarpAffine, WarpPerspective
// and Remap with a constant border, their adjoints, and fused "warp + L2 loss + adjoint"
// steps.
//
// The reference has no F32 warp (its warps validate U8 only, ago_kernel_api.cpp:19255); the
// coordinate conventions are those of its U8 warps.  WarpAffine (ago_haf_cpu_geometric.cpp:
// 679-684, ago_affine_matrix_t m[3][2]):  xs = m00*x + m10*y + m20,  ys = m01*x + m11*y + m21,
// theta holding (m00, m01, m10, m11, m20, m21).  WarpPerspective (ago_haf_cpu_geometric.cpp:
// 1594-1602, ago_perspective_matrix_t m[3][3]):  z = m02*x + m12*y + m22,
// xs = (m00*x + m10*y + m20) / z,  ys = (m01*x + m11*y + m21) / z, theta holding the nine
// entries in storage order; z == 0 samples the border.  Bilinear interpolation from
// floor(xs), floor(ys); each of the four taps outside the source reads the border value.
//
// Adjoint: d/dsrc scatters gout times the tap weights (red.global.add on the source
// gradient); d/dtheta sums gout * (dout/dxs * dxs/dtheta + dout/dys * dys/dtheta) in double
// per thread, warp and block (atomicAdd double per block and image).
#include "agocuda_internal.cuh"
#include <limits.h>

uint64_t agocuda_count_launch(unsigned n);

namespace {

// One sample: the fractions, the four taps, and in `key` the element index of the first tap where
// all four lie inside a source of fewer than 2^31 elements (`wide` is false), else kNoKey.
constexpr int kNoKey = INT_MIN;
struct Sample {
    int key;
    float fx, fy;
    float p00, p01, p10, p11;
};

// Where the taps of a sample lie that has no key: each on its own inside the source or not
struct Place {
    int x0, y0;
    float fx, fy;
    bool k00, k01, k10, k11;
};

// Positions are formed in double: a float position near x = 1000 is only good to ~6e-5 px,
// and the theta gradient is a strongly cancelling sum over every pixel.
__device__ __forceinline__ Place place(int W, int H, double xs, double ys)
{
    Place t;
    const double fx0 = floor(xs), fy0 = floor(ys);
    t.fx = (float)(xs - fx0);
    t.fy = (float)(ys - fy0);
    // positions far outside the source (or NaN): every tap reads the border
    const bool far = !(fx0 > -2.0 && fx0 < (double)W + 1.0 && fy0 > -2.0 && fy0 < (double)H + 1.0);
    t.x0 = far ? -2 : (int)fx0;
    t.y0 = far ? -2 : (int)fy0;
    if (far) { t.fx = 0.f; t.fy = 0.f; }     // NaN / infinite positions: the border, exactly
    const int x1 = t.x0 + 1, y1 = t.y0 + 1;
    const bool cx0 = t.x0 >= 0 && t.x0 < W, cx1 = x1 >= 0 && x1 < W, cy0 = t.y0 >= 0 && t.y0 < H, cy1 = y1 >= 0 && y1 < H;
    t.k00 = cx0 && cy0; t.k01 = cx1 && cy0; t.k10 = cx0 && cy1; t.k11 = cx1 && cy1;
    return t;
}

// floor(v) of a position inside a source of n columns (or rows) without the double-to-int
// conversions and FRND: v + 1.5 * 2^52 rounded down holds floor(v) in its low word, and its
// high word is 0x43380000 exactly for 0 <= floor(v) < 2^32 (any other value, an infinity or
// a NaN has another one).  Returns whether both taps floor(v), floor(v) + 1 lie inside.
__device__ __forceinline__ bool floor_inside(double v, int n, int &i, float &f)
{
    const double magic = 6755399441055744.0;
    const double t = __dadd_rd(v, magic);
    i = __double2loint(t);
    f = (float)(v - (t - magic));
    return __double2hiint(t) == 0x43380000 && (unsigned)i < (unsigned)(n - 1);
}

__device__ __forceinline__ Sample sample(const float *src, int stride, int W, int H, double xs, double ys, float border,
                                         bool wide)
{
    Sample s;
    int x0, y0;
    const bool inx = floor_inside(xs, W, x0, s.fx), iny = floor_inside(ys, H, y0, s.fy);
    if (inx && iny && !wide) {
        s.key = y0 * stride + x0;
        const float *p = src + s.key;
        s.p00 = __ldg(p); s.p01 = __ldg(p + 1);
        s.p10 = __ldg(p + stride); s.p11 = __ldg(p + stride + 1);
    } else {
        const Place t = place(W, H, xs, ys);
        const float *p = src + (long long)t.y0 * stride + t.x0;
        s.p00 = t.k00 ? __ldg(p) : border;
        s.p01 = t.k01 ? __ldg(p + 1) : border;
        s.p10 = t.k10 ? __ldg(p + stride) : border;
        s.p11 = t.k11 ? __ldg(p + stride + 1) : border;
        s.fx = t.fx;
        s.fy = t.fy;
        s.key = kNoKey;
    }
    return s;
}

// The scatter of a warp that walks down the rows of a 32-column strip.  One atomic per tap is
// what bounds the adjoint (4 per pixel); neighbouring samples mostly share taps, so a lane
// keeps its lower two contributions until the next row, where they join the upper two if the
// addresses agree, and hands its right-hand contribution to the lane whose left-hand one has
// that address.  Near a unit-scale map about 1.7 atomics per pixel are left.  Any map is
// right: contributions join only where their addresses are equal.
struct Scatter {
    int key = kNoKey;          // address of the contributions kept from the row above
    float v0 = 0.f, v1 = 0.f;

    // all lanes of the warp take part; a lane without a sample passes key kNoKey and g 0.  where()
    // is the Place of a sample without a key, which few have: it is found again, not carried.
    template <class WHERE>
    __device__ __forceinline__ void row(float *gsrc, int stride, const Sample &t, float g, bool has, WHERE where)
    {
        const float gu = g * (1.f - t.fx), gr = g * t.fx;
        float c00 = gu * (1.f - t.fy), c01 = gr * (1.f - t.fy);
        const float c10 = gu * t.fy, c11 = gr * t.fy;
        const int k = t.key;
        if (key != kNoKey) {
            if (key == k) {
                c00 += v0;
                c01 += v1;
            } else {
                atomicAdd(gsrc + key, v0);
                atomicAdd(gsrc + key + 1, v1);
            }
        }
        const int lane = threadIdx.x & 31;
        const int ku = __shfl_up_sync(0xffffffffu, k, 1), kd = __shfl_down_sync(0xffffffffu, k, 1);
        const float cu = __shfl_up_sync(0xffffffffu, c01, 1);
        key = kNoKey;
        if (k != kNoKey) {
            if (lane > 0 && ku == k - 1) c00 += cu;
            atomicAdd(gsrc + k, c00);
            if (lane == 31 || kd != k + 1) atomicAdd(gsrc + k + 1, c01);
            key = k + stride;
            v0 = c10;
            v1 = c11;
        } else if (has) {
            const Place w = where();
            float *p = gsrc + (long long)w.y0 * stride + w.x0;
            if (w.k00) atomicAdd(p, c00);
            if (w.k01) atomicAdd(p + 1, c01);
            if (w.k10) atomicAdd(p + stride, c10);
            if (w.k11) atomicAdd(p + stride + 1, c11);
        }
    }
    __device__ __forceinline__ void flush(float *gsrc)
    {
        const int lane = threadIdx.x & 31;
        const int ku = __shfl_up_sync(0xffffffffu, key, 1), kd = __shfl_down_sync(0xffffffffu, key, 1);
        const float cu = __shfl_up_sync(0xffffffffu, v1, 1);
        if (key == kNoKey) return;
        atomicAdd(gsrc + key, lane > 0 && ku == key - 1 ? v0 + cu : v0);
        if (lane == 31 || kd != key + 1) atomicAdd(gsrc + key + 1, v1);
    }
};

// a (1 - f) + b f
__device__ __forceinline__ float mix(float a, float b, float f) { return __fmaf_rn(b, f, a * (1.f - f)); }
__device__ __forceinline__ float interp(const Sample &t) { return mix(mix(t.p00, t.p01, t.fx), mix(t.p10, t.p11, t.fx), t.fy); }
__device__ __forceinline__ float dout_dxs(const Sample &t) { return mix(t.p01 - t.p00, t.p11 - t.p10, t.fy); }
__device__ __forceinline__ float dout_dys(const Sample &t) { return mix(t.p10 - t.p00, t.p11 - t.p01, t.fx); }

// block reduction of N per-thread double sums into double atomics at dst[0..N)
template <int N>
__device__ __forceinline__ void block_add(const double (&v)[N], double *dst)
{
    __shared__ double red[N][8];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
    for (int k = 0; k < N; k++) {
        double s = v[k];
#pragma unroll
        for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (lane == 0) red[k][warp] = s;
    }
    __syncthreads();
    if (threadIdx.x < N) {
        double s = 0.0;
        for (int w = 0; w < nw; w++) s += red[threadIdx.x][w];
        atomicAdd(dst + threadIdx.x, s);
    }
}

struct Img32 {
    float *p;                 // image 0 (image i at p + i * batch)
    long long batch;
    int stride, W, H;
};

enum Mode { kForward = 0, kAdjoint = 1, kFusedL2 = 2 };

// Warps of image blockIdx.z.  Modes: forward (out), adjoint (gout -> gsrc, parameter
// gradient), fused L2 step (target -> gsrc, gtheta and loss with gout = 2 (out - target)).
// NT = 6: affine; NT = 9: perspective; NT = 2: displacement field (the gradient is a field).
// Per image the adjoint adds NT theta gradients, the fused step NT gradients and then the loss.
//
// A warp owns a strip of 32 columns and `rows` rows and walks down it, the taps of the next
// row loaded while a row is worked on.  Per pixel a thread adds 2 (affine) or 6 terms to
// double sums of its own; x is fixed per thread, so sum(g x) is x sum(g), and the sums meet
// across lanes once per strip instead of once per pixel (7 double butterflies per pixel were
// the larger half of the fused step).  Products with y are fused into their sums, and a sample
// carries no place of its own, only a key.  Affine L2 step of 32 x 1024^2: 573 us with one pixel
// per thread, 264 us so; issue-bound, and larger bodies (two rows unrolled) are slower, 338 us.
// `rows` is 32 where the batch fills the device with such strips and less where it does not
// (warp_rows): 16 rows, with twice as many sums across lanes, took 267 us.
template <int MODE, int NT>
__global__ void __launch_bounds__(256)
k_warp_f32(int W, int H, int rows, Img32 src, Img32 out, Img32 aux, const float *par, long long parBatch, int parStride,
           float border, Img32 gsrc, void *gpar)
{
    const int x = blockIdx.x * 32 + (threadIdx.x & 31), n = blockIdx.z;
    const int yA = (blockIdx.y * 8 + (threadIdx.x >> 5)) * rows, yB = min(yA + rows, H);
    const bool act = x < W;
    const float *sp = src.p + src.batch * n;
    float *gp = MODE == kForward ? nullptr : gsrc.p + gsrc.batch * n;
    const bool wide = (long long)src.stride * src.H > 0x7fffffffll;
    const float *th = NT == 2 ? nullptr : par + NT * n;
    const float2 *field = NT == 2 ? (const float2 *)par + parBatch * n : nullptr;
    float2 *gfield = NT == 2 && MODE == kAdjoint ? (float2 *)gpar + parBatch * n : nullptr;
    // the parts of the map that do not depend on y (products of 24-bit factors: exact)
    double mx[3] = {}, my[3] = {}, m0[3] = {};
    if (NT != 2) {
        constexpr int D = NT == 9 ? 3 : 2;
#pragma unroll
        for (int k = 0; k < D; k++) {
            mx[k] = (double)th[k] * x;
            my[k] = (double)th[D + k];
            m0[k] = (double)th[2 * D + k];
        }
    }
    struct Pos { double xs, ys, iz; };
    // yd = y; the sums my y + mx round once, like the sum of the exact product and mx
    auto position = [&](int y, double yd) -> Pos {
        if (NT == 2) {
            const float2 d = act ? field[(size_t)y * parStride + x] : make_float2(0.f, 0.f);
            return {(double)x + d.x, (double)y + d.y, 1.0};
        }
        const double xn = __fma_rn(my[0], yd, mx[0]) + m0[0], yn = __fma_rn(my[1], yd, mx[1]) + m0[1];
        if (NT == 6) return {xn, yn, 1.0};
        const double z = __fma_rn(my[2], yd, mx[2]) + m0[2];
        if (z == 0.0) { const double nan = __longlong_as_double(0x7ff8000000000000ll); return {nan, nan, 0.0}; }
        const double iz = 1.0 / z;
        return {xn * iz, yn * iz, iz};
    };
    if constexpr (MODE == kForward) {
        if (!act) return;
        float *o = out.p + out.batch * n + x;
        for (int y = yA; y < yB; y += 2) {                 // two rows at a time: their loads overlap
            const int y1 = min(y + 1, yB - 1);
            const Pos p = position(y, y), q = position(y1, y1);
            const Sample a = sample(sp, src.stride, src.W, src.H, p.xs, p.ys, border, wide);
            const Sample b = sample(sp, src.stride, src.W, src.H, q.xs, q.ys, border, wide);
            o[(size_t)y * out.stride] = interp(a);
            if (y + 1 < yB) o[(size_t)(y + 1) * out.stride] = interp(b);
        }
        return;
    }
    constexpr int NS = NT == 2 ? 1 : NT + (MODE == kFusedL2 ? 1 : 0);
    double sum[NS] = {};
    Scatter sc;
    const float *ap = aux.p + aux.batch * n + x;
    auto load = [&](int y, double yd, Pos &p, Sample &s, float &a) {
        if (act && y < yB) {
            p = position(y, yd);
            a = __ldg(ap + (size_t)y * aux.stride);
            s = sample(sp, src.stride, src.W, src.H, p.xs, p.ys, border, wide);
        } else {
            s = Sample{};
            s.key = kNoKey;
            a = 0.f;
        }
    };
    Pos p, pn;
    Sample s, sn;
    float a, an;
    double yd = yA;
    load(yA, yd, p, s, a);
    for (int y = yA; y < yB; y++) {
        const double yn = yd + 1.0;
        load(y + 1, yn, pn, sn, an);
        float g = a;
        if (MODE == kFusedL2) {
            const float r = act ? interp(s) - a : 0.f;
            sum[NS - 1] = __fma_rn((double)r, (double)r, sum[NS - 1]);
            g = 2.f * r;
        }
        sc.row(gp, gsrc.stride, s, g, act, [&]() {
            const Pos q = position(y, yd);
            return place(src.W, src.H, q.xs, q.ys);
        });
        const float gx = g * dout_dxs(s), gy = g * dout_dys(s);
        if (NT == 2) {
            if (act) gfield[(size_t)y * parStride + x] = make_float2(gx, gy);
        } else if (NT == 6) {
            const double dx = gx, dy = gy;
            sum[4 % NS] += dx;
            sum[5 % NS] += dy;
            sum[2 % NS] = __fma_rn(dx, yd, sum[2 % NS]);
            sum[3 % NS] = __fma_rn(dy, yd, sum[3 % NS]);
        } else if (act && p.iz != 0.0 && (gx != 0.f || gy != 0.f)) {   // a sample on the border has no theta term
            // d(xs)/d(m00, m10, m20) = (x, y, 1) / z; d(xs)/d(m02, m12, m22) = -xs (x, y, 1) / z; same for ys
            const double gxz = gx * p.iz, gyz = gy * p.iz, q = -((double)gx * p.xs + (double)gy * p.ys) * p.iz;
            sum[6 % NS] += gxz;
            sum[7 % NS] += gyz;
            sum[8 % NS] += q;
            sum[3 % NS] = __fma_rn(gxz, yd, sum[3 % NS]);
            sum[4 % NS] = __fma_rn(gyz, yd, sum[4 % NS]);
            sum[5 % NS] = __fma_rn(q, yd, sum[5 % NS]);
        }
        p = pn; s = sn; a = an; yd = yn;
    }
    sc.flush(gp);
    if constexpr (NT != 2) {
        constexpr int D = NT == 9 ? 3 : 2;
#pragma unroll
        for (int k = 0; k < D; k++) sum[k] = sum[2 * D + k] * x;
        block_add<NS>(sum, (double *)gpar + NS * n);
    }
}

// Rows per warp: `most` where the strips still give every SM 32 warps (its latency hiding),
// halved until they do.
int warp_rows(int n, int W, int H, int most)
{
    const long long want = 32ll * agocuda_sm_count();
    int r = most;
    while (r > 1 && (long long)n * div_up(W, 32) * div_up(H, r) < want) r >>= 1;
    return r;
}

dim3 warp_grid(int n, int W, int H, int rows) { return dim3(div_up(W, 32), div_up(H, 8 * rows), n); }

Img32 img32(const float *p, long long batch, int stride, int W, int H) { return Img32{(float *)p, batch, stride, W, H}; }

bool batch_ok(int n, int W, int H, int sW, int sH)
{
    return n > 0 && n <= 65535 && W > 0 && H > 0 && sW > 0 && sH > 0 && W < (1 << 24) && H < (1 << 24) &&
           sW < (1 << 24) && sH < (1 << 24);
}

}  // namespace

extern "C" int agocuda_WarpAffine_F32_Bilinear_Constant_batch(void *stream, int n, int W, int H, float *pDst,
                                                              long long dstBatch, int dstStride, int srcW, int srcH,
                                                              const float *pSrc, long long srcBatch, int srcStride,
                                                              const float *theta, float border)
{
    if (!pDst || !pSrc || !theta || !batch_ok(n, W, H, srcW, srcH) || dstStride < W || srcStride < srcW)
        return AGOCUDA_INVALID_PARAMS;
    const int rows = warp_rows(n, W, H, 4);
    k_warp_f32<kForward, 6><<<warp_grid(n, W, H, rows), 256, 0, as_stream(stream)>>>(
        W, H, rows, img32(pSrc, srcBatch, srcStride, srcW, srcH), img32(pDst, dstBatch, dstStride, W, H), Img32{}, theta, 0, 0,
        border, Img32{}, nullptr);
    agocuda_count_launch(1);
    return agocuda_launch_status();
}

extern "C" int agocuda_WarpAffine_F32_Bilinear_Constant_adjoint_batch(void *stream, int n, int W, int H,
                                                                      const float *pGradOut, long long goBatch, int goStride,
                                                                      int srcW, int srcH, const float *pSrc,
                                                                      long long srcBatch, int srcStride, const float *theta,
                                                                      float border, float *pGradSrc, double *pGradTheta)
{
    if (!pGradOut || !pSrc || !theta || !pGradSrc || !pGradTheta || !batch_ok(n, W, H, srcW, srcH) || goStride < W ||
        srcStride < srcW)
        return AGOCUDA_INVALID_PARAMS;
    const int rows = warp_rows(n, W, H, 32);
    k_warp_f32<kAdjoint, 6><<<warp_grid(n, W, H, rows), 256, 0, as_stream(stream)>>>(
        W, H, rows, img32(pSrc, srcBatch, srcStride, srcW, srcH), Img32{}, img32(pGradOut, goBatch, goStride, W, H), theta, 0, 0,
        border, img32(pGradSrc, srcBatch, srcStride, srcW, srcH), pGradTheta);
    agocuda_count_launch(1);
    return agocuda_launch_status();
}

extern "C" int agocuda_WarpAffine_F32_L2_step_batch(void *stream, int n, int W, int H, const float *pTarget, long long tBatch,
                                                    int tStride, int srcW, int srcH, const float *pSrc, long long srcBatch,
                                                    int srcStride, const float *theta, float border, float *pGradSrc,
                                                    double *pGradThetaLoss)
{
    if (!pTarget || !pSrc || !theta || !pGradSrc || !pGradThetaLoss || !batch_ok(n, W, H, srcW, srcH) || tStride < W ||
        srcStride < srcW)
        return AGOCUDA_INVALID_PARAMS;
    const int rows = warp_rows(n, W, H, 32);
    k_warp_f32<kFusedL2, 6><<<warp_grid(n, W, H, rows), 256, 0, as_stream(stream)>>>(
        W, H, rows, img32(pSrc, srcBatch, srcStride, srcW, srcH), Img32{}, img32(pTarget, tBatch, tStride, W, H), theta, 0, 0,
        border, img32(pGradSrc, srcBatch, srcStride, srcW, srcH), pGradThetaLoss);
    agocuda_count_launch(1);
    return agocuda_launch_status();
}

extern "C" int agocuda_Remap_F32_Bilinear_Constant_batch(void *stream, int n, int W, int H, float *pDst, long long dstBatch,
                                                         int dstStride, int srcW, int srcH, const float *pSrc,
                                                         long long srcBatch, int srcStride, const float *pField,
                                                         long long fieldBatch, int fieldStride, float border)
{
    if (!pDst || !pSrc || !pField || !batch_ok(n, W, H, srcW, srcH) || dstStride < W || srcStride < srcW ||
        fieldStride < W || ((uintptr_t)pField & 7))
        return AGOCUDA_INVALID_PARAMS;
    const int rows = warp_rows(n, W, H, 4);
    k_warp_f32<kForward, 2><<<warp_grid(n, W, H, rows), 256, 0, as_stream(stream)>>>(
        W, H, rows, img32(pSrc, srcBatch, srcStride, srcW, srcH), img32(pDst, dstBatch, dstStride, W, H), Img32{}, pField,
        fieldBatch, fieldStride, border, Img32{}, nullptr);
    agocuda_count_launch(1);
    return agocuda_launch_status();
}

extern "C" int agocuda_Remap_F32_Bilinear_Constant_adjoint_batch(void *stream, int n, int W, int H, const float *pGradOut,
                                                                 long long goBatch, int goStride, int srcW, int srcH,
                                                                 const float *pSrc, long long srcBatch, int srcStride,
                                                                 const float *pField, long long fieldBatch, int fieldStride,
                                                                 float border, float *pGradSrc, float *pGradField)
{
    if (!pGradOut || !pSrc || !pField || !pGradSrc || !pGradField || !batch_ok(n, W, H, srcW, srcH) || goStride < W ||
        srcStride < srcW || fieldStride < W || ((uintptr_t)pField & 7) || ((uintptr_t)pGradField & 7))
        return AGOCUDA_INVALID_PARAMS;
    const int rows = warp_rows(n, W, H, 32);
    k_warp_f32<kAdjoint, 2><<<warp_grid(n, W, H, rows), 256, 0, as_stream(stream)>>>(
        W, H, rows, img32(pSrc, srcBatch, srcStride, srcW, srcH), Img32{}, img32(pGradOut, goBatch, goStride, W, H),
        pField, fieldBatch, fieldStride, border, img32(pGradSrc, srcBatch, srcStride, srcW, srcH), pGradField);
    agocuda_count_launch(1);
    return agocuda_launch_status();
}

extern "C" int agocuda_WarpPerspective_F32_Bilinear_Constant_batch(void *stream, int n, int W, int H, float *pDst,
                                                                   long long dstBatch, int dstStride, int srcW, int srcH,
                                                                   const float *pSrc, long long srcBatch, int srcStride,
                                                                   const float *theta, float border)
{
    if (!pDst || !pSrc || !theta || !batch_ok(n, W, H, srcW, srcH) || dstStride < W || srcStride < srcW)
        return AGOCUDA_INVALID_PARAMS;
    const int rows = warp_rows(n, W, H, 4);
    k_warp_f32<kForward, 9><<<warp_grid(n, W, H, rows), 256, 0, as_stream(stream)>>>(
        W, H, rows, img32(pSrc, srcBatch, srcStride, srcW, srcH), img32(pDst, dstBatch, dstStride, W, H), Img32{}, theta, 0, 0,
        border, Img32{}, nullptr);
    agocuda_count_launch(1);
    return agocuda_launch_status();
}

extern "C" int agocuda_WarpPerspective_F32_Bilinear_Constant_adjoint_batch(void *stream, int n, int W, int H,
                                                                           const float *pGradOut, long long goBatch,
                                                                           int goStride, int srcW, int srcH,
                                                                           const float *pSrc, long long srcBatch,
                                                                           int srcStride, const float *theta, float border,
                                                                           float *pGradSrc, double *pGradTheta)
{
    if (!pGradOut || !pSrc || !theta || !pGradSrc || !pGradTheta || !batch_ok(n, W, H, srcW, srcH) || goStride < W ||
        srcStride < srcW)
        return AGOCUDA_INVALID_PARAMS;
    const int rows = warp_rows(n, W, H, 32);
    k_warp_f32<kAdjoint, 9><<<warp_grid(n, W, H, rows), 256, 0, as_stream(stream)>>>(
        W, H, rows, img32(pSrc, srcBatch, srcStride, srcW, srcH), Img32{}, img32(pGradOut, goBatch, goStride, W, H), theta, 0, 0,
        border, img32(pGradSrc, srcBatch, srcStride, srcW, srcH), pGradTheta);
    agocuda_count_launch(1);
    return agocuda_launch_status();
}

extern "C" int agocuda_WarpPerspective_F32_L2_step_batch(void *stream, int n, int W, int H, const float *pTarget,
                                                         long long tBatch, int tStride, int srcW, int srcH, const float *pSrc,
                                                         long long srcBatch, int srcStride, const float *theta, float border,
                                                         float *pGradSrc, double *pGradThetaLoss)
{
    if (!pTarget || !pSrc || !theta || !pGradSrc || !pGradThetaLoss || !batch_ok(n, W, H, srcW, srcH) || tStride < W ||
        srcStride < srcW)
        return AGOCUDA_INVALID_PARAMS;
    const int rows = warp_rows(n, W, H, 32);
    k_warp_f32<kFusedL2, 9><<<warp_grid(n, W, H, rows), 256, 0, as_stream(stream)>>>(
        W, H, rows, img32(pSrc, srcBatch, srcStride, srcW, srcH), Img32{}, img32(pTarget, tBatch, tStride, W, H), theta, 0, 0,
        border, img32(pGradSrc, srcBatch, srcStride, srcW, srcH), pGradThetaLoss);
    agocuda_count_launch(1);
    return agocuda_launch_status();
}
