// fast.cu -- vxFastCornersNode (org.khronos.openvx.fast_corners) on sm_100a: FAST-9 corners of
// a U8 image with and without non-maximum suppression, as a raster-ordered vx_keypoint_t list.
//
// Reference arithmetic (HafCpu_FastCorners_XY_U8_{NoSupression,Supression},
// ago_haf_cpu_fast_corners.cpp:414, :599): a pixel c is a corner when 9 contiguous pixels of
// the 16-pixel radius-3 circle are all > c + t or all < c - t (16-bit compares, t =
// floor(strength_threshold)).  Without suppression rows 3 .. H-4 and EVERY column are tested
// (the circle of the outer three columns reads across the row end in AGO's layout) and each
// corner's strength is the threshold.  With suppression rows 3 .. H-4 and columns 3 .. W-4
// get a strength -- the reference's binary search (:216) for the largest threshold that
// still gives a corner, which is (max over 9-arcs of the arc's minimum contrast) - 1 on each
// side, the larger side kept -- and a corner survives when its strength is >= its upper and
// left neighbours and > its right and lower ones.  The list is in raster order; the count
// scalar holds every corner, the array min(count, capacity).  The reference's GPU path
// appends with atomics; this one keeps the CPU path's order.
//
// Three launches: k_fast_tile (a 128x13 tile per CTA: circle tests on the four pixels of a word
// at once, strengths of the few corners from a compacted list, suppression inside the tile with
// a one-pixel halo; the corners as a bitmap, their strengths, and a count per tile row),
// k_fast_scan (one CTA: row offsets and counts) and k_fast_emit (a warp per row writes its
// keypoints at its offset, a lane per bitmap word).  A strength map in memory and a second pass
// for the suppression took 25 + 25 us per 1080p frame.
#include "agocuda_internal.cuh"

uint64_t agocuda_count_launch(unsigned n);

namespace {

constexpr int kFtX = 128, kFtY = 13, kFtHalo = 4;             // 15 tested rows of 34 words: 510 of 512 items
constexpr int kFtSW = kFtX + 2 * kFtHalo, kFtTH = kFtY + 2, kFtSH = kFtTH + 6;   // 136 bytes, 15 tested rows, 21 source rows
constexpr int kFtWords = kFtSW / 4;

__device__ __constant__ int8_t kCircleDx[16] = {0, 1, 2, 3, 3, 3, 2, 1, 0, -1, -2, -3, -3, -3, -2, -1};
__device__ __constant__ int8_t kCircleDy[16] = {-3, -3, -2, -1, 0, 1, 2, 3, 3, 3, 2, 1, 0, -1, -2, -3};

// bit i: circle pixels i .. i+8 (mod 16) all set in m
__device__ __forceinline__ bool arc9(uint32_t m)
{
    const uint32_t r = m | (m << 16);
    uint32_t a = r & (r >> 1);
    a &= a >> 2;
    a &= a >> 4;
    a &= r >> 8;
    return (a & 0xFFFFu) != 0;
}

// bit 7 of each byte: a > b (the average of a and ~b, rounded down, is at least 128)
__device__ __forceinline__ uint32_t gt4(uint32_t a, uint32_t b)
{
    const uint32_t n = ~b;
    return (a & n) + (((a ^ n) & 0xfefefefeu) >> 1);
}

// bit 7 of each byte: bit 7 set in nine consecutive words of the circle f
__device__ __forceinline__ uint32_t arc9x4(const uint32_t f[16])
{
    uint32_t a3[16], any = 0;
#pragma unroll
    for (int i = 0; i < 16; i++) a3[i] = f[i] & f[(i + 1) & 15] & f[(i + 2) & 15];
#pragma unroll
    for (int i = 0; i < 16; i++) any |= a3[i] & a3[(i + 3) & 15] & a3[(i + 6) & 15];
    return any;
}

// max over the 16 circular windows of 9 of the window minimum of d
__device__ __forceinline__ int best_arc_min(const int d[16])
{
    int m1[16], m2[16], m4[16];
#pragma unroll
    for (int i = 0; i < 16; i++) m1[i] = min(d[i], d[(i + 1) & 15]);
#pragma unroll
    for (int i = 0; i < 16; i++) m2[i] = min(m1[i], m1[(i + 2) & 15]);
#pragma unroll
    for (int i = 0; i < 16; i++) m4[i] = min(m2[i], m2[(i + 4) & 15]);
    int best = -1 << 20;
#pragma unroll
    for (int i = 0; i < 16; i++) best = max(best, min(m4[i], d[(i + 8) & 15]));
    return best;
}

// Corner flags of the four pixels of tile word q (columns x0-4+4q ..) of tested row tr (image row
// y0-1+tr): bit 7 of each byte of `plus` (brighter arc) and `minus`.
//
// PACKED (0 <= t <= kFtPackedMax): the tests c + t < p and p < c - t in byte lanes, with saturated
// bounds (a bound of 255 or 0 is never passed, as the unsaturated one); the arcs by ANDs of the 16
// circle words.  One pixel at a time takes 16 byte loads and 32 compares each; the thresholds that do
// are negative, or so large that the 16-bit sum c + t can wrap, below every pixel.
constexpr int kFtPackedMax = 32767 - 255;
template <bool PACKED>
__device__ __forceinline__ void fast_flags(const uint8_t (*tile)[kFtSW], int tr, int q, int t, uint32_t &plus, uint32_t &minus)
{
    if constexpr (PACKED) {
        uint32_t f[16], g[16], c = 0, hi = 0, lo = 0;
        const uint32_t T = (uint32_t)min(t, 255) * 0x01010101u;
        const int ql = max(q - 1, 0), qr = min(q + 1, kFtWords - 1);   // outer words: pixels that are not used
        auto row = [&](int dy, uint32_t w[3]) {
            const uint32_t *p = (const uint32_t *)tile[3 + tr + dy];
            w[0] = p[ql]; w[1] = p[q]; w[2] = p[qr];
        };
        auto at = [](const uint32_t w[3], int dx) {        // the four pixels dx columns to the right
            return dx == 0 ? w[1] : dx > 0 ? __funnelshift_r(w[1], w[2], 8 * dx) : __funnelshift_r(w[0], w[1], 32 + 8 * dx);
        };
        auto test = [&](int i, uint32_t v) { f[i] = gt4(v, hi); g[i] = gt4(lo, v); };
        uint32_t w[3];
        row(0, w);
        c = w[1];
        hi = __vaddus4(c, T);
        lo = __vsubus4(c, T);
        test(4, at(w, 3)); test(12, at(w, -3));
        row(-3, w); test(15, at(w, -1)); test(0, at(w, 0)); test(1, at(w, 1));
        row(3, w); test(9, at(w, -1)); test(8, at(w, 0)); test(7, at(w, 1));
        row(-2, w); test(14, at(w, -2)); test(2, at(w, 2));
        row(2, w); test(10, at(w, -2)); test(6, at(w, 2));
        row(-1, w); test(13, at(w, -3)); test(3, at(w, 3));
        row(1, w); test(11, at(w, -3)); test(5, at(w, 3));
        plus = arc9x4(f) & 0x80808080u;
        minus = arc9x4(g) & 0x80808080u;
    } else {
        plus = minus = 0;
        for (int j = 0; j < 4; j++) {
            const int cx = 4 * q + j, cy = 3 + tr;
            if (cx < kFtHalo - 1 || cx > kFtHalo + kFtX) continue;
            const int c = tile[cy][cx], hi = (int16_t)(c + t), lo = (int16_t)(c - t);
            uint32_t p = 0, m = 0;
#pragma unroll
            for (int i = 0; i < 16; i++) {
                const int b = tile[cy + kCircleDy[i]][cx + kCircleDx[i]];
                p |= (uint32_t)(b > hi) << i;
                m |= (uint32_t)(b < lo) << i;
            }
            plus |= arc9(p) ? 0x80u << (8 * j) : 0u;
            minus |= arc9(m) ? 0x80u << (8 * j) : 0u;
        }
    }
}

// Corners: with suppression of rows 3..H-4 and columns 3..W-4, without of rows 3..H-4 and every
// column.  bitmap: 4 words of a tile row; counts[tile column][row]; map: a corner's strength.
template <bool SUP, bool PACKED>
__global__ void __launch_bounds__(256) k_fast_tile(int W, int H, const uint8_t *src, int srcStride, int t, uint8_t *map, int mapStride,
                                                  uint32_t *bitmap, int words, uint32_t *counts)
{
    __shared__ __align__(16) uint8_t tile[kFtSH][kFtSW];
    __shared__ __align__(16) uint8_t str[kFtTH][kFtSW];
    __shared__ uint16_t list[kFtTH * kFtSW];               // tr * 136 + column, bit 14: brighter arc, bit 15: darker arc
    __shared__ uint32_t bits[kFtY][4];
    __shared__ int n;
    const int x0 = blockIdx.x * kFtX, y0 = blockIdx.y * kFtY, yT = y0 - 4, tid = threadIdx.x;
    const bool edge = x0 - kFtHalo < 0 || x0 + kFtX + kFtHalo > W || yT < 0 || yT + kFtSH > H;
    if (!edge) {
        for (int i = tid; i < kFtSH * kFtWords; i += 256) {
            const int r = i / kFtWords, w = i - r * kFtWords;
            *(uint32_t *)&tile[r][4 * w] = ldg_u32(src + (size_t)(yT + r) * srcStride + x0 - kFtHalo + 4 * w);
        }
    } else {
        // image-edge tiles: bytes as AGO's layout holds them (across row ends, zero outside)
        for (int i = tid; i < kFtSH * kFtSW; i += 256) {
            const int r = i / kFtSW, c = i - r * kFtSW;
            tile[r][c] = (uint8_t)ago_byte(src, (size_t)srcStride, W, H, yT + r, x0 - kFtHalo + c);
        }
    }
    for (int i = tid; i < kFtTH * kFtWords; i += 256) ((uint32_t *)&str[0][0])[i] = 0;
    if (tid < kFtY * 4) (&bits[0][0])[tid] = 0;
    if (tid == 0) n = 0;
    __syncthreads();
    for (int i = tid; i < kFtTH * kFtWords; i += 256) {
        const int tr = i / kFtWords, q = i - tr * kFtWords, y = y0 - 1 + tr;
        if (y < 3 || y >= H - 3 || (!SUP && (tr == 0 || tr == kFtTH - 1))) continue;
        uint32_t plus, minus;
        fast_flags<PACKED>(tile, tr, q, t, plus, minus);
        for (uint32_t m = plus | minus; m; m &= m - 1) {
            const int j = (__ffs(m) - 1) >> 3, c = 4 * q + j, x = x0 - kFtHalo + c;
            const bool wanted = SUP ? c >= kFtHalo - 1 && c <= kFtHalo + kFtX && x >= 3 && x < W - 3
                                    : c >= kFtHalo && c < kFtHalo + kFtX && x < W;
            if (!wanted) continue;
            const uint32_t p = (plus >> (8 * j + 7)) & 1, d = (minus >> (8 * j + 7)) & 1;
            list[atomicAdd(&n, 1)] = (uint16_t)(tr * kFtSW + c + (p << 14) + (d << 15));
        }
    }
    __syncthreads();
    const int corners = n;
    if constexpr (SUP) {
        for (int i = tid; i < corners; i += 256) {
            const uint32_t e = list[i];
            const int at = (int)(e & 0x3fff), tr = at / kFtSW, c = at - tr * kFtSW, v = tile[3 + tr][c];
            int d[16], sp = 0, sn = 0;
            if (e & 0x4000) {
#pragma unroll
                for (int k = 0; k < 16; k++) d[k] = (int)tile[3 + tr + kCircleDy[k]][c + kCircleDx[k]] - v;
                sp = max(best_arc_min(d) - 1, t);          // t: the search's lower end, reached where c + t wraps
            }
            if (e & 0x8000) {
#pragma unroll
                for (int k = 0; k < 16; k++) d[k] = v - (int)tile[3 + tr + kCircleDy[k]][c + kCircleDx[k]];
                sn = best_arc_min(d) - 1;
            }
            str[tr][c] = (uint8_t)max(sp, sn);
        }
        __syncthreads();
    }
    for (int i = tid; i < corners; i += 256) {
        const int at = (int)(list[i] & 0x3fff), tr = at / kFtSW, c = at - tr * kFtSW;
        if (tr == 0 || tr == kFtTH - 1 || c < kFtHalo || c >= kFtHalo + kFtX) continue;   // the halo's
        bool keep = true;
        if constexpr (SUP) {
            const uint8_t *s = &str[tr][c], *u = s - kFtSW, *d = s + kFtSW;
            const int v = s[0];
            keep = v && v >= u[-1] && v >= u[0] && v >= u[1] && v >= s[-1] && v > s[1] && v > d[-1] && v > d[0] && v > d[1];
            if (keep) map[(size_t)(y0 - 1 + tr) * mapStride + x0 - kFtHalo + c] = (uint8_t)v;
        }
        if (keep) atomicOr(&bits[tr - 1][(c - kFtHalo) >> 5], 1u << ((c - kFtHalo) & 31));
    }
    __syncthreads();
    if (tid < kFtY * 4) {
        const int r = tid >> 2, w = (x0 >> 5) + (tid & 3), y = y0 + r;
        uint32_t k = __popc(bits[r][tid & 3]);
        if (y < H && w < words) bitmap[(size_t)y * words + w] = bits[r][tid & 3];
        const unsigned quad = 0xfu << (tid & 28);          // the four words of the row
        k += __shfl_xor_sync(quad, k, 1);
        k += __shfl_xor_sync(quad, k, 2);
        if (y < H && (tid & 3) == 0) counts[(size_t)blockIdx.x * H + y] = k;
    }
}

// one CTA of 1024 threads: exclusive scan of the row counts; the totals
__global__ void __launch_bounds__(1024) k_fast_scan(int H, int tiles, const uint32_t *counts, uint32_t *rowStart, uint32_t capacity,
                                                   uint32_t *pCornerCount, uint32_t *pNumCorners)
{
    __shared__ uint32_t warpSum[32];
    const int per = (H + 1023) / 1024, tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int r0 = min(H, tid * per), r1 = min(H, r0 + per);
    auto row_count = [&](int r) {
        uint32_t c = 0;
#pragma unroll 8
        for (int k = 0; k < tiles; k++) c += counts[(size_t)k * H + r];
        return c;
    };
    uint32_t s = 0;
    for (int r = r0; r < r1; r++) {
        const uint32_t c = row_count(r);
        rowStart[r] = c;                                   // its count until the offsets are known
        s += c;
    }
    uint32_t inc = s;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t n = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += n;
    }
    if (lane == 31) warpSum[wid] = inc;
    __syncthreads();
    if (wid == 0) {
        uint32_t v = warpSum[lane], x = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t n = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += n;
        }
        warpSum[lane] = x - v;     // exclusive prefix of the warps
    }
    __syncthreads();
    uint32_t run = warpSum[wid] + inc - s;
    for (int r = r0; r < r1; r++) {
        const uint32_t c = rowStart[r];
        rowStart[r] = run;
        run += c;
    }
    if (tid == 1023) {
        const uint32_t total = warpSum[wid] + inc;
        if (pNumCorners) *pNumCorners = total;
        if (pCornerCount) *pCornerCount = min(total, capacity);
    }
}

template <bool SUP>
__global__ void __launch_bounds__(256) k_fast_emit(int W, int H, const uint8_t *map, int mapStride, const uint32_t *bitmap,
                                                  int words, const uint32_t *rowStart, uint32_t capacity,
                                                  vx_keypoint_like *corners, float threshold)
{
    const int y = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (y >= H) return;
    uint32_t at = rowStart[y];
    if (at >= capacity) return;
    for (int w0 = 0; w0 < words && at < capacity; w0 += 32) {
        uint32_t bits = w0 + lane < words ? bitmap[(size_t)y * words + w0 + lane] : 0;
        const uint32_t n = __popc(bits);
        uint32_t upTo = n;                                 // corners of the lanes up to this one
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t v = __shfl_up_sync(0xffffffffu, upTo, o);
            if (lane >= o) upTo += v;
        }
        for (uint32_t i = at + upTo - n; bits && i < capacity; i++, bits &= bits - 1) {
            const int x = 32 * (w0 + lane) + __ffs(bits) - 1;
            vx_keypoint_like k;
            k.x = x;
            k.y = y;
            k.strength = SUP ? (float)map[(size_t)y * mapStride + x] : threshold;
            k.scale = 0.f;
            k.orientation = 0.f;
            k.tracking_status = 1;
            k.error = 0.f;
            corners[i] = k;
        }
        at += __shfl_sync(0xffffffffu, upTo, 31);
    }
}

size_t align256(size_t v) { return (v + 255) & ~(size_t)255; }

struct FastScratch {
    uint8_t *map;
    uint32_t *bitmap, *counts, *rowStart;
    int mapStride, words, tiles;
    size_t bytes;
};

FastScratch fast_layout(uint32_t W, uint32_t H, void *base)
{
    FastScratch s{};
    s.mapStride = (int)((W + 15) & ~15u);
    s.words = (int)((W + 31) / 32);
    s.tiles = (int)((W + kFtX - 1) / kFtX);
    uint8_t *p = (uint8_t *)base;
    size_t o = 0;
    s.map = p + o; o += align256((size_t)s.mapStride * H);
    s.bitmap = (uint32_t *)(p + o); o += align256((size_t)s.words * H * 4);
    s.counts = (uint32_t *)(p + o); o += align256((size_t)s.tiles * H * 4);
    s.rowStart = (uint32_t *)(p + o); o += align256((size_t)H * 4);
    s.bytes = o;
    return s;
}

}  // namespace

extern "C" size_t agocuda_FastCorners_scratch_size(uint32_t width, uint32_t height)
{
    return fast_layout(width, height, nullptr).bytes;
}

extern "C" int agocuda_FastCorners_XY_U8(void *stream, uint32_t W, uint32_t H, const uint8_t *pSrc, uint32_t srcStride,
                                         float strengthThreshold, int32_t nonmaxSuppression, void *pCorners,
                                         uint32_t cornerCapacity, uint32_t *pCornerCount, uint32_t *pNumCorners,
                                         void *scratch, size_t scratchBytes)
{
    if (!pSrc || !scratch || W < 7 || H < 7 || W > (1u << 20) || H > (1u << 20) || srcStride < W || (srcStride & 3) ||
        ((uintptr_t)pSrc & 3) || ((uintptr_t)scratch & 255) || (cornerCapacity && !pCorners) ||
        !(strengthThreshold > -32768.f && strengthThreshold < 32768.f))
        return AGOCUDA_INVALID_PARAMS;
    const FastScratch s = fast_layout(W, H, scratch);
    if (scratchBytes < s.bytes) return AGOCUDA_INVALID_PARAMS;
    const int t = (int16_t)floorf(strengthThreshold);
    cudaStream_t q = as_stream(stream);
    const dim3 g1(div_up(W, kFtX), div_up(H, kFtY));
    const unsigned g2 = div_up(H, 8);
    vx_keypoint_like *kp = (vx_keypoint_like *)pCorners;
    const bool packed = t >= 0 && t <= kFtPackedMax;
    (nonmaxSuppression ? (packed ? k_fast_tile<true, true> : k_fast_tile<true, false>)
                       : (packed ? k_fast_tile<false, true> : k_fast_tile<false, false>))<<<g1, 256, 0, q>>>(
        (int)W, (int)H, pSrc, (int)srcStride, t, s.map, s.mapStride, s.bitmap, s.words, s.counts);
    k_fast_scan<<<1, 1024, 0, q>>>((int)H, s.tiles, s.counts, s.rowStart, cornerCapacity, pCornerCount, pNumCorners);
    if (nonmaxSuppression)
        k_fast_emit<true><<<g2, 256, 0, q>>>((int)W, (int)H, s.map, s.mapStride, s.bitmap, s.words, s.rowStart,
                                             cornerCapacity, kp, strengthThreshold);
    else
        k_fast_emit<false><<<g2, 256, 0, q>>>((int)W, (int)H, s.map, s.mapStride, s.bitmap, s.words, s.rowStart,
                                              cornerCapacity, kp, strengthThreshold);
    agocuda_count_launch(3);
    return agocuda_launch_status();
}
