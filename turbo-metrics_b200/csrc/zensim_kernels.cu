// zensim_kernels.cu -- the zensim feature extraction of crates/zensim-cuda on
// sm_100a: positive XYB at the SIMD-padded width, a 4-scale box pyramid of
// the padded planes, and per (scale, channel) the radius-5 box blurs and the
// 17 pooled sums + 3 maxima from which the host forms the 228 features.
//
//   zs_prep_kernel   sRGB8 through the reference table, opsin mix, the Halley
//                    cube root of cbrtf_fast, positive XYB (color.rs:70-149);
//                    padding columns take the XYB of their mirror column
//                    (lib.rs:236-252, pad.rs); then the 2x2 box means of
//                    every smaller scale (downscale.rs:21-43, source clamped
//                    at the far edge), one launch per image
//   zs_walk_kernel   the vertical running sums (features.rs:83-193), whose
//                    f32 value depends on every row above: one block walks 32
//                    columns of one (scale, channel) from top to bottom and
//                    saves the four sums every 8 rows
//   zs_feat_kernel   one block per 64 x 32 tile of a (scale, channel): each
//                    thread takes one column and 8 rows, starts from the
//                    saved sums and slides them down its rows exactly as one
//                    walk of the whole column would; per pixel the SSIM,
//                    edge, high-frequency and MSE terms (features.rs:102-176)
//                    go to 17 f64 sums and 3 maxima
//   zs_reduce_kernel per (scale, channel): the tiles' sums in a fixed order
//
// The reference walks every column in one thread, and so did the first form
// of this pass (one thread = one column, with the horizontal sums, the error
// maps and the f64 sums on the walk): a 1080p pair then had 177 blocks of 64
// threads and took 2154 us, waiting on its own chain.  Only the four running
// sums are a chain (two dependent adds per row); with their state saved every
// 8 rows everything else runs in parallel at the same f32 roundings.  Per
// 1080p pair now (B200, each kernel alone, cold): prep 24 us per image (49 + 17
// us as four launches), walk 73 us (its row loads' latency and the barrier per
// chunk), features 104 us (issue: 290 instructions per pixel and channel, of
// them 96 for the horizontal sums, 17 f64 adds and 17 conversions), reduce 10 us.
//
// Sums are reduced in a fixed order -- where the reference adds each column
// with a float atomic -- so results do not depend on scheduling.
//
// Compiled with -fmad=false: every fused multiply-add is explicit (fmaf where
// the reference uses mul_add), divisions are IEEE (__fdiv_rn).
#include <cuda_runtime.h>
#include <stdint.h>

#include "dependent_launch.cuh"
#include "zensim_kernels.h"

namespace zs {

__device__ float g_lut[256];

__device__ __forceinline__ int mirror(int i, int n) {
    if (n <= 1) return 0;
    const int period = 2 * (n - 1);
    const int m = ((i % period) + period) % period;
    return m < n ? m : period - m;
}

// cbrtf_fast (color.rs:70-91): bit seed, two Halley steps
__device__ __forceinline__ float cbrt_fast(float x) {
    if (x == 0.0f) return 0.0f;
    const unsigned ui = __float_as_uint(x);
    const unsigned hx = (ui & 0x7fffffffu) / 3u + 709958130u;
    float t = __uint_as_float((ui & 0x80000000u) | hx);
    float r = t * t * t;
    t = t * __fdiv_rn(fmaf(x, 2.0f, r), fmaf(r, 2.0f, x));
    r = t * t * t;
    t = t * __fdiv_rn(fmaf(x, 2.0f, r), fmaf(r, 2.0f, x));
    return t;
}

// bias: -cbrt_fast(B0), the same for every pixel
__device__ __forceinline__ void positive_xyb(float r, float g, float b, float bias, float o[3]) {
    const float M02 = 0.078f, M00 = 0.30f, M01 = 1.0f - M02 - M00;
    const float M12 = 0.078f, M10 = 0.23f, M11 = 1.0f - M12 - M10;
    const float M20 = 0.24342269f, M21 = 0.20476745f, M22 = 1.0f - M20 - M21;
    const float B0 = 0.0037930734f;
    const float m0 = fmaxf(fmaf(M00, r, fmaf(M01, g, fmaf(M02, b, B0))), 0.0f);
    const float m1 = fmaxf(fmaf(M10, r, fmaf(M11, g, fmaf(M12, b, B0))), 0.0f);
    const float m2 = fmaxf(fmaf(M20, r, fmaf(M21, g, fmaf(M22, b, B0))), 0.0f);
    const float c0 = cbrt_fast(m0) + bias, c1 = cbrt_fast(m1) + bias, c2 = cbrt_fast(m2);
    const float xv = 0.5f * (c0 - c1), yv = 0.5f * (c0 + c1), bv = c2 - yv;
    o[0] = fmaf(xv, 14.0f, 0.42f);
    o[1] = yv + 0.01f;
    o[2] = bv + 0.55f;
}

// The columns that the box sums of a row of n read beyond its ends repeat
// their mirror columns (n >= 8): each is stored with the column it repeats.
__device__ __forceinline__ void store_mirrored(float *row, int x, int n, float v) {
    if (x >= 1 && x <= kZsRadius) row[-x] = v;
    if (x <= n - 2 && x >= n - 1 - kZsRadius) row[2 * (n - 1) - x] = v;
}

// ---------------------------------------------------------------------------
// prep: one block = 64 x 16 pixels of the padded scale-0 plane, one 2x2 quad
// per thread; the smaller scales of the block follow in shared memory.  The
// padded width is a multiple of 16, so only the bottom row can lack a
// neighbour.  The sRGB table lies in shared memory (in constant memory the 32
// lanes' different indexes were read one after the other: 49 us of 66 us per
// 1080p image went to the scale-0 pass).
// ---------------------------------------------------------------------------
constexpr int kPrepW = 64, kPrepH = 16, kPrepT = (kPrepW / 2) * (kPrepH / 2);

__global__ void __launch_bounds__(kPrepT) zs_prep_kernel(const uint8_t *__restrict__ img, size_t pitch, int w, int h,
                                                         const __grid_constant__ ZsPlan plan, int which,
                                                         float bias) {
    __shared__ float lut[256];
    __shared__ float lv[2][3][kPrepT];  // scale-1 block (32 x 8), then scale 2 (16 x 4)
    const int t = threadIdx.x;
    static_assert(kPrepT == 256, "one table entry per thread");
    lut[t] = g_lut[t];
    __syncthreads();
    const int qx = t % (kPrepW / 2), qy = t / (kPrepW / 2);
    const int x = blockIdx.x * kPrepW + 2 * qx, y = blockIdx.y * kPrepH + 2 * qy;
    const ZsPlanes &o0 = which ? plan.sc[0].dis : plan.sc[0].ref;
    const bool on = x < o0.n && y < h, vy = y + 1 < h;
    float m[3] = {0.0f, 0.0f, 0.0f};
    if (on) {
        const int xa = x < w ? x : mirror(x, w), xb = x + 1 < w ? x + 1 : mirror(x + 1, w);
        float q[4][3];
#pragma unroll
        for (int row = 0; row < 2; row++) {
            if (row && !vy) {  // the missing row repeats the one above
#pragma unroll
                for (int c = 0; c < 3; c++) q[2][c] = q[0][c], q[3][c] = q[1][c];
                break;
            }
            const uint8_t *r = img + (size_t)(y + row) * pitch;
            const uint8_t *a = r + 3 * (size_t)xa, *b = r + 3 * (size_t)xb;
            positive_xyb(lut[__ldg(a)], lut[__ldg(a + 1)], lut[__ldg(a + 2)], bias, q[2 * row]);
            positive_xyb(lut[__ldg(b)], lut[__ldg(b + 1)], lut[__ldg(b + 2)], bias, q[2 * row + 1]);
#pragma unroll
            for (int c = 0; c < 3; c++) {
                float *dst = o0.p[c] + (size_t)(y + row) * o0.pitch;
                *(float2 *)(dst + x) = make_float2(q[2 * row][c], q[2 * row + 1][c]);
                store_mirrored(dst, x, o0.n, q[2 * row][c]);
                store_mirrored(dst, x + 1, o0.n, q[2 * row + 1][c]);
            }
        }
#pragma unroll
        for (int c = 0; c < 3; c++) {
            float v = q[0][c] + q[1][c];
            v = v + q[2][c];
            v = v + q[3][c];
            m[c] = v * 0.25f;
        }
    }
    if (plan.ns > 1 && on) {
        const ZsPlanes &o = which ? plan.sc[1].dis : plan.sc[1].ref;
#pragma unroll
        for (int c = 0; c < 3; c++) {
            float *dst = o.p[c] + (size_t)(y >> 1) * o.pitch;
            dst[x >> 1] = m[c];
            store_mirrored(dst, x >> 1, o.n, m[c]);
            lv[0][c][t] = m[c];
        }
    }
    for (int s = 2; s < plan.ns; s++) {
        __syncthreads();
        const int bw = kPrepW >> s, bh = kPrepH >> s, pw = bw * 2;
        const ZsPlanes &o = which ? plan.sc[s].dis : plan.sc[s].ref;
        const int ox = blockIdx.x * bw + t % bw, oy = blockIdx.y * bh + t / bw;
        if (t < bw * bh && ox < o.n && oy < plan.sc[s].h) {
            const int ya = t / bw * 2, yb = 2 * oy + 1 < plan.sc[s - 1].h ? ya + 1 : ya, xa = t % bw * 2;
#pragma unroll
            for (int c = 0; c < 3; c++) {
                const float *p = lv[s & 1][c];
                float v = p[ya * pw + xa] + p[ya * pw + xa + 1];
                v = v + p[yb * pw + xa];
                v = v + p[yb * pw + xa + 1];
                v = v * 0.25f;
                float *dst = o.p[c] + (size_t)oy * o.pitch;
                dst[ox] = v;
                store_mirrored(dst, ox, o.n, v);
                lv[(s & 1) ^ 1][c][t] = v;
            }
        }
    }
}

// ---------------------------------------------------------------------------
// horizontal box sums (blur.rs:40-96) of four adjacent columns
// ---------------------------------------------------------------------------
constexpr float kInv = 1.0f / (float)(2 * kZsRadius + 1);

// out[p][j]: the scaled sum p of column x + j, j < 4 (x a multiple of 4) --
// the sums of s, t, s^2 + t^2 and s t over the columns x + j - 5 .. x + j + 5
// of the rows a (reference) and d (distorted), added left to right as the
// reference adds them.  The rows carry their mirrored columns on both sides,
// so no tap needs an index of its own.  A sample's products are formed once
// for the four columns.  Scalar adds: as f32x2 pairs (s, t) and
// (s^2 + t^2, s t) the sums took half the adds but as many moves to build the
// register pairs.
__device__ __forceinline__ void hsum4(const float *a, const float *d, int x, float4 out[4]) {
    float o[4][4];
#pragma unroll
    for (int q = 0; q < 5; q++) {
        const float4 f = *(const float4 *)(a + x - 8 + 4 * q), g = *(const float4 *)(d + x - 8 + 4 * q);
        const float av[4] = {f.x, f.y, f.z, f.w}, dv[4] = {g.x, g.y, g.z, g.w};
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int k = 4 * q + i;  // column x - 8 + k; columns x - 5 .. x + 8 are used
            if (k < 3 || k > 16) continue;
            const float s = av[i], t = dv[i];
            const float ss = s * s, tt = t * t, st = s * t;
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const int tap = k - 3 - j;
                if (tap == 0) o[0][j] = s, o[1][j] = t, o[2][j] = ss + tt, o[3][j] = st;
                if (tap > 0 && tap < 2 * kZsRadius + 1) {
                    o[0][j] = o[0][j] + s;
                    o[1][j] = o[1][j] + t;
                    o[2][j] = o[2][j] + ss;
                    o[2][j] = o[2][j] + tt;
                    o[3][j] = o[3][j] + st;
                }
            }
        }
    }
#pragma unroll
    for (int p = 0; p < 4; p++) out[p] = make_float4(o[p][0] * kInv, o[p][1] * kInv, o[p][2] * kInv, o[p][3] * kInv);
}

// ---------------------------------------------------------------------------
// walk: the running sums of 32 columns of one (scale, channel), all rows
//
// Warps 4..11 form the horizontal sums of 32 rows at a time (thread = one row,
// four columns) into a ring of such chunks in shared memory; warps 0..3
// (one sum each, lane = column) slide the chunk before down: (sum + entering
// row) - leaving row.  One barrier per chunk; the chain's two dependent adds
// per row run beside the next chunk's sums.
// ---------------------------------------------------------------------------
constexpr int kChunk = 32, kRingRows = 4 * kChunk;  // three chunks are live; a power of two
constexpr size_t kWalkSmem = sizeof(float) * 4 * kRingRows * kZsWalkW;
constexpr int kWalkThreads = 128 + kChunk * (kZsWalkW / 4);

__global__ void __launch_bounds__(kWalkThreads, 3) zs_walk_kernel(const __grid_constant__ ZsPlan plan) {
    extern __shared__ __align__(16) float smem[];
    dep::grid_wait();  // both pyramids are written
    float(*ring)[kRingRows][kZsWalkW] = (float(*)[kRingRows][kZsWalkW])smem;
    int s = 0;
    while (s + 1 < plan.ns && (int)blockIdx.x >= plan.sc[s + 1].walk_first) s++;
    const ZsScale &S = plan.sc[s];
    const int b = blockIdx.x - S.walk_first, ch = b / S.walk_x, x0 = (b - ch * S.walk_x) * kZsWalkW;
    const int n = S.n, h = S.h, t = threadIdx.x;
    const int chunks = (h + kChunk - 1) / kChunk;
    const int nsub = (h + kZsSub - 1) / kZsSub, ylast = kZsSub * (nsub - 1);
    const size_t pitch = S.ref.pitch;
    const float *A = S.ref.p[ch], *D = S.dis.p[ch];
    if (t >= 128) {
        const int r = (t - 128) / (kZsWalkW / 4), c = 4 * ((t - 128) % (kZsWalkW / 4)), x = x0 + c;
        const bool on = x < n;
        for (int it = 0; it <= chunks; it++) {
            const int y = it * kChunk + r;
            if (it < chunks && y < h && on) {
                float4 o[4];
                hsum4(A + (size_t)y * pitch, D + (size_t)y * pitch, x, o);
#pragma unroll
                for (int p = 0; p < 4; p++) *(float4 *)&ring[p][y % kRingRows][c] = o[p];
            }
            __syncthreads();
        }
        return;
    }
    const int p = t >> 5, lane = t & 31, x = x0 + lane;
    const float *R = &ring[p][0][lane];
    float *out = S.state + ((size_t)ch * nsub * 4 + p) * pitch + x;
    float sum = 0.0f;
    int y = 0;  // sum: the window of row y
    auto row = [&](int i) -> const float & { return R[(i & (kRingRows - 1)) * kZsWalkW]; };
    for (int it = 0; it <= chunks; it++) {
        if (it > 0) {
            if (it == 1) {
                for (int k = 0; k < 2 * kZsRadius + 1; k++) sum += row(k < kZsRadius ? kZsRadius - k : k - kZsRadius);
                if (x < n) out[0] = sum;
            }
            // the chunks before `it` hold the rows below `have`; rows past
            // the bottom are mirrored, so the last chunk serves every row left
            const int have = it * kChunk;
            while (y < ylast && (y + kZsSub - 1 + kZsRadius + 1 < have || have >= h)) {
                float in[kZsSub], lv[kZsSub];
                if (y > 0 && y + 2 * kZsSub <= h) {
                    // rows y - 8 .. y + 15, in whole groups of 8 of the ring
                    static_assert(kZsSub == 8 && kZsRadius == 5 && kRingRows % 8 == 0, "rows per group");
                    const float *g0 = &row(y - 8), *g1 = &row(y), *g2 = &row(y + 8);
#pragma unroll
                    for (int k = 0; k < kZsSub; k++) {
                        in[k] = k < 2 ? g1[(k + 6) * kZsWalkW] : g2[(k - 2) * kZsWalkW];
                        lv[k] = k < 5 ? g0[(k + 3) * kZsWalkW] : g1[(k - 5) * kZsWalkW];
                    }
                } else {
#pragma unroll
                    for (int k = 0; k < kZsSub; k++) {
                        const int e = y + k + kZsRadius + 1, l = y + k - kZsRadius;
                        in[k] = row(e < h ? e : 2 * (h - 1) - e);
                        lv[k] = row(l >= 0 ? l : -l);
                    }
                }
#pragma unroll
                for (int k = 0; k < kZsSub; k++) sum = sum + in[k] - lv[k];
                y += kZsSub;
                if (x < n) out[(size_t)(y / kZsSub) * 4 * pitch] = sum;
            }
        }
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------
// features: one 64 x 32 tile of one (scale, channel)
//
// The tile's horizontal sums, with the 5 rows above and below that its
// windows reach, go to shared memory (42 rows for 32); then a thread slides
// the four sums from the saved state of its 8 rows.  f64 adds and their
// conversions are what is left: 17 of each per pixel.
// ---------------------------------------------------------------------------
constexpr int kFeatThreads = kZsTileW * (kZsTileH / kZsSub);
constexpr int kFeatRows = kZsTileH + 2 * kZsRadius;
constexpr int kFeatWarps = kFeatThreads / 32;
constexpr size_t kFeatSums = sizeof(float) * 4 * kFeatRows * kZsTileW;
constexpr size_t kFeatRed = sizeof(double) * kZsOut * kFeatWarps * 33;
constexpr size_t kFeatSmem = kFeatSums > kFeatRed ? kFeatSums : kFeatRed;

__global__ void __launch_bounds__(kFeatThreads, 3) zs_feat_kernel(const __grid_constant__ ZsPlan plan,
                                                                  double *__restrict__ out) {
    extern __shared__ __align__(16) float smem[];
    int s = 0;
    while (s + 1 < plan.ns && (int)blockIdx.x >= plan.sc[s + 1].tile_first) s++;
    const ZsScale &S = plan.sc[s];
    int b = blockIdx.x - S.tile_first;
    const int per = S.tiles_x * S.tiles_y, ch = b / per;
    b -= ch * per;
    const int ty = b / S.tiles_x, x0 = (b - ty * S.tiles_x) * kZsTileW, y0 = ty * kZsTileH;
    const int n = S.n, h = S.h, t = threadIdx.x;
    const size_t pitch = S.ref.pitch;
    const float *A = S.ref.p[ch], *D = S.dis.p[ch];
    const int ybase = y0 - kZsRadius;
    dep::grid_wait();  // the saved sums are written
    for (int i = t; i < kFeatRows * (kZsTileW / 4); i += kFeatThreads) {
        const int r = i / (kZsTileW / 4), c = 4 * (i % (kZsTileW / 4)), x = x0 + c, y = ybase + r;
        if (x >= n || y < 0 || y >= h) continue;
        float4 o[4];
        hsum4(A + (size_t)y * pitch, D + (size_t)y * pitch, x, o);
#pragma unroll
        for (int p = 0; p < 4; p++) *(float4 *)(smem + (p * kFeatRows + r) * kZsTileW + c) = o[p];
    }
    const int col = t % kZsTileW, x = x0 + col, ya = y0 + (t / kZsTileW) * kZsSub;
    double acc[kZsSums];
#pragma unroll
    for (int i = 0; i < kZsSums; i++) acc[i] = 0.0;
    float pk0 = 0.0f, pk1 = 0.0f, pk2 = 0.0f;
    const bool on = x < n && ya < h;
    float sm1 = 0.0f, sm2 = 0.0f, ssq = 0.0f, ss12 = 0.0f;
    if (on) {
        const int nsub = (h + kZsSub - 1) / kZsSub;
        const float *st = S.state + ((size_t)ch * nsub + ya / kZsSub) * 4 * pitch + x;
        sm1 = st[0], sm2 = st[pitch], ssq = st[2 * pitch], ss12 = st[3 * pitch];
    }
    __syncthreads();
    // one pixel: its terms, from the sums of its window
    auto pixel = [&](float sv, float dv) {
        const float C2 = 0.0009f;
        const float mu1 = sm1 * kInv, mu2 = sm2 * kInv, sq = ssq * kInv, s12 = ss12 * kInv;
        const float md = mu1 - mu2;
        const float num_m = fmaf(md, -md, 1.0f);
        const float num_s = fmaf(2.0f, fmaf(-mu1, mu2, s12), C2);
        const float den_s = fmaf(-mu2, mu2, fmaf(-mu1, mu1, sq)) + C2;
        const float sd_raw = 1.0f - __fdiv_rn(num_m * num_s, den_s);
        const float sd = sd_raw > 0.0f ? sd_raw : 0.0f;
        const float sd2 = sd * sd, sd4 = sd2 * sd2;
        acc[0] += (double)sd;
        acc[1] += (double)sd4;
        acc[2] += (double)sd2;
        acc[14] += (double)(sd4 * sd4);
        pk0 = sd > pk0 ? sd : pk0;
        const float vs = sv - mu1, vd = dv - mu2;
        const float d1 = fabsf(vs), d2 = fabsf(vd);
        const float ed = __fdiv_rn(1.0f + d2, 1.0f + d1) - 1.0f;
        const float art = ed > 0.0f ? ed : 0.0f, det = ed < 0.0f ? -ed : 0.0f;
        const float a2 = art * art, l2 = det * det, a4 = a2 * a2, l4 = l2 * l2;
        acc[3] += (double)art;
        acc[4] += (double)a4;
        acc[5] += (double)a2;
        acc[6] += (double)det;
        acc[7] += (double)l4;
        acc[8] += (double)l2;
        acc[15] += (double)(a4 * a4);
        acc[16] += (double)(l4 * l4);
        pk1 = art > pk1 ? art : pk1;
        pk2 = det > pk2 ? det : pk2;
        acc[10] += (double)(vs * vs);
        acc[11] += (double)(vd * vd);
        acc[12] += (double)d1;
        acc[13] += (double)d2;
        const float pd = sv - dv;
        acc[9] += (double)(pd * pd);
    };
    // slide the vertical window: (sum + entering row) - leaving row
    auto slide = [&](const float *in, const float *lv) {
        constexpr int plane = kFeatRows * kZsTileW;
        sm1 = sm1 + in[0] - lv[0];
        sm2 = sm2 + in[plane] - lv[plane];
        ssq = ssq + in[2 * plane] - lv[2 * plane];
        ss12 = ss12 + in[3 * plane] - lv[3 * plane];
    };
    if (on) {
        const float *pa = A + (size_t)ya * pitch + x, *pd = D + (size_t)ya * pitch + x;
        const float *sums = smem + (ya - ybase) * kZsTileW + col;
        if (ya >= kZsRadius && ya + kZsSub + kZsRadius <= h) {  // no mirrored row
            float sv = pa[0], dv = pd[0];
#pragma unroll 2
            for (int k = 0; k < kZsSub; k++) {
                const float s = sv, d = dv;
                if (k + 1 < kZsSub) pa += pitch, pd += pitch, sv = *pa, dv = *pd;
                pixel(s, d);
                if (k + 1 < kZsSub) slide(sums + (kZsRadius + 1) * kZsTileW, sums - kZsRadius * kZsTileW);
                sums += kZsTileW;
            }
        } else {
            for (int k = 0; k < kZsSub && ya + k < h; k++) {
                const int y = ya + k;
                pixel(pa[k * pitch], pd[k * pitch]);
                const int in = y + kZsRadius + 1 < h ? kZsRadius + 1 : 2 * (h - 1 - y) - (kZsRadius + 1);
                const int lv = y >= kZsRadius ? -kZsRadius : kZsRadius - 2 * y;
                if (k + 1 < kZsSub && y + 1 < h) slide(sums + in * kZsTileW, sums + lv * kZsTileW);
                sums += kZsTileW;
            }
        }
    }
    // fixed-order block reduction through shared memory: each (value, warp)'s
    // 32 lanes in order, then the warps in order; sums, and maxima for the peaks
    __syncthreads();  // the horizontal sums are no longer read
    double *red = (double *)smem;
    const int w = t >> 5, lane = t & 31;
#pragma unroll
    for (int i = 0; i < kZsSums; i++) red[(i * kFeatWarps + w) * 33 + lane] = acc[i];
    red[(17 * kFeatWarps + w) * 33 + lane] = (double)pk0;
    red[(18 * kFeatWarps + w) * 33 + lane] = (double)pk1;
    red[(19 * kFeatWarps + w) * 33 + lane] = (double)pk2;
    __syncthreads();
    double v = 0.0;
    const int i = t / kFeatWarps;
    if (i < kZsOut) {
        const double *q = red + t * 33;
        v = q[0];
#pragma unroll 8
        for (int k = 1; k < 32; k++) v = i < kZsSums ? v + q[k] : fmax(v, q[k]);
    }
    __syncthreads();
    if (i < kZsOut) red[t] = v;
    __syncthreads();
    if (t < kZsOut) {
        v = red[t * kFeatWarps];
        for (int k = 1; k < kFeatWarps; k++) v = t < kZsSums ? v + red[t * kFeatWarps + k] : fmax(v, red[t * kFeatWarps + k]);
        out[(size_t)blockIdx.x * kZsOut + t] = v;
    }
}

// per (scale, channel): the tiles' records, 48 strided runs per value added
// in order, then the runs in order
constexpr int kRuns = 48;

__global__ void __launch_bounds__(kZsOut *kRuns) zs_reduce_kernel(const __grid_constant__ ZsPlan plan,
                                                                  const double *__restrict__ in,
                                                                  double *__restrict__ out) {
    __shared__ double red[kRuns][kZsOut];
    dep::grid_wait();
    const ZsScale &S = plan.sc[blockIdx.x / 3];
    const int per = S.tiles_x * S.tiles_y, t = threadIdx.x, i = t % kZsOut, r = t / kZsOut;
    const double *q = in + ((size_t)S.tile_first + (size_t)(blockIdx.x % 3) * per) * kZsOut + i;
    double v = 0.0;
#pragma unroll 4
    for (int k = r; k < per; k += kRuns) v = i < kZsSums ? v + q[(size_t)k * kZsOut] : fmax(v, q[(size_t)k * kZsOut]);
    red[r][i] = v;
    __syncthreads();
    if (t < kZsOut) {
        v = red[0][t];
        for (int k = 1; k < kRuns; k++) v = t < kZsSums ? v + red[k][t] : fmax(v, red[k][t]);
        out[(size_t)blockIdx.x * kZsOut + t] = v;
    }
}

cudaError_t zs_configure() {
    const cudaError_t e =
        cudaFuncSetAttribute(zs_walk_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kWalkSmem);
    if (e != cudaSuccess) return e;
    return cudaFuncSetAttribute(zs_feat_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kFeatSmem);
}

cudaError_t zs_upload_lut(const float *lut256) { return cudaMemcpyToSymbol(g_lut, lut256, 256 * sizeof(float)); }

cudaError_t zs_launch_prep(const uint8_t *img, size_t pitch, int w, int h, const ZsPlan &plan, int which, float bias,
                           cudaStream_t st) {
    dim3 grid((plan.sc[0].n + kPrepW - 1) / kPrepW, (h + kPrepH - 1) / kPrepH);
    zs_prep_kernel<<<grid, kPrepT, 0, st>>>(img, pitch, w, h, plan, which, bias);
    return cudaGetLastError();
}

cudaError_t zs_launch_features(const ZsPlan &plan, double *tile_out, double *out, cudaStream_t st) {
    cudaError_t e = cudaSuccess;
    const int parts = plan.one_channel ? 3 * plan.ns : 1;
    for (int i = 0; i < parts && e == cudaSuccess; i++) {
        ZsPlan part = plan;
        double *part_out = tile_out;
        if (plan.one_channel) {
            // one channel of one scale as a plan of its own; its walk waits for
            // the features that read the states before it
            const int c = i % 3;
            ZsScale &S = part.sc[0] = plan.sc[i / 3];
            S.ref.p[0] = S.ref.p[c];
            S.dis.p[0] = S.dis.p[c];
            part.ns = 1;
            part.walk_blocks = S.walk_x;
            part.tiles = S.tiles_x * S.tiles_y;
            part_out += (size_t)kZsOut * (S.tile_first + c * part.tiles);
            S.walk_first = S.tile_first = 0;
        }
        e = dep::launch(true, zs_walk_kernel, dim3(part.walk_blocks), kWalkThreads, kWalkSmem, st, part);
        if (e == cudaSuccess)
            e = dep::launch(true, zs_feat_kernel, dim3(part.tiles), kFeatThreads, kFeatSmem, st, part, part_out);
    }
    if (e == cudaSuccess)
        e = dep::launch(true, zs_reduce_kernel, dim3(plan.ns * 3), kZsOut * kRuns, 0, st, plan, tile_out, out);
    return e;
}

}  // namespace zs
