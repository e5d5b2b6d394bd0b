// ssim2_device.cuh -- device-side data structures and per-pixel math of the
// B200 SSIMULACRA2 engine.  Shared by the kernels in ssim2_kernels.cu.
//
// Arithmetic is written with explicit fmaf() and the translation unit is
// compiled with -fmad=false, so every rounding step is the one written here
// (the CPU restatement of the same arithmetic reproduces it).
#pragma once
#include <type_traits>

#include <stdint.h>

namespace s2 {

constexpr int kScales = 6;
constexpr int kTileW = 120;          // output columns per fused tile (1920 = 16 tiles)
constexpr int kCols = kTileW + 8;    // columns incl. the 4-px halo on each side (one thread each)
constexpr int kBand = 64;            // rows per shift band (tiles never straddle one)
constexpr int kStep = 8;             // output rows per vertical / horizontal step
constexpr int kSegW = 8;             // output pixels per horizontal task (one f32 partial sum)
constexpr int kSegs = kTileW / kSegW;  // horizontal tasks per row (15)
constexpr int kStripMin = 16, kStripMid = 32, kStripMax = 64;  // tile heights (divide kBand)
constexpr int kPyrBlk = 64;          // scale-0 block edge of the prep kernel, ...
constexpr int kPyrBlkSmall = 32;     // ... and of its form for few blocks (multiples of 2^5)
constexpr float kC2 = 0.0009f;
constexpr int kDsLevels = 5;         // DSSIM scales (dssim-cuda/src/lib.rs:73)

enum Format { FMT_LINEAR_F32 = 0, FMT_SRGB8 = 1, FMT_NV12 = 2, FMT_RGB16 = 3, FMT_P016 = 4 };
enum Storage { ST_F32 = 0, ST_F16 = 1, ST_BF16 = 2 };

// FIR taps of the exact form of the recursive Gaussian (sigma 1.5, N = 5),
// |k| = 0..4, rounded to f32.  The engine re-derives them in double at start
// (ssim2_engine.cpp) and refuses to run if they differ.
#define S2_T0 0x1.0ef8d6p-2f
#define S2_T1 0x1.b413e8p-3f
#define S2_T2 0x1.bfd672p-4f
#define S2_T3 0x1.2700c8p-5f
#define S2_T4 0x1.347d7p-7f

// One pair as the kernels see it.
struct DevPair {
    const void *in[2];       // scale-0 input: ref, dis (NV12: Y plane)
    const void *in_uv[2];    // NV12 CbCr planes
    long long pitch[2];      // bytes
    int fmt, bits;
    int w[kScales], h[kScales];
    int nscales;             // scored scales (>= 1)
    int lp[kScales];         // element pitch of the XYB planes of scale s
    void *lvl[2][kScales];   // planar XYB of scales 0..nscales-1 (3 planes each)
    int tile_base[kScales];  // first global tile of each scale
    int tile_cnt[kScales];
    int blk_base;            // first pyramid block
    int blk_x, blk_y;        // pyramid blocks of this pair (of the submission's block edge)
    int status;
    int prep_mask;           // images the prep pass converts: bit 0 reference, bit 1 distorted
    // 4:2:0 YUV (NV12 / P016): y_coeff, r_coeff, b_coeff, g_coeff1, g_coeff2
    // of the pair's matrix, range and depth, the luma minimum and the chroma
    // neutral value (cuda-colorspace-kernel/src/lib.rs:46-203)
    float yuv[5];
    int yuv_min, yuv_neutral;
    int lvl_ext;             // images whose XYB planes live outside the submission (bit per image)
    // DSSIM, the sibling metric sharing this pyramid: the prep pass also
    // converts levels 0..lab_levels-1 to dssim-core's scaled Lab (3 f32
    // planes per level, pitch lp[s]) and, when DSSIM's later levels are
    // clamped to 8 pixels, keeps the linear RGB of level lab_levels-1 in
    // `keep` (3 planes, pitch lp[s]) for the clamp pass.
    float *lab[2][kDsLevels];
    float *keep[2];
    int lab_levels;          // 0: no Lab output
    int prep_levels;         // levels the prep pass builds (XYB and Lab)
};

// One pair as the DSSIM kernels see it.  Level sizes follow dssim-cuda
// (halved rounding up, never below 8: dssim-cuda/src/lib.rs:184-205).
struct DsPair {
    float *lab[2][kDsLevels];    // 3 planes (L, a, b) per level, `pitch` floats per row
    float *map[kDsLevels];       // SSIM map per level, same pitch
    float *keep[2];              // clamp pass source: linear RGB of level clamp_from - 1
    float *scratch[2];           // clamp pass: two linear-RGB levels, 3 planes each
    long long splane;            // floats per plane of one scratch level
    int w[kDsLevels], h[kDsLevels], pitch[kDsLevels];
    int tile_base[kDsLevels], tile_cnt[kDsLevels];
    int kw, kh, kpitch;          // keep geometry
    int clamp_from;              // first level the clamp pass builds (kDsLevels: none)
    int prep_mask;
    int status;
};

// A run of DSSIM tiles (32 x 32 outputs), and of strips when the submission
// runs in them, of one (pair, level).
struct DsSeg {
    int first_tile;
    int pair;
    int level;
    int tiles_x;
    int first_strip;
};
constexpr int kDsStripW = 120;     // output columns of a strip
constexpr int kDsStripRows = 64;   // output rows of a strip
constexpr int kDsStripBlocks = 4;  // resident strips per SM
__host__ __device__ __forceinline__ int ds_strips_x(int w) { return (w + kDsStripW - 1) / kDsStripW; }

// A run of tiles of one (pair, scale); tiles are numbered across segments.
struct Seg {
    int first_tile;
    int pair;
    int scale;
    int tiles_x;
    int strip_rows;
};

// A run of S2_BLUR_IIR_REF blocks of one (pair, scale): one per (32 columns,
// channel) of the vertical walk, one per (32 rows, channel) of the horizontal.
struct IirSeg {
    int first;     // first block
    int pair;
    int scale;
    int rec_base;  // first row record of this (pair, scale) in the partial sums
    float *v;      // the 15 vertical-walk output planes of this (pair, scale)
};

struct DevResult {
    double score;
    double stats[108];
    double sums[108];
    int n_scales;
    int status;
    double dssim;                // DSSIM of the pair (NaN when not scored)
    double dssim_scale[kDsLevels];  // per-level 1 - mean |avg - ssim|
};

// ---------------------------------------------------------------------------
// colour math
// ---------------------------------------------------------------------------


// Opsin absorbance (crates/ssimulacra2-cuda-kernel/src/xyb.rs:3-36).
#define S2_M00 0.30f
#define S2_M02 0.078f
#define S2_M10 0.23f
#define S2_M12 0.078f
#define S2_M20 0.24342269f
#define S2_M21 0.20476745f
#define S2_B0 0.0037930734f
#define S2_B0_ROOT 0.1559542025327239180319220163705f

// Cube root of x >= 0 (0 for x <= 0 or NaN).  Newton iteration on the
// reciprocal cube root, r <- r + r (1 - x r^3) / 3, which needs no division,
// from the exponent-thirds bit-manipulation seed of W. Kahan ("Computing a
// real cube root", 1991); then y = x r^2 and one Newton correction of y.
// Only IEEE multiplies and fused multiply-adds, and no branches, so every
// platform rounds the same way.  Two iterations from the ~3% seed leave
// ~1e-5, which the final correction squares away: <= 1 ulp over
// [1e-30, 1e30] (checked in the tests).
// i / 3 for i < 2^31 (the bits of a non-negative float) as one high multiply:
// 0x55555556 = (2^32 + 2) / 3, so the high word of i * 0x55555556 is
// floor(i / 3 + 2 i / (3 * 2^32)), and the added fraction is below 1/3.
__device__ __forceinline__ unsigned s2_div3(unsigned i) { return __umulhi(i, 0x55555556u); }

__device__ __forceinline__ float s2_cbrtf(float x) {
    const bool pos = x > 0.0f, tiny = x < 0x1p-100f;
    float xs = tiny ? x * 0x1p102f : x;
    xs = pos ? xs : 1.0f;
    float r = __uint_as_float(0x54a2fa8cu - s2_div3(__float_as_uint(xs)));
    const float third = 0x1.555556p-2f;
#pragma unroll
    for (int k = 0; k < 2; k++) {
        float t = xs * r;
        t = t * r;
        t = t * r;
        r = fmaf(r * third, 1.0f - t, r);
    }
    float y = xs * r;
    y = y * r;
    const float e = fmaf(y * y, y, -xs);
    const float c = (r * r) * third;
    y = fmaf(-e, c, y);
    y = y * (tiny ? 0x1p-34f : 1.0f);
    return pos ? y : 0.0f;
}

// ---- the XYB cube root --------------------------------------------------
// Correctly rounded in all but a few cases per 10^5 (<= 1 ulp always): a
// seed r ~ x^(-1/3) from the SFU, 2^(-log2(x) / 3) (lg2.approx / ex2.approx,
// about 4e-7 relative), y = x r^2, and one Newton step for y^3 = x whose
// residual y^3 - x is formed with y^2 split exactly into hi + lo (the
// FMA-based TwoProduct of Ogita, Rump and Oishi, "Accurate sum and dot
// product", 2005), so the step's error is second order in the seed's: the
// result then no longer depends on how the seed was found, and a CPU can
// check it against the correctly rounded cube root.  (s2_cbrtf above, with a
// plain residual, is within an ulp but its last bit follows its seed.)
__device__ __forceinline__ float s2_rcbrt_sfu(float x) {
    float l, r;
    asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(l) : "f"(x));
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(l * -0x1.555556p-2f));
    return r;
}

__device__ __forceinline__ float s2_cbrt_step(float x, float r) {
    float y = x * r;
    y = y * r;
    const float hi = y * y;
    const float lo = fmaf(y, y, -hi);  // y^2 = hi + lo exactly
    float e = fmaf(hi, y, -x);
    e = fmaf(lo, y, e);  // y^3 - x
    const float c = (r * r) * 0x1.555556p-2f;  // 1 / (3 y^2)
    return fmaf(-e, c, y);
}

// x in [2^-100, 2^100] (the opsin values of non-negative linear RGB, which
// are >= the bias 0.0038)
__device__ __forceinline__ float s2_cbrtf_unit(float x) { return s2_cbrt_step(x, s2_rcbrt_sfu(x)); }

// any x: 0 for x <= 0 or NaN; tiny x scaled by 2^102 and the root by 2^-34
__device__ __forceinline__ float s2_cbrtf_xyb(float x) {
    const bool pos = x > 0.0f, tiny = x < 0x1p-100f;
    float xs = tiny ? x * 0x1p102f : x;
    xs = pos ? xs : 1.0f;
    const float y = s2_cbrt_step(xs, s2_rcbrt_sfu(xs)) * (tiny ? 0x1p-34f : 1.0f);
    return pos ? y : 0.0f;
}

// dssim-core's scaled Lab of one linear-RGB pixel, with the reference GPU's
// f32 operations: fused multiply-adds where dssim-cuda-kernel/src/lab.rs:42-86
// uses mul_add, IEEE divisions, a cube root above the CIE threshold and the
// linear segment below it (lab.rs:37-44).  The cube root is s2_cbrtf (within
// an ulp, like the math library's the reference calls), whose IEEE-only
// operations the CPU restatement reproduces bit for bit: the SSIM map's
// variance terms amplify ulp-level differences of the Lab values.
__device__ __forceinline__ float ds_lab_f(float t) {
    return t > 216.0f / 24389.0f ? s2_cbrtf(t) : fmaf(24389.0f / (27.0f * 116.0f), t, 16.0f / 116.0f);
}

__device__ __forceinline__ void ds_lab(float r, float g, float b, float o[3]) {
    const float x = fmaf(0.4124f, r, fmaf(0.3576f, g, 0.1805f * b)) / 0.9505f;
    const float y = fmaf(0.2126f, r, fmaf(0.7152f, g, 0.0722f * b)) / 1.0f;
    const float z = fmaf(0.0193f, r, fmaf(0.1192f, g, 0.9505f * b)) / 1.089f;
    const float fx = ds_lab_f(x), fy = ds_lab_f(y), fz = ds_lab_f(z);
    o[0] = (fy - 16.0f / 116.0f) * 1.05f;
    o[1] = fmaf(fx - fy, 500.0f / 220.0f, 86.2f / 220.0f);
    o[2] = fmaf(fy - fz, 200.0f / 220.0f, 107.9f / 220.0f);
}

// a / b for b > 0 normal (the error-map denominators: >= 9e-4 and >= 1).
// The reciprocal comes from the SFU approximation (PTX rcp.approx.ftz.f32,
// at most 1 ulp from 1/b); the quotient q = a r then gets one residual
// correction q + (a - b q) r, the final step of Markstein's division
// (P. Markstein, "IA-64 and Elementary Functions", 2000): the residual
// a - b q is exact under FMA, so the corrected quotient is within
// 0.5 ulp + 2^-23 of the residual's weight -- the IEEE quotient except in
// rare near-halfway cases.  4 instructions instead of a division's
// multi-instruction sequence with its slow path.
__device__ __forceinline__ float s2_div(float a, float b) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(b));
    const float q = a * r;
    const float e = fmaf(-b, q, a);
    return fmaf(e, r, q);
}

// KUNIT: the argument is known >= 0.0038 (non-negative linear RGB).
template <bool KUNIT>
__device__ __forceinline__ float opsin_row(int g, float r, float gg, float b) {
    const float m01 = 1.0f - S2_M02 - S2_M00;
    const float m11 = 1.0f - S2_M12 - S2_M10;
    const float m22 = 1.0f - S2_M20 - S2_M21;
    float v;
    if (g == 0)
        v = fmaf(S2_M00, r, fmaf(m01, gg, fmaf(S2_M02, b, S2_B0)));
    else if (g == 1)
        v = fmaf(S2_M10, r, fmaf(m11, gg, fmaf(S2_M12, b, S2_B0)));
    else
        v = fmaf(S2_M20, r, fmaf(S2_M21, gg, fmaf(m22, b, S2_B0)));
    if (KUNIT) return s2_cbrtf_unit(v) - S2_B0_ROOT;
    return s2_cbrtf_xyb(v) - S2_B0_ROOT;
}

// XYB channel g from the three opsin cube roots (xyb.rs:42-78).
__device__ __forceinline__ float xyb_from_opsin(int g, float rg, float gr, float bb) {
    float y = 0.5f * (rg + gr);
    if (g == 0) return fmaf(0.5f * (rg - gr), 14.0f, 0.42f);
    if (g == 1) return y + 0.01f;
    return (bb - y) + 0.55f;
}

// ---- two pixels at once (sm_100 f32x2 operations; each lane rounds exactly
// as the scalar operation, so these return the scalar functions' results) --
__device__ __forceinline__ float2 s2_f2(float a) { return make_float2(a, a); }
__device__ __forceinline__ float2 s2_neg2(float2 a) { return make_float2(-a.x, -a.y); }

// s2_cbrtf of two values at once (f32x2 where both lanes do the same
// operation; each lane rounds as the scalar steps).  The product that
// 1 - t subtracts is formed by two scalar multiplies: a packed product
// feeding a packed add would be fused into one rounding.
__device__ __forceinline__ float2 s2_cbrtf2(float2 x) {
    const bool p0 = x.x > 0.0f, p1 = x.y > 0.0f, t0 = x.x < 0x1p-100f, t1 = x.y < 0x1p-100f;
    float2 xs = make_float2(t0 ? x.x * 0x1p102f : x.x, t1 ? x.y * 0x1p102f : x.y);
    xs = make_float2(p0 ? xs.x : 1.0f, p1 ? xs.y : 1.0f);
    float2 r = make_float2(__uint_as_float(0x54a2fa8cu - s2_div3(__float_as_uint(xs.x))),
                           __uint_as_float(0x54a2fa8cu - s2_div3(__float_as_uint(xs.y))));
    const float2 third = s2_f2(0x1.555556p-2f);
#pragma unroll
    for (int k = 0; k < 2; k++) {
        float2 t = __fmul2_rn(xs, r);
        t = __fmul2_rn(t, r);
        t = make_float2(t.x * r.x, t.y * r.y);
        r = __ffma2_rn(__fmul2_rn(r, third), __fadd2_rn(s2_f2(1.0f), s2_neg2(t)), r);
    }
    float2 y = __fmul2_rn(xs, r);
    y = __fmul2_rn(y, r);
    const float2 e = __ffma2_rn(__fmul2_rn(y, y), y, s2_neg2(xs));
    const float2 c = __fmul2_rn(__fmul2_rn(r, r), third);
    y = __ffma2_rn(s2_neg2(e), c, y);
    y = __fmul2_rn(y, make_float2(t0 ? 0x1p-34f : 1.0f, t1 ? 0x1p-34f : 1.0f));
    return make_float2(p0 ? y.x : 0.0f, p1 ? y.y : 0.0f);
}

__device__ __forceinline__ float2 ds_lab_f2(float2 t) {
    const float thr = 216.0f / 24389.0f;
    const float2 c = s2_cbrtf2(t);
    const float2 l = __ffma2_rn(s2_f2(24389.0f / (27.0f * 116.0f)), t, s2_f2(16.0f / 116.0f));
    return make_float2(t.x > thr ? c.x : l.x, t.y > thr ? c.y : l.y);
}

// ds_lab of two pixels (lanes), each lane rounding as ds_lab: the products
// of the colour matrix feed the addends of FMAs, never a packed add.
__device__ __forceinline__ void ds_lab2(float2 r, float2 g, float2 b, float2 o[3]) {
    const float2 xn = __ffma2_rn(s2_f2(0.4124f), r, __ffma2_rn(s2_f2(0.3576f), g, __fmul2_rn(s2_f2(0.1805f), b)));
    const float2 y = __ffma2_rn(s2_f2(0.2126f), r, __ffma2_rn(s2_f2(0.7152f), g, __fmul2_rn(s2_f2(0.0722f), b)));
    const float2 zn = __ffma2_rn(s2_f2(0.0193f), r, __ffma2_rn(s2_f2(0.1192f), g, __fmul2_rn(s2_f2(0.9505f), b)));
    const float2 fx = ds_lab_f2(make_float2(xn.x / 0.9505f, xn.y / 0.9505f));
    const float2 fy = ds_lab_f2(y);
    const float2 fz = ds_lab_f2(make_float2(zn.x / 1.089f, zn.y / 1.089f));
    o[0] = __fmul2_rn(__fadd2_rn(fy, s2_f2(-(16.0f / 116.0f))), s2_f2(1.05f));
    o[1] = __ffma2_rn(__fadd2_rn(fx, s2_neg2(fy)), s2_f2(500.0f / 220.0f), s2_f2(86.2f / 220.0f));
    o[2] = __ffma2_rn(__fadd2_rn(fy, s2_neg2(fz)), s2_f2(200.0f / 220.0f), s2_f2(107.9f / 220.0f));
}


// Packed f32x2 arithmetic (__fmul2_rn, __fadd2_rn, __ffma2_rn): each lane
// rounds as the scalar operation, but the compiler contracts a packed
// multiply whose result feeds a packed add into one fused multiply-add (one
// rounding instead of two), even in a -fmad=false build (measured on sm_100a
// with CUDA 12.9).  So no packed product here feeds a packed sum: products
// that are summed are formed by scalar multiplies (never contracted under
// -fmad=false), or the sum is the addend of a packed FMA, or the product is
// exact (a multiplication by 0.5).
// The same operations as inline PTX (add / mul / fma .rn.f32x2).  Each lane
// rounds as the scalar operation -- but the assembler, too, was measured to
// fuse a packed multiply whose result feeds a packed add into one fused
// multiply-add (a probe over 1.7e7 operand triples on sm_100a, CUDA 12.9:
// every case where the two roundings differ from one came out fused).  So
// here as well no packed product feeds a packed sum: the fused tile pass
// feeds products to the multiplicand or addend of an explicit FMA, or sums
// the two lanes of a product with a scalar add.
__device__ __forceinline__ float2 s2_padd(float2 a, float2 b) {
    float2 d;
    asm("{.reg .b64 ra, rb, rd;\n\tmov.b64 ra, {%2, %3};\n\tmov.b64 rb, {%4, %5};\n\t"
        "add.rn.f32x2 rd, ra, rb;\n\tmov.b64 {%0, %1}, rd;}"
        : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return d;
}
__device__ __forceinline__ float2 s2_pmul(float2 a, float2 b) {
    float2 d;
    asm("{.reg .b64 ra, rb, rd;\n\tmov.b64 ra, {%2, %3};\n\tmov.b64 rb, {%4, %5};\n\t"
        "mul.rn.f32x2 rd, ra, rb;\n\tmov.b64 {%0, %1}, rd;}"
        : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return d;
}
__device__ __forceinline__ float2 s2_pfma(float2 a, float2 b, float2 c) {
    float2 d;
    asm("{.reg .b64 ra, rb, rc, rd;\n\tmov.b64 ra, {%2, %3};\n\tmov.b64 rb, {%4, %5};\n\t"
        "mov.b64 rc, {%6, %7};\n\tfma.rn.f32x2 rd, ra, rb, rc;\n\tmov.b64 {%0, %1}, rd;}"
        : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
    return d;
}

__device__ __forceinline__ float2 s2_mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 s2_add2(float2 a, float2 b) { return __fadd2_rn(a, b); }

// The negated quotients -(a.x / b.x, a.y / b.y) by s2_div's steps on both
// lanes, with the reciprocals of -b: r' = -r, q' = a r' = -q, e = b q' + a =
// a - b q, e r' + q' = -(e r + q); each step rounds to the negation of the
// scalar step's result (round-to-nearest is symmetric, and so is the
// hardware reciprocal), so -n is s2_div of each lane.
__device__ __forceinline__ float2 s2_div2_neg(float2 a, float2 b) {
    float2 r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r.x) : "f"(-b.x));
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r.y) : "f"(-b.y));
    const float2 q = s2_pmul(a, r);
    const float2 e = s2_pfma(b, q, a);
    return s2_pfma(e, r, q);
}

// BT.709 inverse OETF (crates/cuda-colorspace-kernel/src/lib.rs:223-238) of
// two samples: ((v + (alpha - 1)) / alpha)^(1/0.45) from the threshold on,
// v / 4.5 below; the two divisions are multiplications by the f32 reciprocals
// 1/alpha and 2/9 (<= 1 ulp from dividing), and both branches are evaluated and
// selected.  p^(1/0.45) = p^(20/9) with p = m 2^e, m in [1, 2): m^(20/9) is a
// degree-7 polynomial in t = m - 1.5 (Chebyshev interpolation at 8 nodes,
// converted to monomials and rounded to f32; Horner with fmaf), times
// 2^(20e/9), one f32 constant per exponent (a power of two times a rounded
// 2^(r/9)); <= 3.3 ulp on [0.1, 2].
//
// pw: s2_pow_table() of every exponent field, sign bit included, so that no
// value needs a clamp before the lookup: the selected branch has p >= 0.164
// (e >= -3), and where p >= 2 the factor only has to give a result above 1.
// An entry also holds 2^-e, which turns p into m in the multiply-add that
// forms t (exact; picking m's bits out of p took a logic instruction more).
//
// SAT: the result clamped to [0, 1] (the 4:2:0 family), which the last
// multiplications do for nothing.  Without SAT the power's base is clamped to
// [1/8, 1.5], its value for samples beyond the nominal range.
constexpr int kPowTable = 512;
__host__ __device__ __forceinline__ float2 s2_pow_table(int field) {
    if (field < 124 || field > 255) return make_float2(0.0f, 0.0f);
    if (field > 127) return make_float2(4.0f, 0.5f);
    return field == 127 ? make_float2(1.0f, 1.0f)
                        : (field == 126 ? make_float2(0x1.b6e8aep-3f, 2.0f)
                                        : (field == 125 ? make_float2(0x1.784086p-5f, 4.0f)
                                                        : make_float2(0x1.428a3p-7f, 8.0f)));
}

template <bool SAT>
__device__ __forceinline__ float2 bt709_eotf2(float2 v, const float2 *pw) {
    const float thr = 0.08124285829863521110029445797874f;
    // alpha - 1 and 1 / alpha, alpha = 1 + 5.5 * 0.018053968510807
    float2 q = s2_mul2(s2_add2(v, s2_f2(0x1.96b84p-4f)), s2_f2(0x1.d1c096p-1f));
    if (!SAT) q = make_float2(fminf(fmaxf(q.x, 0.125f), 1.5f), fminf(fmaxf(q.y, 0.125f), 1.5f));
    const float2 fx = pw[__float_as_uint(q.x) >> 23], fy = pw[__float_as_uint(q.y) >> 23];
    const float2 t = make_float2(fmaf(q.x, fx.y, -1.5f), fmaf(q.y, fy.y, -1.5f));
    float2 y = __ffma2_rn(s2_f2(0x1.1eb37ap-12f), t, s2_f2(-0x1.88e318p-11f));
    y = __ffma2_rn(y, t, s2_f2(0x1.2713a6p-9f));
    y = __ffma2_rn(y, t, s2_f2(-0x1.37717ep-7f));
    y = __ffma2_rn(y, t, s2_f2(0x1.2c9724p-4f));
    y = __ffma2_rn(y, t, s2_f2(0x1.7c6f02p+0f));
    y = __ffma2_rn(y, t, s2_f2(0x1.d2e55cp+1f));
    y = __ffma2_rn(y, t, s2_f2(0x1.3b279ep+1f));
    const float slope = 0x1.c71c72p-3f;
    if (SAT) {
        const float hx = __saturatef(y.x * fx.x), hy = __saturatef(y.y * fy.x);
        const float lx = __saturatef(v.x * slope), ly = __saturatef(v.y * slope);
        return make_float2(v.x >= thr ? hx : lx, v.y >= thr ? hy : ly);
    }
    const float2 hi = make_float2(y.x * fx.x, y.y * fy.x), lo = s2_mul2(v, s2_f2(slope));
    return make_float2(v.x >= thr ? hi.x : lo.x, v.y >= thr ? hi.y : lo.y);
}

// s2_cbrtf_unit of both lanes (each lane rounds as the scalar steps: no
// packed product feeds a packed sum)
__device__ __forceinline__ float2 s2_cbrtf_unit2(float2 x) {
    float2 l, r;  // s2_rcbrt_sfu of both lanes
    asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(l.x) : "f"(x.x));
    asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(l.y) : "f"(x.y));
    l = s2_mul2(l, s2_f2(-0x1.555556p-2f));
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r.x) : "f"(l.x));
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r.y) : "f"(l.y));
    float2 y = s2_mul2(x, r);
    y = s2_mul2(y, r);
    const float2 hi = s2_mul2(y, y);
    // the two subtractions as scalar FMAs, whose operands negate for nothing
    // (a packed operand takes a logic instruction per lane to negate)
    const float2 lo = make_float2(fmaf(y.x, y.x, -hi.x), fmaf(y.y, y.y, -hi.y));
    float2 e = make_float2(fmaf(hi.x, y.x, -x.x), fmaf(hi.y, y.y, -x.y));
    e = __ffma2_rn(lo, y, e);
    const float2 nc = s2_mul2(s2_mul2(r, r), s2_f2(-0x1.555556p-2f));
    return __ffma2_rn(e, nc, y);
}

// XYB of two pixels of non-negative linear RGB (opsin_row<true> and
// xyb_from_opsin per lane): out[c] = (pixel a, pixel b) of channel c.
__device__ __forceinline__ void xyb_pair_unit(float2 r, float2 g, float2 b, float2 out[3]) {
    const float m01 = 1.0f - S2_M02 - S2_M00;
    const float m11 = 1.0f - S2_M12 - S2_M10;
    const float m22 = 1.0f - S2_M20 - S2_M21;
    const float2 v0 = __ffma2_rn(s2_f2(S2_M00), r, __ffma2_rn(s2_f2(m01), g, __ffma2_rn(s2_f2(S2_M02), b, s2_f2(S2_B0))));
    const float2 v1 = __ffma2_rn(s2_f2(S2_M10), r, __ffma2_rn(s2_f2(m11), g, __ffma2_rn(s2_f2(S2_M12), b, s2_f2(S2_B0))));
    const float2 v2 = __ffma2_rn(s2_f2(S2_M20), r, __ffma2_rn(s2_f2(S2_M21), g, __ffma2_rn(s2_f2(m22), b, s2_f2(S2_B0))));
    const float2 nroot = s2_f2(-S2_B0_ROOT);
    const float2 rg = s2_add2(s2_cbrtf_unit2(v0), nroot);
    const float2 gr = s2_add2(s2_cbrtf_unit2(v1), nroot);
    const float2 bb = s2_add2(s2_cbrtf_unit2(v2), nroot);
    const float2 y = s2_mul2(s2_f2(0.5f), s2_add2(rg, gr));
    // a - b as b * -1 + a: one rounding, that of the subtraction
    out[0] = __ffma2_rn(s2_mul2(s2_f2(0.5f), __ffma2_rn(gr, s2_f2(-1.0f), rg)), s2_f2(14.0f), s2_f2(0.42f));
    out[1] = s2_add2(y, s2_f2(0.01f));
    out[2] = s2_add2(__ffma2_rn(y, s2_f2(-1.0f), bb), s2_f2(0.55f));
}

struct ColorConsts {
    // BT.2020 -> BT.709 linear matrix (row-major)
    float m2020[9];
};

template <typename T> __device__ __forceinline__ float ld_store(const T *p);
template <> __device__ __forceinline__ float ld_store<float>(const float *p) { return __ldg(p); }
template <typename T> __device__ __forceinline__ T to_store(float v);
template <> __device__ __forceinline__ float to_store<float>(float v) { return v; }

// A 2x2 quad of linear RGB: [row][channel], lanes = left and right pixel.
struct Quad {
    float2 c[2][3];
};

// Sample `i` (0 low half, 1 high half) of a word of two samples of ES bytes,
// plus 2^23, as a float: the sample is the float's low mantissa bits, and
// subtracting 2^23 (exact) leaves it (a conversion would go through the SFU).
template <int ES>
__device__ __forceinline__ float s2_sample(unsigned w, int i) {
    return __uint_as_float(__byte_perm(w, 0x4b000000u, ES == 1 ? (i ? 0x7441 : 0x7440) : (i ? 0x7432 : 0x7410)));
}
constexpr float kSample0 = 8388608.0f;

// RGB16: two pixels (words lo: r0 g0, mid: b0 r1, hi: g1 b1) of samples of
// `bits` bits, BT.709/BT.2020 inverse OETF, then BT.2020 -> BT.709 primaries,
// clamped >= 0.  inv = 1 / (2^bits - 1) in f32.  The scaled samples are scalar
// products: the OETF adds to them.
__device__ __forceinline__ void rgb16_linear2(unsigned lo, unsigned mid, unsigned hi, float inv, const ColorConsts &cc,
                                              const float2 *pw, float2 o[3]) {
    const float2 r = make_float2((s2_sample<2>(lo, 0) - kSample0) * inv, (s2_sample<2>(mid, 1) - kSample0) * inv);
    const float2 g = make_float2((s2_sample<2>(lo, 1) - kSample0) * inv, (s2_sample<2>(hi, 0) - kSample0) * inv);
    const float2 b = make_float2((s2_sample<2>(mid, 0) - kSample0) * inv, (s2_sample<2>(hi, 1) - kSample0) * inv);
    const float2 p0 = bt709_eotf2<false>(r, pw), p1 = bt709_eotf2<false>(g, pw), p2 = bt709_eotf2<false>(b, pw);
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const float *m = cc.m2020 + 3 * k;
        const float2 v = __ffma2_rn(s2_f2(m[0]), p0, __ffma2_rn(s2_f2(m[1]), p1, __fmul2_rn(s2_f2(m[2]), p2)));
        o[k] = make_float2(fmaxf(v.x, 0.0f), fmaxf(v.y, 0.0f));
    }
}

// The six samples of a 4:2:0 quad (x, y even): luma of rows y and y + 1 and
// the shared CbCr pair, two samples per word (low half = left sample / Cb).
// ES = bytes per sample (1 NV12, 2 P016); read as one word per pair when the
// plane bases and the pitch are aligned to it (always for the engine's own
// staging), else sample by sample.
struct Nv12Quad {
    unsigned y0, y1, uv;
};
template <int ES>
__device__ __forceinline__ Nv12Quad yuv_load_quad(const DevPair &P, int img, int x, int y) {
    using W = typename std::conditional<ES == 1, unsigned short, unsigned>::type;
    using S = typename std::conditional<ES == 1, uint8_t, uint16_t>::type;
    const char *yp = (const char *)P.in[img] + (long long)y * P.pitch[img] + ES * x;
    const char *uv = (const char *)P.in_uv[img] + (long long)(y >> 1) * P.pitch[img] + ES * x;
    Nv12Quad q;
    if ((((unsigned long long)P.in[img] | (unsigned long long)P.in_uv[img] | (unsigned long long)P.pitch[img]) &
         (2 * ES - 1)) == 0) {
        q.y0 = __ldg((const W *)yp);
        q.y1 = __ldg((const W *)(yp + P.pitch[img]));
        q.uv = __ldg((const W *)uv);
    } else {
        const S *a = (const S *)yp, *b = (const S *)(yp + P.pitch[img]), *c = (const S *)uv;
        q.y0 = (unsigned)__ldg(a) | ((unsigned)__ldg(a + 1) << (8 * ES));
        q.y1 = (unsigned)__ldg(b) | ((unsigned)__ldg(b + 1) << (8 * ES));
        q.uv = (unsigned)__ldg(c) | ((unsigned)__ldg(c + 1) << (8 * ES));
    }
    return q;
}

// Limited / full range YUV of the pair's matrix (cuda-colorspace-kernel/src/
// biplanar.rs:8-70: nearest chroma, luma floored at the range minimum, BT.709
// inverse OETF, clamp to [0, 1]) of a loaded quad.
template <int ES>
__device__ __forceinline__ void yuv_quad_linear(const Nv12Quad &q, const DevPair &P, const float2 *pw, Quad &o) {
    const float neutral = kSample0 + (float)P.yuv_neutral, ymin = kSample0 + (float)P.yuv_min, yc = P.yuv[0];
    const float cb = s2_sample<ES>(q.uv, 0) - neutral, cr = s2_sample<ES>(q.uv, 1) - neutral;
    const float ar = P.yuv[1] * cr;
    const float ag = fmaf(P.yuv[3], cb, P.yuv[4] * cr);
    const float ab = P.yuv[2] * cb;
#pragma unroll
    for (int row = 0; row < 2; row++) {
        const unsigned w = row ? q.y1 : q.y0;
        // scalar products: luma is summed with the chroma terms below
        const float2 luma = make_float2(fmaxf(s2_sample<ES>(w, 0) - ymin, 0.0f) * yc,
                                        fmaxf(s2_sample<ES>(w, 1) - ymin, 0.0f) * yc);
        o.c[row][0] = bt709_eotf2<true>(s2_add2(luma, s2_f2(ar)), pw);
        o.c[row][1] = bt709_eotf2<true>(s2_add2(luma, s2_f2(ag)), pw);
        o.c[row][2] = bt709_eotf2<true>(s2_add2(luma, s2_f2(ab)), pw);
    }
}

// Linear RGB of the 2x2 quad whose top-left pixel is (x, y) (inside the
// image) for the packed formats.  A column or row outside the image (vx / vy
// false) is not read: it repeats the left pixel, the upper row.  lut: the
// sRGB8 table; pw: the s2_pow_table.
template <int FMT>
__device__ __forceinline__ void lin_quad(const DevPair &P, int img, int x, int y, bool vx, bool vy, const float *lut,
                                         const float2 *pw, const ColorConsts &cc, Quad &o) {
    // a complete row of the quad whose rows are aligned for the format's word
    // size is read as three words: sRGB8 16-bit, RGB16 32-bit, linear f32
    // 64-bit (x is even: the row pair starts 6, 12 or 24 bytes x/2 in)
    constexpr int kAlign = FMT == FMT_SRGB8 ? 2 : (FMT == FMT_RGB16 ? 4 : 8);
    const bool words = vx && ((((unsigned long long)P.in[img]) | (unsigned long long)P.pitch[img]) & (kAlign - 1)) == 0;
    const float inv = FMT == FMT_RGB16 ? 1.0f / (float)((1 << P.bits) - 1) : 0.0f;
    const int right = vx ? 3 : 0;  // samples from the left pixel to the right one
#pragma unroll
    for (int row = 0; row < 2; row++) {
        const char *rp = (const char *)P.in[img] + (long long)(y + (vy ? row : 0)) * P.pitch[img];
        if (FMT == FMT_SRGB8) {
            unsigned w0, w1, w2;
            if (words) {
                const unsigned short *q = (const unsigned short *)(rp + 3 * x);
                w0 = __ldg(q), w1 = __ldg(q + 1), w2 = __ldg(q + 2);
            } else {
                const uint8_t *q = (const uint8_t *)rp + 3 * x;
                w0 = __ldg(q) | (unsigned)__ldg(q + 1) << 8;
                w1 = __ldg(q + 2) | (unsigned)__ldg(q + right) << 8;
                w2 = __ldg(q + right + 1) | (unsigned)__ldg(q + right + 2) << 8;
            }
            o.c[row][0] = make_float2(lut[w0 & 0xffu], lut[w1 >> 8]);
            o.c[row][1] = make_float2(lut[w0 >> 8], lut[w2 & 0xffu]);
            o.c[row][2] = make_float2(lut[w1 & 0xffu], lut[w2 >> 8]);
        } else if (FMT == FMT_RGB16) {
            unsigned w0, w1, w2;
            if (words) {
                const unsigned *q = (const unsigned *)(rp + 6 * x);
                w0 = __ldg(q), w1 = __ldg(q + 1), w2 = __ldg(q + 2);
            } else {
                const uint16_t *q = (const uint16_t *)rp + 3 * x;
                w0 = __ldg(q) | (unsigned)__ldg(q + 1) << 16;
                w1 = __ldg(q + 2) | (unsigned)__ldg(q + right) << 16;
                w2 = __ldg(q + right + 1) | (unsigned)__ldg(q + right + 2) << 16;
            }
            rgb16_linear2(w0, w1, w2, inv, cc, pw, o.c[row]);
        } else {
            float2 a, b, c;
            if (words) {
                const float2 *q = (const float2 *)(rp + 12 * x);
                a = __ldg(q), b = __ldg(q + 1), c = __ldg(q + 2);
            } else {
                const float *q = (const float *)rp + 3 * x;
                a = make_float2(__ldg(q), __ldg(q + 1));
                b = make_float2(__ldg(q + 2), __ldg(q + right));
                c = make_float2(__ldg(q + right + 1), __ldg(q + right + 2));
            }
            o.c[row][0] = make_float2(a.x, b.y);
            o.c[row][1] = make_float2(a.y, c.x);
            o.c[row][2] = make_float2(b.x, c.y);
        }
    }
}

// Sum of the exact-form FIR taps over the valid positions around x in
// [0, n) (the blur's response to a constant 1 under zero padding), rounded
// to f32: exactly 1.0f in the interior, where all nine taps are inside.
// Prefix sums S[m] = t0 + ... + tm of the double-precision taps.
// (The prefix sums are picked by selects: an indexed local array would be
// built in local memory on every call.)
__device__ __forceinline__ double border_prefix(int k) {
    return k == 0 ? 0x1.0ef8d5c79cdafp-2
                  : (k == 1 ? 0x1.e902c9b3e2946p-2
                            : (k == 2 ? 0x1.2c7c332eb15f4p-1 : (k == 3 ? 0x1.3eec3fae31770p-1 : 0x1.43be3571e736ap-1)));
}
__device__ __forceinline__ float border_gain(int x, int n) {
    int lo = min(x, 4), hi = min(n - 1 - x, 4);
    if (lo == 4 && hi == 4) return 1.0f;
    double s = border_prefix(lo) + border_prefix(hi);
    return (float)(s - 0x1.0ef8d5c79cdafp-2);
}

}  // namespace s2
