// ssim2_iir.cu -- S2_BLUR_IIR_REF: the reference's own f32 arithmetic.
//
// The default blur of this engine is the exact closed form of the recursive
// Gaussian (a 9-tap FIR), which is far closer to the FP64 result than the
// reference's f32 recursion.  This mode instead reproduces the reference's
// recursion step for step, so that the 108 statistics match the arithmetic
// of crates/ssimulacra2-cuda:
//
//   iir_vertical_kernel    block per (32 columns, channel) of a (pair, scale): the
//                          walk of ssimulacra2-cuda-kernel/src/blur.rs:95-136
//                          (sum of the entering and leaving samples, three
//                          second-order recursions with the same FMA order,
//                          sum of the three outputs) down the column of one of
//                          the 15 blurred inputs (XYB of ref and dis, their
//                          squares and product, as NPP Mul forms them,
//                          ssimulacra2-cuda/src/lib.rs:868-886).  Output
//                          planes in HBM (the reference's img[3..7]).
//   iir_horizontal_kernel  block per (32 rows, channel): five warps (one per
//                          blurred plane, lane = row) walk along the rows of
//                          the five vertical outputs (the reference
//                          transposes and walks down again, lib.rs:911-947 --
//                          identical arithmetic), eleven more form the error
//                          maps of error_maps.rs:36-59 as written and the
//                          pooling of lib.rs:986-1016 (f64 sums of d and of
//                          the f32 (d*d)*(d*d)); one partial-sum record per 32 rows.
//
// What bounds them: a line is walked by one lane in order, and its warp issues
// a sample's instructions one after the other, most of them dependent.  Only
// one multiply-add of them is the recursion itself (about 4 cycles); the loads,
// products, window sum, three filters and output sum come to about 25 a sample
// in the vertical walk, issued 4 to 5 cycles apart: 115 cycles.  What was done
// is to keep memory latency and the maps off that stream.  One 1280x853 pair
// (B200, each kernel alone, cold): the vertical walk 50 us with its rows copied
// ahead (505 us with a load per step on the stream), the horizontal walk 91 us
// (1487 us as a thread per row and channel, whose five planes' loads were
// uncoalesced, with the maps on the stream): 139 cycles a sample, where the
// walkers and the helpers wait for one another at a barrier per 32 columns and
// a little over half of the issue slots are used.
//
// The XYB planes come from prep_kernel (same pyramid and XYB arithmetic as the
// reference, with the engine's own cube root); finalize_kernel reduces the row
// records in order.  The translation unit is compiled with -fmad=false: every
// FMA below is explicit, as in the reference (Rust never contracts).
#include "dependent_launch.cuh"
#include "ssim2_device.cuh"
#include "ssim2_launch.h"

namespace s2 {

// f32 recursion constants (ssimulacra2-cuda-kernel/build.rs:28-145 evaluated
// in double and rounded, as printed in examples/cpu.rs:931-948).
#define S2_MUL_IN_1 0x1.c4fa84p-5f
#define S2_MUL_IN_3 -0x1.e1fd7ap-5f
#define S2_MUL_IN_5 0x1.a8894ap-7f
#define S2_MUL_PREV_1 0x1.e6f0e2p+0f
#define S2_MUL_PREV_3 0x1.2cf23p+0f
#define S2_MUL_PREV_5 0x1.1a6264p-53f
#define S2_MUL_PREV2 (-1.0f)

struct IirState {
    float p1, p3, p5, q1, q3, q5;  // prev, prev2
    __device__ __forceinline__ void zero() { p1 = p3 = p5 = q1 = q3 = q5 = 0.f; }
    // one step of blur.rs:95-136; returns out_1 + out_3 + out_5
    __device__ __forceinline__ float step(float sum) {
        float o1 = sum * S2_MUL_IN_1, o3 = sum * S2_MUL_IN_3, o5 = sum * S2_MUL_IN_5;
        o1 = fmaf(S2_MUL_PREV2, q1, o1);
        o3 = fmaf(S2_MUL_PREV2, q3, o3);
        o5 = fmaf(S2_MUL_PREV2, q5, o5);
        q1 = p1;
        q3 = p3;
        q5 = p5;
        o1 = fmaf(S2_MUL_PREV_1, p1, o1);
        o3 = fmaf(S2_MUL_PREV_3, p3, o3);
        o5 = fmaf(S2_MUL_PREV_5, p5, o5);
        p1 = o1;
        p3 = o3;
        p5 = o5;
        return (o1 + o3) + o5;
    }
};

constexpr int kN = 5;  // radius of the recursion

__device__ __forceinline__ int find_iseg(const IirSeg *segs, int nseg, int t) {
    int lo = 0, hi = nseg - 1;
    while (lo < hi) {
        int mid = (lo + hi + 1) >> 1;
        if (segs[mid].first <= t) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// The vertical walk of one channel's five planes over 32 columns: warp =
// plane, lane = column.  The rows of both images are copied (cp.async, 16
// bytes) into a ring of four stages of 16 rows, three stages ahead, once for
// the five planes that are formed from them; the left sample, 10 rows back,
// is still in a register.  An output plane is stored as [32 columns][row]
// [column], so a walk's rows are 128 bytes apart (immediate offsets) and the
// horizontal walk's 32 x 32 chunk is one run of 4 KB.
constexpr int kVRows = 16, kVStages = 4, kVThreads = 160;

template <typename ST>
__global__ void __launch_bounds__(kVThreads) iir_vertical_kernel(const DevPair *__restrict__ pairs,
                                                                 const IirSeg *__restrict__ segs, int nseg) {
    static_assert(sizeof(ST) == 4, "16-byte copies of four samples");
    __shared__ __align__(16) float ring[kVStages][2][kVRows][32];
    const IirSeg sg = segs[find_iseg(segs, nseg, blockIdx.x)];
    const DevPair &P = pairs[sg.pair];
    const int s = sg.scale, W = P.w[s], H = P.h[s], lp = P.lp[s];
    const int local = blockIdx.x - sg.first;
    const int c = local % 3, x0 = local / 3 * 32;
    const int kind = threadIdx.x >> 5, lane = threadIdx.x & 31;  // x, y, x^2, y^2, xy
    const long long plane = (long long)lp * H;
    const ST *xr = (const ST *)P.lvl[0][s] + c * plane + x0, *xd = (const ST *)P.lvl[1][s] + c * plane + x0;
    // step i: right = i, left = i - 2N, output row y = i - N + 1
    const int batches = (H + kN - 1 + kVRows - 1) / kVRows;
    auto fetch = [&](int b) {  // rows b * 16 .. + 15 (the planes' pitch is a multiple of 64 samples)
        if (b < batches) {
            for (int i = threadIdx.x; i < 2 * kVRows * 8; i += kVThreads) {
                const int img = i / (kVRows * 8), r = i / 8 % kVRows, q = 4 * (i % 8), y = b * kVRows + r;
                if (y >= H) continue;
                const unsigned d = (unsigned)__cvta_generic_to_shared(&ring[b % kVStages][img][r][q]);
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d),
                             "l"((img ? xd : xr) + (long long)y * lp + q)
                             : "memory");
            }
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    const int ia = kind == 1 || kind == 3, ib = kind >= 3;
    const bool mul = kind >= 2, on = x0 + lane < W;
    float *dst = sg.v + (c * 5 + kind) * plane + (long long)x0 * H + lane;
    IirState st;
    st.zero();
    float tail[2 * kN];  // the last 2N samples of the batch before (0 before the start)
#pragma unroll
    for (int k = 0; k < 2 * kN; k++) tail[k] = 0.f;
    for (int b = 0; b < kVStages - 1; b++) fetch(b);
    for (int b = 0; b < batches; b++) {
        asm volatile("cp.async.wait_group %0;\n" ::"n"(kVStages - 2) : "memory");
        __syncthreads();  // batch b has landed for every warp, and batch b - 1 is walked
        fetch(b + kVStages - 1);
        const float *pa = &ring[b % kVStages][ia][0][lane], *pb = &ring[b % kVStages][ib][0][lane];
        float v[kVRows];
#pragma unroll
        for (int k = 0; k < kVRows; k++) {
            const float a = pa[k * 32];
            v[k] = mul ? a * pb[k * 32] : a;
        }
        float *d = dst + (long long)(b * kVRows - kN + 1) * 32;
        if (b > 0 && (b + 1) * kVRows <= H) {
#pragma unroll
            for (int k = 0; k < kVRows; k++) {
                const float out = st.step((k >= 2 * kN ? v[k - 2 * kN] : tail[k]) + v[k]);
                if (on) d[k * 32] = out;
            }
        } else {
#pragma unroll
            for (int k = 0; k < kVRows; k++) {
                const int i = b * kVRows + k, y = i - kN + 1;
                if (i >= H) v[k] = 0.f;
                const float out = st.step((k >= 2 * kN ? v[k - 2 * kN] : tail[k]) + v[k]);
                if (on && y >= 0 && y < H) d[k * 32] = out;
            }
        }
#pragma unroll
        for (int k = 0; k < 2 * kN; k++) tail[k] = v[kVRows - 2 * kN + k];
    }
}

// The horizontal walk: chunks of 32 columns of the block's 32 rows, the five
// planes copied two chunks ahead (cp.async, 16 bytes); the left sample, 10
// columns back, is still in a register, and the outputs replace the samples
// they were walked from.  Rows are 36 floats apart in shared memory, so the
// walk's 16-byte accesses (lane = row) and the maps' 4-byte ones (lane =
// column) both cover all banks.  While warps 0..4 walk chunk c, the eleven
// others issue the copies of chunk c + 2 and form the maps of chunk c - 1,
// whose XYB samples they loaded a chunk before; one barrier per chunk.  Both
// sides are dependent instructions (about one every five cycles a warp): with
// five helpers, and the copies on the walkers, the pass took 109 us instead
// of 91 us.
constexpr int kHc = 32, kHp = kHc + 4, kHSlots = 4;
constexpr int kHPlane = kHc * kHp;                     // floats of one plane of a chunk
constexpr int kWalkers = 5, kHelpers = 11;
constexpr int kHThreads = 32 * (kWalkers + kHelpers);
constexpr size_t kHSmem = sizeof(float) * 5 * kHSlots * kHPlane;

template <typename ST>
__global__ void __launch_bounds__(kHThreads, 2) iir_horizontal_kernel(const DevPair *__restrict__ pairs,
                                                                const IirSeg *__restrict__ segs, int nseg,
                                                             double *__restrict__ partials) {
    extern __shared__ __align__(16) float hsm[];
    __shared__ double red[kHelpers][6];
    dep::grid_wait();  // the vertical walk is done
    const IirSeg sg = segs[find_iseg(segs, nseg, blockIdx.x)];
    const DevPair &P = pairs[sg.pair];
    const int s = sg.scale, W = P.w[s], H = P.h[s], lp = P.lp[s];
    const int local = blockIdx.x - sg.first;
    const int c = local % 3, y0 = local / 3 * kHc, rows = min(kHc, H - y0);
    const long long plane = (long long)lp * H;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // step i of a row: right = i, left = i - 2N, output column x = i - N + 1
    const int chunks = (W + kN - 1 + kHc - 1) / kHc;
    const bool walker = warp < kWalkers;
    const int helper = warp - kWalkers;
    constexpr int kMapRows = (kHc + kHelpers - 1) / kHelpers;  // rows of a helper: helper, helper + kHelpers, ...
    // columns ch * 32 .. + 31 of the five planes' rows (what lies past a row's
    // end is replaced by zeros in the walk)
    const float *const v = sg.v + c * 5 * plane + (long long)y0 * 32;
    auto fetch = [&](int ch) {
        if (ch * kHc < W) {
            const int slot = ch % kHSlots;
            const float *q = v + (long long)ch * 32 * H;
            for (int i = threadIdx.x - 32 * kWalkers; i < 5 * kHc * 8; i += 32 * kHelpers) {
                const int p = i / (kHc * 8), r = i / 8 % kHc, x = 4 * (i % 8);
                if (r >= rows) continue;
                const unsigned d = (unsigned)__cvta_generic_to_shared(hsm + (p * kHSlots + slot) * kHPlane + r * kHp + x);
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(q + p * plane + r * 32 + x)
                             : "memory");
            }
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    IirState st;
    st.zero();
    double acc[6] = {0, 0, 0, 0, 0, 0};
    const float C2 = 0.0009f;
    float tail[2 * kN];  // the last 2N samples of the chunk before
#pragma unroll
    for (int k = 0; k < 2 * kN; k++) tail[k] = 0.f;
    float src[kMapRows], dis[kMapRows];
    const ST *xr = (const ST *)P.lvl[0][s] + c * plane + (long long)y0 * lp;
    const ST *xd = (const ST *)P.lvl[1][s] + c * plane + (long long)y0 * lp;
    auto samples = [&](int ch) {  // the XYB samples under the maps of chunk ch
        const int x = min(max(ch * kHc + lane - kN + 1, 0), W - 1);
#pragma unroll
        for (int k = 0; k < kMapRows; k++) {
            const long long o = (long long)min(helper + kHelpers * k, rows - 1) * lp + x;
            src[k] = ld_store<ST>(xr + o);
            dis[k] = ld_store<ST>(xd + o);
        }
    };
    if (!walker) {
        fetch(0);
        fetch(1);
        asm volatile("cp.async.wait_group 1;\n" ::: "memory");
    }
    __syncthreads();
    for (int ch = 0; ch <= chunks; ch++) {
        if (walker) {
            if (ch < chunks) {
                float4 *cur = (float4 *)(hsm + (warp * kHSlots + ch % kHSlots) * kHPlane + lane * kHp);
                float ring[kHc];
                const int have = W - ch * kHc;  // columns of the chunk inside the row
#pragma unroll
                for (int k = 0; k < kHc; k += 4) {
                    const float4 f = cur[k / 4];
                    ring[k] = f.x, ring[k + 1] = f.y, ring[k + 2] = f.z, ring[k + 3] = f.w;
                    if (have < kHc) {
#pragma unroll
                        for (int j = 0; j < 4; j++) ring[k + j] = k + j < have ? ring[k + j] : 0.f;
                    }
                    float o[4];
#pragma unroll
                    for (int j = 0; j < 4; j++)
                        o[j] = st.step((k + j >= 2 * kN ? ring[(k + j - 2 * kN) & (kHc - 1)] : tail[(k + j) % (2 * kN)]) +
                                       ring[k + j]);
                    cur[k / 4] = make_float4(o[0], o[1], o[2], o[3]);
                }
#pragma unroll
                for (int k = 0; k < 2 * kN; k++) tail[k] = ring[kHc - 2 * kN + k];
            }
        } else {
            fetch(ch + 2);  // into the slot of chunk ch - 2, whose maps were formed before the last barrier
            if (ch > 0) {
                const int x = (ch - 1) * kHc + lane - kN + 1;
                const float *o = hsm + (ch - 1) % kHSlots * kHPlane + lane;
#pragma unroll
                for (int k = 0; k < kMapRows; k++) {
                    const int r = helper + kHelpers * k;
                    if (r >= rows || x < 0 || x >= W) continue;
                    // error_maps.rs:36-59, as written
                    const float source = src[k], distorted = dis[k];
                    const float *q = o + r * kHp;
                    constexpr int kP = kHSlots * kHPlane;
                    const float mu1 = q[0], mu2 = q[kP], sigma11 = q[2 * kP], sigma22 = q[3 * kP], sigma12 = q[4 * kP];
                    const float mu11 = mu1 * mu1, mu22 = mu2 * mu2, mu12 = mu1 * mu2, mu_diff = mu1 - mu2;
                    const float num_m = fmaf(mu_diff, -mu_diff, 1.0f);
                    const float num_s = fmaf(2.0f, sigma12 - mu12, C2);
                    const float denom_s = ((sigma11 - mu11) + (sigma22 - mu22)) + C2;
                    const float d = fmaxf(1.0f - (num_m * num_s) / denom_s, 0.0f);
                    const float denom = 1.0f / (1.0f + fabsf(source - mu1));
                    const float numer = 1.0f + fabsf(distorted - mu2);
                    const float d1 = fmaf(numer, denom, -1.0f);
                    const float vals[3] = {d, fmaxf(d1, 0.0f), fmaxf(-d1, 0.0f)};
                    // lib.rs:986-1016: f64 sum of d, f64 sum of the f32 (d*d)*(d*d)
#pragma unroll
                    for (int m = 0; m < 3; m++) {
                        const float sq = vals[m] * vals[m];
                        acc[m] += (double)vals[m];
                        acc[3 + m] += (double)(sq * sq);
                    }
                }
            }
            if (ch < chunks) samples(ch);
            asm volatile("cp.async.wait_group 1;\n" ::: "memory");  // chunk ch + 1 has landed
        }
        __syncthreads();
    }
    if (!walker) {
#pragma unroll
        for (int m = 0; m < 6; m++) {
            double t = acc[m];
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) t += __shfl_down_sync(0xffffffffu, t, off);
            if (lane == 0) red[helper][m] = t;
        }
    }
    __syncthreads();
    // the plan keeps one record per row: the group's sums in its first, zeros in the others
    double *out = partials + (long long)(sg.rec_base + y0) * 18 + c * 6;
    for (int i = threadIdx.x; i < rows * 6; i += kHThreads) {
        const int r = i / 6, m = i % 6;
        double t = 0.0;
        if (r == 0)
            for (int w = 0; w < kHelpers; w++) t += red[w][m];
        out[(long long)r * 18 + m] = t;
    }
}

cudaError_t configure_iir_kernels() {
    return cudaFuncSetAttribute(iir_horizontal_kernel<float>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)kHSmem);
}

cudaError_t launch_iir(int storage, const DevPair *pairs, const IirSeg *vsegs, int nvseg, int vtotal,
                       const IirSeg *hsegs, int nhseg, int htotal, double *partials, cudaStream_t st) {
    (void)storage;  // f32 planes only
    if (vtotal > 0) {
        const cudaError_t e =
            dep::launch(false, iir_vertical_kernel<float>, dim3(vtotal), kVThreads, 0, st, pairs, vsegs, nvseg);
        if (e != cudaSuccess) return e;
    }
    if (htotal > 0) {
        return dep::launch(true, iir_horizontal_kernel<float>, dim3(htotal), kHThreads, kHSmem, st, pairs, hsegs, nhseg,
                           partials);
    }
    return cudaSuccess;
}

}  // namespace s2
