// zensim_engine.cu -- C ABI of the zensim feature path (s2_zensim_*):
// Zensim::new / set_reference / compute_with_reference / compute_features /
// has_reference / clear_reference / debug_compute_raw of crates/zensim-cuda
// (src/lib.rs:168-819).  The reference's XYB pyramid stays resident after
// set_reference; every compute converts the distorted image and its pyramid
// (one launch), walks the vertical sums, scores the tiles and reduces them
// (three launches), and forms the 228 features on the host from the sums of
// each (scale, channel).
#include <cuda_runtime.h>

#include <cmath>
#include <cstring>

#include "../../include/ssim2b200.h"
#include "zensim_kernels.h"

using namespace zs;

s2_status s2_cuda_fail(cudaError_t e, const char *what);
void s2_set_last_error(const char *msg);
extern const float s2_srgb8_lut[256];

#define ZS_CUDA(call)                                          \
    do {                                                       \
        cudaError_t e_ = (call);                               \
        if (e_ != cudaSuccess) return s2_cuda_fail(e_, #call); \
    } while (0)

namespace {

size_t align_up(size_t v, size_t a) { return (v + a - 1) / a * a; }

// crates/zensim-cuda/src/lib.rs:58-66
int simd_padded_width(int w) {
    const int aligned = (w + 15) & ~15;
    return (aligned >= 512 && (aligned / 16) % 2 == 0) ? aligned + 16 : aligned;
}

// cbrtf_fast of the opsin bias, negated, with the device's operations (this
// unit's host code is built with -ffp-contract=off)
float opsin_bias() {
    const float x = 0.0037930734f;
    uint32_t u;
    std::memcpy(&u, &x, 4);
    u = u / 3u + 709958130u;
    float t;
    std::memcpy(&t, &u, 4);
    for (int k = 0; k < 2; k++) {
        const float r = t * t * t;
        t = t * (std::fmaf(x, 2.0f, r) / std::fmaf(r, 2.0f, x));
    }
    return -t;
}

}  // namespace

struct s2_zensim {
    int device = 0;
    uint32_t w = 0, h = 0;
    ZsPlan plan = {};
    void *planes = nullptr;       // both pyramids, then the work area unless it lies in `stage`
    size_t plane_bytes = 0;
    uint8_t *stage = nullptr;     // device copy of host inputs (w * 3 * h bytes)
    size_t stage_bytes() const { return (size_t)w * 3 * h; }
    double *tile_out = nullptr;   // work area: kZsOut doubles per tile, then per (scale, channel)
    double out_h[kZsScales * 3 * kZsOut];  // host copy of the latter
    bool has_ref = false;
    double raw_acc[kZsScales][3][kZsSums];
    uint32_t raw_peak[kZsScales][3][3];

    size_t out_doubles() const { return (size_t)kZsOut * 3 * plan.ns; }
    size_t tile_doubles() const { return (size_t)kZsOut * plan.tiles; }
};

static bool g_zs_lut_ready[64];

// Bytes of saved sums up to which every channel of every scale has its own.
// They add a quarter to the planes' memory, 34 GB at 65536 x 65536, where the
// planes alone take 137; above this, and where the device has no room for them,
// the channels take turns in those of one channel of scale 0 (a sixteenth).
// The line is at 2^30 pixels, where a channel's walk has blocks for every SM
// (16384 columns: 512) and the turns cost little; an image below it is short of
// blocks, not of memory.
constexpr size_t kZsMaxState = (size_t)8 << 30;

// The device buffers of z, the saved sums by channels in turns (one_channel)
// or all beside each other (states bytes, the first `state` of each scale).
// What the features need besides the planes -- the saved sums and the tiles'
// records -- follows the planes, or, in turns, lies in the host inputs' copy
// where that is large enough (2.4 of its 3 bytes per pixel): the copy is read by
// the prep pass and free afterwards, so an image then needs no more memory
// than its planes and inputs.
static cudaError_t zs_allocate(s2_zensim *z, size_t planes, size_t states, const size_t *state, bool one_channel) {
    ZsPlan &P = z->plan;
    P.one_channel = one_channel;
    if (one_channel)
        states = align_up((size_t)((P.sc[0].h + kZsSub - 1) / kZsSub) * 4 * P.sc[0].ref.pitch * sizeof(float), 256);
    const size_t work = states + sizeof(double) * (z->tile_doubles() + z->out_doubles());
    const bool shared = one_channel && work <= z->stage_bytes();
    z->plane_bytes = planes + (shared ? 0 : work);
    cudaError_t e = cudaMalloc(&z->planes, z->plane_bytes);
    if (e == cudaSuccess) e = cudaMalloc((void **)&z->stage, z->stage_bytes());
    if (e != cudaSuccess) {
        cudaGetLastError();  // not an error of the launches that follow
        cudaFree(z->planes);
        z->planes = nullptr;
        return e;
    }
    char *const area = shared ? (char *)z->stage : (char *)z->planes + planes;
    for (int s = 0; s < P.ns; s++) P.sc[s].state = (float *)(area + (one_channel ? 0 : state[s]));
    z->tile_out = (double *)(area + states);
    return cudaSuccess;
}

s2_status s2_zensim_create(int32_t device, uint32_t width, uint32_t height, s2_zensim **out) {
    return s2_zensim_create_limited(device, width, height, kZsMaxState, out);
}

s2_status s2_zensim_create_limited(int32_t device, uint32_t width, uint32_t height, size_t max_state,
                                   s2_zensim **out) {
    if (!out) return S2_ERR_INVALID_ARG;
    *out = nullptr;
    // zensim-cuda/src/lib.rs:200-205
    if (width < 8 || height < 8 || width > (1u << 16) || height > (1u << 16)) return S2_ERR_INVALID_SIZE;
    ZS_CUDA(cudaSetDevice(device));
    if (device >= 0 && device < 64 && !g_zs_lut_ready[device]) {
        ZS_CUDA(zs_upload_lut(s2_srgb8_lut));
        ZS_CUDA(zs_configure());
        g_zs_lut_ready[device] = true;
    }
    s2_zensim *z = new s2_zensim();
    std::memset(z->raw_acc, 0, sizeof z->raw_acc);
    std::memset(z->raw_peak, 0, sizeof z->raw_peak);
    z->device = device;
    z->w = width;
    z->h = height;
    // scales while the logical width and the height are >= 8 (lib.rs:222-233)
    ZsPlan &P = z->plan;
    int lw = (int)width, n = simd_padded_width((int)width), h = (int)height;
    size_t bytes = 0, states = 0, off[kZsScales][2], state[kZsScales];
    for (int s = 0; s < kZsScales; s++) {
        if (lw < 8 || h < 8) break;
        ZsScale &S = P.sc[s];
        S.n = S.ref.n = S.dis.n = n;
        S.h = h;
        S.ref.pitch = S.dis.pitch = align_up((size_t)(kZsLeft + n + kZsRight), 64);
        for (int img = 0; img < 2; img++) {
            off[s][img] = bytes;
            bytes += 3 * align_up(S.ref.pitch * h * sizeof(float), 256);
        }
        state[s] = states;
        states += align_up((size_t)3 * ((h + kZsSub - 1) / kZsSub) * 4 * S.ref.pitch * sizeof(float), 256);
        S.walk_x = (n + kZsWalkW - 1) / kZsWalkW;
        S.walk_first = P.walk_blocks;
        P.walk_blocks += 3 * S.walk_x;
        S.tiles_x = (n + kZsTileW - 1) / kZsTileW;
        S.tiles_y = (h + kZsTileH - 1) / kZsTileH;
        S.tile_first = P.tiles;
        P.tiles += 3 * S.tiles_x * S.tiles_y;
        P.ns++;
        lw = (lw + 1) / 2;
        n = n / 2;
        h = (h + 1) / 2;
    }
    cudaError_t e = zs_allocate(z, bytes, states, state, states > max_state);
    if (e == cudaErrorMemoryAllocation && !P.one_channel) e = zs_allocate(z, bytes, states, state, true);
    if (e != cudaSuccess) {
        s2_zensim_destroy(z);
        return e == cudaErrorMemoryAllocation ? S2_ERR_OOM : s2_cuda_fail(e, "zensim buffers");
    }
    for (int s = 0; s < P.ns; s++) {
        ZsScale &S = P.sc[s];
        const size_t plane = align_up(S.ref.pitch * S.h * sizeof(float), 256);
        ZsPlanes *pl[2] = {&S.ref, &S.dis};
        for (int img = 0; img < 2; img++)
            for (int c = 0; c < 3; c++) pl[img]->p[c] = (float *)((char *)z->planes + off[s][img] + c * plane) + kZsLeft;
    }
    *out = z;
    return S2_OK;
}

void s2_zensim_destroy(s2_zensim *z) {
    if (!z) return;
    cudaSetDevice(z->device);
    cudaDeviceSynchronize();
    cudaFree(z->planes);
    cudaFree(z->stage);
    delete z;
}

// Convert one image (img 0 reference, 1 distorted) and build its pyramid.
static s2_status zs_pyramid(s2_zensim *z, int img, const uint8_t *src, size_t pitch, int32_t on_host,
                            cudaStream_t st) {
    if (!src) return S2_ERR_INVALID_ARG;
    const size_t row = (size_t)z->w * 3;
    if (pitch < row) return S2_ERR_DIM_MISMATCH;
    if (on_host) {
        ZS_CUDA(cudaMemcpy2DAsync(z->stage, row, src, pitch, row, z->h, cudaMemcpyHostToDevice, st));
        src = z->stage;
        pitch = row;
    }
    static const float bias = opsin_bias();
    ZS_CUDA(zs_launch_prep(src, pitch, (int)z->w, (int)z->h, z->plan, img, bias, st));
    return S2_OK;
}

s2_status s2_zensim_set_reference_srgb8(s2_zensim *z, const uint8_t *ref, size_t pitch, int32_t on_host,
                                        void *stream) {
    if (!z) return S2_ERR_INVALID_ARG;
    ZS_CUDA(cudaSetDevice(z->device));
    z->has_ref = false;
    cudaStream_t st = (cudaStream_t)stream;
    s2_status r = zs_pyramid(z, 0, ref, pitch, on_host, st);
    if (r != S2_OK) return r;
    ZS_CUDA(cudaStreamSynchronize(st));
    z->has_ref = true;
    return S2_OK;
}

// lib.rs:686-819: the 228 features from the sums of each (scale, channel)
static void zs_assemble(s2_zensim *z, double *feat) {
    std::memset(feat, 0, sizeof(double) * kZsFeatures);
    const int basic_total = z->plan.ns * 13 * 3;
    for (int s = 0; s < z->plan.ns; s++) {
        const double inv_n = 1.0 / ((double)z->plan.sc[s].n * (double)z->plan.sc[s].h);
        for (int c = 0; c < 3; c++) {
            const double *r = z->raw_acc[s][c];
            const uint32_t *pk = z->raw_peak[s][c];
            const double l2 = std::fabs(r[10]) > 0.0 ? r[11] / r[10] : 0.0;
            const double l1 = std::fabs(r[12]) > 0.0 ? r[13] / r[12] : 0.0;
            double *o = feat + s * 3 * 13 + c * 13;
            o[0] = std::fabs(r[0] * inv_n);
            o[1] = std::pow(std::fmax(r[1] * inv_n, 0.0), 0.25);
            o[2] = std::sqrt(std::fmax(r[2] * inv_n, 0.0));
            o[3] = std::fabs(r[3] * inv_n);
            o[4] = std::pow(std::fmax(r[4] * inv_n, 0.0), 0.25);
            o[5] = std::sqrt(std::fmax(r[5] * inv_n, 0.0));
            o[6] = std::fabs(r[6] * inv_n);
            o[7] = std::pow(std::fmax(r[7] * inv_n, 0.0), 0.25);
            o[8] = std::sqrt(std::fmax(r[8] * inv_n, 0.0));
            o[9] = r[9] * inv_n;
            o[10] = std::fmax(1.0 - l2, 0.0);
            o[11] = std::fmax(1.0 - l1, 0.0);
            o[12] = std::fmax(l2 - 1.0, 0.0);
            double *p = feat + basic_total + s * 3 * 6 + c * 6;
            float f;
            for (int k = 0; k < 3; k++) {
                std::memcpy(&f, &pk[k], 4);
                p[k] = (double)f;
            }
            p[3] = std::pow(std::fmax(r[14] * inv_n, 0.0), 0.125);
            p[4] = std::pow(std::fmax(r[15] * inv_n, 0.0), 0.125);
            p[5] = std::pow(std::fmax(r[16] * inv_n, 0.0), 0.125);
        }
    }
}

s2_status s2_zensim_compute_with_reference_srgb8(s2_zensim *z, const uint8_t *dis, size_t pitch, int32_t on_host,
                                                 void *stream, double *features, int32_t *n_scales) {
    if (!z || !features) return S2_ERR_INVALID_ARG;
    if (!z->has_ref) return S2_ERR_NO_REFERENCE;
    ZS_CUDA(cudaSetDevice(z->device));
    cudaStream_t st = (cudaStream_t)stream;
    s2_status r = zs_pyramid(z, 1, dis, pitch, on_host, st);
    if (r != S2_OK) return r;
    double *const out_d = z->tile_out + z->tile_doubles();
    ZS_CUDA(zs_launch_features(z->plan, z->tile_out, out_d, st));
    ZS_CUDA(cudaMemcpyAsync(z->out_h, out_d, sizeof(double) * z->out_doubles(), cudaMemcpyDeviceToHost, st));
    ZS_CUDA(cudaStreamSynchronize(st));
    std::memset(z->raw_acc, 0, sizeof z->raw_acc);
    std::memset(z->raw_peak, 0, sizeof z->raw_peak);
    for (int s = 0; s < z->plan.ns; s++)
        for (int c = 0; c < 3; c++) {
            const double *o = z->out_h + (size_t)kZsOut * (3 * s + c);
            std::memcpy(z->raw_acc[s][c], o, sizeof(double) * kZsSums);
            for (int k = 0; k < 3; k++) {
                const float peak = (float)o[kZsSums + k];
                std::memcpy(&z->raw_peak[s][c][k], &peak, 4);
            }
        }
    zs_assemble(z, features);
    if (n_scales) *n_scales = z->plan.ns;
    return S2_OK;
}

s2_status s2_zensim_compute_features_srgb8(s2_zensim *z, const uint8_t *ref, size_t ref_pitch, const uint8_t *dis,
                                           size_t dis_pitch, int32_t on_host, void *stream, double *features,
                                           int32_t *n_scales) {
    s2_status r = s2_zensim_set_reference_srgb8(z, ref, ref_pitch, on_host, stream);
    if (r != S2_OK) return r;
    return s2_zensim_compute_with_reference_srgb8(z, dis, dis_pitch, on_host, stream, features, n_scales);
}

int32_t s2_zensim_has_reference(const s2_zensim *z) { return z && z->has_ref ? 1 : 0; }

s2_status s2_zensim_clear_reference(s2_zensim *z) {
    if (!z) return S2_ERR_INVALID_ARG;
    z->has_ref = false;
    return S2_OK;
}

s2_status s2_zensim_raw(const s2_zensim *z, double *acc, uint32_t *peaks) {
    if (!z || !acc || !peaks) return S2_ERR_INVALID_ARG;
    std::memcpy(acc, z->raw_acc, sizeof z->raw_acc);
    std::memcpy(peaks, z->raw_peak, sizeof z->raw_peak);
    return S2_OK;
}

s2_status s2_zensim_mem_usage(const s2_zensim *z, size_t *bytes) {
    if (!z || !bytes) return S2_ERR_INVALID_ARG;
    *bytes = z->stage_bytes() + z->plane_bytes;
    return S2_OK;
}
