// zensim_kernels.h -- device descriptors and launch entry points of the
// zensim feature path (zensim_kernels.cu).
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

namespace zs {

constexpr int kZsScales = 4;
constexpr int kZsRadius = 5;   // box radius of the V0.2 profile (crates/zensim-cuda/src/lib.rs:36-50)
constexpr int kZsSums = 17;    // pooled sums per (scale, channel)
constexpr int kZsOut = 20;     // + the 3 maxima
constexpr int kZsFeatures = 228;
constexpr int kZsTileW = 64;   // columns of a feature tile
constexpr int kZsTileH = 32;   // rows of a feature tile
constexpr int kZsSub = 8;      // rows between two saved states of the vertical sums
constexpr int kZsWalkW = 32;   // columns of a walk block

// Three planar f32 planes (X, Y, B) of width n (the padded width), rows of
// `pitch` floats; p points at column 0 of row 0, which kZsLeft floats precede
// and kZsRight follow column n - 1 in every row: the mirrored columns.
constexpr int kZsLeft = 32, kZsRight = 12;

struct ZsPlanes {
    float *p[3];
    int n;
    size_t pitch;
};

struct ZsScale {
    ZsPlanes ref, dis;
    int n, h;
    // states of the vertical sums every kZsSub rows: [channel][row / kZsSub][sum 0..3][pitch]
    float *state;
    int walk_first, walk_x;           // first walk block of the scale, walk blocks per channel
    int tile_first, tiles_x, tiles_y; // first feature tile, tiles per row / column of a channel
};

// The work of one image size, passed to the kernels by value.
struct ZsPlan {
    ZsScale sc[kZsScales];
    int ns;
    int walk_blocks, tiles;
    bool one_channel;  // the scales' channels share one channel's states (scale 0's): a walk and a feature launch each
};

cudaError_t zs_configure();
cudaError_t zs_upload_lut(const float *lut256);
// sRGB8 -> the XYB planes of every scale (img 0 reference, 1 distorted)
cudaError_t zs_launch_prep(const uint8_t *img, size_t pitch, int w, int h, const ZsPlan &plan, int which, float bias,
                           cudaStream_t st);
// the features of the two pyramids: tile_out holds kZsOut doubles per tile,
// out kZsOut doubles per (scale, channel) (17 sums, then the 3 maxima)
cudaError_t zs_launch_features(const ZsPlan &plan, double *tile_out, double *out, cudaStream_t st);

}  // namespace zs
