// bh_display.h - Launch descriptor of the display transform (bh_display.cu).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "../../include/bh_gpu.h"

namespace bhg {

// Device state of one frame's exposure meter (a radix select); zero between
// uses.
constexpr int kMeterBits = 11;
constexpr int kMeterBins = 1 << kMeterBits;
struct ExposureState {
    unsigned long long count;        // positive finite luminances
    unsigned long long k[2];         // remaining rank of the 99.9th and 99.99th percentile
    unsigned long long prefix[2];    // their bits found so far
    unsigned long long mask;         // which bits are found
    unsigned int ticket;             // blocks of the current pass that are done
    unsigned int pad;
    double exposure;                 // the result
    unsigned long long hist[2][kMeterBins];
};

// One frame of a display launch.
struct DisplayFrame {
    bh_xyz* pixels;                  // W x H, row-major (glare writes it in place)
    uint8_t* rgb;                    // W x H x 3
    long long scratch;               // its first pixel in the glare scratch
    int width, height;
    int index, pad;                  // its exposure state
};

// Glare weights that fit the kernels' parameters: 2 r + 1 each.
constexpr int kGlareMaxRadius = 60;
struct GlareWeights {
    double near_w[2 * kGlareMaxRadius + 1], far_w[2 * kGlareMaxRadius + 1];
    int r_near, r_far;
    double core, a, b;               // the weights of the image, the near and the far blur
};

struct DisplayLaunch {
    const DisplayFrame* frames;      // device, n of them
    const DisplayFrame* h_frames;    // the same on the host
    int n;
    int max_width, max_height;
    long long max_pixels;
    // add_glare: off, in the tiled kernels (GlareWeights), or for wider radii
    // one tap per load with the weights on the device
    int glare;                       // 0, 1 (tiled), 2 (wide)
    GlareWeights w;
    const double* k_near;            // wide: normalised weights, 2 r + 1 each
    const double* k_far;
    bh_xyz *tmp_near, *tmp_far;      // scratch, one pixel per pixel of the frames
    bh_xyz* tmp;                     // wide: a third
    // exposure: fixed when > 0, else metered with `key` into states[index].exposure
    double exposure, key;
    ExposureState* states;
    int sm_count;
    // develop (skipped when not `develop`)
    int develop;
    int tonemap;
    double log_k, denom;             // 10^clamp(log_decades, 1, 20), log10(1 + log_k)
};

cudaError_t launch_display(const DisplayLaunch& L, cudaStream_t stream);

}  // namespace bhg
