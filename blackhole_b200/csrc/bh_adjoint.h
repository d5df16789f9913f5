// bh_adjoint.h - Frame constants of the discrete adjoint (host and device).
//
// The adjoint differentiates the luminance loss of one frame with respect to
// four scene parameters: the spin a, the camera inclination (its polar angle
// theta, radians), the accretion rate in Eddington units and the disc's outer
// radius.  Everything per frame that depends on a parameter carries its
// derivative here, computed on the host with dual numbers; the per-ray part
// runs on the device (bh_adjoint.cuh).
#pragma once

#include <cuda_runtime.h>

#include <string>

#include "../../include/bh_gpu.h"
#include "bh_frame.h"

namespace bhg {

// Index of a parameter in the tangent arrays below.
enum { kParSpin = 0, kParIncl = 1 };

struct AdjointFrame {
    // d/d(spin) and d/d(inclination) of the camera's non-zero ZAMO tetrad legs
    // (tet00, tet03, tet11, tet22, tet33) and of g_{mu nu} at the camera
    // (tt, t phi, rr, theta theta, phi phi).
    double d_tet[5][2];
    double d_ml[5][2];
    // d/d(spin) of the disc constants; the disc's spin is clamped to
    // +-0.9999 (disc.h:75), beyond which they do not move.
    double d_disc_a;
    double d_x0;
    double d_pt_x[3], d_pt_c[3], d_pt_den[3];
    double d_mdot_da;                // d(accretion rate in kg/s) / d(spin), through the efficiency
    double d_mdot_dedd;              // d(accretion rate) / d(Eddington ratio)
    int32_t checkpoint_interval;     // accepted steps between stored states (doubles when full)
    int32_t checkpoint_slots;        // stored states per ray in flight
};

// Checks that the scene is one the adjoint covers (a disc and/or a sky; no
// Sun, neutron star or hot spot) and fills the derivatives.  Returns a
// bh_status; `F` must come from make_frame for the same config.
int make_adjoint_frame(const bh_render_config& c, const FrameParams& F, AdjointFrame& X, std::string& err);

// One adjoint launch over the rays of one frame.
struct AdjointLaunch {
    FrameParams frame;               // binary64 frame constants (ray_begin 0)
    AdjointFrame X;
    SkyData sky;
    const bh_xyz* pixels;            // the rendered frame, row-major W x H (device)
    const float* target;             // target luminance, row-major W x H (device)
    double* ray_grad;                // 4 per ray, pixel-major then sample (device)
    double* ray_Y;                   // luminance per ray in the same order, or nullptr
    double* ckpt;                    // ckpt_warps * 32 * checkpoint_slots * kAdjSlotWords doubles: the stored
                                     // states of the grid's last ckpt_warps warps
    int ckpt_warps;
    const HitRecord* hits;           // the render's hit records, work order (device)
    // The rays that have a gradient (work order ids; n_rays entries): those whose
    // steps the render recorded from the front, the others from the back.
    int* rays;
    const double* traj;              // the recorded steps (TraceLaunch::traj), or null
    int traj_cap;
    const int* abort;                // nonzero: the render was stopped and its records are not complete
    const int* xing_step;            // TraceLaunch::xing_step, disc_end
    const double* disc_end;
    // The edge pass: per crossing slot (2 per ray, slot = 2 * ray + crossing,
    // rays in work order) the radius of the ray's first two equatorial
    // crossings as the render found them (0: none; zeroed before the
    // render; the second one's sign is set when a third followed), the
    // candidate list ((slot << 2) | kEdge* bits; those in recorded steps from the
    // front, the others from the back) and 3 edge contributions per slot.
    double* xing_r;
    unsigned long long* cand;
    double* edge_out;
    // 1 for a ray whose event came after its third or later equatorial
    // crossing (an image of order three or higher), in ray_grad order
    unsigned char* high_order;
    // By index: 0 next recorded candidate, 1 accepted steps, 2 replayed steps, 3 disc
    // rays, 4 sky rays, 5 largest interval, 6 recorded candidates, 7 steps of the
    // edge pass, 8 edge cells, 9 high-order rays, 10 recorded rays with a
    // gradient, 11 other rays with a gradient, 12 next recorded ray, 13 other
    // candidates, 14 next job without records.
    unsigned long long* counters;
    // loss; the four per-ray gradient sums (spin and inclination over the
    // rays of image order one and two); the three edge sums; the spin and
    // inclination sums over the rays of order three and higher
    double* sums;
    long long n_rays;
    int grid, block;
    int grid_reverse;                // blocks of the kernel over the recorded rays
    cudaStream_t side_stream;        // that kernel runs here, beside the edge terms and the rays without records
    cudaEvent_t fork_event, join_event;
};

constexpr int kAdjCounters = 15;
constexpr int kAdjSlotWords = 11;         // doubles per stored state
constexpr int kAdjSums = 10;

// Enqueues the edge pass's candidate selection over the sample grid, the
// adjoint kernel (rays without records, then edge terms), the sweeps over the
// recorded rays beside it and the deterministic reduction of the per-ray
// gradients, the edge contributions and the loss; `counters` and `edge_out`
// must be zeroed before.
cudaError_t launch_adjoint(const AdjointLaunch& L, cudaStream_t stream);
// Threads per block of the adjoint kernel, and its resident blocks per SM at
// `block_size` threads.
int adjoint_block_size();
int reverse_blocks_per_sm();
int adjoint_blocks_per_sm(int block_size);

}  // namespace bhg
