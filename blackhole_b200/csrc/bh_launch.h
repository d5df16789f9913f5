// bh_launch.h - Host-side launch wrappers of the trace, shade and stats kernels.
#pragma once

#include <cuda_runtime.h>

#include "bh_frame.h"

struct bh_xyz;
struct bh_ray_result;

namespace bhg {

struct TraceLaunch {
    const FrameParams* frames;       // device array
    const long long* frame_ray_end;  // device array: cumulative ray counts (exclusive end)
    int nframes;
    long long total_rays;
    HitRecord* hits;                 // device, total_rays entries
    QueueState* queue;               // device
    int precision;                   // BH_PRECISION_*
    int block_size;
    int grid;                        // blocks
    int draws;                       // batches of rays a warp takes before it ends, with refill 32 and a
                                     // grid to match (0: until none is left)
    int rays_per_thread;
    int refill;
    unsigned long long budget;       // step-attempt budget of the launch, 0 = none
    int reg_variant;                 // 0: default register cap, 1: the wider one
    void* deferred;                  // mixed precision: total_rays deferred records
    int grid_resume;                 // blocks of the binary64 resume launch
    int block_resume;                // its threads per block
    cudaEvent_t resume_event;        // recorded between the two launches (optional)
    double* jet;                     // jet emission per ray (total_rays), or null when no
                                     // frame of the launch has a jet
    double* xing;                    // radii of each ray's first two equatorial crossings
                                     // (2 per ray, zeroed before; 0 = none), or null
    // With xing: the accepted steps of each ray are recorded too, the first
    // traj_cap of them, kTrajWords doubles each (r, th, p_r, p_th, the step's
    // size, sin and cos of th, at its start; word w of step j of ray i at
    // traj[(j kTrajWords + w) total_rays + i]), but for those of a ray that is
    // falling in (it has no gradient, and the creep to the horizon is most of
    // its steps).  Null: not.  xing_step: the step of each crossing (2 per ray),
    // kNotRecorded while falling in; disc_end: where a ray that hit the disc
    // would go on, kEndWords doubles each (the state at the end of its last
    // step, the next step's size, the controller's memory, sin and cos of th;
    // word w of ray i at disc_end[w total_rays + i]).
    double* traj;
    int traj_cap;
    int* xing_step;
    double* disc_end;
    int surfaces;                    // 1 when a frame of the launch has the Sun or a neutron star
    int expanded;                    // 1 when a frame of the launch has a^2 >= 1 (Delta has no pair of roots)
    // Mixed precision: near-critical rays (escaping rays that circle close to
    // the photon shell) traced by a binary64 kernel of grid_side blocks of 64
    // on `stream`, beside the binary32 kernel on side_stream (fork_event and
    // join_event order it against `stream`, start_event fires once the binary64
    // blocks have begun), or before it on `stream` when side_stream is null.
    int near_critical;
    int grid_side;
    const FrameParams* frames_side;  // device: the frames under binary64_treatment
    unsigned char* sel_flag;         // device, total_rays: near-critical flags (classification
                                     // pass), or null: then both kernels test each ray themselves
    int* sel_list;                   // device, total_rays: the near-critical rays' ids
    cudaStream_t side_stream;
    cudaEvent_t fork_event, start_event, join_event;
    // Row bands of a single-frame launch whose pixels are shaded and copied
    // out while the rest of the frame is traced: each finished ray adds one
    // to band_done[gid / rays_per_band]; after the last trace kernel every
    // counter is raised to its band's size (so a wait on it always ends).
    // Null: no counting.
    unsigned int* band_done;
    long long rays_per_band;
    int nbands;
};

// Bytes of one deferred-ray record.
size_t deferred_record_bytes();
constexpr size_t kDeferredRecordBytes = 96;   // checked against the record in bh_trace.cu

constexpr int kTrajWords = 7, kEndWords = 10, kNotRecorded = 0x7fffffff;

// Persistent trace kernel over all rays of all frames.
cudaError_t launch_trace(const TraceLaunch& L, cudaStream_t stream);

// Blocks per SM that fit for a precision and block size (occupancy query;
// the least over the plain, surface and jet kernels of that precision and cap).
int trace_blocks_per_sm(int precision, int block_size, int variant);
// Registers per thread of the trace kernels of a precision (the most over
// the plain, surface and jet kernels).
int trace_registers(int precision, int variant);

// Shades the frame-local pixels [pixel_lo, pixel_hi) (work order) of each
// frame on `blocks` blocks, and adds those pixels' counts and maxima to the
// frame's stats (zeroed before); each block's flux goes to a partial of its own
// (flux_per_frame of them per frame, this launch's first one at `flux`).
struct ShadeLaunch {
    const FrameParams* frames;
    int nframes;
    int blocks;
    long long pixel_lo, pixel_hi;
    const HitRecord* hits;
    SkyData sky;
    bh_xyz* pixels;                  // device (frame-major, row-major)
    bh_ray_result* rays;             // optional device per-sample results (single frame)
    const double* jet;               // jet emission per ray (TraceLaunch::jet), or null
    FrameStats* stats;
    double* flux;
    int flux_per_frame;
};

// Blocks for `pixels` of one frame, `most` at most.
int shade_blocks(long long pixels, int most);
cudaError_t launch_shade(const ShadeLaunch& L, cudaStream_t stream);

// Sums each frame's flux partials into its stats.
struct ReduceLaunch {
    int nframes;
    int flux_per_frame;
    const double* flux;              // nframes * flux_per_frame
    FrameStats* stats;
};

cudaError_t launch_reduce(const ReduceLaunch& L, cudaStream_t stream);

// Known-answer evaluation of device functions (bh_gpu_eval): the trace
// kernels' right-hand side at n states of 8 doubles (8 derivatives each),
// and the shading's disc temperature (what 0: n radii -> n kelvin) or
// blackbody lookup (what 1: n kelvin -> 3n XYZ).
cudaError_t launch_eval_rhs(int precision, const FrameParams* d_frame, const double* d_in, long long n,
                            double* d_out, cudaStream_t stream);
cudaError_t launch_eval_shade(int what, const FrameParams* d_frame, const double* d_table, const double* d_in,
                              long long n, double* d_out, cudaStream_t stream);

}  // namespace bhg
