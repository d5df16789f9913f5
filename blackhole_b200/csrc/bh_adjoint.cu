// bh_adjoint.cu - The discrete-adjoint kernels and reductions (sm_100a).
//
// adjoint_select_kernel: one thread per ray.  The render's hit record says
// which rays have a gradient at all: those that ended on the disc or saw a sky
// that varies at their direction.  A captured ray, or one that met the uniform
// background, is done here; the others are listed.
//
// reverse_kernel: the listed rays whose steps the render recorded, backwards.
// Nothing is integrated again: at 512^2 the forward pass per ray that each
// sweep started with was 5 of 12.2 ms, its trajectory going through the same
// memory; the record costs the render 0.2 ms.
//
// adjoint_kernel: the edge terms, and the listed rays without records (more
// steps than the record holds, or a frame too large for one), which are
// integrated again.  A lane that does so owns `checkpoint_slots` stored states
// (45 KB) in global memory, interleaved over the warp, for the job it is
// working on (bh_adjoint.cuh has the per-ray algorithm).  Beside a record of 512
// steps per ray few jobs need them (15 rays at 512^2), so an eighth of the
// warps own states; every warp does elsewhere.
//
// In both a warp takes 32 jobs at a time from a global atomic counter.  A
// ray's loss weight is 2 (Y_pixel - target) / S^2 for Loss = sum over pixels
// of (Y_pixel - target)^2, Y_pixel being the sample mean of the rendered frame
// (bh_gpu_render's output).
//
// The edge pass: a point-sampled frame has no derivative with respect to
// r_out, and its derivatives with respect to the spin and the inclination
// miss the motion of the disc's edges; the derivative of the frame averaged
// over each sample's cell has both.  edge_candidates_kernel picks each
// sample's first two equatorial crossings near an edge (adj::edge_mask,
// against the spread of the neighbouring samples' same crossing; the render
// records the crossings), and the adjoint kernel takes their edge terms
// (weight 2 (Y_pixel - target)): edge_recorded where the render recorded the
// steps up to the crossing, adj::edge_sample elsewhere.  reverse_kernel runs
// beside it on a second stream, since both are long chains that leave issue
// slots free: 512^2 takes 8.3 ms so and 10.9 ms with the edge terms after the
// rays (the frame before the records: 12.2 ms; 128^2 5.6 -> 3.5 ms).
//
// The edge pass covers the edges of the first two equatorial crossings (the
// direct image of the disc and its first lensed image).  Images of order
// three and higher are rings so thin that a sample's derivative holds over a
// small part of its cell, and their edges are not in the edge pass, so their
// per-ray spin and inclination terms are summed apart (the held-out sums)
// rather than into the frame gradient.
//
// adjoint_reduce_kernel: ten blocks, each summing one quantity (the loss,
// the four per-ray gradient components, the three edge components, the two
// held-out components) over a fixed thread-to-element assignment and a fixed
// tree, so the result does not depend on the order rays finished in.
#include <cuda_runtime.h>

#include "bh_adjoint.cuh"
#include "bh_launch.h"

namespace bhg {

namespace {

using adj::kAdjBlock;
constexpr size_t kAdjShared = sizeof(double) * adj::kScratch * kAdjBlock;
// 8 warps per SM with 255 registers; 10 and 12 with 200 and 168 took 5 and 9% longer
// per 512^2 gradient, 6 the same.
constexpr int kAdjBlocksPerSm = 4;
constexpr int kReduceThreads = 1024;
static_assert(adj::kCkWords == kAdjSlotWords, "kAdjSlotWords is stale");

// Candidate selection: one thread per sample (work order); each of its first
// two equatorial crossings, as the render recorded them, is compared with the
// same crossing of its four neighbours in the W S x H S sample grid
// (adj::edge_mask).
__global__ void __launch_bounds__(256) edge_candidates_kernel(const __grid_constant__ AdjointLaunch L) {
    const long long id = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (id >= L.n_rays || *(const volatile int*)L.abort) return;
    const int S = L.frame.S;
    const int SS = S * S;
    const int W = L.frame.width, H = L.frame.height;
    const long long pixel = id / SS;
    const int k = (int)(id - pixel * SS);
    int px, py;
    pixel_xy(W, H, pixel, &px, &py);
    const int gx = px * S + k % S;
    const int gy = py * S + k / S;
    const int GW = W * S, GH = H * S;
    for (int j = 0; j < 2; ++j) {
        const double rc = fabs(L.xing_r[2 * id + j]);
        if (rc == 0.0) break;
        double dmax = 0.0;
        #pragma unroll
        for (int n = 0; n < 4; ++n) {
            const int nx = gx + (n == 0) - (n == 1);
            const int ny = gy + (n == 2) - (n == 3);
            if (nx < 0 || nx >= GW || ny < 0 || ny >= GH) continue;
            const long long nid = pixel_index(W, H, nx / S, ny / S) * SS + (ny % S) * S + nx % S;
            const double rn = fabs(L.xing_r[2 * nid + j]);
            if (rn == 0.0) continue;
            const double d = fabs(rc - rn);
            if (d > dmax) dmax = d;
        }
        const int m = adj::edge_mask(L.frame, rc, dmax);
        if (m) {
            const unsigned long long c = ((unsigned long long)(2 * id + j) << 2) | (unsigned long long)m;
            if (L.traj && L.xing_step[2 * id + j] <= L.traj_cap) L.cand[atomicAdd(&L.counters[6], 1ull)] = c;
            else L.cand[2 * L.n_rays - 1 - (long long)atomicAdd(&L.counters[13], 1ull)] = c;
        }
    }
}

// The pixel (index, row-major) and sample of a ray (work order).
__device__ __forceinline__ long long ray_pixel(const AdjointLaunch& L, long long id, int* px, int* py, int* k) {
    const int SS = L.frame.S * L.frame.S;
    const long long pixel = id / SS;
    *k = (int)(id - pixel * SS);
    pixel_xy(L.frame.width, L.frame.height, pixel, px, py);
    return (long long)*py * L.frame.width + *px;
}

// What the render's hit record says of each ray: its class counts, whether
// its image is of order three or higher, and whether it has a gradient.
// Rays without one get their (zero) gradient and their luminance here; the
// rest are listed, 32 consecutive rays at a time.
__global__ void __launch_bounds__(256) adjoint_select_kernel(const __grid_constant__ AdjointLaunch L) {
    const long long id = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const int SS = L.frame.S * L.frame.S;
    bool listed = false;
    unsigned steps = 0;
    int what = BH_HIT_EXHAUSTED;
    bool high = false;
    if (id < L.n_rays && !*(const volatile int*)L.abort) {
        int px, py, k;
        const long long pix = ray_pixel(L, id, &px, &py, &k);
        const long long o = pix * SS + k;
        const HitRecord& h = L.hits[id];
        what = h.what;
        steps = (unsigned)h.steps;
        const bool event = what == BH_HIT_DISC || what == BH_HIT_SKY;
        high = event && L.xing_r[2 * id + 1] < 0.0;
        const double w = 2.0 * (L.pixels[pix].y - (double)L.target[pix]) / (double)SS;
        double Y = 0.0;
        if (what == BH_HIT_DISC) {
            listed = w != 0.0;
            if (!listed && L.ray_Y)
                Y = adj::disc_luminance(L.frame, L.X, L.sky.table, h.y[1], -h.y[4], h.y[7]).v;
        } else if (what == BH_HIT_SKY) {
            const double y6[6] = {h.y[0], h.y[1], h.y[2], h.y[3], h.y[5], h.y[6]};
            double d[3], gY[3];
            if (adj::escape_direction_value(y6, -h.y[4], h.y[7], L.frame.a, d)) {
                Y = adj::sky_luminance(L.sky, L.frame, d, gY);
                // (a weight that is not finite has a gradient on any sky)
                listed = w != 0.0 && (!isfinite(w) || gY[0] != 0.0 || gY[1] != 0.0 || gY[2] != 0.0);
            }
        }
        L.high_order[o] = high ? 1 : 0;
        if (!listed) {
            #pragma unroll
            for (int q = 0; q < 4; ++q) L.ray_grad[o * 4 + q] = 0.0;
            if (L.ray_Y) L.ray_Y[o] = Y;
        }
    }
    const unsigned lane = threadIdx.x & 31;
    const bool recorded = L.traj && steps <= (unsigned)L.traj_cap;
    const unsigned m = __ballot_sync(kFull, listed && recorded);
    const unsigned m2 = __ballot_sync(kFull, listed && !recorded);
    const unsigned nd = __popc(__ballot_sync(kFull, what == BH_HIT_DISC));
    const unsigned ns = __popc(__ballot_sync(kFull, what == BH_HIT_SKY));
    const unsigned nh = __popc(__ballot_sync(kFull, high));
    const unsigned st = __reduce_add_sync(kFull, steps);
    unsigned long long base = 0, base2 = 0;
    if (lane == 0) {
        if (m) base = atomicAdd(&L.counters[10], (unsigned long long)__popc(m));
        if (m2) base2 = atomicAdd(&L.counters[11], (unsigned long long)__popc(m2));
        if (st) atomicAdd(&L.counters[1], (unsigned long long)st);
        if (nd) atomicAdd(&L.counters[3], (unsigned long long)nd);
        if (ns) atomicAdd(&L.counters[4], (unsigned long long)ns);
        if (nh) atomicAdd(&L.counters[9], (unsigned long long)nh);
    }
    base = __shfl_sync(kFull, base, 0);
    base2 = __shfl_sync(kFull, base2, 0);
    const unsigned before = (1u << lane) - 1u;
    if (listed && recorded) L.rays[base + __popc(m & before)] = (int)id;
    else if (listed) L.rays[L.n_rays - 1 - (long long)(base2 + __popc(m2 & before))] = (int)id;
}

// The edge term of a crossing in a recorded step: what the ray meets beyond it
// is the render's own record, unless the render ended the ray there, and the
// sweep goes over the recorded steps.  Returns the steps integrated.
__device__ __noinline__ long long edge_recorded(const AdjointLaunch& L, long long id, int px, int py, int k, int which,
                                                int edges, double w, double out[3], int* cells) {
    out[0] = out[1] = out[2] = 0.0;
    *cells = 0;
    const HitRecord& h = L.hits[id];
    const int N = L.xing_step[2 * id + which];
    const adj::RayC c = adj::ray_consts(L.frame, -h.y[4], h.y[7]);
    long long work = 0;
    double Y_beyond;
    if (h.what == BH_HIT_DISC && h.steps == N) {
        adj::Integ t;
        for (int i = 0; i < 6; ++i) t.y[i] = L.disc_end[i * L.n_rays + id];
        t.h = L.disc_end[6 * L.n_rays + id];
        t.errp_mem = L.disc_end[7 * L.n_rays + id];
        t.sn0 = L.disc_end[8 * L.n_rays + id];
        t.c0 = L.disc_end[9 * L.n_rays + id];
        t.h_acc = 0.0;
        t.have_k1 = 0;
        t.tries = 0;
        t.steps = N;
        double r_hit = 0.0;
        const int what = (N >= L.frame.max_steps) ? BH_HIT_EXHAUSTED
                                                  : adj::forward_run(L.frame, c, t, nullptr, nullptr, 0, &r_hit, true);
        work = t.steps - N;
        Y_beyond = adj::luminance(L.frame, L.X, L.sky, what, r_hit, t.y, c.E, c.Lz);
    } else {
        const double y[6] = {h.y[0], h.y[1], h.y[2], h.y[3], h.y[5], h.y[6]};
        Y_beyond = adj::luminance(L.frame, L.X, L.sky, h.what, h.y[1], y, c.E, c.Lz);
    }
    double dY[2];
    adj::edge_jumps(L.frame, L.X, L.sky, edges, Y_beyond, c.E, c.Lz, dY);
    if (dY[0] == 0.0 && dY[1] == 0.0) return work;
    double yb[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0}, Eb = 0.0, Lzb = 0.0, ab = 0.0, rstar = 1.0;
    #pragma unroll 1
    for (int j = N - 1; j >= 0; --j) {
        const double* p = L.traj + (long long)j * kTrajWords * L.n_rays + id;
        double v[kTrajWords];
        #pragma unroll
        for (int q = 0; q < kTrajWords; ++q) v[q] = p[q * L.n_rays];
        adj::step_vjp(c, v, v[5], v[6], v[4], yb, &Eb, &Lzb, &ab, rstar);
        rstar = 0.0;
    }
    adj::edge_finish(L.frame, L.X, px, py, k, edges, w, fabs(L.xing_r[2 * id + which]), dY, yb, Eb, Lzb, ab, out,
                     cells, nullptr);
    return work;
}

// Two queues of jobs.  First the listed rays and the edge candidates without
// recorded steps (a forward pass and a reverse sweep: the longest jobs), for the
// warps that own stored states; then, for every warp, the candidates with
// recorded steps.  Results go to per-ray and per-crossing slots, so the sums do
// not depend on which lane took which job.
__global__ void __launch_bounds__(kAdjBlock, kAdjBlocksPerSm) adjoint_kernel(const __grid_constant__ AdjointLaunch L) {
    const int lane = threadIdx.x & 31;
    const long long warp = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int slots = L.X.checkpoint_slots;
    const long long owner = warp - ((long long)gridDim.x * (kAdjBlock / 32) - L.ckpt_warps);
    double* ck = L.ckpt + owner * slots * adj::kCkWords * 32 + lane;
    const int SS = L.frame.S * L.frame.S;
    // rays and candidates start on a warp of their own
    const unsigned long long n_rays = L.counters[11], first_cand = (n_rays + 31) & ~31ull,
                             n_stored = first_cand + L.counters[13], n_recorded = L.counters[6];
    unsigned long long replay = 0, max_int = 0, edge_steps = 0, edge_cells = 0;
    bool stored = owner >= 0;                // which queue the warp takes from
    for (;;) {
        unsigned long long job = 0;
        if (lane == 0) job = atomicAdd(&L.counters[stored ? 14 : 0], 32ull);
        job = __shfl_sync(kFull, job, 0);
        if (job >= (stored ? n_stored : n_recorded)) {
            if (!stored) break;
            stored = false;
            continue;
        }
        job += lane;
        int px, py, k;
        if (stored ? (job >= first_cand && job < n_stored) : job < n_recorded) {
            const unsigned long long c = L.cand[stored ? 2 * L.n_rays - 1 - (long long)(job - first_cand)
                                                       : (long long)job];
            const long long xs = (long long)(c >> 2);     // 2 * ray + crossing
            const long long pix = ray_pixel(L, xs >> 1, &px, &py, &k);
            const double w = 2.0 * (L.pixels[pix].y - (double)L.target[pix]);
            double out[3];
            int n_cells = 0;
            edge_steps += (unsigned long long)(
                stored ? adj::edge_sample(L.frame, L.X, L.sky, px, py, k, (int)(xs & 1) + 1, (int)(c & 3ull), w, ck,
                                          slots, 32, out, &n_cells)
                       : edge_recorded(L, xs >> 1, px, py, k, (int)(xs & 1), (int)(c & 3ull), w, out, &n_cells));
            edge_cells += (unsigned long long)n_cells;
            L.edge_out[3 * xs] = out[0];
            L.edge_out[3 * xs + 1] = out[1];
            L.edge_out[3 * xs + 2] = out[2];
        } else if (stored && job < n_rays) {
            const long long id = L.rays[L.n_rays - 1 - (long long)job];
            const long long pix = ray_pixel(L, id, &px, &py, &k);
            const double w = 2.0 * (L.pixels[pix].y - (double)L.target[pix]) / (double)SS;
            adj::RayResult res;
            adj::adjoint_ray(L.frame, L.X, L.sky, id, w, ck, slots, 32, false, &res);
            const long long o = pix * SS + k;
            #pragma unroll
            for (int q = 0; q < 4; ++q) L.ray_grad[o * 4 + q] = res.grad[q];
            if (L.ray_Y) L.ray_Y[o] = res.Y;
            replay += (unsigned long long)res.replay;
            if ((unsigned long long)res.interval > max_int) max_int = (unsigned long long)res.interval;
        }
        __syncwarp();
    }
    if (replay) atomicAdd(&L.counters[2], replay);
    if (max_int) atomicMax(&L.counters[5], max_int);
    if (edge_steps) atomicAdd(&L.counters[7], edge_steps);
    if (edge_cells) atomicAdd(&L.counters[8], edge_cells);
}

// The listed rays whose steps the render recorded: the seed from the hit
// record, then each step backwards from its record.  The lanes of a warp walk
// the same step numbers, from the longest ray's last, so that their loads
// coalesce (56 bytes a ray and step, 2.3 GB at 512^2: 0.35 ms of the kernel's
// 4.4).  Bound by the latency of a step's chain of binary64 operations.  At
// least 5 blocks per SM: 168 registers, with which 6 fit (12 warps), 8.3 ms per
// 512^2 gradient; at least 4 (8 warps) 8.8.
constexpr int kReverseBlocksPerSm = 5;
__global__ void __launch_bounds__(kAdjBlock, kReverseBlocksPerSm)
reverse_kernel(const __grid_constant__ AdjointLaunch L) {
    const int lane = threadIdx.x & 31;
    const int SS = L.frame.S * L.frame.S;
    const unsigned long long n_jobs = L.counters[10];
    for (;;) {
        unsigned long long job = 0;
        if (lane == 0) job = atomicAdd(&L.counters[12], 32ull);
        job = __shfl_sync(kFull, job, 0);
        if (job >= n_jobs) break;
        job += lane;
        long long id = 0, o = 0;
        int N = 0;
        adj::RayC c = {};
        adj::Seed sd = {};
        if (job < n_jobs) {
            id = L.rays[job];
            int px, py, k;
            const long long pix = ray_pixel(L, id, &px, &py, &k);
            o = pix * SS + k;
            const double w = 2.0 * (L.pixels[pix].y - (double)L.target[pix]) / (double)SS;
            const HitRecord& h = L.hits[id];
            const double y[6] = {h.y[0], h.y[1], h.y[2], h.y[3], h.y[5], h.y[6]};
            c = adj::ray_consts(L.frame, -h.y[4], h.y[7]);
            adj::seed_ray(L.frame, L.X, L.sky, h.what, h.y[1], y, c.E, c.Lz, w, sd);
            if (sd.any()) N = h.steps;
        }
        double yb[6], Eb = sd.Eb, Lzb = sd.Lzb, ab = sd.ab, rstar = sd.rstar_b;
        #pragma unroll
        for (int i = 0; i < 6; ++i) yb[i] = sd.yb[i];
        const int most = __reduce_max_sync(kFull, N);
        #pragma unroll 1
        for (int j = most - 1; j >= 0; --j) {
            if (j < N) {
                const double* p = L.traj + (long long)j * kTrajWords * L.n_rays + id;
                double v[kTrajWords];
                #pragma unroll
                for (int q = 0; q < kTrajWords; ++q) v[q] = p[q * L.n_rays];
                adj::step_vjp(c, v, v[5], v[6], v[4], yb, &Eb, &Lzb, &ab, rstar);
                rstar = 0.0;
            }
            __syncwarp();
        }
        if (job < n_jobs) {
            double y0[6], E, Lz, dy0[2][6], dE[2], dLz[2], grad[4] = {0.0, 0.0, sd.d_edd, 0.0};
            if (N > 0) {
                adj::ray_start(L.frame, L.X, id, y0, &E, &Lz, dy0, dE, dLz);
                for (int q = 0; q < 2; ++q) {
                    double gq = Eb * dE[q] + Lzb * dLz[q];
                    for (int i = 0; i < 6; ++i) gq += yb[i] * dy0[q][i];
                    grad[q] = gq;
                }
                grad[kParSpin] += ab;
            }
            #pragma unroll
            for (int q = 0; q < 4; ++q) L.ray_grad[o * 4 + q] = grad[q];
            if (L.ray_Y) L.ray_Y[o] = sd.Y;
        }
    }
}

__global__ void after_kernel() {}

__global__ void __launch_bounds__(kReduceThreads)
adjoint_reduce_kernel(const double* __restrict__ grad, const double* __restrict__ edge,
                      const unsigned char* __restrict__ high, long long n_rays, const bh_xyz* __restrict__ pixels,
                      const float* __restrict__ target, long long n_pix, double* out) {
    __shared__ double part[kReduceThreads];
    const int b = blockIdx.x;
    double acc = 0.0;
    if (b == 0) {
        for (long long p = threadIdx.x; p < n_pix; p += kReduceThreads) {
            const double d = pixels[p].y - (double)target[p];
            acc += d * d;
        }
    } else if (b <= 2) {           // spin, inclination: images of order one and two
        for (long long i = threadIdx.x; i < n_rays; i += kReduceThreads)
            if (!high[i]) acc += grad[i * 4 + (b - 1)];
    } else if (b <= 4) {           // Eddington ratio, r_out: every ray
        for (long long i = threadIdx.x; i < n_rays; i += kReduceThreads) acc += grad[i * 4 + (b - 1)];
    } else if (b <= 7) {
        for (long long i = threadIdx.x; i < 2 * n_rays; i += kReduceThreads) acc += edge[i * 3 + (b - 5)];
    } else {                       // spin, inclination: order three and higher
        for (long long i = threadIdx.x; i < n_rays; i += kReduceThreads)
            if (high[i]) acc += grad[i * 4 + (b - 8)];
    }
    part[threadIdx.x] = acc;
    __syncthreads();
    for (int s = kReduceThreads / 2; s > 0; s >>= 1) {
        if (threadIdx.x < s) part[threadIdx.x] += part[threadIdx.x + s];
        __syncthreads();
    }
    if (threadIdx.x == 0) out[b] = part[0];
}

}  // namespace

int adjoint_block_size() { return kAdjBlock; }

int reverse_blocks_per_sm() {
    int n = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, reverse_kernel, kAdjBlock, kAdjShared);
    return n;
}

int adjoint_blocks_per_sm(int block_size) {
    int n = 0;
    if (block_size != kAdjBlock) return 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, adjoint_kernel, block_size, kAdjShared);
    return n;
}

cudaError_t launch_adjoint(const AdjointLaunch& L, cudaStream_t stream) {
    if (L.block != kAdjBlock) return cudaErrorInvalidValue;
    if (L.n_rays > 0) {
        edge_candidates_kernel<<<(unsigned)((L.n_rays + 255) / 256), 256, 0, stream>>>(L);
        adjoint_select_kernel<<<(unsigned)((L.n_rays + 255) / 256), 256, 0, stream>>>(L);
        // The edge terms and the rays without records beside the recorded rays:
        // long chains both, that share no output.  The empty kernel lets the
        // few long chains be placed first; the other way round they wait for
        // the persistent reverse_kernel's blocks to end (512^2 9.7 against 8.4 ms).
        // On the context's own streams that order held on each of 60 contexts;
        // waiting for the chains' launch-completion event instead, as launch_trace
        // does on a caller's stream, costs 1% (8.46 against 8.34 ms).
        cudaError_t e;
        const bool side = L.traj && L.side_stream;
        cudaStream_t s2 = side ? L.side_stream : stream;
        if (side) {
            if ((e = cudaEventRecord(L.fork_event, stream)) != cudaSuccess) return e;
            if ((e = cudaStreamWaitEvent(s2, L.fork_event, 0)) != cudaSuccess) return e;
        }
        adjoint_kernel<<<L.grid, L.block, kAdjShared, stream>>>(L);
        if (side) after_kernel<<<1, 32, 0, s2>>>();
        if (L.traj) reverse_kernel<<<L.grid_reverse, kAdjBlock, kAdjShared, s2>>>(L);
        if (side) {
            if ((e = cudaEventRecord(L.join_event, s2)) != cudaSuccess) return e;
            if ((e = cudaStreamWaitEvent(stream, L.join_event, 0)) != cudaSuccess) return e;
        }
    }
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    const long long n_pix = (long long)L.frame.width * L.frame.height;
    adjoint_reduce_kernel<<<kAdjSums, kReduceThreads, 0, stream>>>(L.ray_grad, L.edge_out, L.high_order,
                                                                  L.n_rays, L.pixels, L.target, n_pix, L.sums);
    return cudaGetLastError();
}

}  // namespace bhg
