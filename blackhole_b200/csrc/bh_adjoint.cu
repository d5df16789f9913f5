// bh_adjoint.cu - The discrete-adjoint kernels and reductions (sm_100a).
//
// adjoint_select_kernel: one thread per ray.  The render's hit record says
// which rays have a gradient at all: those that ended on the disc or saw a sky
// that varies at their direction.  A captured ray, or one that met the uniform
// background, is done here; the others are listed.
//
// adjoint_kernel: a warp takes 32 jobs at a time from a global atomic counter;
// each lane owns `checkpoint_slots` stored states in global memory, interleaved
// over the warp, for the job it is working on (bh_adjoint.cuh has the per-ray
// algorithm).  A ray's loss weight is 2 (Y_pixel - target) / S^2 for
// Loss = sum over pixels of (Y_pixel - target)^2, Y_pixel being the sample
// mean of the rendered frame (bh_gpu_render's output).
//
// The edge pass: a point-sampled frame has no derivative with respect to
// r_out, and its derivatives with respect to the spin and the inclination
// miss the motion of the disc's edges; the derivative of the frame averaged
// over each sample's cell has both.  edge_candidates_kernel picks each
// sample's first two equatorial crossings near an edge (adj::edge_mask,
// against the spread of the neighbouring samples' same crossing; the render
// records the crossings), and the adjoint kernel takes their edge terms
// (adj::edge_sample, weight 2 (Y_pixel - target)) as its first jobs, so the
// long ones overlap the per-ray work instead of forming a tail of their own.
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
    if (id >= L.n_rays) return;
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
            const unsigned long long at = atomicAdd(&L.counters[6], 1ull);
            L.cand[at] = ((unsigned long long)(2 * id + j) << 2) | (unsigned long long)m;
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
    if (id < L.n_rays) {
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
                listed = w != 0.0 && (gY[0] != 0.0 || gY[1] != 0.0 || gY[2] != 0.0);
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
    const unsigned m = __ballot_sync(kFull, listed);
    const unsigned nd = __popc(__ballot_sync(kFull, what == BH_HIT_DISC));
    const unsigned ns = __popc(__ballot_sync(kFull, what == BH_HIT_SKY));
    const unsigned nh = __popc(__ballot_sync(kFull, high));
    const unsigned st = __reduce_add_sync(kFull, steps);
    unsigned long long base = 0;
    if (lane == 0) {
        if (m) base = atomicAdd(&L.counters[10], (unsigned long long)__popc(m));
        if (st) atomicAdd(&L.counters[1], (unsigned long long)st);
        if (nd) atomicAdd(&L.counters[3], (unsigned long long)nd);
        if (ns) atomicAdd(&L.counters[4], (unsigned long long)ns);
        if (nh) atomicAdd(&L.counters[9], (unsigned long long)nh);
    }
    base = __shfl_sync(kFull, base, 0);
    if (listed) L.rays[base + __popc(m & ((1u << lane) - 1u))] = (int)id;
}

// One queue of jobs: first the edge candidates (each a forward pass to its
// crossing, the continuation past it and a reverse sweep: the longest jobs),
// then the listed rays.  Results go to per-ray and per-crossing slots, so the
// sums do not depend on which lane took which job.
__global__ void __launch_bounds__(kAdjBlock, kAdjBlocksPerSm) adjoint_kernel(const __grid_constant__ AdjointLaunch L) {
    const int lane = threadIdx.x & 31;
    const long long warp = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int slots = L.X.checkpoint_slots;
    double* ck = L.ckpt + warp * slots * adj::kCkWords * 32 + lane;
    const int SS = L.frame.S * L.frame.S;
    const unsigned long long n_cand = L.counters[6], n_jobs = n_cand + L.counters[10];
    unsigned long long replay = 0, max_int = 0, edge_steps = 0, edge_cells = 0;
    for (;;) {
        unsigned long long job = 0;
        if (lane == 0) job = atomicAdd(&L.counters[0], 32ull);
        job = __shfl_sync(kFull, job, 0);
        if (job >= n_jobs) break;
        job += lane;
        int px, py, k;
        if (job < n_cand) {
            const unsigned long long c = L.cand[job];
            const long long xs = (long long)(c >> 2);     // 2 * ray + crossing
            const long long pix = ray_pixel(L, xs >> 1, &px, &py, &k);
            const double w = 2.0 * (L.pixels[pix].y - (double)L.target[pix]);
            double out[3];
            int n_cells = 0;
            edge_steps += (unsigned long long)adj::edge_sample(L.frame, L.X, L.sky, px, py, k, (int)(xs & 1) + 1,
                                                               (int)(c & 3ull), w, ck, slots, 32, out, &n_cells);
            edge_cells += (unsigned long long)n_cells;
            L.edge_out[3 * xs] = out[0];
            L.edge_out[3 * xs + 1] = out[1];
            L.edge_out[3 * xs + 2] = out[2];
        } else if (job < n_jobs) {
            const long long id = L.rays[job - n_cand];
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
        adjoint_kernel<<<L.grid, L.block, kAdjShared, stream>>>(L);
    }
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    const long long n_pix = (long long)L.frame.width * L.frame.height;
    adjoint_reduce_kernel<<<kAdjSums, kReduceThreads, 0, stream>>>(L.ray_grad, L.edge_out, L.high_order,
                                                                  L.n_rays, L.pixels, L.target, n_pix, L.sums);
    return cudaGetLastError();
}

}  // namespace bhg
