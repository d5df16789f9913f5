// bh_display.cu - The display transform on the GPU (image.cpp:22-191).
//
// A rendered frame stays on the device and leaves it as 8-bit sRGB (3 bytes
// per pixel instead of 24):
//
//   glare      add_glare (image.cpp:47-104): two separable Gaussian blurs with
//              clamped edges (sigma = radius and 3 radius), then
//              p core + near 0.7 s + far 0.3 s.  Two kernels: the rows of both
//              blurs from one tile, then the columns of both and the sum.  The
//              taps are summed in the reference's order without contraction,
//              with the reference's normalised weights computed on the host.
//   exposure   auto_exposure (image.cpp:22-45): the order statistics
//              k = (size_t)(q (n - 1)), q = 0.999 and 0.9999, of the n positive
//              finite luminances, found by a 6-pass most-significant-digit
//              radix select on the binary64 bit patterns (positive doubles
//              order like their bits).  A pass is one kernel: histograms of 11
//              bits (shared-memory bins, one global add per bin per block),
//              and the block that finishes last picks the digit.  No host round
//              trip, so the whole transform can run inside a stream or graph.
//   develop    develop (image.cpp:117-191, spectrum.cpp:137-152): exposure,
//              XYZ -> linear sRGB, gamut clamp, tone curve, sRGB transfer,
//              rounding to 8 bits; one thread per pixel.
//
// The frames of a film go through each kernel together (the grid's third
// dimension), so that small frames fill the GPU.
//
// The arithmetic is binary64 with the reference's operand order and no fused
// multiply-add, so the output equals the reference's byte for byte except
// where the device's pow/log10/tanh and the host libm's differ in the last
// bit at a rounding boundary of 255 v.
#include <cuda_runtime.h>

#include <cstdint>

#include "../../include/bh_gpu.h"
#include "bh_display.h"

namespace bhg {

namespace {

constexpr int kThreads = 256;

__device__ __forceinline__ double mul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double add(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double sub(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ int clampi(int v, int lo, int hi) { return (v < lo) ? lo : (hi < v) ? hi : v; }
__device__ __forceinline__ double clampd(double v, double lo, double hi) {
    return (v < lo) ? lo : (hi < v) ? hi : v;
}

// One pass of the separable blur for radii beyond the tiled kernels': along x
// (dir 0) or y (dir 1), one thread per pixel.
__global__ void blur_pass(const bh_xyz* __restrict__ src, bh_xyz* __restrict__ dst, int w, int h,
                          const double* __restrict__ k, int r, int dir) {
    const long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= (long long)w * h) return;
    const int y = (int)(p / w), x = (int)(p - (long long)y * w);
    double ax = 0.0, ay = 0.0, az = 0.0;
    for (int i = -r; i <= r; ++i) {
        const long long q = dir == 0 ? (long long)y * w + clampi(x + i, 0, w - 1)
                                     : (long long)clampi(y + i, 0, h - 1) * w + x;
        const double kk = __ldg(&k[i + r]);
        const bh_xyz s = src[q];
        ax = add(ax, mul(kk, s.x));
        ay = add(ay, mul(kk, s.y));
        az = add(az, mul(kk, s.z));
    }
    dst[p] = bh_xyz{ax, ay, az};
}

__global__ void glare_combine(bh_xyz* __restrict__ px, const bh_xyz* __restrict__ nearp,
                              const bh_xyz* __restrict__ farp, long long n, double core, double a, double b) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    bh_xyz p = px[i];
    const bh_xyz q = nearp[i], f = farp[i];
    p.x = add(add(mul(p.x, core), mul(q.x, a)), mul(f.x, b));
    p.y = add(add(mul(p.y, core), mul(q.y, a)), mul(f.y, b));
    p.z = add(add(mul(p.z, core), mul(q.z, a)), mul(f.z, b));
    px[i] = p;
}

// The tiled blur.  A row is 3 W doubles (x, y, z of each pixel), so a tap i of
// element e lies at e + 3 i and lanes read side by side.  One thread per pixel with
// every tap from L1 was bound by those loads (24 bytes a lane at a stride of 24)
// and by its five small launches: 66 us per 512 x 288 frame at radius 3, these two
// kernels 22 (six frames at a time); the binary64 adds and products alone need 7.
//
// Rows of both blurs: a block has 256 elements of a row and the taps on
// either side in shared memory.
__global__ void __launch_bounds__(kThreads) glare_rows(const DisplayFrame* __restrict__ frames, bh_xyz* tmp_near,
                                                       bh_xyz* tmp_far, const __grid_constant__ GlareWeights G) {
    __shared__ double tile[kThreads + 6 * kGlareMaxRadius];
    const DisplayFrame F = frames[blockIdx.z];
    const int n = 3 * F.width, e0 = (int)blockIdx.x * kThreads, rf = G.r_far, rn = G.r_near;
    if (e0 >= n) return;
    for (int y = blockIdx.y; y < F.height; y += gridDim.y) {
        const double* row = reinterpret_cast<const double*>(F.pixels + (long long)y * F.width);
        for (int t = threadIdx.x; t < kThreads + 6 * rf; t += kThreads) {
            int e = e0 - 3 * rf + t;
            // beyond either end: the edge pixel's same component
            if (e < 0) e = (e + 3 * rf) % 3;
            else if (e >= n) e = n - 3 + e % 3;
            tile[t] = row[e];
        }
        __syncthreads();
        const int e = e0 + (int)threadIdx.x;
        if (e < n) {
            const double* c = tile + threadIdx.x + 3 * rf;
            double f = 0.0, q = 0.0;
            int i = -rf;
            #pragma unroll 4
            for (; i < -rn; ++i) f = add(f, mul(G.far_w[i + rf], c[3 * i]));
            #pragma unroll 4
            for (; i <= rn; ++i) {
                const double v = c[3 * i];
                f = add(f, mul(G.far_w[i + rf], v));
                q = add(q, mul(G.near_w[i + rn], v));
            }
            #pragma unroll 4
            for (; i <= rf; ++i) f = add(f, mul(G.far_w[i + rf], c[3 * i]));
            const long long at = 3 * (F.scratch + (long long)y * F.width) + e;
            reinterpret_cast<double*>(tmp_far)[at] = f;
            reinterpret_cast<double*>(tmp_near)[at] = q;
        }
        __syncthreads();
    }
}

// Columns of both blurs and the sum: a block has 32 columns of 64 rows and the
// taps above and below in shared memory, first of the far blur's rows, then of
// the near one's; a thread has eight rows.
constexpr int kColRows = 64, kColThreads = 8, kColPer = kColRows / kColThreads;
__global__ void __launch_bounds__(32 * kColThreads) glare_cols(const DisplayFrame* __restrict__ frames,
                                                               const bh_xyz* __restrict__ tmp_near,
                                                               const bh_xyz* __restrict__ tmp_far,
                                                               const __grid_constant__ GlareWeights G) {
    extern __shared__ double ctile[];
    const DisplayFrame F = frames[blockIdx.z];
    const int n = 3 * F.width, col = (int)blockIdx.x * 32 + (int)threadIdx.x;
    if ((int)blockIdx.x * 32 >= n) return;
    const int c = (col < n) ? col : n - 1;
    for (int y0 = (int)blockIdx.y * kColRows; y0 < F.height; y0 += (int)gridDim.y * kColRows) {
        double acc[2][kColPer];
        #pragma unroll
        for (int which = 0; which < 2; ++which) {
            const int r = which ? G.r_near : G.r_far;
            const double* w = which ? G.near_w : G.far_w;
            const double* src = reinterpret_cast<const double*>(which ? tmp_near : tmp_far) + 3 * F.scratch + c;
            for (int j = threadIdx.y; j < kColRows + 2 * r; j += kColThreads)
                ctile[j * 32 + threadIdx.x] = src[(long long)n * clampi(y0 - r + j, 0, F.height - 1)];
            __syncthreads();
            #pragma unroll
            for (int q = 0; q < kColPer; ++q) acc[which][q] = 0.0;
            const double* t = ctile + threadIdx.y * 32 + threadIdx.x;
            for (int i = 0; i <= 2 * r; ++i) {
                const double k = w[i];
                #pragma unroll
                for (int q = 0; q < kColPer; ++q)
                    acc[which][q] = add(acc[which][q], mul(k, t[(i + q * kColThreads) * 32]));
            }
            __syncthreads();
        }
        if (col < n) {
            double* px = reinterpret_cast<double*>(F.pixels);
            #pragma unroll
            for (int q = 0; q < kColPer; ++q) {
                const int y = y0 + (int)threadIdx.y + q * kColThreads;
                if (y < F.height) {
                    const long long at = (long long)y * n + col;
                    px[at] = add(add(mul(px[at], G.core), mul(acc[1][q], G.a)), mul(acc[0][q], G.b));
                }
            }
        }
    }
}

__device__ __forceinline__ bool metered(double y) { return y > 0.0 && isfinite(y); }

// One digit of the radix select: histograms of the digit at `shift` (width
// `bits`) of the keys that match each target's prefix; the block that finishes
// last picks the digits that hold the targets' ranks.  With a histogram and a
// picking kernel per 8 bits and a counting kernel before them the meter took 17
// launches and 66 us per frame.
__global__ void __launch_bounds__(kThreads) exposure_pass(const DisplayFrame* __restrict__ frames, ExposureState* states,
                                                          int shift, int bits, int first, int last, double key) {
    __shared__ unsigned int bins[2][kMeterBins];
    __shared__ unsigned long long part[2][kThreads];
    __shared__ unsigned int s_last;
    const DisplayFrame F = frames[blockIdx.z];
    ExposureState* st = &states[F.index];
    const bh_xyz* px = F.pixels;
    const long long n = (long long)F.width * F.height;
    const int nb = 1 << bits;
    for (int i = threadIdx.x; i < nb; i += kThreads) bins[0][i] = bins[1][i] = 0u;
    __syncthreads();
    const unsigned long long mask = st->mask, p0 = st->prefix[0], p1 = st->prefix[1];
    const bool one = p0 == p1;               // the targets have not parted yet: one histogram
    for (long long i = (long long)blockIdx.x * kThreads + threadIdx.x; i < n; i += (long long)gridDim.x * kThreads) {
        const double y = px[i].y;
        if (!metered(y)) continue;
        const unsigned long long k = (unsigned long long)__double_as_longlong(y);
        const unsigned d = (unsigned)(k >> shift) & (unsigned)(nb - 1);
        if ((k & mask) == p0) atomicAdd(&bins[0][d], 1u);
        if (!one && (k & mask) == p1) atomicAdd(&bins[1][d], 1u);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < nb; i += kThreads) {
        if (bins[0][i]) atomicAdd(&st->hist[0][i], (unsigned long long)bins[0][i]);
        if (bins[1][i]) atomicAdd(&st->hist[1][i], (unsigned long long)bins[1][i]);
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) s_last = atomicAdd(&st->ticket, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    // Per thread the counts of `per` consecutive digits, then an inclusive scan.
    const int per = nb / kThreads;
    unsigned long long own[2] = {0ull, 0ull};
    for (int j = 0; j < per; ++j) {
        const int d = threadIdx.x * per + j;
        own[0] += __ldcg(&st->hist[0][d]);
        own[1] += __ldcg(&st->hist[one ? 0 : 1][d]);
    }
    part[0][threadIdx.x] = own[0];
    part[1][threadIdx.x] = own[1];
    __syncthreads();
    for (int off = 1; off < kThreads; off <<= 1) {
        unsigned long long v[2] = {0ull, 0ull};
        if ((int)threadIdx.x >= off) {
            v[0] = part[0][threadIdx.x - off];
            v[1] = part[1][threadIdx.x - off];
        }
        __syncthreads();
        part[0][threadIdx.x] += v[0];
        part[1][threadIdx.x] += v[1];
        __syncthreads();
    }
    // the first digit's histogram counts every metered luminance
    const unsigned long long m = first ? part[0][kThreads - 1] : st->count;
    unsigned long long rank[2];
    #pragma unroll
    for (int q = 0; q < 2; ++q) {
        if (first) {
            const unsigned long long k = m ? (unsigned long long)((q == 0 ? 0.999 : 0.9999) * (double)(m - 1)) : 0ull;
            rank[q] = (m && k > m - 1) ? m - 1 : k;
        } else {
            rank[q] = st->k[q];
        }
    }
    __syncthreads();
    if (m > 0) {
        #pragma unroll
        for (int q = 0; q < 2; ++q) {
            unsigned long long below = part[q][threadIdx.x] - own[q];
            if (rank[q] >= below && rank[q] < below + own[q]) {
                int d = threadIdx.x * per;
                const unsigned long long* hist = st->hist[one ? 0 : q];
                for (unsigned long long c; rank[q] >= below + (c = __ldcg(&hist[d])); ++d) below += c;
                st->prefix[q] |= (unsigned long long)d << shift;
                st->k[q] = rank[q] - below;
            }
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < nb; i += kThreads) st->hist[0][i] = st->hist[1][i] = 0ull;
    if (threadIdx.x == 0) {
        st->count = m;
        st->mask = mask | ((unsigned long long)(nb - 1) << shift);
        st->ticket = 0u;
        if (last) {
            double e = 1.0;
            if (m > 0) {
                const double hi = __longlong_as_double((long long)st->prefix[0]);
                const double peak = __longlong_as_double((long long)st->prefix[1]);
                if (hi > 0.0) e = key / hi;
                if (peak > 0.0) {
                    const double c = 3.0 * key / peak;
                    if (c < e) e = c;
                }
            }
            st->exposure = e;
        }
    }
}

__device__ __forceinline__ double aces_curve(double x) {
    const double a = 2.51, b = 0.03, c = 2.43, d = 0.59, e = 0.14;
    return clampd(mul(x, add(mul(a, x), b)) / add(mul(x, add(mul(c, x), d)), e), 0.0, 1.0);
}

__device__ __forceinline__ double srgb_encode(double v) {
    v = clampd(v, 0.0, 1.0);
    return (v <= 0.0031308) ? mul(12.92, v) : sub(mul(1.055, pow(v, 1.0 / 2.4)), 0.055);
}

__global__ void develop_kernel(const DisplayFrame* __restrict__ frames, const ExposureState* __restrict__ states,
                               double fixed, int tonemap, double log_k, double denom) {
    const DisplayFrame F = frames[blockIdx.z];
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (long long)F.width * F.height) return;
    const double ex = (fixed > 0.0) ? fixed : states[F.index].exposure;
    uint8_t* __restrict__ out = F.rgb;
    bh_xyz c = F.pixels[i];
    if (!isfinite(c.x) || !isfinite(c.y) || !isfinite(c.z)) c = bh_xyz{0.0, 0.0, 0.0};
    c.x = mul(c.x, ex);
    c.y = mul(c.y, ex);
    c.z = mul(c.z, ex);
    double v[3];
    v[0] = sub(sub(mul(3.2404542, c.x), mul(1.5371385, c.y)), mul(0.4985314, c.z));
    v[1] = add(add(mul(-0.9692660, c.x), mul(1.8760108, c.y)), mul(0.0415560, c.z));
    v[2] = add(sub(mul(0.0556434, c.x), mul(0.2040259, c.y)), mul(1.0572252, c.z));
    double m = v[0];
    if (v[1] < m) m = v[1];
    if (v[2] < m) m = v[2];
    if (!(m >= 0.0)) {
        v[0] = sub(v[0], m);
        v[1] = sub(v[1], m);
        v[2] = sub(v[2], m);
    }
    #pragma unroll
    for (int ch = 0; ch < 3; ++ch) {
        double x = (v[ch] < 0.0) ? 0.0 : v[ch];
        switch (tonemap) {
        case BH_TONEMAP_LINEAR: x = clampd(x, 0.0, 1.0); break;
        case BH_TONEMAP_REINHARD: x = x / add(1.0, x); break;
        case BH_TONEMAP_ACES: x = aces_curve(x); break;
        case BH_TONEMAP_LOG:
            x = clampd(log10(add(1.0, mul(log_k, (x < 0.0) ? 0.0 : x))) / denom, 0.0, 1.0);
            break;
        default: {
            const double cap = 0.12, wt = 0.5;
            const double f = aces_curve(x);
            const double l = clampd(log10(add(1.0, mul(log_k, (x < 0.0) ? 0.0 : x))) / denom, 0.0, 1.0);
            const double lift = mul(cap, tanh(mul(wt, l) / cap));
            x = clampd(add(f, mul(lift, sub(1.0, f))), 0.0, 1.0);
            break;
        }
        }
        out[i * 3 + ch] = (uint8_t)lround(mul(255.0, srgb_encode(x)));
    }
}

}  // namespace

cudaError_t launch_display(const DisplayLaunch& L, cudaStream_t s) {
    if (L.n <= 0 || L.max_pixels <= 0) return cudaSuccess;
    const unsigned blocks = (unsigned)((L.max_pixels + kThreads - 1) / kThreads);
    const unsigned rows = (unsigned)(L.max_height < 65535 ? L.max_height : 65535);
    if (L.glare == 1) {
        const size_t shared = sizeof(double) * 32 * (kColRows + 2 * L.w.r_far);
        glare_rows<<<dim3((3 * L.max_width + kThreads - 1) / kThreads, rows, L.n), kThreads, 0, s>>>(
            L.frames, L.tmp_near, L.tmp_far, L.w);
        glare_cols<<<dim3((3 * L.max_width + 31) / 32, (L.max_height + kColRows - 1) / kColRows, L.n),
                     dim3(32, kColThreads), shared, s>>>(L.frames, L.tmp_near, L.tmp_far, L.w);
    } else if (L.glare == 2) {
        for (int i = 0; i < L.n; ++i) {
            const DisplayFrame& F = L.h_frames[i];
            const long long n = (long long)F.width * F.height;
            const unsigned b = (unsigned)((n + kThreads - 1) / kThreads);
            bh_xyz *t = L.tmp + F.scratch, *nr = L.tmp_near + F.scratch, *fr = L.tmp_far + F.scratch;
            blur_pass<<<b, kThreads, 0, s>>>(F.pixels, t, F.width, F.height, L.k_near, L.w.r_near, 0);
            blur_pass<<<b, kThreads, 0, s>>>(t, nr, F.width, F.height, L.k_near, L.w.r_near, 1);
            blur_pass<<<b, kThreads, 0, s>>>(F.pixels, t, F.width, F.height, L.k_far, L.w.r_far, 0);
            blur_pass<<<b, kThreads, 0, s>>>(t, fr, F.width, F.height, L.k_far, L.w.r_far, 1);
            glare_combine<<<b, kThreads, 0, s>>>(F.pixels, nr, fr, n, L.w.core, L.w.a, L.w.b);
        }
    }
    if (!(L.exposure > 0.0)) {
        // enough blocks to fill the GPU over all frames, each with a few
        // thousand pixels at least
        const long long want = (L.max_pixels + 8 * kThreads - 1) / (8 * kThreads);
        const long long most = (4LL * L.sm_count + L.n - 1) / L.n;
        const unsigned grid = (unsigned)(want < most ? want : most);
        static_assert(512 % kThreads == 0, "a thread takes whole digits of the scan");
        for (int pass = 0; pass < 6; ++pass) {
            // five digits of 11 bits and one of 9
            const int bits = pass < 5 ? kMeterBits : 9, shift = pass < 5 ? 53 - kMeterBits * pass : 0;
            exposure_pass<<<dim3(grid, 1, L.n), kThreads, 0, s>>>(L.frames, L.states, shift, bits, pass == 0,
                                                                 pass == 5, L.key);
        }
    }
    if (L.develop)
        develop_kernel<<<dim3(blocks, 1, L.n), kThreads, 0, s>>>(L.frames, L.states, L.exposure, L.tonemap, L.log_k,
                                                                L.denom);
    return cudaGetLastError();
}

}  // namespace bhg
