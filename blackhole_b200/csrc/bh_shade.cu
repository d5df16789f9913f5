// bh_shade.cu - Shading and stats kernels of the render path.
//
//   shade_kernel      per-pixel shading of the terminated rays (render.cpp:265-393,
//                     disc.h:94-126, spectrum.cpp:123-134, scene.h:111-223) and the
//                     sample average of render.cpp:456-462.
//                     It sums the per-frame stats (render.cpp:481-494) on the way.
//   flux_kernel       a fixed-order sum of a frame's flux.
//
// Everything here is binary64: it runs once per ray, after the integration.
#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>

#include "../../include/bh_gpu.h"
#include "bh_common.cuh"
#include "bh_frame.h"
#include "bh_launch.h"

namespace bhg {

namespace {

__device__ void blackbody(const double* __restrict__ tab, double T, double o[3]) {
    // spectrum.cpp:123-134
    const double kLogTMin = 1.6989700043360187, kLogTMax = 9.4771212547196626;
    const double lg = log10(dclamp(T, 50.0, 3.0e9));
    const double f = (lg - kLogTMin) / (kLogTMax - kLogTMin) * (kTableN - 1);
    int i = (int)f;
    i = (i < 0) ? 0 : (i > kTableN - 2 ? kTableN - 2 : i);
    const double u = f - i;
    o[0] = exp(__ldg(&tab[i]) * (1.0 - u) + __ldg(&tab[i + 1]) * u);
    o[1] = exp(__ldg(&tab[kTableN + i]) * (1.0 - u) + __ldg(&tab[kTableN + i + 1]) * u);
    o[2] = exp(__ldg(&tab[2 * kTableN + i]) * (1.0 - u) + __ldg(&tab[2 * kTableN + i + 1]) * u);
}

__device__ double circ_energy(double a, double r, int sigma) {
    const double sr = sqrt(r);
    const double num = r * r - 2.0 * r + sigma * a * sr;
    const double den = r * sqrt(r * r - 3.0 * r + 2.0 * sigma * a * sr);
    return num / den;
}
__device__ double circ_angmom(double a, double r, int sigma) {
    const double sr = sqrt(r);
    const double num = sigma * sr * (r * r - 2.0 * sigma * a * sr + a * a);
    const double den = r * sqrt(r * r - 3.0 * r + 2.0 * sigma * a * sr);
    return num / den;
}

// Novikov-Thorne effective temperature (disc.h:94-121, W from disc.h:46-64).
__device__ double disc_temperature(const FrameParams& F, double r) {
    if (r <= F.r_in || r > F.r_out) return 0.0;
    const double a = F.disc_a;
    const int sg = F.disc_sigma;
    const double x = sqrt(r);
    double W = x - F.x0 - 1.5 * a * log(x / F.x0);
    #pragma unroll
    for (int i = 0; i < 3; ++i)
        if (F.pt_c[i] != 0.0) W = W - F.pt_c[i] * log((x - F.pt_x[i]) / F.pt_den[i]);
    const double r32 = r * sqrt(r);
    const double Om = sg / (r32 + sg * a);
    const double dd = r32 + sg * a;
    const double dOm = -sg * 1.5 * sqrt(r) / (dd * dd);
    const double E = circ_energy(a, r, sg);
    const double L = circ_angmom(a, r, sg);
    const double den = E - Om * L;
    if (!(den > 0.0)) return 0.0;
    double Fd = (-dOm) / (4.0 * kPi * r * den * den) * W;
    if (!(Fd > 0.0 && isfinite(Fd))) Fd = 0.0;
    const double Fl = Fd * F.disc_mdot * 2.99792458e8 * 2.99792458e8 / F.disc_rg2;
    if (Fl <= 0.0) return 0.0;
    return pow(Fl / 5.670374419e-8, 0.25);
}

// Position derivatives dr, dth, dphi at a state (the RHS of geodesic.h:58-61).
__device__ void position_rates(const FrameParams& F, const double* y, double d[3]) {
    const double a = F.a, a2 = F.a2;
    const double r = y[1], th = y[2];
    double sn, cs;
    sincos(th, &sn, &cs);
    if (fabs(sn) < 1e-9) sn = (sn < 0.0) ? -1e-9 : 1e-9;
    const double sn2 = sn * sn, cs2 = cs * cs;
    const double Sig = r * r + a2 * cs2;
    const double Del = r * r - 2.0 * r + a2;
    const double SD = Sig * Del;
    const double gtp = -2.0 * a * r / SD;
    const double gpp = (Del - a2 * sn2) / (SD * sn2);
    d[0] = (Del / Sig) * y[5];
    d[1] = (1.0 / Sig) * y[6];
    d[2] = gtp * y[4] + gpp * y[7];
}

// render.cpp:15-26 (normalised at render.cpp:364-366).
__device__ bool sky_direction(const FrameParams& F, const double* y, double v[3]) {
    double dd[3];
    position_rates(F, y, dd);
    const double a = F.a;
    const double r = y[1], th = y[2], ph = y[3];
    const double R = sqrt(r * r + a * a);
    double sn, cs, sp, cp;
    sincos(th, &sn, &cs);
    sincos(ph, &sp, &cp);
    const double dr = dd[0], dth = dd[1], dph = dd[2];
    const double dR = (R > 0.0) ? r / R * dr : dr;
    v[0] = dR * sn * cp + R * cs * dth * cp - R * sn * sp * dph;
    v[1] = dR * sn * sp + R * cs * dth * sp + R * sn * cp * dph;
    v[2] = dr * cs - r * sn * dth;
    const double vn = sqrt(v[0] * v[0] + v[1] * v[1] + v[2] * v[2]);
    if (!(vn > 0.0)) return false;
    v[0] /= vn; v[1] /= vn; v[2] /= vn;
    return true;
}

// Star field + diffuse background along direction d (scene.h:111-158, 202-223).
__device__ void sky_radiance(const SkyData& sky, const FrameParams& F, const double d[3], double o[3]) {
    o[0] = o[1] = o[2] = 0.0;
    if (sky.n_stars > 0) {
        const double cutoff = F.cutoff, inv2s2 = F.inv2s2, norm = F.psf_norm;
        const double theta = acos(dclamp(d[2], -1.0, 1.0));
        const double phi = atan2(d[1], d[0]);
        const int it = (int)(theta / kPi * kLat);
        const double sn = dmaxr(sin(theta), 1e-6);
        const double dlon = 2.0 * kPi / kLon;
        int span_p = (int)ceil(cutoff / (sn * dlon));
        if (span_p < 1) span_p = 1;
        const int sp = (span_p * 2 + 1 >= kLon) ? kLon / 2 : span_p;
        const int pbase = (int)((phi + kPi) / (2.0 * kPi) * kLon);
        // The stars k0 <= k < k1, in catalogue order.
        auto stars = [&](int k0, int k1) {
            for (int k = k0; k < k1; ++k) {
                const double4 s = sky.star_pos[k];
                const double dot = dclamp(d[0] * s.x + d[1] * s.y + d[2] * s.z, -1.0, 1.0);
                if (dot < F.cut_dot) continue;   // outside the cutoff, without the acos
                const double ang = (dot > 0.9999995) ? sqrt(dmaxr(0.0, 2.0 * (1.0 - dot))) : acos(dot);
                if (ang > cutoff) continue;
                const double w = norm * exp(-ang * ang * inv2s2) * s.w;
                const double4 c = sky.star_col[k];
                o[0] += w * c.x * c.z;
                o[1] += w;
                o[2] += w * c.y * c.z;
            }
        };
        if (whole_window(pbase, sp, kLon)) {
            // the window's bins of a row are neighbours, and so are their stars:
            // one run per row
            for (int a = -F.span_t; a <= F.span_t; ++a) {
                const int ti = it + a;
                if (ti < 0 || ti >= kLat) continue;
                const int bin = ti * kLon + pbase;
                stars(__ldg(&sky.bin_start[bin - sp]), __ldg(&sky.bin_start[bin + sp + 1]));
            }
        } else {
            const int base = ((pbase % kLon) + kLon) % kLon;
            for (int a = -F.span_t; a <= F.span_t; ++a) {
                const int ti = it + a;
                if (ti < 0 || ti >= kLat) continue;
                for (int b = base - sp; b <= base + sp; ++b) {
                    const int pi = ((b % kLon) + kLon) % kLon;
                    const int bin = ti * kLon + pi;
                    stars(__ldg(&sky.bin_start[bin]), __ldg(&sky.bin_start[bin + 1]));
                }
            }
        }
    }
    if (F.milky_way) {
        double amp;
        if (F.sky_mode == BH_SKY_UNIFORM) {
            amp = sky.diffuse_L;
        } else {
            const double ca = 0.8660254037844387, sa = 0.5;
            const double g1 = ca * d[1] + sa * d[2];
            const double g2 = -sa * d[1] + ca * d[2];
            const double sin_b = dclamp(g2, -1.0, 1.0);
            const double band = exp(-fabs(sin_b) / 0.055);
            const double l = atan2(g1, d[0]);
            const double bulge = 0.55 + 0.45 * exp(-(l * l) / (2.0 * 0.45 * 0.45));
            const double lane = 0.65 + 0.35 * sin(l * 7.3 + sin_b * 41.0) * sin(l * 3.1 - sin_b * 17.0);
            amp = sky.diffuse_L * band * bulge * dmaxr(0.0, lane);
        }
        o[0] += amp * sky.mw_x * sky.mw_inv;
        o[1] += amp;
        o[2] += amp * sky.mw_z * sky.mw_inv;
    }
}

// render.cpp:265-375 for one terminated ray.  Returns g (disc/surface hits)
// and the sky direction (escaped rays) for the per-sample results.
__device__ void shade_one(const SkyData& sky, const FrameParams& F, const HitRecord& hr, double c[3],
                          double* g_out, double dir[3]) {
    c[0] = c[1] = c[2] = 0.0;
    *g_out = 0.0;
    dir[0] = dir[1] = dir[2] = 0.0;
    const double* y = hr.y;
    switch (hr.what) {
    case BH_HIT_DISC: {
        const double r = y[1];
        double T = disc_temperature(F, r);
        if (T <= 0.0) return;
        if (F.hs_enabled) {
            const double t_emit = F.observer_time + y[0];
            const double phi_s = F.hs_phi0 + F.hs_omega * t_emit;
            const double dx = r * cos(y[3]) - F.hs_r * cos(phi_s);
            const double dy = r * sin(y[3]) - F.hs_r * sin(phi_s);
            const double d2 = dx * dx + dy * dy;
            const double f = 1.0 + F.hs_contrast * exp(-0.5 * d2 / (F.hs_sigma * F.hs_sigma));
            T *= pow(f, 0.25);
        }
        // keplerian_four_velocity (kerr.h:260-266) and redshift_factor (render.cpp:31-34)
        const double a = F.disc_a;
        const int sg = F.disc_sigma;
        const double r32 = r * sqrt(r);
        const double Om = sg / (r32 + sg * a);
        const double dsc = r * r * r - 3.0 * r * r + 2.0 * sg * a * r32;
        const double ut = (r32 + sg * a) / sqrt(dmaxr(1e-300, dsc));
        const double ku = y[4] * ut + y[5] * 0.0 + y[6] * 0.0 + y[7] * (Om * ut);
        const double g = (ku > 1e-12) ? 1.0 / ku : 0.0;
        if (g <= 0.0) return;
        *g_out = g;
        blackbody(sky.table, g * T, c);
        return;
    }
    case BH_HIT_SUN: {
        const double a = F.a, r = y[1], th = y[2];
        double sn = sin(th);
        if (fabs(sn) < 1e-9) sn = (sn < 0.0) ? -1e-9 : 1e-9;
        const double cs = cos(th);
        const double Sig = r * r + F.a2 * cs * cs;
        const double mtt = -(1.0 - 2.0 * r / Sig);
        if (mtt >= 0.0) return;
        const double ut = 1.0 / sqrt(-mtt);
        const double ku = y[4] * ut;
        const double g = (ku > 1e-12) ? 1.0 / ku : 0.0;
        if (g <= 0.0) return;
        *g_out = g;
        // Viewing direction (normalised when non-zero, render.cpp:311-316) and
        // Eddington limb darkening (scene.h:266-276).
        double v[3];
        (void)sky_direction(F, y, v);
        const double rr = sqrt(r * r + a * a);
        const double p[3] = {rr * sin(th) * cos(y[3]), rr * sin(th) * sin(y[3]), r * cos(th)};
        double limb = 1.0;
        double nrm[3] = {p[0] - F.sun_c[0], p[1] - F.sun_c[1], p[2] - F.sun_c[2]};
        const double len = sqrt(nrm[0] * nrm[0] + nrm[1] * nrm[1] + nrm[2] * nrm[2]);
        if (len > 0.0) {
            nrm[0] /= len; nrm[1] /= len; nrm[2] /= len;
            const double mu = dclamp(-(nrm[0] * v[0] + nrm[1] * v[1] + nrm[2] * v[2]), 0.0, 1.0);
            limb = (2.0 + 3.0 * mu) / 5.0;
        }
        blackbody(sky.table, g * F.sun_T_eff / F.sun_redshift_div, c);
        c[0] *= limb; c[1] *= limb; c[2] *= limb;
        return;
    }
    case BH_HIT_STAR: {
        const double r = y[1], th = y[2], ph = y[3];
        const double sn = sin(th);
        const double norm2 = 1.0 - 2.0 / F.ns_R - F.ns_Omega * F.ns_Omega * F.ns_R * F.ns_R * sn * sn;
        const double ut = (norm2 > 1e-12) ? 1.0 / sqrt(norm2) : 1.0;
        const double ku = y[4] * ut + y[7] * (F.ns_Omega * ut);
        if (!(ku > 1e-12)) return;
        const double g = 1.0 / ku;
        *g_out = g;
        double T = F.ns_T_eff;
        if (F.ns_caps) {
            const double t_emit = F.observer_time + y[0];
            const double phase = F.ns_cap_phase0 + F.ns_Omega * t_emit;
            const double m0 = sin(F.ns_cap_tilt) * cos(phase), m1 = sin(F.ns_cap_tilt) * sin(phase),
                         m2 = cos(F.ns_cap_tilt);
            const double n0 = sin(th) * cos(ph), n1 = sin(th) * sin(ph), n2 = cos(th);
            double ang = acos(dclamp(n0 * m0 + n1 * m1 + n2 * m2, -1.0, 1.0));
            if (F.ns_two_caps) ang = dminr(ang, kPi - ang);
            if (ang <= F.ns_cap_radius) {
                const double edge = 0.9 * F.ns_cap_radius;
                if (ang <= edge) {
                    T = F.ns_cap_T;
                } else {
                    const double u = (ang - edge) / (F.ns_cap_radius - edge);
                    const double w = 0.5 * (1.0 + cos(kPi * u));
                    T = F.ns_T_eff + (F.ns_cap_T - F.ns_T_eff) * w;
                }
            }
        }
        const double f = 1.0 - 2.0 / r;
        const double mu = (f > 0.0) ? dclamp(-y[5] * sqrt(f) / ku, 0.0, 1.0) : 1.0;
        const double limb = (2.0 + 3.0 * mu) / 5.0;
        blackbody(sky.table, g * T, c);
        c[0] *= limb; c[1] *= limb; c[2] *= limb;
        return;
    }
    case BH_HIT_SKY: {
        double v[3];
        if (!sky_direction(F, y, v)) return;
        dir[0] = v[0]; dir[1] = v[1]; dir[2] = v[2];
        if (!F.stars_enabled) return;
        sky_radiance(sky, F, v, c);
        return;
    }
    default:
        return;
    }
}

// A thread's share of a frame's stats (render.cpp:481-494).
struct StatsAcc {
    unsigned long long steps = 0, attempts = 0;
    unsigned rays = 0, cls[6] = {0, 0, 0, 0, 0, 0}, jet = 0;
    double mn = 0.0, mq = 0.0, flux = 0.0;
};

__device__ __forceinline__ unsigned long long dbits(double x) { return (unsigned long long)__double_as_longlong(x); }

__device__ __forceinline__ unsigned long long warp_sum(unsigned long long v) {
    #pragma unroll
    for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
    return v;
}
__device__ __forceinline__ double warp_sum(double v) {
    #pragma unroll
    for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
    return v;
}
__device__ __forceinline__ unsigned long long warp_max(unsigned long long v) {
    #pragma unroll
    for (int o = 16; o; o >>= 1) {
        const unsigned long long u = __shfl_xor_sync(kFull, v, o);
        if (u > v) v = u;
    }
    return v;
}

constexpr int kShadeThreads = 128;
constexpr int kShadeWarps = kShadeThreads / 32;

static_assert(offsetof(FrameStats, steps) == 8 && offsetof(FrameStats, attempts) == 16 &&
                  offsetof(FrameStats, captured) == 24 && offsetof(FrameStats, disc_hits) == 32 &&
                  offsetof(FrameStats, sun_hits) == 40 && offsetof(FrameStats, star_hits) == 48 &&
                  offsetof(FrameStats, escaped) == 56 && offsetof(FrameStats, exhausted) == 64 &&
                  offsetof(FrameStats, jet_rays) == 72 && BH_HIT_HORIZON == 0 && BH_HIT_DISC == 1 && BH_HIT_SUN == 2 &&
                  BH_HIT_STAR == 3 && BH_HIT_SKY == 4 && BH_HIT_EXHAUSTED == 5,
              "block_stats adds the counters in this order");

// The block's sum of its threads' stats: counts and maxima, whose sums do not
// depend on the order, are added to the frame's stats; the flux goes to the
// block's partial.
__device__ void block_stats(const StatsAcc& t, FrameStats* out, double* flux) {
    __shared__ unsigned long long s_sum[10], s_max[2];
    __shared__ double s_flux[kShadeWarps];
    if (threadIdx.x < 10) s_sum[threadIdx.x] = 0ull;
    if (threadIdx.x < 2) s_max[threadIdx.x] = 0ull;
    __syncthreads();
    unsigned long long v[10] = {__reduce_add_sync(kFull, t.rays), warp_sum(t.steps), warp_sum(t.attempts)};
    #pragma unroll
    for (int q = 0; q < 6; ++q) v[3 + q] = __reduce_add_sync(kFull, t.cls[q]);
    v[9] = __reduce_add_sync(kFull, t.jet);
    // non-negative doubles order like their bits
    const unsigned long long mn = warp_max(dbits(t.mn)), mq = warp_max(dbits(t.mq));
    const double f = warp_sum(t.flux);
    if ((threadIdx.x & 31) == 0) {
        s_flux[threadIdx.x >> 5] = f;
        #pragma unroll
        for (int q = 0; q < 10; ++q)
            if (v[q]) atomicAdd(&s_sum[q], v[q]);
        atomicMax(&s_max[0], mn);
        atomicMax(&s_max[1], mq);
    }
    __syncthreads();
    if (threadIdx.x < 10) {
        // rays, steps, attempts, the six classes in BH_HIT_* order, jet rays:
        // the order of FrameStats' counters
        if (s_sum[threadIdx.x]) atomicAdd(&out->rays + threadIdx.x, s_sum[threadIdx.x]);
    } else if (threadIdx.x == 32) {
        atomicMax(&out->max_norm_bits, s_max[0]);
    } else if (threadIdx.x == 64) {
        atomicMax(&out->max_q_bits, s_max[1]);
    } else if (threadIdx.x == 96) {
        double s = s_flux[0];
        for (int i = 1; i < kShadeWarps; ++i) s += s_flux[i];
        *flux = s;
    }
}

struct ShadeArgs {
    const FrameParams* frames;
    long long pixel_lo, pixel_hi;
    const HitRecord* hits;
    SkyData sky;
    bh_xyz* pixels;
    bh_ray_result* rays;
    const double* jet;
    FrameStats* stats;
    double* flux;
    int flux_per_frame;
};

// The frame's pixels (grid.y: frames) shaded, 128 at a time per block, and
// its stats summed on the way: the hit records (96 bytes a ray) are read once.
// With the stats in a pass of their own over the records a 1024^2 mixed frame
// took 162 us for both, now 128, a 2048^2 one 445 and 290.  What is left is the
// shading's binary64 chains (20 warps per SM; 16 and 24 the same within 5%).
__global__ void __launch_bounds__(kShadeThreads, 5) shade_kernel(ShadeArgs A) {
    const FrameParams& F = A.frames[blockIdx.y];
    const long long npx = (long long)F.width * F.height;
    const long long hi = (A.pixel_hi < npx) ? A.pixel_hi : npx;
    const int SS = F.S * F.S;
    StatsAcc st;
    for (long long p = A.pixel_lo + (long long)blockIdx.x * kShadeThreads + threadIdx.x; p < hi;
         p += (long long)gridDim.x * kShadeThreads) {      // frame-local pixel, band order
        int px, py;
        pixel_xy(F.width, F.height, p, &px, &py);
        double acc[3] = {0.0, 0.0, 0.0};
        for (int k = 0; k < SS; ++k) {
            const long long rid = F.ray_begin + p * SS + k;
            const HitRecord hr = A.hits[rid];
            double c[3], g, dir[3];
            shade_one(A.sky, F, hr, c, &g, dir);
            // Whatever the ray ended on, the jet light it collected on the way is
            // added in the jet's one colour (render.cpp:377-392).
            const double jet = (F.jet_enabled && A.jet) ? A.jet[rid] : 0.0;
            if (jet > 0.0) {
                c[0] += F.jet_col[0] * jet;
                c[1] += F.jet_col[1] * jet;
                c[2] += F.jet_col[2] * jet;
                st.jet += 1;
            }
            acc[0] += c[0]; acc[1] += c[1]; acc[2] += c[2];
            st.rays += 1;
            st.steps += (unsigned long long)hr.steps;
            st.attempts += (unsigned long long)hr.attempts;
            #pragma unroll
            for (int q = 0; q < 6; ++q) st.cls[q] += (hr.what == q) ? 1u : 0u;
            st.mn = dmaxr(st.mn, hr.max_norm);
            st.mq = dmaxr(st.mq, hr.max_q);
            if (A.rays) {
                bh_ray_result& o = A.rays[((long long)py * F.width + px) * SS + k];
                o.what = hr.what;
                o.steps = hr.steps;
                #pragma unroll
                for (int i = 0; i < 8; ++i) o.y[i] = hr.y[i];
                o.g = g;
                o.dir[0] = dir[0]; o.dir[1] = dir[1]; o.dir[2] = dir[2];
                o.xyz.x = c[0]; o.xyz.y = c[1]; o.xyz.z = c[2];
                o.attempts = hr.attempts;
                o.reserved = 0;
                o.max_norm = hr.max_norm;
                o.max_q = hr.max_q;
                o.jet = jet;
            }
        }
        const double w = F.inv_SS;
        bh_xyz& out = A.pixels[F.pixel_begin + (long long)py * F.width + px];
        out.x = acc[0] * w;
        out.y = acc[1] * w;
        out.z = acc[2] * w;
        st.flux += acc[1] * w;
    }
    block_stats(st, &A.stats[blockIdx.y], &A.flux[(long long)blockIdx.y * A.flux_per_frame + blockIdx.x]);
}

constexpr int kRedThreads = 256;

// The flux of a frame, one block each: thread t sums the partials t,
// t + kRedThreads, ... in that order, then a fixed tree combines the threads:
// the same bits on every run.
__global__ void __launch_bounds__(kRedThreads) flux_kernel(const double* __restrict__ partials, int count,
                                                           FrameStats* __restrict__ out) {
    __shared__ double s_flux[kRedThreads / 32];
    const double* mine = partials + (long long)blockIdx.x * count;
    double f = 0.0;
    for (int b = threadIdx.x; b < count; b += kRedThreads) f += mine[b];
    f = warp_sum(f);
    if ((threadIdx.x & 31) == 0) s_flux[threadIdx.x >> 5] = f;
    __syncthreads();
    if (threadIdx.x != 0) return;
    for (int i = 1; i < kRedThreads / 32; ++i) f += s_flux[i];
    out[blockIdx.x].total_flux = f;
}


// Device shading functions at given inputs (known-answer tests): what 0,
// the disc's effective temperature at radii in[i]; what 1, the blackbody
// XYZ of temperatures in[i] from the device table (3 per input).
__global__ void eval_shade_kernel(int what, const FrameParams* __restrict__ Fp, const double* __restrict__ tab,
                                  const double* __restrict__ in, long long n, double* __restrict__ out) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    if (what == 0) out[i] = disc_temperature(*Fp, in[i]);
    else blackbody(tab, in[i], out + 3 * i);
}

}  // namespace

cudaError_t launch_eval_shade(int what, const FrameParams* d_frame, const double* d_table, const double* d_in,
                              long long n, double* d_out, cudaStream_t stream) {
    if (n <= 0) return cudaSuccess;
    eval_shade_kernel<<<(unsigned)((n + 127) / 128), 128, 0, stream>>>(what, d_frame, d_table, d_in, n, d_out);
    return cudaGetLastError();
}

int shade_blocks(long long pixels, int most) {
    const long long want = (pixels + kShadeThreads - 1) / kShadeThreads;
    return (int)(want < 1 ? 1 : (want < most ? want : most));
}

cudaError_t launch_shade(const ShadeLaunch& L, cudaStream_t stream) {
    if (L.pixel_hi <= L.pixel_lo || L.nframes <= 0) return cudaSuccess;
    ShadeArgs A;
    A.frames = L.frames;
    A.pixel_lo = L.pixel_lo;
    A.pixel_hi = L.pixel_hi;
    A.hits = L.hits;
    A.sky = L.sky;
    A.pixels = L.pixels;
    A.rays = L.rays;
    A.jet = L.jet;
    A.stats = L.stats;
    A.flux = L.flux;
    A.flux_per_frame = L.flux_per_frame;
    shade_kernel<<<dim3((unsigned)L.blocks, (unsigned)L.nframes), kShadeThreads, 0, stream>>>(A);
    return cudaGetLastError();
}

cudaError_t launch_reduce(const ReduceLaunch& L, cudaStream_t stream) {
    flux_kernel<<<L.nframes, kRedThreads, 0, stream>>>(L.flux, L.flux_per_frame, L.stats);
    return cudaGetLastError();
}

}  // namespace bhg
