// bh_adjoint.cuh - The per-ray discrete adjoint of the binary64 render path.
//
// For one camera ray this computes the ray's luminance Y (the CIE Y of its
// shaded colour) and, for a loss weight w = dLoss/dY, the ray's contribution
// to dLoss/d(spin, inclination, Eddington ratio, r_out):
//
//   1. forward: the ray is integrated with the render path's DP5(4) scheme,
//      PI controller, step limiter and events (render.cpp:69-260,
//      geodesic.h:123-204); the state (y, h, controller memory) before each
//      accepted step and the step's size are stored in the ray's slots.
//      When the slots are full every second state is dropped and the interval
//      between the stored ones doubles, so memory stays bounded for any step
//      count;
//   2. seed: the shading of the hit (disc: Novikov-Thorne temperature,
//      Keplerian redshift, blackbody table, disc.h:94-126, render.cpp:31-34,
//      spectrum.cpp:123-134; sky: the escape direction and the star field,
//      render.cpp:15-26, scene.h:111-158) is differentiated in forward mode
//      (dual numbers) with respect to the hit state and the parameters;
//   3. reverse: step by step from the last (replayed from the stored states
//      where those were thinned), the adjoint state is carried back
//      through each DP5 step in reverse (the vector-Jacobian products of its
//      six stages), with the accepted step sizes held fixed: the discrete
//      adjoint of the step sequence the forward pass took.  The disc-crossing
//      root s* (theta(s*) = pi/2 on the dense-output polynomial) is
//      differentiated by the implicit-function theorem;
//   4. the adjoint of the initial photon is contracted with the derivatives of
//      the initial state (camera tetrad and metric at the camera).
//
// The disc's edges are steps in the image: a ray's luminance does not depend
// on r_out except when its crossing radius passes r_out, so the derivative of
// a point-sampled frame with respect to r_out is zero, and the edges move
// with the spin and the inclination too.  The edge term (edge_sample below)
// is the derivative of the frame averaged over each sample's cell: for a
// crossing near an edge, the luminance jump times the edge's length in the
// cell times its speed, the image-plane gradient of the crossing radius and
// its parameter derivatives coming from a reverse sweep seeded with that
// radius.
//
// All arithmetic is binary64.  The functions compile for the host as well, so
// the same code can be checked against finite differences on a CPU.
#pragma once

#include <cmath>
#include <cstdint>
#include <type_traits>

#include "../../include/bh_gpu.h"
#include "bh_adjoint.h"
#include "bh_common.cuh"
#include "bh_dp5.cuh"
#include "bh_dual.cuh"
#include "bh_frame.h"

#if defined(__CUDA_ARCH__)
#define BHA_NOINLINE __noinline__
#else
#define BHA_NOINLINE
#endif

namespace bhg {
namespace adj {

// Exact (non-contracted) binary64 products and sums for the ray set-up, so the
// initial photon is the render path's to the last bit.
__host__ __device__ __forceinline__ double xm(double a, double b) {
#if defined(__CUDA_ARCH__)
    return __dmul_rn(a, b);
#else
    return a * b;
#endif
}
__host__ __device__ __forceinline__ double xa(double a, double b) {
#if defined(__CUDA_ARCH__)
    return __dadd_rn(a, b);
#else
    return a + b;
#endif
}
__host__ __device__ __forceinline__ double xs(double a, double b) {
#if defined(__CUDA_ARCH__)
    return __dsub_rn(a, b);
#else
    return a - b;
#endif
}
__host__ __device__ __forceinline__ double xd(double a, double b) {
#if defined(__CUDA_ARCH__)
    return __ddiv_rn(a, b);
#else
    return a / b;
#endif
}
__host__ __device__ __forceinline__ double xsqrt(double a) {
#if defined(__CUDA_ARCH__)
    return __dsqrt_rn(a);
#else
    return std::sqrt(a);
#endif
}
__host__ __device__ __forceinline__ bool is_finite(double x) {
#if defined(__CUDA_ARCH__)
    return isfinite(x);
#else
    return std::isfinite(x);
#endif
}
__host__ __device__ __forceinline__ void sc(double x, double* s, double* c) {
#if defined(__CUDA_ARCH__)
    sincos(x, s, c);
#else
    *s = std::sin(x);
    *c = std::cos(x);
#endif
}

// Constants of a ray's right-hand side.
struct RayC {
    double a, a2, E, Lz, rp, rm;
    int factored;
};

// Hamilton's equations in Carter's separated form (the render path's
// right-hand side, geodesic.h:50-71):
//   2 Sigma H = Delta p_r^2 + p_th^2 + (L_z - a E sin^2)^2 / sin^2
//               - ((r^2 + a^2) E - a L_z)^2 / Delta,
// at sin(th) = sn, cos(th) = cs, with one reciprocal (of Sigma Delta sin^2)
// for the three quotients.  RhsMid holds what the derivatives and their
// vector-Jacobian products share.
struct RhsMid {
    double sn, sn2, D, iS, iD, isn2, r2a2, K, Lp, KiD, B;
};
__host__ __device__ __forceinline__ RhsMid rhs_mid(const RayC& c, double r, double sn, double cs, double pr,
                                                   double pth) {
    RhsMid m;
    if (fabs(sn) < 1e-9) sn = (sn < 0.0) ? -1e-9 : 1e-9;   // kerr.h:51
    m.sn = sn;
    m.sn2 = sn * sn;
    const double cs2 = cs * cs, r2 = r * r;
    const double S = r2 + c.a2 * cs2;
    m.D = c.factored ? (r - c.rp) * (r - c.rm) : (r2 - 2.0 * r + c.a2);
    const double SD = S * m.D;
    const double inv = rcp_nr(SD * m.sn2);
    m.iS = inv * m.D * m.sn2;
    m.iD = inv * S * m.sn2;
    m.isn2 = inv * SD;
    m.r2a2 = r2 + c.a2;
    m.K = m.r2a2 * c.E - c.a * c.Lz;
    m.Lp = c.Lz - c.a * c.E * m.sn2;
    m.KiD = m.K * m.iD;
    m.B = m.D * pr * pr + pth * pth + m.Lp * m.Lp * m.isn2 - m.K * m.KiD;
    return m;
}
// (dr, dth, dp_r, dp_th) / dlambda: the components the stages depend on.
__host__ __device__ __forceinline__ void rhs4(const RayC& c, double r, double sn, double cs, double pr, double pth,
                                              double d[4]) {
    const RhsMid m = rhs_mid(c, r, sn, cs, pr, pth);
    const double Dr = 2.0 * r - 2.0;
    d[0] = m.D * pr * m.iS;
    d[1] = pth * m.iS;
    d[2] = -0.5 * m.iS * (Dr * (pr * pr + m.KiD * m.KiD) - 2.0 * r * (2.0 * c.E * m.KiD + m.B * m.iS));
    const double q = c.Lz * m.isn2;
    d[3] = -m.sn * cs * m.iS * (c.a2 * (c.E * c.E + m.B * m.iS) - q * q);
}
// d = (dt, dr, dth, dphi, dp_r, dp_th) / dlambda.
__host__ __device__ __forceinline__ void rhs6(const RayC& c, double r, double sn, double cs, double pr, double pth,
                                              double d[6]) {
    const RhsMid m = rhs_mid(c, r, sn, cs, pr, pth);
    const double Dr = 2.0 * r - 2.0;
    d[0] = m.iS * (c.a * m.Lp + m.r2a2 * m.KiD);
    d[1] = m.D * pr * m.iS;
    d[2] = pth * m.iS;
    d[3] = m.iS * (m.Lp * m.isn2 + c.a * m.KiD);
    d[4] = -0.5 * m.iS * (Dr * (pr * pr + m.KiD * m.KiD) - 2.0 * r * (2.0 * c.E * m.KiD + m.B * m.iS));
    const double q = c.Lz * m.isn2;
    d[5] = -m.sn * cs * m.iS * (c.a2 * (c.E * c.E + m.B * m.iS) - q * q);
}

// The right-hand side at angle th; *sn_out, *cs_out receive sin(th), cos(th).
__host__ __device__ __forceinline__ void rhs6_th(const RayC& c, double r, double th, double pr, double pth,
                                                 double d[6], double* sn_out, double* cs_out) {
    double sn, cs;
    sc(th, &sn, &cs);
    rhs6(c, r, sn, cs, pr, pth, d);
    *sn_out = sn;
    *cs_out = cs;
}

// Vector-Jacobian product of rhs6 at (r, th, p_r, p_th) given sin(th) = sn
// and cos(th) = cs: for db = dLoss/d(d), adds dLoss/d(r, th, p_r, p_th) into
// g[0..3] and dLoss/d(E, L_z, a) into *Eb, *Lzb, *ab.  Reverse-mode
// differentiation of the expressions of rhs6, written out.  TIME: whether
// db[0] can be non-zero; nothing the loss sees depends on t, so the reverse
// sweep runs without.
template <bool TIME>
__host__ __device__ __forceinline__ void rhs_vjp(const RayC& c, double r, double sn_true, double cs, double pr,
                                                 double pth, const double db[6], double g[4], double* Eb,
                                                 double* Lzb, double* ab) {
    const RhsMid m = rhs_mid(c, r, sn_true, cs, pr, pth);
    const bool clamped = fabs(sn_true) < 1e-9;
    const double a = c.a, a2 = c.a2, E = c.E, Lz = c.Lz;
    const double sn = m.sn, sn2 = m.sn2, cs2 = cs * cs, D = m.D, iS = m.iS, iD = m.iD, isn2 = m.isn2;
    const double r2a2 = m.r2a2, K = m.K, Lp = m.Lp, KiD = m.KiD, B = m.B;
    const double Dr = 2.0 * r - 2.0;
    const double BiS = B * iS, q = Lz * isn2, pk = pr * pr + KiD * KiD;
    const double X3 = Lp * isn2 + a * KiD;
    const double X4 = Dr * pk - 2.0 * r * (2.0 * E * KiD + BiS);
    const double X5 = a2 * (E * E + BiS) - q * q;
    const double P5 = -sn * cs;

    // outputs
    double b_iS = db[1] * D * pr + db[2] * pth + db[3] * X3 - 0.5 * db[4] * X4 + db[5] * P5 * X5;
    double bD = db[1] * pr * iS;
    double bpr = db[1] * D * iS;
    double bpth = db[2] * iS;
    const double bX3 = db[3] * iS;
    const double bX4 = -0.5 * db[4] * iS;
    const double bP5 = db[5] * iS * X5;
    const double bX5 = db[5] * P5 * iS;
    // X3 = Lp isn2 + a KiD
    double bLp = bX3 * isn2;
    double bisn2 = bX3 * Lp;
    double ba = bX3 * KiD;
    double bKiD = bX3 * a;
    double br2a2 = 0.0;
    if (TIME) {
        // X0 = a Lp + r2a2 KiD
        b_iS += db[0] * (a * Lp + r2a2 * KiD);
        const double bX0 = db[0] * iS;
        ba += bX0 * Lp;
        bLp += bX0 * a;
        br2a2 += bX0 * KiD;
        bKiD += bX0 * r2a2;
    }
    // X4 = Dr (pr^2 + KiD^2) - 2 r (2 E KiD + B iS)
    const double bDr = bX4 * pk;
    bpr += 2.0 * bX4 * Dr * pr;
    const double br4 = -2.0 * bX4;
    double br = br4 * (2.0 * E * KiD + BiS) + 2.0 * bDr;
    const double rb4 = r * br4;
    double bE = 2.0 * rb4 * KiD;
    bKiD += 2.0 * (rb4 * E + bX4 * Dr * KiD);
    // X5 = a2 (E^2 + B iS) - (Lz isn2)^2
    double ba2 = bX5 * (E * E + BiS);
    const double a2b5 = a2 * bX5;
    bE += 2.0 * a2b5 * E;
    const double bq = -2.0 * bX5 * q;
    double bLz = bq * isn2;
    bisn2 += bq * Lz;
    // B iS in both
    const double bBiS = rb4 + a2b5;
    const double bB = bBiS * iS;
    b_iS += bBiS * B;
    // P5 = -sn cs
    double bsn = -bP5 * cs;
    double bcs = -bP5 * sn;
    // B = D pr^2 + pth^2 + Lp^2 isn2 - K KiD
    bD += bB * pr * pr;
    bpr += 2.0 * bB * D * pr;
    bpth += 2.0 * bB * pth;
    const double bLp2 = bB * Lp;
    bLp += 2.0 * bLp2 * isn2;
    bisn2 += bLp2 * Lp;
    bKiD -= bB * K;
    // KiD = K iD
    const double bK = bKiD * iD - bB * KiD;
    const double biD = bKiD * K;
    // Lp = Lz - a E sn2
    bLz += bLp - bK * a;
    const double bLps = bLp * sn2;
    ba -= bLps * E + bK * Lz;
    bE += bK * r2a2 - bLps * a;
    // K = r2a2 E - a Lz; r2a2 = r2 + a2
    br2a2 += bK * E;
    ba2 += br2a2;
    // the reciprocals
    const double bS = -b_iS * iS * iS;
    bD -= biD * iD * iD;
    const double bsn2 = -bLp * a * E - bisn2 * isn2 * isn2;
    // Delta = r^2 - 2 r + a^2 (the factored form has the same value)
    br += bD * Dr;
    ba2 += bD;
    // Sigma = r2 + a2 cs2
    ba2 += bS * cs2;
    br += 2.0 * r * (br2a2 + bS);
    bsn += 2.0 * sn * bsn2;
    bcs += 2.0 * cs * (bS * a2);
    ba += 2.0 * a * ba2;
    const double bth = (clamped ? 0.0 : cs * bsn) - sn_true * bcs;
    g[0] += br;
    g[1] += bth;
    g[2] += bpr;
    g[3] += bpth;
    *Eb += bE;
    *Lzb += bLz;
    *ab += ba;
}
__host__ __device__ BHA_NOINLINE void rhs6_vjp(const RayC& c, double r, double sn, double cs, double pr, double pth,
                                               const double db[6], double g[4], double* Eb, double* Lzb,
                                               double* ab) {
    rhs_vjp<true>(c, r, sn, cs, pr, pth, db, g, Eb, Lzb, ab);
}

// sin and cos of a stage's angle th from those of the step's base angle th0.
__host__ __device__ __forceinline__ bool near_angle(double dth) { return fabs(dth) <= kMaxShift; }
// The full form for an angle that moved further: out of line on the device.
__host__ __device__ BHA_NOINLINE void far_sincos(double th, double* s, double* c) { sc(th, s, c); }
__host__ __device__ __forceinline__ void stage_sincos(double th, double th0, double sn0, double cs0, double* s,
                                                      double* c) {
    const double dth = th - th0;
    if (near_angle(dth)) shift_sincos(sn0, cs0, dth, s, c);
    else far_sincos(th, s, c);
}

// The Runge-Kutta tableau for the stage loops (row j: stage j + 1), the
// fifth-order weights (row 6) and the error weights (row 7).
__host__ __device__ constexpr double tableau(int row, int col) {
    const double t[8][7] = {
        {0, 0, 0, 0, 0, 0, 0}, {A21, 0, 0, 0, 0, 0, 0}, {A31, A32, 0, 0, 0, 0, 0},
        {A41, A42, A43, 0, 0, 0, 0}, {A51, A52, A53, A54, 0, 0, 0}, {A61, A62, A63, A64, A65, 0, 0},
        {B1, 0, B3, B4, B5, B6, 0}, {E1, 0, E3, E4, E5, E6, E7}};
    return t[row][col];
}
// f(std::integral_constant<int, j>) for a stage number 1 <= j <= 6 that is not
// known before the loop runs.
template <class Fn>
__host__ __device__ __forceinline__ void by_stage(int j, Fn&& f) {
    switch (j) {
    case 1: f(std::integral_constant<int, 1>{}); break;
    case 2: f(std::integral_constant<int, 2>{}); break;
    case 3: f(std::integral_constant<int, 3>{}); break;
    case 4: f(std::integral_constant<int, 4>{}); break;
    case 5: f(std::integral_constant<int, 5>{}); break;
    default: f(std::integral_constant<int, 6>{}); break;
    }
}
__host__ __device__ __forceinline__ double weight5(int j) {
    return (j == 0) ? B1 : (j == 2) ? B3 : (j == 3) ? B4 : (j == 4) ? B5 : (j == 5) ? B6 : 0.0;
}

// A ray's stage values live in shared memory on the device (kScratch doubles
// per thread, threads side by side: no bank conflicts) and the stage loops
// stay rolled around one copy of the right-hand side and of its
// vector-Jacobian product.  Unrolled, with the stages in registers, the forward
// and the reverse step were 20 to 30 KB of code each and the instruction fetch
// stalled the kernel (1.4 of 4.2 cycles per issue): 13.2 against 8.6 ms per 512^2
// gradient on one B200, the dependent binary64 chain of a warp (39% of the issue
// slots, 41% of the binary64 pipe at 8 warps per SM) bounding what is left.
constexpr int kScratch = 60;
constexpr int kAdjBlock = 64;
#if defined(__CUDA_ARCH__)
#define BHA_SCRATCH(name)                        \
    extern __shared__ double bha_scratch_smem[]; \
    double* const name = bha_scratch_smem + threadIdx.x;
constexpr int kScratchStride = kAdjBlock;
#else
inline double* host_scratch() {
    static thread_local double buf[kScratch];
    return buf;
}
#define BHA_SCRATCH(name) double* const name = host_scratch();
constexpr int kScratchStride = 1;
#endif

// Integrator state of one ray.
struct Integ {
    double y[6];        // t, r, th, phi, p_r, p_th
    double k1[6];       // FSAL stage at y
    double h;
    double errp_mem;    // beta ln err_prev, err_prev the last accepted error norm (>= 1e-4)
    double sn0, c0;     // sin(th), cos(th) at y
    double h_acc;       // the last accepted step's size
    int have_k1;
    int tries;
    int steps;
};

// One accepted step: its ends' r, th and cosines; its stages are left in the
// scratch (component i of k_(j+1) at 6 j + i) until the next attempt.
struct StepRec {
    double r0, th0, r1, th1;
    double h;
    double c0, c7;      // cos(th) at y and at yn
};

// Attempt steps from `s` until one is accepted (render.cpp:127-137 with
// geodesic.h:123-204), then advance `s`.  Returns false when no acceptable
// step was found (more than 40 rejections or |h| < 1e-14).  The sin/cos of the
// stages and of the step's end come from the step's base angle by angle
// addition, like the render's; a stored state holds them, so that a step
// started from it repeats the one that passed it.
__host__ __device__ __forceinline__ bool advance_step(const FrameParams& F, const RayC& c, Integ& s,
                                                      StepRec* rec) {
    BHA_SCRATCH(scr)
    auto K = [&](int j, int i) -> double& { return scr[(6 * j + i) * kScratchStride]; };
    if (!s.have_k1) {
        rhs6(c, s.y[1], s.sn0, s.c0, s.y[4], s.y[5], s.k1);
        s.have_k1 = 1;
    }
    for (;;) {
        if (s.tries == 0) {
            const double hmax = 0.05 * dmaxr(1.0, s.y[1] - F.r_h) + 0.01;
            if (s.h > hmax) s.h = hmax;
        }
        const double h = s.h;
        double yn[6], e[6], c7 = 0.0, sn7 = 0.0;
        #pragma unroll
        for (int i = 0; i < 6; ++i) K(0, i) = s.k1[i];
        #pragma unroll 1
        for (int j = 1; j < 7; ++j) {
            double acc[6] = {0, 0, 0, 0, 0, 0};
            if (j == 6) {
                #pragma unroll
                for (int i = 0; i < 6; ++i) e[i] = 0.0;
            }
            // one case per stage, so that the loads and sums overlap
            auto sums = [&](auto stage) {
                constexpr int n = decltype(stage)::value;
                #pragma unroll
                for (int l = 0; l < n; ++l) {
                    #pragma unroll
                    for (int i = 0; i < 6; ++i) {
                        if (n < 6 && (i == 0 || i == 3)) continue;   // t and phi enter no stage
                        const double kk = K(l, i);
                        acc[i] += tableau(n, l) * kk;
                        if (n == 6) e[i] += tableau(7, l) * kk;
                    }
                }
            };
            by_stage(j, sums);
            #pragma unroll
            for (int i = 0; i < 6; ++i) yn[i] = s.y[i] + h * acc[i];
            double d[6], sn, cs;
            stage_sincos(yn[2], s.y[2], s.sn0, s.c0, &sn, &cs);
            rhs6(c, yn[1], sn, cs, yn[4], yn[5], d);
            #pragma unroll
            for (int i = 0; i < 6; ++i) K(j, i) = d[i];
            sn7 = sn;
            c7 = cs;
        }
        double err2 = 0.0;
        #pragma unroll
        for (int i = 0; i < 6; ++i) {
            const double ei = h * (e[i] + E7 * K(6, i));
            const double scl = F.atol + F.rtol * dmaxr(fabs(s.y[i]), fabs(yn[i]));
            const double q = ei * rcp_nr(scl);
            err2 += q * q;
        }
        // err: the square of the RMS norm; the PI factor 0.9 err^-alpha
        // err_prev^beta (geodesic.h:171-173) as one exp of logarithms, the
        // forward pass and every replay alike
        double err = err2 * 0.125;
        if (!is_finite(err)) err = 1e10;
        const double lq = log(dmaxr(err, 1e-32));
        double fac = 0.9 * exp(fma(-0.5 * kAlpha, lq, s.errp_mem));
        fac = dclamp(fac, 0.2, 5.0);
        if (!(err <= 1.0)) {
            s.h *= dminr(fac, 1.0);
            if (++s.tries > 40 || fabs(s.h) < 1e-14) return false;
            continue;
        }
        s.tries = 0;
        ++s.steps;
        if (rec) {
            rec->r0 = s.y[1];
            rec->th0 = s.y[2];
            rec->r1 = yn[1];
            rec->th1 = yn[2];
            rec->h = h;
            rec->c0 = s.c0;
            rec->c7 = c7;
        }
        #pragma unroll
        for (int i = 0; i < 6; ++i) {
            s.y[i] = yn[i];
            s.k1[i] = K(6, i);
        }
        s.c0 = c7;
        s.sn0 = sn7;
        s.errp_mem = kBeta * dmaxr(0.5 * lq, kLnErrFloor);
        s.h_acc = h;
        s.h = h * fac;
        return true;
    }
}
// The same for the replays, out of line.
__host__ __device__ BHA_NOINLINE bool advance(const FrameParams& F, const RayC& c, Integ& s) {
    return advance_step(F, c, s, nullptr);
}
// The dense output of component i (1: r, 2: th) of the step that advance_step
// has just recorded.
__host__ __device__ __forceinline__ DenseC step_dense(const StepRec& q, int i) {
    BHA_SCRATCH(scr)
    auto K = [&](int j) { return scr[(6 * j + i) * kScratchStride]; };
    return dense_coef(q.h, i == 1 ? q.r0 : q.th0, i == 1 ? q.r1 : q.th1, K(0), K(2), K(3), K(4), K(5), K(6));
}

// Equatorial target angle pi/2 + m pi between th0 and th1 (render.cpp:180-189).
__host__ __device__ __forceinline__ double crossing_target(double th0, double th1) {
    const double m = (th1 > th0) ? ceil((th0 - 0.5 * kPi) / kPi) : floor((th0 - 0.5 * kPi) / kPi);
    return 0.5 * kPi + m * kPi;
}

// What the render records of a ray's accepted step (kTrajWords doubles): r, th,
// p_r, p_th at its start, its size, and sin and cos of the angle.  Word w of
// step j of ray i lies at traj[(j kTrajWords + w) n_rays + i], so that the lanes
// of a warp write and read side by side.

// Carries the adjoint yb of the state after one accepted step (from ys with
// step h; sn0, cs0: sin and cos of its angle) back to the state before it,
// accumulating the E, L_z and spin adjoints.  The six stages are computed again and their vector-Jacobian
// products taken in reverse.  rstar_b != 0 marks the step that ends on the
// disc: the hit radius r* = P_r(s*) at the crossing theta(s*) = target of the
// dense polynomials then receives the weight rstar_b (and yb, the adjoint of
// the step's end state, is zero).  yb[0] is zero throughout and yb[3] stays what
// it is: nothing depends on t, and no right-hand side on phi.
// Scratch: the stages' derivatives, then their adjoints, component i of stage j
// at 4 j + i; from 24 on the stages' (r, th, p_r, p_th, sin, cos), 6 each.
__host__ __device__ __forceinline__ void step_vjp(const RayC& c, const double y0[4], double sn0, double cs0, double h,
                                                  double yb[6], double* Eb, double* Lzb, double* ab, double rstar_b) {
    constexpr int kC[4] = {1, 2, 4, 5};      // r, th, p_r, p_th in the state
    BHA_SCRATCH(scr)
    auto K = [&](int j, int i) -> double& { return scr[(4 * j + i) * kScratchStride]; };
    auto Y = [&](int j, int i) -> double& { return scr[(24 + 6 * j + i) * kScratchStride]; };
    const bool event = rstar_b != 0.0;
    double yn[4];
    #pragma unroll 1
    for (int j = 0; j < 6; ++j) {
        double acc[4] = {0, 0, 0, 0}, t[4], sn = sn0, cs = cs0;
        auto sums = [&](auto stage) {
            constexpr int n = decltype(stage)::value;
            #pragma unroll
            for (int l = 0; l < n; ++l) {
                #pragma unroll
                for (int i = 0; i < 4; ++i) acc[i] += tableau(n, l) * K(l, i);
            }
        };
        if (j > 0) by_stage(j, sums);
        #pragma unroll
        for (int i = 0; i < 4; ++i) t[i] = y0[i] + h * acc[i];
        if (j > 0) stage_sincos(t[1], y0[1], sn0, cs0, &sn, &cs);
        #pragma unroll
        for (int i = 0; i < 4; ++i) Y(j, i) = t[i];
        Y(j, 4) = sn;
        Y(j, 5) = cs;
        if (j == 5 && !event) break;         // k_6 enters the step's end alone
        double d[4];
        rhs4(c, t[0], sn, cs, t[2], t[3], d);
        #pragma unroll
        for (int i = 0; i < 4; ++i) K(j, i) = d[i];
    }

    // The weights of the step's end (the adjoint of yn) and of the state at the
    // start of the step, and the event's own weights of the stages: all of them
    // D_j r5 of one component each, D_1 and D_7 with more.
    double ynb[4], ybar[4], r5r = 0.0, r5th = 0.0, k1r = 0.0, k1th = 0.0;
    #pragma unroll
    for (int i = 0; i < 4; ++i) {
        ynb[i] = yb[kC[i]];
        ybar[i] = 0.0;
    }
    if (event) {
        #pragma unroll
        for (int i = 0; i < 4; ++i) {
            double acc = 0.0;
            for (int l = 0; l < 6; ++l) acc += weight5(l) * K(l, i);
            yn[i] = y0[i] + h * acc;
        }
        double sn7, cs7, k7[4];
        sc(yn[1], &sn7, &cs7);
        rhs4(c, yn[0], sn7, cs7, yn[2], yn[3], k7);
        const DenseC cth = dense_coef(h, y0[1], yn[1], K(0, 1), K(2, 1), K(3, 1), K(4, 1), K(5, 1), k7[1]);
        const DenseC crr = dense_coef(h, y0[0], yn[0], K(0, 0), K(2, 0), K(3, 0), K(4, 0), K(5, 0), k7[0]);
        const double target = crossing_target(cth.r1, cth.r1 + cth.r2);
        const double s = dense_crossing(cth, target), s1 = 1.0 - s;
        const double dth = dense_deriv(cth, s), dr = dense_deriv(crr, s);
        // the reverse of a component's dense output at s with weight v (its
        // coefficients as dense_coef forms them)
        const double v[2] = {rstar_b, (dth != 0.0) ? -rstar_b * dr / dth : 0.0};
        double r5[2], k1w[2], k7b[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
        #pragma unroll
        for (int q = 0; q < 2; ++q) {
            const double r4b = s * s * s1 * v[q], r3b = s * s1 * v[q] - r4b;
            r5[q] = h * s * s * s1 * s1 * v[q];
            k1w[q] = h * r3b;
            k7b[1 + q] = D7 * r5[q] - h * r4b;
            const double r2b = s * v[q] + r4b - r3b;
            ynb[q] += r2b;
            ybar[q] += v[q] - r2b;
        }
        r5r = r5[0]; r5th = r5[1];
        k1r = k1w[0]; k1th = k1w[1];
        double g4[4] = {0.0, 0.0, 0.0, 0.0};
        rhs_vjp<false>(c, yn[0], sn7, cs7, yn[2], yn[3], k7b, g4, Eb, Lzb, ab);
        #pragma unroll
        for (int i = 0; i < 4; ++i) ynb[i] += g4[i];
    }
    #pragma unroll
    for (int i = 0; i < 4; ++i) ybar[i] += ynb[i];
    #pragma unroll
    for (int j = 0; j < 6; ++j) {
        constexpr double Dw[6] = {D1, 0.0, D3, D4, D5, D6};
        const double hb = h * weight5(j);
        #pragma unroll
        for (int i = 0; i < 4; ++i) {
            double v = hb * ynb[i];
            if (i == 0) v += Dw[j] * r5r + (j == 0 ? k1r : 0.0);
            if (i == 1) v += Dw[j] * r5th + (j == 0 ? k1th : 0.0);
            K(j, i) = v;
        }
    }
    const double hphi = h * yb[3];
    #pragma unroll 1
    for (int j = 5; j >= 0; --j) {
        double g4[4] = {0.0, 0.0, 0.0, 0.0};
        const double db[6] = {0.0, K(j, 0), K(j, 1), weight5(j) * hphi, K(j, 2), K(j, 3)};
        rhs_vjp<false>(c, Y(j, 0), Y(j, 4), Y(j, 5), Y(j, 2), Y(j, 3), db, g4, Eb, Lzb, ab);
        #pragma unroll
        for (int i = 0; i < 4; ++i) ybar[i] += g4[i];
        #pragma unroll
        for (int i = 0; i < 4; ++i) g4[i] *= h;
        auto spread = [&](auto stage) {
            constexpr int n = decltype(stage)::value;
            #pragma unroll
            for (int l = 0; l < n; ++l) {
                #pragma unroll
                for (int i = 0; i < 4; ++i) K(l, i) += tableau(n, l) * g4[i];
            }
        };
        if (j > 0) by_stage(j, spread);
    }
    #pragma unroll
    for (int i = 0; i < 4; ++i) yb[kC[i]] = ybar[i];
}

// ---- shading in forward mode ---------------------------------------------------

using D5 = Dual<5>;   // slots: r, E, L_z, spin, Eddington ratio
using D8 = Dual<8>;   // slots: r, th, phi, p_r, p_th, E, L_z, spin
enum { kS5R = 0, kS5E = 1, kS5L = 2, kS5A = 3, kS5M = 4 };

template <class T>
__host__ __device__ T circ_energy_t(const T& a, const T& r, int sg) {
    const T sr = sqrt(r);
    const T num = r * r - 2.0 * r + (double)sg * a * sr;
    const T den = r * sqrt(r * r - 3.0 * r + 2.0 * (double)sg * a * sr);
    return num / den;
}
template <class T>
__host__ __device__ T circ_angmom_t(const T& a, const T& r, int sg) {
    const T sr = sqrt(r);
    const T num = (double)sg * sr * (r * r - 2.0 * (double)sg * a * sr + a * a);
    const T den = r * sqrt(r * r - 3.0 * r + 2.0 * (double)sg * a * sr);
    return num / den;
}

// CIE Y of the blackbody table at temperature T (spectrum.cpp:123-134).
template <class T>
__host__ __device__ T blackbody_Y(const double* tab, const T& Tk) {
    const double kLogTMin = 1.6989700043360187, kLogTMax = 9.4771212547196626;
    T Tc = Tk;
    if (Tk.v < 50.0) Tc = T(50.0);
    if (Tk.v > 3.0e9) Tc = T(3.0e9);
    const T f = (log10(Tc) - kLogTMin) / (kLogTMax - kLogTMin) * (double)(kTableN - 1);
    int i = (int)f.v;
    i = (i < 0) ? 0 : (i > kTableN - 2 ? kTableN - 2 : i);
    const T u = f - (double)i;
    return exp(tab[kTableN + i] * (1.0 - u) + tab[kTableN + i + 1] * u);
}

// Luminance of a disc hit at radius r (disc.h:94-121, kerr.h:260-266,
// render.cpp:31-34, 277-297) as a dual over (r, E, L_z, spin, Eddington).
__host__ __device__ inline D5 disc_luminance(const FrameParams& F, const AdjointFrame& X, const double* tab,
                                             double r_hit, double E_, double Lz_) {
    if (r_hit <= F.r_in || r_hit > F.r_out) return D5(0.0);
    const D5 r = D5::var(r_hit, kS5R);
    const D5 E = D5::var(E_, kS5E);
    const D5 Lz = D5::var(Lz_, kS5L);
    auto par = [](double v, double da) {
        D5 q(v);
        q.d[kS5A] = da;
        return q;
    };
    const int sg = F.disc_sigma;
    const D5 a = par(F.disc_a, X.d_disc_a);
    const D5 x0 = par(F.x0, X.d_x0);
    const D5 x = sqrt(r);
    D5 W = x - x0 - 1.5 * a * log(x / x0);
    for (int i = 0; i < 3; ++i)
        if (F.pt_c[i] != 0.0) {
            const D5 ci = par(F.pt_c[i], X.d_pt_c[i]);
            const D5 xi = par(F.pt_x[i], X.d_pt_x[i]);
            const D5 di = par(F.pt_den[i], X.d_pt_den[i]);
            W = W - ci * log((x - xi) / di);
        }
    const D5 r32 = r * sqrt(r);
    const D5 dd = r32 + (double)sg * a;
    const D5 Om = (double)sg / dd;
    const D5 dOm = -(double)sg * 1.5 * sqrt(r) / (dd * dd);
    const D5 Ec = circ_energy_t(a, r, sg);
    const D5 Lc = circ_angmom_t(a, r, sg);
    const D5 den = Ec - Om * Lc;
    if (!(den.v > 0.0)) return D5(0.0);
    const D5 Fd = (-dOm) / (4.0 * kPi * r * den * den) * W;
    if (!(Fd.v > 0.0 && is_finite(Fd.v))) return D5(0.0);
    D5 mdot(F.disc_mdot);
    mdot.d[kS5A] = X.d_mdot_da;
    mdot.d[kS5M] = X.d_mdot_dedd;
    const D5 Fl = Fd * mdot * (2.99792458e8 * 2.99792458e8) / F.disc_rg2;
    if (!(Fl.v > 0.0)) return D5(0.0);
    const D5 T = pow(Fl / 5.670374419e-8, 0.25);
    // Keplerian four-velocity and g = 1 / (p . u), p_t = -E, p_phi = L_z.
    const D5 dsc = r * r * r - 3.0 * r * r + 2.0 * (double)sg * a * r32;
    const D5 ut = dd / sqrt(dsc.v > 1e-300 ? dsc : D5(1e-300));
    const D5 ku = (-E) * ut + Lz * (Om * ut);
    if (!(ku.v > 1e-12)) return D5(0.0);
    const D5 g = 1.0 / ku;
    return blackbody_Y(tab, g * T);
}

// Escape direction (render.cpp:15-26, normalised as render.cpp:364-366) as a
// dual over (r, th, phi, p_r, p_th, E, L_z, spin).  False if degenerate.
__host__ __device__ inline bool escape_direction(const double y[6], double E_, double Lz_, double a_, D8 v[3]) {
    const D8 r = D8::var(y[1], 0), th = D8::var(y[2], 1), ph = D8::var(y[3], 2);
    const D8 pr = D8::var(y[4], 3), pth = D8::var(y[5], 4);
    const D8 E = D8::var(E_, 5), Lz = D8::var(Lz_, 6), a = D8::var(a_, 7);
    const D8 a2 = a * a;
    const D8 sn_raw = sin(th), cs = cos(th);
    D8 sn = sn_raw;
    if (fabs(sn.v) < 1e-9) sn = D8((sn.v < 0.0) ? -1e-9 : 1e-9);
    const D8 sn2 = sn * sn, cs2 = cs * cs;
    const D8 Sig = r * r + a2 * cs2;
    const D8 Del = r * r - 2.0 * r + a2;
    const D8 SD = Sig * Del;
    const D8 gtp = -2.0 * a * r / SD;
    const D8 gpp = (Del - a2 * sn2) / (SD * sn2);
    const D8 dr = (Del / Sig) * pr;
    const D8 dth = pth / Sig;
    const D8 dph = gtp * (-E) + gpp * Lz;
    const D8 R = sqrt(r * r + a * a);
    const D8 sp = sin(ph), cp = cos(ph);
    const D8 dR = (R.v > 0.0) ? r / R * dr : dr;
    v[0] = dR * sn_raw * cp + R * cs * dth * cp - R * sn_raw * sp * dph;
    v[1] = dR * sn_raw * sp + R * cs * dth * sp + R * sn_raw * cp * dph;
    v[2] = dr * cs - r * sn_raw * dth;
    const D8 vn = sqrt(v[0] * v[0] + v[1] * v[1] + v[2] * v[2]);
    if (!(vn.v > 0.0)) return false;
    v[0] = v[0] / vn;
    v[1] = v[1] / vn;
    v[2] = v[2] / vn;
    return true;
}

// The escape direction alone.
__host__ __device__ inline bool escape_direction_value(const double y[6], double E, double Lz, double a,
                                                       double v[3]) {
    const double r = y[1], a2 = a * a;
    double sn_raw, cs, sp, cp;
    sc(y[2], &sn_raw, &cs);
    sc(y[3], &sp, &cp);
    const double sn = (fabs(sn_raw) < 1e-9) ? ((sn_raw < 0.0) ? -1e-9 : 1e-9) : sn_raw;
    const double sn2 = sn * sn;
    const double Sig = r * r + a2 * cs * cs;
    const double Del = r * r - 2.0 * r + a2;
    const double SD = Sig * Del;
    const double dr = (Del / Sig) * y[4];
    const double dth = y[5] / Sig;
    const double dph = -2.0 * a * r / SD * (-E) + (Del - a2 * sn2) / (SD * sn2) * Lz;
    const double R = std::sqrt(r * r + a2);
    const double dR = (R > 0.0) ? r / R * dr : dr;
    v[0] = dR * sn_raw * cp + R * cs * dth * cp - R * sn_raw * sp * dph;
    v[1] = dR * sn_raw * sp + R * cs * dth * sp + R * sn_raw * cp * dph;
    v[2] = dr * cs - r * sn_raw * dth;
    const double vn = std::sqrt(v[0] * v[0] + v[1] * v[1] + v[2] * v[2]);
    if (!(vn > 0.0)) return false;
    v[0] /= vn;
    v[1] /= vn;
    v[2] /= vn;
    return true;
}

// CIE Y of the sky along unit direction d and its gradient with respect to d
// (scene.h:111-158, 202-223; the star field's Gaussian point-spread function
// and the diffuse background).
__host__ __device__ inline double sky_luminance(const SkyData& sky, const FrameParams& F, const double d[3],
                                                double gY[3]) {
    using D3 = Dual<3>;
    gY[0] = gY[1] = gY[2] = 0.0;
    double Y = 0.0;
    if (sky.n_stars > 0 && F.stars_enabled) {
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
        for (int a = -F.span_t; a <= F.span_t; ++a) {
            const int ti = it + a;
            if (ti < 0 || ti >= kLat) continue;
            for (int b = -sp; b <= sp; ++b) {
                int pi = pbase + b;
                pi = ((pi % kLon) + kLon) % kLon;
                const int bin = ti * kLon + pi;
                const int k0 = sky.bin_start[bin], k1 = sky.bin_start[bin + 1];
                for (int k = k0; k < k1; ++k) {
                    const double4 s = sky.star_pos[k];
                    const double dot_raw = d[0] * s.x + d[1] * s.y + d[2] * s.z;
                    const double dot = dclamp(dot_raw, -1.0, 1.0);
                    if (dot < F.cut_dot) continue;   // outside the cutoff, without the acos
                    double ang, dang2;   // angle and d(angle^2)/d(dot)
                    if (dot > 0.9999995) {
                        ang = sqrt(dmaxr(0.0, 2.0 * (1.0 - dot)));
                        dang2 = -2.0;
                    } else {
                        ang = acos(dot);
                        const double q = 1.0 - dot * dot;
                        dang2 = (q > 0.0) ? -2.0 * ang / sqrt(q) : 0.0;
                    }
                    if (ang > cutoff) continue;
                    const double w = norm * exp(-ang * ang * inv2s2) * s.w;
                    Y += w;
                    if (dot_raw > -1.0 && dot_raw < 1.0) {
                        const double dw = -w * inv2s2 * dang2;   // dw / d(dot)
                        gY[0] += dw * s.x;
                        gY[1] += dw * s.y;
                        gY[2] += dw * s.z;
                    }
                }
            }
        }
    }
    if (F.milky_way) {
        if (F.sky_mode == BH_SKY_UNIFORM) {
            Y += sky.diffuse_L;
        } else {
            const D3 d0 = D3::var(d[0], 0), d1 = D3::var(d[1], 1), d2 = D3::var(d[2], 2);
            const double ca = 0.8660254037844387, sa = 0.5;
            const D3 g1 = ca * d1 + sa * d2;
            D3 g2 = -sa * d1 + ca * d2;
            if (g2.v < -1.0) g2 = D3(-1.0);
            if (g2.v > 1.0) g2 = D3(1.0);
            const D3 band = exp(-fabs(g2) / 0.055);
            const D3 l = atan2(g1, d0);
            const D3 bulge = 0.55 + 0.45 * exp(-(l * l) / (2.0 * 0.45 * 0.45));
            const D3 lane = 0.65 + 0.35 * sin(l * 7.3 + g2 * 41.0) * sin(l * 3.1 - g2 * 17.0);
            if (lane.v > 0.0) {
                const D3 amp = sky.diffuse_L * band * bulge * lane;
                Y += amp.v;
                for (int i = 0; i < 3; ++i) gY[i] += amp.d[i];
            }
        }
    }
    return Y;
}

// ---- the ray ----------------------------------------------------------------------

struct RayResult {
    double Y;               // luminance of the ray
    double grad[4];         // w * dY/d(spin, inclination, Eddington ratio, r_out)
    int what;               // BH_HIT_*
    int steps;              // accepted steps of the forward pass
    long long replay;       // accepted steps replayed by the reverse pass
    int interval;           // final checkpoint interval
};

// Initial photon of frame-local ray `local_id` (render.cpp:440-451,
// scene.h:356-384, geodesic.h:215-231) and its derivatives with respect to
// the spin and the inclination.
// The image-plane position of sample k of pixel (px, py) (scene.h:356-384
// with the render path's jitter): su, sv in [-1, 1]; *x_pix, *y_pix in pixels.
__host__ __device__ inline void sample_position_at(const FrameParams& F, int px, int py, int k, double* su,
                                                   double* sv, double* x_pix, double* y_pix) {
    const int S = F.S;
    const int sy = k / S, sx = k - (k / S) * S;
    const uint64_t s0 = F.seed ^ ((uint64_t)py << 32) ^ ((uint64_t)px * 0x9E3779B97F4A7C15ull);
    const uint64_t g = 0x9E3779B97F4A7C15ull;
    const double u1 = u53(mix64(s0 + (uint64_t)(2 * k + 1) * g));
    const double u2 = u53(mix64(s0 + (uint64_t)(2 * k + 2) * g));
    const double jx = xm(xa((double)sx, u1), F.inv_S);
    const double jy = xm(xa((double)sy, u2), F.inv_S);
    *x_pix = xa((double)px, jx);
    *y_pix = xa((double)py, jy);
    *su = xs(xd(xm(2.0, *x_pix), (double)F.width), 1.0);
    *sv = xs(1.0, xd(xm(2.0, *y_pix), (double)F.height));
}

// The same for frame-local sample `local_id` (work order).
__host__ __device__ inline void sample_position(const FrameParams& F, long long local_id, double* su, double* sv,
                                                double* x_pix, double* y_pix) {
    const int S = F.S;
    const long long pixel = local_id / (S * S);
    const int k = (int)(local_id - pixel * (S * S));
    int px, py;
    pixel_xy(F.width, F.height, pixel, &px, &py);
    sample_position_at(F, px, py, k, su, sv, x_pix, y_pix);
}

// The initial photon at image-plane position (su, sv) and its derivatives
// with respect to the spin and the inclination.
__host__ __device__ inline void ray_start_at(const FrameParams& F, const AdjointFrame& X, double su, double sv,
                                             double y[6], double* E, double* Lz, double dy[2][6], double dE[2],
                                             double dLz[2]) {
    double x = xm(su, F.tanf);
    double yy = xd(xm(sv, F.tanf), F.aspect);
    const double z = 1.0;
    if (F.has_roll) {
        const double xr = xs(xm(F.cr, x), xm(F.sr, yy));
        const double yr = xa(xm(F.sr, x), xm(F.cr, yy));
        x = xr; yy = yr;
    }
    const double y2 = xs(xm(F.cp, yy), xm(F.sp, z));
    const double z2 = xa(xm(F.sp, yy), xm(F.cp, z));
    const double x2 = xa(xm(F.cy, x), xm(F.sy, z2));
    const double z3 = xa(xm(-F.sy, x), xm(F.cy, z2));
    const double v0 = -z3, v1 = -y2, v2 = x2;
    const double n = xsqrt(xa(xa(xm(v0, v0), xm(v1, v1)), xm(v2, v2)));
    const double d0 = xd(v0, n), d1 = xd(v1, n), d2 = xd(v2, n);
    // p^mu = -(e_0 - d^i e_i), lowered: the same expressions as the render path
    const double zero = 0.0;
    const double p0 = -xa(F.tet00, xm(-1.0, xa(xa(xm(d0, zero), xm(d1, zero)), xm(d2, zero))));
    const double p1 = -xa(zero, xm(-1.0, xa(xa(xm(d0, F.tet11), xm(d1, zero)), xm(d2, zero))));
    const double p2 = -xa(zero, xm(-1.0, xa(xa(xm(d0, zero), xm(d1, F.tet22)), xm(d2, zero))));
    const double p3 = -xa(F.tet03, xm(-1.0, xa(xa(xm(d0, zero), xm(d1, zero)), xm(d2, F.tet33))));
    const double pt = xa(xm(F.ml_tt, p0), xm(F.ml_tp, p3));
    const double pph = xa(xm(F.ml_tp, p0), xm(F.ml_pp, p3));
    y[0] = 0.0;
    y[1] = F.cam_r;
    y[2] = F.cam_th;
    y[3] = F.cam_ph;
    y[4] = xm(F.ml_rr, p1);
    y[5] = xm(F.ml_thth, p2);
    *E = -pt;
    *Lz = pph;
    for (int q = 0; q < 2; ++q) {
        const double p0q = -X.d_tet[0][q];
        const double p1q = d0 * X.d_tet[2][q];
        const double p2q = d1 * X.d_tet[3][q];
        const double p3q = -X.d_tet[1][q] + d2 * X.d_tet[4][q];
        const double ptq = X.d_ml[0][q] * p0 + F.ml_tt * p0q + X.d_ml[1][q] * p3 + F.ml_tp * p3q;
        const double pphq = X.d_ml[1][q] * p0 + F.ml_tp * p0q + X.d_ml[4][q] * p3 + F.ml_pp * p3q;
        dy[q][0] = 0.0;
        dy[q][1] = 0.0;
        dy[q][2] = (q == kParIncl) ? 1.0 : 0.0;
        dy[q][3] = 0.0;
        dy[q][4] = X.d_ml[2][q] * p1 + F.ml_rr * p1q;
        dy[q][5] = X.d_ml[3][q] * p2 + F.ml_thth * p2q;
        dE[q] = -ptq;
        dLz[q] = pphq;
    }
}

// The initial photon of frame-local sample `local_id`.
__host__ __device__ inline void ray_start(const FrameParams& F, const AdjointFrame& X, long long local_id,
                                          double y[6], double* E, double* Lz, double dy[2][6], double dE[2],
                                          double dLz[2]) {
    double su, sv, xp, yp;
    sample_position(F, local_id, &su, &sv, &xp, &yp);
    ray_start_at(F, X, su, sv, y, E, Lz, dy, dE, dLz);
}

// Accepted steps of the replay buffer: where states were thinned the reverse
// pass recomputes a segment in pieces of at most this many steps.
constexpr int kReplay = 16;

// Stored states of one ray: y, sin and cos of its angle, the proposed h and
// beta ln err_prev after every `interval` accepted steps, and the size of the
// step taken from there.  With
// the interval at one, as every ray starts, the reverse sweep reads each
// step's state and size back and integrates nothing again; full slots drop
// every second state and double the interval, and a segment's steps are then
// replayed from its first state.  Word w of slot j lies at
// ck[(j kCkWords + w) stride]: on the device the lanes of a warp interleave
// (stride 32), so that their accesses coalesce.
constexpr int kCkWords = 11;
struct Checkpoints {
    double* ck;
    int slots;
    int interval;
    int n;
    int stride;
    __host__ __device__ __forceinline__ double* at(int slot, int word) const {
        return ck + ((long long)slot * kCkWords + word) * stride;
    }
    __host__ __device__ __forceinline__ void push(const Integ& st) {
        for (int i = 0; i < 6; ++i) *at(n, i) = st.y[i];
        *at(n, 6) = st.h;
        *at(n, 7) = st.errp_mem;
        *at(n, 9) = st.sn0;
        *at(n, 10) = st.c0;
        ++n;
    }
    __host__ __device__ __forceinline__ void after_step(const Integ& st) {
        if (interval == 1) *at(n - 1, 8) = st.h_acc;
        if (st.steps % interval != 0) return;
        if (n == slots) thin();
        if (st.steps % interval == 0) push(st);
    }
    __host__ __device__ BHA_NOINLINE void thin() {
        for (int j = 0; j < slots / 2; ++j)
            for (int i = 0; i < kCkWords; ++i) *at(j, i) = *at(2 * j, i);
        n = slots / 2;
        interval *= 2;
    }
};

// The first two equatorial crossings of a ray: their radii and the accepted
// steps they lie in (0: none); `count` counts all of them.
struct Crossings {
    double r[2];
    int step[2];
    int n;
    int count;
};

// Integrates from `s` with the render path's events (render.cpp:158-257)
// until the ray ends, returning its class, or until its equatorial crossing
// number `stop_crossing` (counted from `s`; 0: none), returning -1 after that
// crossing's step with its radius in *r_hit and without looking at whether
// it hits the disc.  The crossing radius of a disc hit goes to *r_hit.
// Checkpoints (cp) and the first two equatorial crossings (xr) are recorded
// when given.  end_falling: a ray moving inwards inside the innermost photon
// orbit ends there as captured; no turning point is left to it and nothing
// lies on its way (the disc ends at the ISCO), and the creep to the horizon it
// is spared is most of a captured ray's steps.
__host__ __device__ BHA_NOINLINE int forward_run(const FrameParams& F, const RayC& ray, Integ& state, Checkpoints* cp_io,
                                                    Crossings* xr, int stop_crossing, double* r_hit,
                                                    bool end_falling = false) {
    if (F.max_steps <= 0) return BH_HIT_EXHAUSTED;
    // the ray in registers; handed back at its end
    const RayC c = ray;
    Integ s = state;
    Checkpoints cps{nullptr, 0, 1, 0, 1};
    if (cp_io) cps = *cp_io;
    Checkpoints* const cp = cp_io ? &cps : nullptr;
    auto end = [&](int what) {
        state = s;
        if (cp_io) *cp_io = cps;
        return what;
    };
    StepRec rec;
    int crossings = 0;
    for (;;) {
        if (!advance_step(F, c, s, &rec)) return end(BH_HIT_HORIZON);   // no acceptable step (render.cpp:133-136)
        const double rn = rec.r1;
        if (rn <= F.r_stop) return end(BH_HIT_HORIZON);
        if (F.disc_enabled && rec.c0 * rec.c7 < 0.0) {
            const DenseC cth = step_dense(rec, 2);
            const double s_end = dense_crossing(cth, crossing_target(cth.r1, cth.r1 + cth.r2));
            const DenseC crr = step_dense(rec, 1);
            const double rc = dense_eval(crr, s_end);
            if (xr) {
                if (xr->n < 2) {
                    xr->r[xr->n] = rc;
                    xr->step[xr->n++] = s.steps;
                }
                ++xr->count;
            }
            if (++crossings == stop_crossing) {
                *r_hit = rc;
                return end(-1);
            }
            if (rc >= F.r_in && rc <= F.r_out) {
                *r_hit = rc;
                return end(BH_HIT_DISC);
            }
        }
        if (rn > F.r_escape) return end(BH_HIT_SKY);
        if (s.steps >= F.max_steps) return end(BH_HIT_EXHAUSTED);
        if (end_falling && rn < F.r_promote && s.k1[1] < 0.0) return end(BH_HIT_HORIZON);
        if (cp) cp->after_step(s);
    }
}

// The reverse pass: carries the adjoint yb of the state after accepted step N
// of size h_last (and, when rstar_b != 0, the weight of the disc-crossing
// radius of step N) back to the initial photon, with the E, L_z and spin
// adjoints accumulated.  Returns the steps replayed (none where every state
// was kept).
__host__ __device__ BHA_NOINLINE long long reverse_sweep(const FrameParams& F, const RayC& ray, const Checkpoints& cps,
                                                         int N, double h_last, double rstar_b, double yb[6],
                                                         double* Eb, double* Lzb, double* ab) {
    constexpr int kC[4] = {1, 2, 4, 5};
    const RayC c = ray;
    const Checkpoints cp = cps;
    long long replay = 0;
    double buf[kReplay][7];                  // a replayed piece: r, th, p_r, p_th, the step's size, sin, cos
    int first = 0, m = 0;                    // its steps: first + 1 .. first + m
    double yv[6], Ev = *Eb, Lv = *Lzb, av = *ab;
    for (int i = 0; i < 6; ++i) yv[i] = yb[i];
    for (int j = N - 1; j >= 0; --j) {       // step j + 1, from state j
        double y0[4], h, sn, cs;
        if (cp.interval == 1) {
            #pragma unroll
            for (int i = 0; i < 4; ++i) y0[i] = *cp.at(j, kC[i]);
            h = (j == N - 1) ? h_last : *cp.at(j, 8);
            sn = *cp.at(j, 9);
            cs = *cp.at(j, 10);
        } else {
            if (j < first || m == 0) {
                // replay the piece that ends with step j + 1 from the last
                // stored state before it
                const int seg = j / cp.interval, off = j - seg * cp.interval;
                const int skip = (off / kReplay) * kReplay;
                first = seg * cp.interval + skip;
                m = j - first + 1;
                Integ r;
                for (int i = 0; i < 6; ++i) r.y[i] = *cp.at(seg, i);
                r.h = *cp.at(seg, 6);
                r.errp_mem = *cp.at(seg, 7);
                r.sn0 = *cp.at(seg, 9);
                r.c0 = *cp.at(seg, 10);
                r.have_k1 = 0;
                r.tries = 0;
                r.steps = 0;
                for (int q = 0; q < skip; ++q) advance(F, c, r);
                for (int q = 0; q < m; ++q) {
                    for (int i = 0; i < 4; ++i) buf[q][i] = r.y[kC[i]];
                    buf[q][5] = r.sn0;
                    buf[q][6] = r.c0;
                    advance(F, c, r);
                    buf[q][4] = r.h_acc;
                }
                replay += skip + m;
            }
            for (int i = 0; i < 4; ++i) y0[i] = buf[j - first][i];
            h = buf[j - first][4];
            sn = buf[j - first][5];
            cs = buf[j - first][6];
        }
        step_vjp(c, y0, sn, cs, h, yv, &Ev, &Lv, &av, (j == N - 1) ? rstar_b : 0.0);
    }
    for (int i = 0; i < 6; ++i) yb[i] = yv[i];
    *Eb = Ev;
    *Lzb = Lv;
    *ab = av;
    return replay;
}

__host__ __device__ inline RayC ray_consts(const FrameParams& F, double E, double Lz) {
    RayC c;
    c.a = F.a;
    c.a2 = F.a2;
    c.E = E;
    c.Lz = Lz;
    c.rp = F.r_plus;
    c.rm = F.r_minus;
    c.factored = F.factored_delta;
    return c;
}

__host__ __device__ inline void integ_start(const FrameParams& F, const double y0[6], Integ& s) {
    for (int i = 0; i < 6; ++i) s.y[i] = y0[i];
    sc(y0[2], &s.sn0, &s.c0);
    s.h = F.h0;
    s.errp_mem = kBeta * kLnErrFloor;
    s.h_acc = 0.0;
    s.have_k1 = 0;
    s.tries = 0;
    s.steps = 0;
}

// The luminance of a ray that ended in `what` (disc: at radius r_hit; sky: in
// state y = (t, r, th, phi, p_r, p_th)) and, times the loss weight w, its
// derivatives: where the reverse pass starts.
struct Seed {
    double Y, d_edd;
    double yb[6];        // with respect to the state at the end of the last step (sky)
    double rstar_b;      // with respect to the hit radius (disc)
    double Eb, Lzb, ab;
    __host__ __device__ bool any() const {
        return rstar_b != 0.0 || Eb != 0.0 || Lzb != 0.0 || ab != 0.0 || yb[1] != 0.0 || yb[2] != 0.0 ||
               yb[3] != 0.0 || yb[4] != 0.0 || yb[5] != 0.0;
    }
};
__host__ __device__ BHA_NOINLINE void seed_ray(const FrameParams& F, const AdjointFrame& X, const SkyData& sky,
                                               int what, double r_hit, const double y[6], double E, double Lz,
                                               double w, Seed& o) {
    o = Seed{};
    if (what == BH_HIT_DISC) {
        const D5 Y = disc_luminance(F, X, sky.table, r_hit, E, Lz);
        o.Y = Y.v;
        o.rstar_b = w * Y.d[kS5R];
        o.Eb = w * Y.d[kS5E];
        o.Lzb = w * Y.d[kS5L];
        o.ab = w * Y.d[kS5A];
        o.d_edd = w * Y.d[kS5M];
    } else if (what == BH_HIT_SKY) {
        D8 v[3];
        if (escape_direction(y, E, Lz, F.a, v)) {
            const double d[3] = {v[0].v, v[1].v, v[2].v};
            double gY[3];
            o.Y = sky_luminance(sky, F, d, gY);
            double gs[8];
            for (int k = 0; k < 8; ++k)
                gs[k] = w * (gY[0] * v[0].d[k] + gY[1] * v[1].d[k] + gY[2] * v[2].d[k]);
            for (int k = 0; k < 5; ++k) o.yb[k + 1] = gs[k];
            o.Eb = gs[5];
            o.Lzb = gs[6];
            o.ab = gs[7];
        }
    }
}

// The forward pass, the seed and the reverse pass of one ray.  `ck` holds
// `slots` states of kCkWords doubles.  With w == 0 (or forward_only) only the
// luminance is computed.  xr (may be null) receives the ray's first two
// equatorial crossings.
__host__ __device__ inline void adjoint_ray(const FrameParams& F, const AdjointFrame& X, const SkyData& sky,
                                            long long local_id, double w, double* ck, int slots, int stride,
                                            bool forward_only, RayResult* out, Crossings* xr = nullptr) {
    double y0[6], E, Lz, dy0[2][6], dE[2], dLz[2];
    ray_start(F, X, local_id, y0, &E, &Lz, dy0, dE, dLz);
    const RayC c = ray_consts(F, E, Lz);
    out->Y = 0.0;
    for (int q = 0; q < 4; ++q) out->grad[q] = 0.0;
    out->replay = 0;

    Integ s;
    integ_start(F, y0, s);
    Checkpoints cp{ck, slots, X.checkpoint_interval, 0, stride};
    cp.push(s);
    double r_hit = 0.0;
    const int what = forward_run(F, c, s, &cp, xr, 0, &r_hit);
    out->what = what;
    out->steps = s.steps;
    out->interval = cp.interval;

    Seed sd;
    seed_ray(F, X, sky, what, r_hit, s.y, E, Lz, w, sd);
    out->Y = sd.Y;
    out->grad[2] = sd.d_edd;
    double Eb = sd.Eb, Lzb = sd.Lzb, ab = sd.ab;
    double* const yb = sd.yb;
    const double rstar_b = sd.rstar_b;
    if (forward_only || w == 0.0 || (what != BH_HIT_DISC && what != BH_HIT_SKY)) return;
    if (!sd.any()) return;

    // ---- reverse and the initial photon ------------------------------------------------
    out->replay = reverse_sweep(F, c, cp, s.steps, s.h_acc, rstar_b, yb, &Eb, &Lzb, &ab);
    for (int q = 0; q < 2; ++q) {
        double gq = Eb * dE[q] + Lzb * dLz[q];
        for (int i = 0; i < 6; ++i) gq += yb[i] * dy0[q][i];
        out->grad[q] += gq;
    }
    out->grad[kParSpin] += ab;
}

// ---- the edge term ---------------------------------------------------------------------
//
// A point-sampled frame changes with r_out only where a sample's equatorial
// crossing radius r_c passes the edge, so the discrete adjoint above has no
// r_out term.  The derivative of the frame averaged over each sample's cell
// of the pixel has one: with r_c linear in the image plane across the cell,
//   d(pixel)/d(r_out)  =  (Y_in - Y_out) L / |grad r_c|,
// L the length of the line r_c = r_out inside the cell (pixel units), Y_in
// the disc's luminance at r_out along the ray (the same E, L_z), Y_out what
// the ray sees when this crossing misses the disc (its continuation traced
// on).  The same edge moves with any parameter q that moves r_c, which adds
//   -(Y_in - Y_out) (d r_c/d q) L / |grad r_c|
// to d(pixel)/dq.  grad r_c and d r_c/dq come from a reverse sweep seeded
// with the crossing radius alone.

// d(initial p_r, p_th, E, L_z)/d(su, sv): the image-plane coordinates of
// scene.h:356-384 (su = 2 (x + jx)/W - 1, sv = 1 - 2 (y + jy)/H).
__host__ __device__ inline void ray_start_pixel_tangents(const FrameParams& F, double su0, double sv0,
                                                         double dpr[2], double dpth[2], double dE[2],
                                                         double dLz[2]) {
    using D2 = Dual<2>;
    const D2 su = D2::var(su0, 0), sv = D2::var(sv0, 1);
    D2 x = su * F.tanf;
    D2 yy = sv * F.tanf / F.aspect;
    if (F.has_roll) {
        const D2 xr = F.cr * x - F.sr * yy;
        const D2 yr = F.sr * x + F.cr * yy;
        x = xr;
        yy = yr;
    }
    const D2 y2 = F.cp * yy - F.sp;
    const D2 z2 = F.sp * yy + F.cp;
    const D2 x2 = F.cy * x + F.sy * z2;
    const D2 z3 = -F.sy * x + F.cy * z2;
    const D2 v0 = -z3, v1 = -y2, v2 = x2;
    const D2 n = sqrt(v0 * v0 + v1 * v1 + v2 * v2);
    const D2 d0 = v0 / n, d1 = v1 / n, d2 = v2 / n;
    for (int k = 0; k < 2; ++k) {
        const double p1 = d0.d[k] * F.tet11, p2 = d1.d[k] * F.tet22, p3 = d2.d[k] * F.tet33;
        dpr[k] = F.ml_rr * p1;
        dpth[k] = F.ml_thth * p2;
        dE[k] = -(F.ml_tp * p3);
        dLz[k] = F.ml_pp * p3;
    }
}

// Length of the line g . (x - c) = rhs inside the rectangle [x0, x1] x [y0, y1].
__host__ __device__ inline double line_in_cell(double gx, double gy, double cx, double cy, double rhs, double x0,
                                               double x1, double y0, double y1) {
    double px[4], py[4];
    int n = 0;
    if (gy != 0.0) {
        for (int e = 0; e < 2; ++e) {
            const double x = e ? x1 : x0;
            const double y = cy + (rhs - gx * (x - cx)) / gy;
            if (y >= y0 && y <= y1) { px[n] = x; py[n] = y; ++n; }
        }
    }
    if (gx != 0.0) {
        for (int e = 0; e < 2; ++e) {
            const double y = e ? y1 : y0;
            const double x = cx + (rhs - gy * (y - cy)) / gx;
            if (x >= x0 && x <= x1) { px[n] = x; py[n] = y; ++n; }
        }
    }
    double best = 0.0;
    for (int i = 0; i < n; ++i)
        for (int j = i + 1; j < n; ++j) {
            const double dx = px[i] - px[j], dy = py[i] - py[j];
            const double l = sqrt(dx * dx + dy * dy);
            if (l > best) best = l;
        }
    return best;
}

// Edges of the disc an equatorial crossing can be near.
enum { kEdgeOuter = 1, kEdgeInner = 2 };

// The luminance of a ray that ended in `what` (as seed_ray).
__host__ __device__ BHA_NOINLINE double luminance(const FrameParams& F, const AdjointFrame& X, const SkyData& sky,
                                                  int what, double r_hit, const double y[6], double E, double Lz) {
    if (what == BH_HIT_DISC) return disc_luminance(F, X, sky.table, r_hit, E, Lz).v;
    double d[3], gY[3];
    if (what == BH_HIT_SKY && escape_direction_value(y, E, Lz, F.a, d)) return sky_luminance(sky, F, d, gY);
    return 0.0;
}

// The luminance jumps across the edges in `edges`: the disc's side is its
// luminance at r_out along this ray; the Novikov-Thorne flux vanishes at r_in.
__host__ __device__ BHA_NOINLINE void edge_jumps(const FrameParams& F, const AdjointFrame& X, const SkyData& sky,
                                                 int edges, double Y_beyond, double E, double Lz, double dY[2]) {
    dY[0] = (edges & kEdgeOuter) ? disc_luminance(F, X, sky.table, F.r_out, E, Lz).v - Y_beyond : 0.0;
    dY[1] = (edges & kEdgeInner) ? -Y_beyond : 0.0;
}

// The edge terms of a sample's crossing at radius rc with jumps dY, from
// d r_c / d(initial state, E, L_z, spin) = (yb, Eb, Lzb, ab); see edge_sample.
__host__ __device__ BHA_NOINLINE void edge_finish(const FrameParams& F, const AdjointFrame& X, int px, int py, int k,
                                                  int edges, double w, double rc, const double dY[2],
                                                  const double yb[6], double Eb, double Lzb, double ab,
                                                  double out[3], int* cells, double* diag) {
    double su, sv, xp, yp;
    sample_position_at(F, px, py, k, &su, &sv, &xp, &yp);
    double y0[6], E, Lz, dy0[2][6], dE[2], dLz[2];
    ray_start_at(F, X, su, sv, y0, &E, &Lz, dy0, dE, dLz);
    double dpr[2], dpth[2], dEp[2], dLzp[2];
    ray_start_pixel_tangents(F, su, sv, dpr, dpth, dEp, dLzp);
    double drc[2];
    for (int j = 0; j < 2; ++j) drc[j] = yb[4] * dpr[j] + yb[5] * dpth[j] + Eb * dEp[j] + Lzb * dLzp[j];
    // grad r_c in pixel units: su = 2 x / W - 1, sv = 1 - 2 y / H
    const double gx = drc[0] * (2.0 / F.width), gy = drc[1] * (-2.0 / F.height);
    const double gn = sqrt(gx * gx + gy * gy);
    double drq[2];
    for (int q = 0; q < 2; ++q) {
        drq[q] = Eb * dE[q] + Lzb * dLz[q];
        for (int i = 0; i < 6; ++i) drq[q] += yb[i] * dy0[q][i];
    }
    drq[kParSpin] += ab;
    // the sample's cell in pixel units
    const int S = F.S;
    const int sy = k / S, sx = k - (k / S) * S;
    const double x0 = px + sx * F.inv_S, x1 = px + (sx + 1) * F.inv_S;
    const double y0c = py + sy * F.inv_S, y1 = py + (sy + 1) * F.inv_S;
    double L[2] = {0.0, 0.0};
    for (int e = 0; e < 2; ++e) {
        if (!(edges & (e == 0 ? kEdgeOuter : kEdgeInner)) || !(gn > 0.0)) continue;
        const double r_edge = (e == 0) ? F.r_out : F.r_in;
        L[e] = line_in_cell(gx, gy, xp, yp, r_edge - rc, x0, x1, y0c, y1);
        if (!(L[e] > 0.0) || dY[e] == 0.0) continue;
        ++*cells;
        const double swept = w * dY[e] * L[e] / gn;
        if (e == 0) {
            out[0] += swept;
            out[1] -= swept * drq[kParSpin];
            out[2] -= swept * drq[kParIncl];
        } else {
            out[1] += swept * (drq[kParSpin] - 2.0 * F.x0 * X.d_x0);
            out[2] += swept * drq[kParIncl];
        }
    }
    if (diag) {
        diag[0] = rc;
        diag[1] = gn;
        diag[2] = drq[0];
        diag[3] = drq[1];
        diag[4] = drc[0];
        diag[5] = drc[1];
        diag[6] = L[0];
        diag[7] = dY[0];
        diag[8] = L[1];
        diag[9] = dY[1];
    }
}

// The edge term of equatorial crossing number `crossing` (1 or 2) of sample k
// of pixel (px, py), for the disc edges in `edges` (kEdgeOuter: r_out;
// kEdgeInner: r_in, the ISCO) and pixel weight w = dLoss/d(pixel).  With
// phi = r_out - r_c (outer) or r_c - r_in (inner), positive on the disc side,
//   d(pixel)/dq = (Y_disc - Y_beyond) (d phi/d q) L / |grad r_c|.
// out[0..2] receive the contributions to dLoss/d(r_out), d(spin),
// d(inclination); *cells the number of edges that cross the sample's cell.
// diag (may be null) receives r_c, |grad r_c| (per pixel), d r_c/d(spin,
// inclination), d r_c/d(su, sv), and per edge (outer, inner) L and
// Y_disc - Y_beyond.  Returns the accepted steps integrated (forward,
// continuation and replay).
__host__ __device__ BHA_NOINLINE long long edge_sample(const FrameParams& F, const AdjointFrame& X, const SkyData& sky,
                                                 int px, int py, int k, int crossing, int edges, double w,
                                                 double* ck, int slots, int stride, double out[3], int* cells,
                                                 double* diag = nullptr) {
    out[0] = out[1] = out[2] = 0.0;
    *cells = 0;
    double su, sv, xp, yp;
    sample_position_at(F, px, py, k, &su, &sv, &xp, &yp);
    double y0[6], E, Lz, dy0[2][6], dE[2], dLz[2];
    ray_start_at(F, X, su, sv, y0, &E, &Lz, dy0, dE, dLz);
    const RayC c = ray_consts(F, E, Lz);
    Integ s;
    integ_start(F, y0, s);
    Checkpoints cp{ck, slots, X.checkpoint_interval, 0, stride};
    cp.push(s);
    double rc = 0.0;
    if (forward_run(F, c, s, &cp, nullptr, crossing, &rc) != -1) return s.steps;
    const int step = s.steps;
    const double h_step = s.h_acc;

    // What the ray meets when this crossing misses the disc: its
    // continuation traced on from there.
    Integ t = s;
    double r_hit = 0.0;
    const int what = forward_run(F, c, t, nullptr, nullptr, 0, &r_hit, true);
    long long work = t.steps;
    const double Y_beyond = luminance(F, X, sky, what, r_hit, t.y, E, Lz);
    double dY[2];
    edge_jumps(F, X, sky, edges, Y_beyond, E, Lz, dY);
    if (dY[0] == 0.0 && dY[1] == 0.0 && !diag) return work;

    // d r_c / d(initial state, E, L_z, spin) by a reverse sweep seeded with r_c
    double yb[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    double Eb = 0.0, Lzb = 0.0, ab = 0.0;
    work += reverse_sweep(F, c, cp, step, h_step, 1.0, yb, &Eb, &Lzb, &ab);

    edge_finish(F, X, px, py, k, edges, w, rc, dY, yb, Eb, Lzb, ab, out, cells, diag);
    return work;
}

// Whether the crossing at radius rc (sample grid neighbours' same crossing
// differing by at most dmax; 0 when none has one) is examined for the disc's
// edges: within twice that spread of an edge, or within a tenth of the edge
// radius when no neighbour has the crossing.  Returns kEdge* bits.
__host__ __device__ inline int edge_mask(const FrameParams& F, double rc, double dmax) {
    int m = 0;
    auto near = [&](double re) { return dmax > 0.0 ? fabs(rc - re) <= 2.0 * dmax : fabs(rc - re) <= 0.1 * re; };
    if (rc >= F.r_in && near(F.r_out)) m |= kEdgeOuter;
    if (rc <= F.r_out && near(F.r_in)) m |= kEdgeInner;
    return m;
}

}  // namespace adj
}  // namespace bhg
