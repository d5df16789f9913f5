// bh_jet.cuh - The jet's volumetric emission on the device (binary64).
//
// jet.h:96-315 and render.cpp:44-62, 107-122: the prescribed parabolic jet
// (radius and Lorentz factor ~ z^k, limb-brightened Gaussian sheath,
// emissivity ~ Gamma^-(2+alpha) R^-(3+alpha) (z/z_base)^zeta with soft ends),
// its plasma four-velocity built in the ZAMO frame, and the optically thin
// transfer integral  j_nu0 Integral shape g^(2+alpha) dlambda  accumulated
// with four-point Gauss-Legendre quadrature on each accepted step's dense
// output, truncated at an occluding event.
#pragma once

#include <cuda_runtime.h>

#include "bh_common.cuh"
#include "bh_dp5.cuh"
#include "bh_frame.h"

namespace bhg {

// Four-point Gauss-Legendre nodes and weights on [0, 1] (render.cpp:46-50).
__device__ __forceinline__ double gl_x(int q) {
    return q == 0 ? 0.06943184420297371 : q == 1 ? 0.33000947820757187 : q == 2 ? 0.66999052179242813
                                                                                 : 0.93056815579702629;
}
__device__ __forceinline__ double gl_w(int q) {
    return (q == 0 || q == 3) ? 0.17392742256872693 : 0.32607257743127307;
}

__device__ __forceinline__ double jet_smoothstep(double t) {
    t = dclamp(t, 0.0, 1.0);
    return t * t * (3.0 - 2.0 * t);
}
// Emissivity of the jet at one quadrature node (jet.h:194-240): the comoving
// profile at cylindrical (z, rho) times g^(2 + alpha), g = 1 / (p . u) for the jet
// plasma at (r, th); p = (p_t, p_r, p_th, p_phi).  Zero outside the jet.
//
// The binary64 special functions bound the jet kernels, so the powers are
// collected into one: with l = ln(|z| / z_base), R / R_base = e^(k l) and
// everything that is a power of z, Gamma or g is
//   exp((zeta - (3 + alpha) k) l - (2 + alpha) ln(Gamma (p . u) / Gamma_base)),
// two logarithms and four exponentials (with the sheath's two) where the
// factors taken one by one are seven powers and two exponentials; the metric's
// square roots come from three rsqrt.  Frames move by a few 1e-15 of their
// norm.  With jet_may_touch: quasar preset at 320 x 180 in binary64 10.7 -> 4.3 ms, M87
// preset at 1024 x 576 mixed 20.8 -> 8.0 ms.
__device__ __forceinline__ double jet_node(const FrameParams& F, double r, double th, double p_t, double p_phi,
                                           const DenseC& cpr, const DenseC& cpth, double s) {
    double sn, cs;
    sincos(th, &sn, &cs);
    const double a = F.a, a2 = F.a2;
    const double z = r * cs;
    const double az = fabs(z);
    if (az <= F.jet_z_base || az >= F.jet_z_top) return 0.0;
    const double r2a2 = r * r + a2;
    const double rho = sqrt(r2a2) * sn;
    const double zc = dmaxr(az, 1e-6);
    const double l = log(zc * F.jet_inv_zb);
    const double pk = exp(F.jet_k * l);                    // (z / z_base)^k
    const double u = rho / (F.jet_R_base * pk);
    const double es = (u - F.jet_u_peak) / F.jet_u_wid, et = u / F.jet_spine_wid;
    const double f = exp(-es * es) + F.jet_spine * exp(-et * et);
    if (f < 1e-9) return 0.0;
    const double ramp = jet_smoothstep((az - F.jet_z_base) / (0.5 * F.jet_z_base)) *
                        jet_smoothstep((F.jet_z_top - az) / (0.15 * F.jet_z_top));
    if (!(f * ramp > 0.0)) return 0.0;
    const double G_at = 1.0 + (F.jet_gamma_max - 1.0) * dminr(1.0, pk * F.jet_ck);

    // the plasma's velocity in the ZAMO frame (kerr.h:283-292)
    if (fabs(sn) < 1e-9) sn = (sn < 0.0) ? -1e-9 : 1e-9;
    const double sn2 = sn * sn;
    const double Sigma = r2a2 - a2 * sn2;
    const double Delta = r * r - 2.0 * r + a2;
    const double A = r2a2 * r2a2 - a2 * Delta * sn2;
    const double rS = rsqrt(Sigma), rD = rsqrt(Delta), rA = rsqrt(A);
    const double sD = Delta * rD;                          // sqrt(Delta)
    const double q = A * rA * rS;                          // sqrt(A / Sigma)
    const double ilapse = q * rD;                          // lapse = sqrt(Sigma Delta / A)
    const double omega = 2.0 * a * r * rA * rA;
    const double iG = 1.0 / G_at;
    const double v2 = dmaxr(0.0, 1.0 - iG * iG);
    const double v = sqrt(v2);
    const double v_phi = dclamp((F.jet_Omega_F - omega) * sn * q * dminr(ilapse, 1e12), -0.5 * v, 0.5 * v);
    const double v_pol = sqrt(dmaxr(0.0, v2 - v_phi * v_phi));
    const double G = dclamp(G_at, 1.0, 1e6);               // 1 / sqrt(max(1e-12, 1 - v^2))
    const double sgn = (cs >= 0.0) ? 1.0 : -1.0;
    const double p_r = dense_eval(cpr, s), p_th = dense_eval(cpth, s);
    const double pol = sgn * v_pol * rS * (p_r * cs * sD - p_th * sn);
    const double ku = G * ((p_t + p_phi * omega) * ilapse + pol + p_phi * v_phi * (rA * rS * Sigma) / sn);
    if (!(ku > 1e-12)) return 0.0;
    const double lz = (az < 1e-6) ? log(az * F.jet_inv_zb) : l;
    const double e = F.jet_zeta * lz - (3.0 + F.jet_alpha) * F.jet_k * l -
                     (2.0 + F.jet_alpha) * log(G_at * ku * F.jet_inv_gb);
    return f * ramp * exp(e);
}

// Shortest distance from the origin to the segment p0 -> p1 (render.cpp:55-62).
__device__ __forceinline__ double segment_distance_to_origin(const double p0[3], const double p1[3]) {
    const double d0 = p1[0] - p0[0], d1 = p1[1] - p0[1], d2 = p1[2] - p0[2];
    const double dd = d0 * d0 + d1 * d1 + d2 * d2;
    double t = 0.0;
    if (dd > 0.0) t = dclamp(-(p0[0] * d0 + p0[1] * d1 + p0[2] * d2) / dd, 0.0, 1.0);
    const double q0 = p0[0] + t * d0, q1 = p0[1] + t * d1, q2 = p0[2] + t * d2;
    return sqrt(q0 * q0 + q1 * q1 + q2 * q2);
}

// Pseudo-Cartesian position (geodesic.h:256-262).
__device__ __forceinline__ void bl_cartesian(double a, double r, double th, double ph, double q[3]) {
    const double rr = sqrt(r * r + a * a);
    double sn, cs, sp, cp;
    sincos(th, &sn, &cs);
    sincos(ph, &sp, &cp);
    q[0] = rr * sn * cp;
    q[1] = rr * sn * sp;
    q[2] = r * cs;
}

// Whether a step from cylindrical (z0, rho0) to (z1, rho1), azimuth difference
// dphi, may touch the jet; false only where every quadrature node of the step has
// zero emissivity for certain.  A point of the step lies within about the
// chord of either end; the margin allows for the curvature of a capped step
// and the roundings of binary32.  Steps longer than a quarter of the distance
// are not judged.  Beyond u_cut jet radii the sheath's profile is below its
// cut-off, and the radius grows with |z| (k >= 0).  Without the test every
// step inside the bounding sphere (all of them, for a camera inside it) went
// through the quadrature's special functions.
__device__ __forceinline__ bool jet_may_touch(const FrameParams& F, float z0, float rho0, float z1, float rho1,
                                              float dphi) {
    if (!(F.jet_r_bound > 0.0)) return false;
    const float dz = z1 - z0;
    const float c2 = fmaf(dz, dz, fmaf(rho0, rho0, rho1 * rho1) - 2.f * rho0 * rho1 * cosf(dphi));
    const float rm = fmaxf(rho0, rho1), zm = fmaxf(fabsf(z0), fabsf(z1));
    const float size = rm + zm;
    const float c = sqrtf(fmaxf(c2, 0.f)) + 3e-3f * size;
    if (!(4.f * c < size)) return true;
    const float zmax = zm + 0.25f * c;
    if (zmax < 0.999f * (float)F.jet_z_base) return false;
    const float zmin = ((z0 < 0.f) != (z1 < 0.f)) ? 0.f : fminf(fabsf(z0), fabsf(z1)) - 0.25f * c;
    if (zmin > 1.001f * (float)F.jet_z_top) return false;
    return rm - 1.5f * c < F.jet_f_cut * __powf(zmax, (float)F.jet_k) || F.jet_f_cut < 0.f;
}

// The transfer integral over [0, s_end] of one step of size h from the dense
// polynomials of r, th, p_r, p_th (render.cpp:107-122); p_t = -E, p_phi = L_z.
__device__ __noinline__ double jet_step_integral(const FrameParams& F, const DenseC& cr, const DenseC& cth,
                                                 const DenseC& cpr, const DenseC& cpth, double E, double Lz,
                                                 double h, double s_end) {
    double sum = 0.0;
    #pragma unroll 1
    for (int q = 0; q < 4; ++q) {
        const double s = gl_x(q) * s_end;
        sum += gl_w(q) * jet_node(F, dense_eval(cr, s), dense_eval(cth, s), -E, Lz, cpr, cpth, s);
    }
    return F.jet_j_nu0 * sum * h * s_end;
}

}  // namespace bhg
