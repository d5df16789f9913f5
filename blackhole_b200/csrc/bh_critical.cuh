// bh_critical.cuh - Which rays of a mixed frame pass close to the photon shell: the
// bounds, and the test in binary32 (it also compiles for the host, where the
// tests compare it with the test in binary64 ray by ray).
#pragma once

#include <cmath>
#include <cstdint>

#include "bh_common.cuh"
#include "bh_frame.h"

namespace bhg {

// Bounds on |R_min| / r*^4 (near_critical, bh_trace.cu): under kNearCritical a ray
// is traced in binary64; under kNearCriticalTight a binary32 ray runs at a quarter
// of the frame's tolerances.
constexpr double kNearCritical = 0.1;
constexpr double kNearCriticalTight = 0.2;
enum { kRayPlain = 0, kRayBinary64 = 1, kRayTight = 2 };

// near_critical of a ray in binary32, where that decides it: the class, or -1
// for a ray that has to be looked at in binary64.  The photon's constants come out
// with relative errors of about 1e-6, R(r*) / r*^4 with a few of those (its terms
// are at most three, and r* is its minimum, so an error in r* enters squared); kMargin
// is a thousand of them.  The direction's components are differences where the
// hole lies off the axis of the field, and their absolute error is that times the
// distance at the hole: it is carried along (db, dq) and widens the margins, by 1%
// more undecided rays for a field of 20,000 M at the hole's distance (without it
// one ray in 2,000 near the hole fell into a wrong class at 10^6 M).  Every
// comparison asks for the certain case, so that a NaN, an overflow or a cancelled E
// decides nothing.
__host__ __device__ __forceinline__ int near_critical_quick(const FrameParams& F, long long local_id) {
    constexpr float kMargin = 4e-3f;
    constexpr float kComponent = 6e-7f;                        // ten roundings, each of 2^-24
    const int S = F.S;
    const long long pixel = local_id / (S * S);
    const int k = (int)(local_id - pixel * (S * S));
    const int sy = k / S, sx = k - sy * S;
    int px, py;
    pixel_xy(F.width, F.height, pixel, &px, &py);
    const uint64_t s0 = F.seed ^ ((uint64_t)py << 32) ^ ((uint64_t)px * 0x9E3779B97F4A7C15ull);
    const uint64_t g = 0x9E3779B97F4A7C15ull;
    const float u1 = (float)(unsigned)(mix64(s0 + (uint64_t)(2 * k + 1) * g) >> 40) * 0x1p-24f;
    const float u2 = (float)(unsigned)(mix64(s0 + (uint64_t)(2 * k + 2) * g) >> 40) * 0x1p-24f;
    const FrameParams::QuickCamera& C = F.quick;
    // 2 (px + jx) / W - 1 with the integer part exact
    const float su = ((float)(2 * px - F.width) + 2.f * ((float)sx + u1) * C.inv_s) * C.inv_w;
    const float sv = ((float)(F.height - 2 * py) - 2.f * ((float)sy + u2) * C.inv_s) * C.inv_h;
    const float x = su * C.tanf, y = sv * C.tanf * C.inv_aspect;
    const float xr = C.cr * x - C.sr * y, yr = C.sr * x + C.cr * y;
    const float y2 = C.cp * yr - C.sp, z2 = C.sp * yr + C.cp;
    const float x2 = C.cy * xr + C.sy * z2, z3 = C.cy * z2 - C.sy * xr;
    const float in = rsqrtf(x2 * x2 + y2 * y2 + z3 * z3);
    const float d0 = -z3 * in, d1 = -y2 * in, d2 = x2 * in;
    const float p0 = -C.tet00, p3 = d2 * C.tet33 - C.tet03;
    const float pt0 = C.ml_tt * p0, pt3 = C.ml_tp * p3;
    const float E = -(pt0 + pt3);
    const float Lz0 = C.ml_tp * p0, Lz3 = C.ml_pp * p3, Lz = Lz0 + Lz3;
    if (d0 > 1e-3f) return kRayPlain;                          // outgoing
    // cancelled sums (a camera in the ergosphere) and a grazing d0 are not judged
    if (!(d0 < -1e-3f) || !(fabsf(E) > 0.05f * (fabsf(pt0) + fabsf(pt3)))) return -1;
    const float a = C.a, a2 = C.a2;
    const float iE = 1.f / E, b = Lz * iE;
    const float pth = C.ml_thth * (d1 * C.tet22);
    // errors of the components, of b (the size of what was summed into L_z bounds
    // its own) and of p_th / E
    const float e1 = kComponent * (fabsf(x) + fabsf(y) + fabsf(C.sp)) * in;
    const float e2 = kComponent * (fabsf(x) + fabsf(y) + fabsf(C.sy) * (1.f + fabsf(y))) * in;
    const float db = (4e-6f * (fabsf(Lz0) + fabsf(Lz3)) + fabsf(C.ml_pp * C.tet33) * e2) * fabsf(iE);
    const float dp = fabsf(C.ml_thth * C.tet22 * iE) * e1;
    const float q = (pth * pth + C.cs2 * (Lz * Lz * C.inv_sn2 - a2 * E * E)) * iE * iE;
    const float bma = b - a;
    const float c2 = a2 - b * b - q, c1 = 2.f * (q + bma * bma), c0 = -a2 * q;
    const float dq = (2.f * fabsf(pth * iE) + dp) * dp + C.cs2 * C.inv_sn2 * (2.f * fabsf(b) + db) * db;
    const float dc = (2.f * fabsf(b) + db) * db + dq;
    const float lim = 1e-3f * (a2 + b * b + fabsf(q) + 1.f) + dc;
    if (c2 > lim) return kRayPlain;                            // no minimum
    if (!(c2 < -lim)) return -1;
    // R' is least at sqrt(-c_2 / 6): above zero there, no minimum either
    const float ri = sqrtf(c2 * (-1.f / 6.f)), ri3 = 8.f * ri * ri * ri;
    const float dl = 1e-3f * (fabsf(c1) + ri3) + 2.f * dq + (4.f * fabsf(bma) + 2.f * db) * db + 2.f * ri * dc;
    if (c1 - ri3 > dl) return kRayPlain;
    if (!(c1 - ri3 < -dl)) return -1;
    float r = sqrtf(-c2), last = 0.f;
    #pragma unroll 1
    for (int it = 0; it < 12; ++it) {
        const float r2 = r * r;
        const float step = (4.f * r2 * r + 2.f * c2 * r + c1) / (12.f * r2 + 2.f * c2);
        r -= step;
        last = fabsf(step);
        if (!(last > 1e-5f * r)) break;
    }
    if (!(last <= 1e-5f * r)) return -1;
    const float ir = 1.f / r;
    // an error db of b moves R(r*) / r*^4 by about 2 |b| db / r^2 (and as much through
    // c_1), one of q by about dq / r^2
    const float margin = kMargin + (16.f * (fabsf(b) + 1.f + db) * db + 4.f * dq) * ir * ir;
    const float Rn = 1.f + (c2 + (c1 + c0 * ir) * ir) * ir * ir;
    // below the horizon, beyond the camera, or certainly not a near miss
    if (Rn > margin || Rn < -(float)kNearCriticalTight - margin) return kRayPlain;
    if (!(margin < 0.04f)) return -1;
    if (r < 0.999f * C.r_plus || r > 1.001f * C.cam_r) return kRayPlain;
    if (!(r > 1.001f * C.r_plus) || !(r < 0.999f * C.cam_r)) return -1;
    if (Rn < -margin && Rn > -(float)kNearCritical + margin) return kRayBinary64;
    if (Rn < -(float)kNearCritical - margin && Rn > -(float)kNearCriticalTight + margin) return kRayTight;
    return -1;
}

}  // namespace bhg
