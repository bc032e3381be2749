// Pieces of the Mohr-Coulomb point evaluation that the return mapping and the potential energy share.
#pragma once

#include "ssp_internal.cuh"

namespace ssp {

struct Mat3 {
    double c_bar, sin_phi, shear, lame;
};

// sin and cos of a Lode angle theta in [0, pi/3] from their Taylor series, Horner in theta^2: the
// first omitted terms, theta^19 / 19! and theta^20 / 20!, are below 2e-17 there, and without a
// branch every lane of a warp runs the same instructions (a general sincos reduces its argument by
// quadrants, and pi/4 < pi/3).  Within one ulp of the correctly rounded values on [0, pi/3].
__device__ __forceinline__ void sincos_lode(double theta, double &s, double &c) {
    const double z = theta * theta;
    double ps = 1.0 / 355687428096000.0;  // 1/17!
    ps = fma(ps, z, -1.0 / 1307674368000.0);
    ps = fma(ps, z, 1.0 / 6227020800.0);
    ps = fma(ps, z, -1.0 / 39916800.0);
    ps = fma(ps, z, 1.0 / 362880.0);
    ps = fma(ps, z, -1.0 / 5040.0);
    ps = fma(ps, z, 1.0 / 120.0);
    ps = fma(ps, z, -1.0 / 6.0);
    s = fma(theta * z, ps, theta);
    double pc = -1.0 / 6402373705728000.0;  // -1/18!
    pc = fma(pc, z, 1.0 / 20922789888000.0);
    pc = fma(pc, z, -1.0 / 87178291200.0);
    pc = fma(pc, z, 1.0 / 479001600.0);
    pc = fma(pc, z, -1.0 / 3628800.0);
    pc = fma(pc, z, 1.0 / 40320.0);
    pc = fma(pc, z, -1.0 / 720.0);
    pc = fma(pc, z, 1.0 / 24.0);
    pc = fma(pc, z, -0.5);
    c = fma(z, pc, 1.0);
}

// Elastic screen from invariants, before any eigen-decomposition, in FP32.  With principal trial
// strains e1 >= e2 >= e3, Q = J2/3 and Lode angle a, the trial yield function is
//   f = 2G[(e1 - e3) + s(e1 + e3)] + 2 lambda s I1 - c_bar,
//   (e1 - e3) + s(e1 + e3) = 2 sqrt(Q) (sqrt(3) sin a + s cos a) + 2 s I1 / 3,
// and sqrt(3) sin a + s cos a <= sqrt(3 + s^2) for every a (Cauchy-Schwarz), so
//   f <= bound = 2G[2 sqrt(Q) sqrt(3 + s^2) + 2 s I1 / 3] + 2 lambda s I1 - c_bar.
// The bound is evaluated in FP32 from inputs truncated to 24 bits (J2 from differences of the
// normal components, so no cancellation against I1): its absolute error stays below ~4e-6 of
//   size = 2|G| (2 sqrt(Q) sqrt(3 + s^2) + 3 max|t_i|) + 2|lambda s I1| + |c_bar|.
// A point with bound <= -1e-4 size is therefore elastic however the FP64 eigenvalues of the full
// path round (their error is at most ~1e-8 sqrt(Q), near repeated roots): the full path's branch
// test would say elastic too.  Such a point is finished from t and I1 in FP64 with the elastic
// branch's own arithmetic, so S and DS are bitwise those of the full path, and it costs about a
// dozen FP64 instructions instead of an eigen-decomposition.
__device__ __forceinline__ bool screen_elastic(const double *E, const Mat3 &m) {
    float t[6];
#pragma unroll
    for (int i = 0; i < 6; ++i) t[i] = df_from_f64(E[i]).hi * (i < 3 ? 1.0f : 0.5f);
    const float G = df_from_f64(m.shear).hi, L = df_from_f64(m.lame).hi;
    const float s = df_from_f64(m.sin_phi).hi, c = df_from_f64(m.c_bar).hi;
    const float d01 = t[0] - t[1], d12 = t[1] - t[2], d20 = t[2] - t[0];
    const float J2 = (d01 * d01 + d12 * d12 + d20 * d20) * (1.0f / 6.0f) + t[3] * t[3] + t[4] * t[4] + t[5] * t[5];
    const float I1 = t[0] + t[1] + t[2];
    const float dev = 2.0f * sqrtf(J2 * (1.0f / 3.0f)) * sqrtf(3.0f + s * s);
    const float bound = 2.0f * G * (dev + (2.0f / 3.0f) * s * I1) + 2.0f * L * s * I1 - c;
    const float tmax = fmaxf(fmaxf(fabsf(t[0]), fabsf(t[1])), fmaxf(fabsf(t[2]), fmaxf(fabsf(t[3]), fmaxf(fabsf(t[4]), fabsf(t[5])))));
    const float size = 2.0f * fabsf(G) * (dev + 3.0f * tmax) + 2.0f * fabsf(L * s * I1) + fabsf(c);
    return bound <= -1e-4f * size;
}

}  // namespace ssp
