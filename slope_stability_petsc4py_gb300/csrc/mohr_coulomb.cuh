// Pieces of the Mohr-Coulomb point evaluation that the return mapping and the potential energy share.
#pragma once

#include "ssp_internal.cuh"

namespace ssp {

struct Mat3 {
    double c_bar, sin_phi, shear, lame;
};

// Roots and reciprocals in FP64 by Newton steps from an FP32 start: the FP64 pipe does 1.6 operations a clock on an
// SM, and what bounds the return mapping is their number.  A square root and its reciprocal together take six, a
// reciprocal three (a division of the compiler's takes about eight, measured as time); errors below 1.5 ulp.
// Arguments outside FP32's comfortable range (zero, negative, not finite) take the routines.
__device__ __forceinline__ bool f32_range(double x) {
    const int e = (__double2hiint(x) >> 20) - 1023;
    return e > -110 && e < 110;
}
// root = sqrt(x), inv = 1 / sqrt(x): with e = 1 - x v^2, v <- v (1 + e / 2 + 3 e^2 / 8)
__device__ __forceinline__ void roots_newton(double x, double &root, double &inv) {
    if (!f32_range(x)) {
        root = sqrt(x);
        inv = 1.0 / root;
        return;
    }
    const double v = f32_widen(rsqrtf(df_from_f64(x).hi));
    const double g = x * v, e = fma(-g, v, 1.0), c = e * fma(0.375, e, 0.5);
    root = fma(g, c, g);
    inv = fma(v, c, v);
}
__device__ __forceinline__ double recip_newton(double x) {
    if (!f32_range(fabs(x))) return 1.0 / x;
    const double r = f32_widen(1.0f / df_from_f64(x).hi);
    const double e = fma(-x, r, 1.0);
    return fma(r, fma(e, e, e), r);
}

// Invariants of the deviator of the symmetric tensor t = [11, 22, 33, 12, 23, 13]: Q = J2 / 3, R = -J3 / 2.
struct Deviator {
    double I1, third, Q, R;
};
__device__ __forceinline__ Deviator deviator_invariants(const double *t) {
    Deviator d;
    d.I1 = t[0] + t[1] + t[2];
    d.third = d.I1 * (1.0 / 3.0);
    const double a = t[0] - d.third, b = t[1] - d.third, c = t[2] - d.third;
    const double sq = fma(a, a, fma(b, b, c * c)), sh = fma(t[3], t[3], fma(t[4], t[4], t[5] * t[5]));
    d.Q = fma(sq, 1.0 / 6.0, sh * (1.0 / 3.0));
    const double bc = fma(b, c, -(t[4] * t[4])), m1 = fma(t[3], c, -(t[4] * t[5])), m2 = fma(t[3], t[4], -(t[5] * b));
    d.R = -0.5 * fma(a, bc, fma(-t[3], m1, t[5] * m2));
    return d;
}

// Ordered principal values third + rq (cos(a) + sqrt(3) sin(a)), third + rq (cos(a) - sqrt(3) sin(a)),
// third - 2 rq cos(a) for the Lode angle a = acos(c) / 3 (c clamped to [-1, 1]).  With phi = acos(|c|) / 3 in
// [0, pi/6], y = cos(phi) is the root of 4 y^3 - 3 y = |c| in [0.86, 1], where its slope is at least 6, so an FP32
// estimate and two Newton steps give it: ten multiply-adds against the forty of an FP64 acos and series for sine
// and cosine.  The steps are on w = 1 - y, which keeps its own digits near an edge:
// w (9 - 12 w + 4 w^2) = 1 - |c|, sin(phi)^2 = w (2 - w).  c < 0 is a = pi/3 - phi: the values' signs and order
// reversed.  Returns 1 or 2 where e1, e2 or e2, e3 are a close pair (phi < 2^-7.5, their gap below a fiftieth of
// rq), else 0.
__device__ __forceinline__ int lode_values(double c, double rq, double third, double &e1, double &e2, double &e3) {
    const bool reversed = __double2hiint(c) < 0;
    c = fabs(c);
    const bool repeated = __double2hiint(c) >= 0x3FF00000;  // |c| >= 1, or NaN
    const float y0 = __cosf(acosf(repeated ? 1.0f : df_from_f64(c).hi) * (1.0f / 3.0f));
    const double slope = f32_widen(1.0f / fmaf(12.0f * y0, y0, -3.0f)), c1 = 1.0 - c;
    double w = f32_widen(1.0f - y0);
#pragma unroll
    for (int k = 0; k < 2; ++k) w = fma(fma(-fma(fma(4.0, w, -12.0), w, 9.0), w, c1), slope, w);
    if (repeated) w = 0.0;
    const double s2 = fma(-w, w, w + w);
    double z = 0.0;
    if (__double2hiint(s2) > 0) {  // sin(phi) by Newton steps on z^2 = s2
        const float r = sqrtf(df_from_f64(s2).hi);
        const double h = f32_widen(0.5f / r);
        z = f32_widen(r);
        z = fma(fma(-z, z, s2), h, z);
        z = fma(fma(-z, z, s2), h, z);
    }
    const double y = reversed ? w - 1.0 : 1.0 - w;
    const double a = rq * y, b = rq * (1.7320508075688772 * z);
    const double ta = third + a, hi = ta + b, lo = ta - b, single = fma(-2.0, a, third);
    e1 = reversed ? single : hi;
    e2 = reversed ? hi : lo;
    e3 = reversed ? lo : single;
    return __double2hiint(s2) >= 0x3F000000 ? 0 : 1 + reversed;
}

// t t (the squared tensor) as [11, 22, 33, 12, 23, 13].  Contractions are written out here and on the way to the
// stresses, so that every kernel that shares this code has the same bits.
__device__ __forceinline__ void square3(const double *t, double *sq) {
    sq[0] = fma(t[0], t[0], fma(t[3], t[3], t[5] * t[5]));
    sq[1] = fma(t[1], t[1], fma(t[3], t[3], t[4] * t[4]));
    sq[2] = fma(t[2], t[2], fma(t[4], t[4], t[5] * t[5]));
    sq[3] = fma(t[3], t[0] + t[1], t[4] * t[5]);
    sq[4] = fma(t[4], t[1] + t[2], t[3] * t[5]);
    sq[5] = fma(t[5], t[0] + t[2], t[3] * t[4]);
}

// The close pair (hi, lo) of t's principal values again, from its third one: an ulp of the invariants moves the pair
// by ulp / (gap / rq), and the tangent divides by the gap twice more.  With the pair at m +- b and the third at
// m - 3a, N = t - m has the values +-b and -3a, N (N + 3a) has b (b + 3a), b (b - 3a) and 0, and its squared
// Frobenius norm F = b^2 (18 a^2 + 2 b^2) gives b to a few ulps of the largest value.
__device__ __forceinline__ void refine_pair(const double *t, double third, double single, double &hi, double &lo) {
    const double a = 0.5 * (third - single), m = third + a, a3 = 3.0 * a;
    double n[6], sq[6];
#pragma unroll
    for (int i = 0; i < 6; ++i) n[i] = i < 3 ? t[i] - m : t[i];
    square3(n, sq);
    double f = 0.0;
#pragma unroll
    for (int i = 0; i < 6; ++i) {
        const double v = fma(a3, n[i], sq[i]);
        f = fma(i < 3 ? v : 2.0 * v, v, f);
    }
    if (!(f < 1e300)) return;  // strains from 1e75 up: the pair as it was
    const double b0 = 0.5 * (hi - lo);
    double b, inv;
    roots_newton(f * recip_newton(fma(2.0 * b0, b0, 18.0 * a * a)), b, inv);
    hi = m + b;
    lo = m - b;
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
// Where this bound does not settle a point, the Lode angle does better: with cos(3 b) = c = R / Q^(3/2) and
// a = b + pi/3, sqrt(3) sin(a) - s cos(a) replaces sqrt(3 + s^2).  FP32 gives c to about 4e-6 (1 + max|t| / sqrt(Q)),
// so b lies between acos(c +- twice that) / 3, and the form's slope, at most sqrt(3 + s^2), times that interval is
// added.  (With the first bound alone most listed points were found elastic in FP64: 196 us to decide them on a
// slope of 3.0 M points, now 74.)  ENERGY: Q^(3/2) is
// at least 1e-15, as the potential energy divides.
// A point with bound <= -1e-4 size is therefore elastic however the FP64 eigenvalues of the full
// path round (their error is at most ~1e-8 sqrt(Q), near repeated roots): the full path's branch
// test would say elastic too.  Such a point is finished from t and I1 in FP64 with the elastic
// branch's own arithmetic, so S and DS are bitwise those of the full path, and it costs about a
// dozen FP64 instructions instead of an eigen-decomposition.
template <bool ENERGY>
__device__ __forceinline__ bool screen_elastic(const double *E, const Mat3 &m) {
    float t[6];
#pragma unroll
    for (int i = 0; i < 6; ++i) t[i] = df_from_f64(E[i]).hi * (i < 3 ? 1.0f : 0.5f);
    const float G = df_from_f64(m.shear).hi, L = df_from_f64(m.lame).hi;
    const float s = df_from_f64(m.sin_phi).hi, c = df_from_f64(m.c_bar).hi;
    const float d01 = t[0] - t[1], d12 = t[1] - t[2], d20 = t[2] - t[0];
    const float J2 = (d01 * d01 + d12 * d12 + d20 * d20) * (1.0f / 6.0f) + t[3] * t[3] + t[4] * t[4] + t[5] * t[5];
    const float I1 = t[0] + t[1] + t[2];
    const float rq = sqrtf(J2 * (1.0f / 3.0f)), most = sqrtf(3.0f + s * s);
    const float dev = 2.0f * rq * most;
    const float rest = 2.0f * (2.0f / 3.0f * G + L) * s * I1 - c;
    const float tmax = fmaxf(fmaxf(fabsf(t[0]), fabsf(t[1])), fmaxf(fabsf(t[2]), fmaxf(fabsf(t[3]), fmaxf(fabsf(t[4]), fabsf(t[5])))));
    const float size = 2.0f * fabsf(G) * (dev + 3.0f * tmax) + 2.0f * fabsf(L * s * I1) + fabsf(c);
    if (2.0f * G * dev + rest <= -1e-4f * size) return true;
    if (!(rq > 1e-10f && rq < 1e10f)) return false;  // rq^3 is a normal float
    const float d0 = (d01 - d20) * (1.0f / 3.0f), d1 = (d12 - d01) * (1.0f / 3.0f), d2 = (d20 - d12) * (1.0f / 3.0f);
    const float R = -0.5f * (d0 * (d1 * d2 - t[4] * t[4]) - t[3] * (t[3] * d2 - t[4] * t[5]) + t[5] * (t[3] * t[4] - t[5] * d1));
    const float cs = R / (ENERGY ? fmaxf(1e-15f, rq * rq * rq) : rq * rq * rq), slack = 8e-6f * (1.0f + tmax / rq);
    const float b0 = acosf(fminf(1.0f, cs + slack)), b1 = acosf(fmaxf(-1.0f, cs - slack));
    float sn, cn;
    __sincosf(b0 * (1.0f / 3.0f) + 1.0471976f, &sn, &cn);
    const float dev2 = 2.0f * rq * (1.7320508f * sn - s * cn + most * (b1 - b0) * (1.0f / 3.0f));
    return 2.0f * G * dev2 + rest <= -1e-4f * size;
}

}  // namespace ssp
