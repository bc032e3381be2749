// 58-bit fixed-point arithmetic on the integer pipe (not part of the public C ABI).
//
// GB300 issues FP64 at 1.6 multiply-adds per clock and SM.  A sum of products of about 58 significant bits
// takes three 32 x 32 -> 64-bit integer multiply-adds per term here, 22 to 29 per clock and SM (measured): five
// times the rate, beside an idle FP64 pipe, and more exact: FP64 rounds every step to 53 bits.
//
// A block of values that belong together (an element's tangents, its gradients) shares one exponent, that
// of its largest; a value is a 64-bit integer in units of the block's last place.  Operands of a product
// are split into two limbs, x = h 2^29 + l with a signed lower limb; a sum of products keeps the h h and the
// h l + l h parts in two 64-bit accumulators and drops l l (a quarter of a unit of the result per term, of either
// sign, so that long sums have no bias).  n products of a-bit and b-bit factors in units of 2^(2 LIMB) stay below 2^63
// for n < 2^(63 + 2 LIMB - a - b): 31 terms of two 58-bit factors (limbs of 29), 127 of two of 56 bits, 63 of 57 and 56
// (limbs of 28).  Every stage is brought back to 58 bits by the block's largest
// value (fx_warp_bits, fx_room): without that the losses of the stages add up (three of them left 40 bits of
// the P2 moment form).
//
// Errors are relative to the largest value of a block.  What FP64 keeps apart, displacement components,
// directions of thin elements, stress components, is therefore a block each in the strains and forces, whose components
// are as exact as FP64's one by one.  The tangents' blocks are an element's gradients (P4: a node's) and its
// tangents: an element matrix is as exact as FP64's relative to its largest entry, not entry by entry (a
// thousand times thinner than wide, gradients along the wide directions have ten of their 57 bits less).
//
// Conversions from and to FP64 are integer operations, too: the hardware's 64-bit conversions run at 1.9 per
// clock and SM at best, and a warp waited some 50 to 60 clocks of the FP64 pipe for each.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace ssp {

constexpr int kFxLimb = 29;
constexpr int kFxDrop = 2 * kFxLimb;  // a product sum's unit is 2^58 times the product of its factors' units

// biased exponent of x (2047: infinity or nan; 0: subnormal or zero, whose unit is exponent 1's)
__device__ __forceinline__ int fx_exponent(double x) { return (__double2hiint(x) >> 20) & 0x7FF; }

// x in units of 2^(e_block - 1022 - bits), truncated: |x| < 2^(e_block - 1022) maps below 2^bits (bits <= 62; at
// 60 a value is exact down to 2^-7 of the largest).  x is finite with an exponent of at most e_block.
__device__ __forceinline__ long long fx_from_f64(double x, int e_block, int bits) {
    const int hi = __double2hiint(x), e = (hi >> 20) & 0x7FF;
    const int d = min(max(e_block, 1) - max(e, 1), 63);
    const unsigned long long m =
        (static_cast<unsigned long long>((hi & 0xFFFFF) | (e ? 0x100000 : 0)) << 32) | static_cast<unsigned>(__double2loint(x));
    const long long v = static_cast<long long>((m << (bits - 53)) >> d), sign = hi >> 31;
    return (v ^ sign) - sign;
}
// the exponent of fx_from_f64's unit
__device__ __forceinline__ int fx_unit(int e_block, int bits) { return max(e_block, 1) - 1022 - bits; }

// x 2^unit, |x| < 2^63, rounded to nearest (ties away from zero).  unit is the same for a block: only where a
// result could leave the normal range the general form is taken (not for a block of zeros, whose unit is as low: with
// it the P2 strain of a slope that moves in a plane took 135 us instead of 123).  A negative x counts as its one's
// complement, one unit smaller in magnitude.
__device__ __forceinline__ double fx_to_f64(long long x, int unit) {
    if (unit <= -1022 || unit >= 950) return x == 0 ? 0.0 : scalbn(__ll2double_rn(x), unit);
    const int sign = static_cast<int>(x >> 32) >> 31;
    const unsigned xh = static_cast<unsigned>(static_cast<unsigned long long>(x) >> 32) ^ sign,
                   xl = static_cast<unsigned>(x) ^ sign;
    const bool small = xh == 0u;
    const unsigned hi = small ? xl : xh, lo = small ? 0u : xl;
    const int s = __clz(static_cast<int>(hi));
    const unsigned h = __funnelshift_l(lo, hi, s), l = lo << s;  // leading one at bit 63 of (h, l)
    // 53 bits, rounded; the leading one is added into the exponent field, and so is a carry of the rounding
    const unsigned long long m = (static_cast<unsigned long long>(h >> 11) << 32 | __funnelshift_r(l, h, 11)) + ((l >> 10) & 1u);
    const int e = unit + (small ? 1022 + 31 : 1022 + 63) - s;
    const unsigned oh = (static_cast<unsigned>(m >> 32) + static_cast<unsigned>(e) * (1u << 20)) |
                        (static_cast<unsigned>(sign) & 0x80000000u);
    return hi == 0u ? 0.0 : __hiloint2double(static_cast<int>(oh), static_cast<int>(m));
}

// x = h 2^LIMB + l, -2^(LIMB-1) <= l < 2^(LIMB-1)
template <int LIMB = kFxLimb>
__device__ __forceinline__ int2 fx_split(long long x) {
    const int h = static_cast<int>((x + (1ll << (LIMB - 1))) >> LIMB);
    return make_int2(h, static_cast<int>(x) - static_cast<int>(static_cast<unsigned>(h) << LIMB));
}

// Bits of the largest magnitude of a block: the magnitudes' bits (one's complement of negative values) are
// OR-ed by each lane (fx_mag), then across the warp.
__device__ __forceinline__ unsigned long long fx_mag(long long x) { return static_cast<unsigned long long>(x ^ (x >> 63)); }
__device__ __forceinline__ int fx_warp_bits(unsigned long long mags) {
    const unsigned hi = __reduce_or_sync(0xffffffffu, static_cast<unsigned>(mags >> 32));
    if (hi) return 64 - __clz(hi);
    return 32 - __clz(__reduce_or_sync(0xffffffffu, static_cast<unsigned>(mags)));
}
// x 2^s for 0 <= s < 32: two funnel shifts (a 64-bit shift by a variable also looks at larger s)
__device__ __forceinline__ long long fx_scale(long long x, int s) {
    const unsigned lo = static_cast<unsigned>(x), hi = static_cast<unsigned>(static_cast<unsigned long long>(x) >> 32);
    return static_cast<long long>(static_cast<unsigned long long>(__funnelshift_l(lo, hi, s)) << 32 | (lo << s));
}
// the shift that brings a block of `bits` bits to 62, at most 31
__device__ __forceinline__ int fx_room(int bits) { return min(31, 62 - bits); }
// x 2^-s rounded: truncated operands have a bias that every product of a sum repeats (the full P2 contraction
// with truncated 55-bit factors was 16 times as far from the exact sums as FP64; rounded to 56 it is nearer)
template <int S>
__device__ __forceinline__ long long fx_round(long long x) { return (x + (1ll << (S - 1))) >> S; }
// fx_split<LIMB>(fx_round<S>(x)), its upper limb from x's upper word alone
template <int LIMB, int S>
__device__ __forceinline__ int2 fx_round_split(long long x) {
    static_assert(LIMB + S > 32, "the rounding of the upper limb is in the upper word");
    const long long w = x + (1ll << (S - 1));
    const int wh = static_cast<int>(w >> 32), h = (wh + (1 << (LIMB + S - 33))) >> (LIMB + S - 32);
    return make_int2(h, static_cast<int>(__funnelshift_r(static_cast<unsigned>(w), static_cast<unsigned>(wh), S) -
                                         (static_cast<unsigned>(h) << LIMB)));
}
// x of up to 62 bits as limbs of x 2^(BITS - 62), rounded, and the exponent of that unit after fx_scale by s
template <int BITS>
__device__ __forceinline__ int2 fx_split_top(long long x) {
    if constexpr (kFxLimb + 62 - BITS > 32) return fx_round_split<kFxLimb, 62 - BITS>(x);
    else return fx_split(fx_round<62 - BITS>(x));
}
template <int BITS>
__device__ __forceinline__ int fx_top_unit(int s) { return (62 - BITS) - s; }

// 32 x 32 -> 64-bit product and multiply-add, one IMAD.WIDE each (written out: from the C++ expressions the
// compiler made about half as many instructions again)
__device__ __forceinline__ long long fx_mul(int a, int b) {
    long long r;
    asm("mul.wide.s32 %0, %1, %2;" : "=l"(r) : "r"(a), "r"(b));
    return r;
}
__device__ __forceinline__ long long fx_mad(int a, int b, long long c) {
    long long r;
    asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(r) : "r"(a), "r"(b), "l"(c));
    return r;
}

// a sum of products
struct FxSum {
    long long hh, mid;
    __device__ __forceinline__ FxSum() : hh(0), mid(0) {}
    __device__ __forceinline__ FxSum(int2 a, int2 b) : hh(fx_mul(a.x, b.x)), mid(fx_mad(a.y, b.x, fx_mul(a.x, b.y))) {}
    __device__ __forceinline__ void add_prod(int2 a, int2 b) {
        hh = fx_mad(a.x, b.x, hh);
        mid = fx_mad(a.y, b.x, fx_mad(a.x, b.y, mid));
    }
    template <int LIMB = kFxLimb>
    __device__ __forceinline__ long long value() const { return hh + fx_round<LIMB>(mid); }
    // the same with UP bits more, where hh has them to spare
    template <int LIMB, int UP>
    __device__ __forceinline__ long long value_up() const { return (hh << UP) + fx_round<LIMB - UP>(mid); }
};

}  // namespace ssp
