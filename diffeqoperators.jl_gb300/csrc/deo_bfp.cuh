// deo_bfp.cuh -- block fixed point: Float64 stencil sums on the integer pipes.
//
// The FP64 pipe of this part issues 2 instructions per clock per SM; 32 x 32 ->
// 64-bit integer multiply-adds issue 60.  A block of values that share one
// exponent E (the largest of the block) is held as integers
//     v = x * 2^(E - 1075 - BFP_G),  x = h * 2^30 + l,  |l| <= 2^29, |h| <= 2^29,
// so a value at the block's largest exponent keeps BFP_G bits below its 53-bit
// mantissa and smaller ones are truncated at that unit.  A weight is held as
// W = round(w * 2^s) = Wh * 2^30 + Wl the same way, s such that the sum of |W|
// over a row stays below 2^60.  The row's sum of W x then takes four
// multiply-adds per tap into three 64-bit columns (hh, cross, ll), none of
// which can overflow, and the total is rounded once by one int64 -> double
// conversion: the only FP64 instruction of a point.
//
// Error, in units of x times the sum of |W|: below 1 from the truncated values,
// below 1/2 from the total's unit.  It is at most 2 ulp of the row's sum |w u| when
// that sum is at least 2^52 units; the kernels test a lower bound of it (one
// tap, or a sum of taps of one weight) and evaluate the points that fail in the
// reference's order, unless the whole block is zero.  (That no value of the
// block lost a bit is not enough: a point whose only nonzero tap has a small
// weight falls below the total's own unit.)
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace deo {

constexpr int BFP_G = 6;

struct Limbs {
    int h, l;
};

// hi word without sign, its lowest bit set when the low word is not zero: orders
// values by exponent, and is zero for zeros alone
__device__ __forceinline__ unsigned bfp_key(double v) {
    const unsigned hi = (unsigned)__double2hiint(v), lo = (unsigned)__double2loint(v);
    return (hi & 0x7fffffffu) | min(lo, 1u);
}

// v in units of 2^(E - 1075 - BFP_G), truncated toward zero, as balanced limbs;
// key: bfp_key(v).  E >= 64 and E >= v's exponent field (a larger one gives
// garbage, no fault); a subnormal v then shifts out entirely.
// G: bits kept below the mantissa of a value at the block's exponent.  BFP_G
// where the kernel adds up to three values, or subtracts two, before the
// product; 7 (|h| <= 2^30) where every value is multiplied by itself.
template <int G = BFP_G>
__device__ __forceinline__ Limbs bfp_convert(double v, unsigned key, int E) {
    const unsigned hi = (unsigned)__double2hiint(v), lo = (unsigned)__double2loint(v);
    const unsigned d = (unsigned)((E << 20) + 0xfffff - (int)key) >> 20;
    unsigned long long m = ((unsigned long long)((hi & 0xfffffu) | 0x100000u) << 32) | lo;
    m <<= G;
    asm("shr.u64 %0, %0, %1;" : "+l"(m) : "r"(d));  // (PTX clamps the amount)
    m += 1ull << 29;
    const int sg = ((int)hi >> 31) | 1;
    Limbs r;
    r.h = (int)(unsigned)(m >> 30) * sg;
    r.l = ((int)((unsigned)m & 0x3fffffffu) - (1 << 29)) * sg;
    return r;
}

// The same rounded to nearest, for points on an exponent E of their own (the largest of the
// point's taps): where the values are small against the block's.
template <int G>
__device__ __forceinline__ Limbs bfp_nearest(double v, int E) {
    const unsigned hi = (unsigned)__double2hiint(v), lo = (unsigned)__double2loint(v);
    const unsigned d = (unsigned)E - ((hi >> 20) & 0x7ffu);
    unsigned long long m = ((unsigned long long)((hi & 0xfffffu) | 0x100000u) << 32) | lo;
    m <<= G + 1;
    asm("shr.u64 %0, %0, %1;" : "+l"(m) : "r"(d));
    m += (1ull << 30) + 1;  // half a unit, and the limbs' balance
    const int sg = ((int)hi >> 31) | 1;
    Limbs r;
    r.h = (int)(unsigned)(m >> 31) * sg;
    r.l = ((int)(((unsigned)m & 0x7fffffffu) >> 1) - (1 << 29)) * sg;
    return r;
}

// Columns of a row's sum: hh * 2^60 + cr * 2^30 + ll.
struct BfpAcc {
    long long hh, cr, ll;
};
__device__ __forceinline__ void bfp_mad(BfpAcc& a, int wh, int wl, int h, int l) {
    a.hh += (long long)wh * h;
    a.cr += (long long)wh * l;
    a.cr += (long long)wl * h;
    a.ll += (long long)wl * l;
}
// The sum in units of 2^(51 + G) (below 2^62 in magnitude); ll enters by its high
// word.
template <int G = BFP_G>
__device__ __forceinline__ long long bfp_total(const BfpAcc& a) {
    const long long cr = a.cr + (long long)(int)(a.ll >> 32) * 4;
    return (a.hh << (9 - G)) + (cr >> (21 + G));
}
// Of values from bfp_nearest, in units of 2^(50 + G), rounded to nearest: within 3/4 of a
// unit of x times the sum of |W|, so a row's sum |w u| of 2^51 units is enough for 2 ulp of
// it.  It is that large where the largest tap's |W| is 2^-(G + 1) of the sum, or where the
// total reaches bfp_own_limit(G) << 32.
template <int G>
__device__ __forceinline__ long long bfp_total_own(const BfpAcc& a) {
    const long long cr = a.cr + (long long)(int)(a.ll >> 32) * 4;
    return (a.hh << (10 - G)) + ((cr + (1LL << (19 + G))) >> (20 + G));
}
__host__ __device__ constexpr int bfp_own_limit(int G) { return 1 << (51 + 59 - (50 + G) - 32); }

// Where the neighbours at one distance are added before the product: the values as signed
// 64-bit integers with 8 bits kept, |x| <= 2^61, rounded down; the limbs of a sum of three are
// its words, |h| < 2^31, |l| <= 2^31.  Columns: hh * 2^62 + hl * 2^30 + lh * 2^32 + ll.
struct BfpOwn {
    long long hh, hl, lh, ll;
};
// v's words, on exponent E
__device__ __forceinline__ long long bfp_shift(Limbs v, int E) {
    const unsigned hi = (unsigned)v.h, d = ((unsigned)(E << 20) + 0xfffffu - (hi & 0x7fffffffu)) >> 20;
    unsigned long long m = ((unsigned long long)((hi & 0xfffffu) | 0x100000u) << 32) | (unsigned)v.l;
    m <<= 8;
    asm("shr.u64 %0, %0, %1;" : "+l"(m) : "r"(d));
    return (long long)m ^ (long long)(v.h >> 31);  // -x - 1 for -x: within a unit like the bits shifted out
}
__device__ __forceinline__ void bfp_mad(BfpOwn& a, int wh, int wl, long long x) {
    const int l = (int)x, h = (int)(x >> 32) + (l < 0);
    a.hh += (long long)wh * h;
    a.hl += (long long)wh * l;
    a.lh += (long long)wl * h;
    a.ll += (long long)wl * l;
}
// In units of 2^58, rounded to nearest (below 2^62 in magnitude): within 3/2 units of x times
// the sum of |W|, so 2^52 units of the row's sum |w u| are enough; reached where the largest
// tap's |W| is 1 / 256 of the sum, or where the total reaches BFP_OWN_LIMIT << 32.
__device__ __forceinline__ long long bfp_total(const BfpOwn& a) {
    return (a.hh << 4) + ((a.lh + (a.hl >> 2) + (a.ll >> 32) + (1LL << 25)) >> 26);
}
constexpr int BFP_OWN_LIMIT = 1 << (52 + 59 - 58 - 32);
// t * 2^k (scale = 2^k; no nonzero t leaves the normal range, see bfp_range_ok).
__device__ __forceinline__ double bfp_double(long long t, double scale) { return __ll2double_rn(t) * scale; }
// The same by the exponent field, without FP64: k20 = k * 2^20.
__device__ __forceinline__ double bfp_double(long long t, int k20) {
    const double r = __ll2double_rn(t);
    int hi = __double2hiint(r);
    asm("{\n\t.reg .pred p;\n\tsetp.ne.s32 p, %0, 0;\n\t@p add.s32 %0, %0, %1;\n\t}" : "+r"(hi) : "r"(k20));
    return __hiloint2double(hi, __double2loint(r));
}
// 2^k, k in the normal range
__device__ __forceinline__ double bfp_pow2(int k) { return __hiloint2double((1023 + k) << 20, 0); }
__host__ __device__ __forceinline__ bool bfp_range_ok(int k) { return 1023 + k >= 1 && 1023 + 62 + k <= 2046; }

}  // namespace deo
