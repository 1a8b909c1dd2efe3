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
// below 2^-5 from the rest.  It is at most 2 ulp of the row's sum |w u| when
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
