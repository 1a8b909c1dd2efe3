// deo_nldfx.cu -- nonlinear_diffusion! on a uniform grid, Float64, in block fixed
// point (deo_bfp.cuh): orders N of p and M of q as k_nld (deo_kernels.cu), for the
// orders and approximation orders instantiated below.
//
// CTA = 128 threads over 512 points; the tiles of p and q with their halo are
// converted once to limbs on their own exponents; a thread evaluates pairs of
// points, every derivative of a pair from the same window, read with 16-byte
// loads.  A derivative's band is symmetric (even orders) or antisymmetric (odd) up
// to a few units, so the two taps of a distance are added or subtracted before the
// product.  Each derivative is rounded once; the products and sums follow the
// reference's order in FP64.  Points whose bound fails take the row tables, and so
// do the boundary rows, in a block of their own: in the tiles' blocks their chain
// of table reads came after the tile's (12 us instead of 6.5 for a short line).
//
// What bounds it (2^22 points, N = 2, M = 1, order 4): the FP64 pipe.  k_nld issues
// 34 FP64 instructions a point there and took 245 us; here it is 5 conversions and 3
// for the products and sums (54 us at the pipe's rate), beside 66 integer
// multiply-adds (15 us): 64.6 us.  Doubling the middle product's factor in FP64
// instead of its exponent: 72.3; so also tiles of 256 points 73.7, 1024 points on 256
// threads 74.2, 512 points on 256 threads 79.6.  The other orders at 2^22 points:
// N = 1, M = 0: 92 -> 37; N = 1, M = 1: 130 -> 43; N = 2, M = 0: 189 -> 57; at order 2
// 67 -> 35, 87 -> 42, 131 -> 57 and, N = 2, M = 1, 168 -> 64 us.
#include <cuda_runtime.h>
#include <limits.h>
#include <stdint.h>

#include "deo_bfp.cuh"
#include "deo_eval.cuh"

namespace deo {
namespace nld {

constexpr int T = 512, NT = 128;

// half-width of the order-k centred band of approximation order A
__host__ __device__ constexpr int half(int k, int A) { return (k + A - 1 + (k + A) % 2) / 2; }

// The order-K derivative, times 2^up, at the centre x of its window.
template <int K, int A>
__device__ __forceinline__ double deriv(const NldBand& b, const Limbs* x, int E, int up = 0) {
    constexpr int H = half(K, A);
    constexpr bool odd = K % 2 == 1;
    BfpAcc s{0, 0, 0};
    if constexpr (odd) s.cr = (long long)b.wd[0] * x[0].h;
    else bfp_mad(s, b.wh[0], b.wl[0], x[0].h, x[0].l);
#pragma unroll
    for (int o = 1; o <= H; ++o) {
        const Limbs p = x[o], m = x[-o];
        bfp_mad(s, b.wh[o], b.wl[o], odd ? p.h - m.h : p.h + m.h, odd ? p.l - m.l : p.l + m.l);
        s.cr += (long long)b.wd[o] * m.h;
    }
    return bfp_double(bfp_total(s), (b.k + E + up) * (1 << 20));
}

template <int N, int M, int A>
__global__ void __launch_bounds__(NT, 8) k_nld_fx(const __grid_constant__ NldBfp B, const PlanDev* __restrict__ P, int len,
                                                  const double* __restrict__ p, const double* __restrict__ q,
                                                  double* __restrict__ du) {
    constexpr int HQ = half(M + N, A), HP = half(N, A), H = HQ > HP ? HQ : HP;
    constexpr int PAD = (H + 1) / 2 * 2, W = T + 2 * PAD, NLD = (W + NT - 1) / NT;
    __shared__ __align__(16) Limbs s[2][W];
    __shared__ unsigned s_max[2];
    const int tid = threadIdx.x;
    auto D = [&](int k, const double* x, int i) { return eval_row_padded<double>(P->t[k - 1].tab[0], x, 1, i + 1); };
    auto ref = [&](int i) {  // k_nld's point
        double acc = (M > 0 ? D(M, q, i) : q[i + 1]) * D(N, p, i);
        if (N == 2) acc = acc + (2.0 * D(M + 1, q, i)) * D(1, p, i);
        du[i] = acc + D(M + N, q, i) * p[i + 1];
    };
    if (blockIdx.x == 0) {  // the boundary rows
        for (int j = tid; j < B.lo + len - B.hi; j += NT) ref(j < B.lo ? j : B.hi + j - B.lo);
        return;
    }
    const int i0 = (blockIdx.x - 1) * T;  // output i has its centre at padded index i + 1
    if (tid < 2) s_max[tid] = 0;
    double raw[2][NLD];
#pragma unroll
    for (int j = 0; j < NLD; ++j) {
        const int64_t at = min(max((int64_t)i0 + 1 - PAD + tid + j * NT, (int64_t)0), (int64_t)len + 1);
        raw[0][j] = __ldg(q + at);
        raw[1][j] = __ldg(p + at);
    }
    __syncthreads();
#pragma unroll
    for (int a = 0; a < 2; ++a) {
        unsigned mx = 0;
#pragma unroll
        for (int j = 0; j < NLD; ++j) mx = max(mx, bfp_key(raw[a][j]));
        mx = __reduce_max_sync(0xffffffffu, mx);
        if (tid % 32 == 0) atomicMax(&s_max[a], mx);
    }
    __syncthreads();
    int E[2], lim[2];
#pragma unroll
    for (int a = 0; a < 2; ++a) {
        E[a] = max((int)(s_max[a] >> 20), 64);
        bool special = E[a] >= 2047;
#pragma unroll
        for (int k = 0; k < (a == 0 ? N + 1 : N); ++k)
            if (a == 1 || M + k > 0) {
                const int e = (a == 0 ? B.q[k].k : B.p[k].k) + E[a];
                special |= !bfp_range_ok(e) || !bfp_range_ok(e + 1);
            }
        lim[a] = special ? INT_MAX : (s_max[a] == 0 ? 0 : (a == 0 ? B.tq : B.tp));
#pragma unroll
        for (int j = 0; j < NLD; ++j)
            if (j + 1 < NLD || tid + j * NT < W) s[a][tid + j * NT] = bfp_convert(raw[a][j], bfp_key(raw[a][j]), E[a]);
    }
    __syncthreads();
    for (int b = 0; b < T; b += 2 * NT) {
        const int at = b + 2 * tid;
        Limbs wq[2 + 2 * PAD], wp[2 + 2 * PAD];  // the pair's window
#pragma unroll
        for (int m = 0; m < 1 + PAD; ++m) {
            const int4 a = *reinterpret_cast<const int4*>(&s[0][at + 2 * m]), c = *reinterpret_cast<const int4*>(&s[1][at + 2 * m]);
            wq[2 * m] = Limbs{a.x, a.y};
            wq[2 * m + 1] = Limbs{a.z, a.w};
            wp[2 * m] = Limbs{c.x, c.y};
            wp[2 * m + 1] = Limbs{c.z, c.w};
        }
#pragma unroll
        for (int v = 0; v < 2; ++v) {
            const int i = i0 + at + v;
            const Limbs *xq = wq + PAD + v, *xp = wp + PAD + v;
            if (i < B.lo || i >= B.hi) continue;
            if (max(abs(xq[-1].h), abs(xq[1].h)) >= lim[0] && max(abs(xp[-1].h), abs(xp[1].h)) >= lim[1]) {
                double acc;
                // the reference's order (k_nld), each derivative from its band
                const double dn = deriv<N, A>(B.p[N - 1], xp, E[1]);
                if constexpr (M > 0) acc = deriv<M, A>(B.q[0], xq, E[0]) * dn;
                else acc = __ldg(q + i + 1) * dn;
                if constexpr (N == 2)  // binomial(2, 1) = 2 by the exponent
                    acc = acc + deriv<M + 1, A>(B.q[1], xq, E[0], 1) * deriv<1, A>(B.p[0], xp, E[1]);
                acc = acc + deriv<M + N, A>(B.q[N], xq, E[0]) * __ldg(p + i + 1);
                du[i] = acc;
            } else {
                ref(i);
            }
        }
    }
}

}  // namespace nld
}  // namespace deo

using namespace deo;

extern "C" int deo_k_nld_fx(const NldBfp* B, const PlanDev* d_plan, int len, int n, int m, int a, const void* p,
                            const void* q, void* du, void* stream) {
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    auto go = [&](auto kernel) {
        kernel<<<(unsigned)(1 + (len + nld::T - 1) / nld::T), nld::NT, 0, st>>>(*B, d_plan, len, (const double*)p,
                                                                            (const double*)q, (double*)du);
        return (int)cudaGetLastError();
    };
    if (a == 2) {
        if (n == 1 && m == 0) return go(nld::k_nld_fx<1, 0, 2>);
        if (n == 1 && m == 1) return go(nld::k_nld_fx<1, 1, 2>);
        if (n == 2 && m == 0) return go(nld::k_nld_fx<2, 0, 2>);
        if (n == 2 && m == 1) return go(nld::k_nld_fx<2, 1, 2>);
    } else if (a == 4) {
        if (n == 1 && m == 0) return go(nld::k_nld_fx<1, 0, 4>);
        if (n == 1 && m == 1) return go(nld::k_nld_fx<1, 1, 4>);
        if (n == 2 && m == 0) return go(nld::k_nld_fx<2, 0, 4>);
        if (n == 2 && m == 1) return go(nld::k_nld_fx<2, 1, 4>);
    }
    return (int)cudaErrorNotSupported;
}
