// deo_rowsfx.cu -- Float64 2-D plans in block fixed point (deo_bfp.cuh): any
// number of terms along the two axes, uniform or not, and one upwind term along
// axis 1 whose coefficient is a field.
//
// The host folds every row (boundary rows, ghosts through the boundary
// condition's map, the terms of one axis added) into a window of K points of its
// line with integer weights on a scale of its own (BfpRows), so the device has one
// kind of row; a ghost that adds a constant sends its few rows to the list below.  CTA = 32 x 8 threads over a 32 x 32 tile: the tile and
// its halo are loaded once, converted to limbs on the tile's exponent and read
// from shared memory; a thread owns one column of 4 rows, keeps its axis-1
// weights in registers and reads axis 2's, the same for its warp, through L1.
// The last tile along an axis starts early enough to be full (its windows then
// fit the halo) and leaves the points of the tile before it alone.  The sum along
// each axis and the field term's are rounded once each, as the reference rounds
// its terms, then added: 5 FP64 instructions a point.
//
// Points whose bound fails go through a list to the generic evaluator at the end
// of the tile.  A tile whose values are mostly small against its largest keeps them as they
// are and sums every row on the largest exponent of its own taps.  2048 x 2048, a Gaussian of
// width 0.02 of the box, us: before this kernel / without that / now: the graded plan below
// 361 / 406 / 154, a Laplacian of order 4 86 / 138 / 78; 4096 x 4096, order 2, 249 / 304 / 210.
//
// What bounds it (2048 x 2048, graded: four centred terms of order 6 and an upwind
// one with a field; 36 FP64 instructions a point in the reference's order, 359 us):
// 108 us; 385 instructions a point -- 72 multiply-adds, 18 shared loads, 9 loads of
// weights -- at 41 % issue, and 5.4 FP64 instructions (36 us at 2 per clock per SM).
// 3 or 5 CTAs an SM (80 or 48 registers) measured 125 / 108 us, 8 rows a thread 118;
// constants of the ghosts added to every point 202 (predicated FP64 adds
// take the pipe's full time).
#include <cuda_runtime.h>
#include <limits.h>
#include <stdint.h>

#include <type_traits>

#include "deo_bfp.cuh"
#include "deo_eval.cuh"

namespace deo {
namespace rows {

constexpr int T = 32, RY = 4, G = 7;

// One axis's row: the sum in int64 units, and whether its bound holds: the larger
// of two taps reaches the row's threshold, or the sum itself shows that
// the row's sum |W x| is large enough.
template <int K, int KP>
__device__ __forceinline__ long long dot(const Limbs* x, int step, const Limbs (&w)[KP], int limit, int limit_t,
                                         bool& ok) {
    constexpr int A = (K - 2) / 2, Z = K - 1 - A;  // the two taps the threshold is for
    BfpAcc s{0, 0, 0};
    int far = 0;
#pragma unroll
    for (int k = 0; k < K; ++k) {
        const Limbs v = x[k * step];
        bfp_mad(s, w[k].h, w[k].l, v.h, v.l);
        if (k == A || k == Z) far = max(far, abs(v.h));
    }
    const long long t = bfp_total<G>(s);
    ok = ok && (far >= limit || abs((int)(t >> 32)) >= limit_t);
    return t;
}

// The same from the values themselves (their words), on the exponent of the row's own taps;
// the result's exponent field, in 2^20, in k20 (0 for zeros, whose sum is 0).
template <int K, int KP>
__device__ __forceinline__ long long dot_own(const Limbs* x, int step, const Limbs (&w)[KP], const BfpRowMeta& m, int& k20,
                                             bool& ok) {
    constexpr int A = (K - 2) / 2, Z = K - 1 - A;
    unsigned mx = 0, lo = 0;
#pragma unroll
    for (int k = 0; k < K; ++k) {
        mx = max(mx, (unsigned)x[k * step].h & 0x7fffffffu);
        lo |= (unsigned)x[k * step].l;
    }
    const int e = (int)(mx >> 20), E = max(e, 64), kexp = m.k - 1 + E;
    BfpAcc s{0, 0, 0};
    int far = 0;
#pragma unroll
    for (int k = 0; k < K; ++k) {
        const Limbs u = x[k * step], v = bfp_nearest<G>(__hiloint2double(u.h, u.l), E);
        bfp_mad(s, w[k].h, w[k].l, v.h, v.l);
        if (k == A || k == Z) far = max(far, abs(v.h));
    }
    const long long t = bfp_total_own<G>(s);
    const bool zero = (mx | lo) == 0;
    ok = ok && !m.always &&
         (zero || (e >= 64 && e < 2047 && bfp_range_ok(kexp) && (far >= m.t || abs((int)(t >> 32)) >= bfp_own_limit(G))));
    k20 = kexp * (1 << 20);
    return zero ? 0 : t;
}

template <int KP>
__device__ __forceinline__ void weights(const BfpRows& R, int row, Limbs (&w)[KP]) {
    const int4* p = reinterpret_cast<const int4*>(R.w) + (int64_t)row * (KP / 2);
#pragma unroll
    for (int k = 0; k < KP / 2; ++k) {
        const int4 v = __ldg(p + k);
        w[2 * k] = Limbs{v.x, v.y};
        w[2 * k + 1] = Limbs{v.z, v.w};
    }
}

__device__ __forceinline__ BfpRowMeta row_meta(const BfpRows& R, int row) {
    const int4 a = __ldg(reinterpret_cast<const int4*>(R.meta) + row);
    return BfpRowMeta{a.x, a.y, a.z, a.w};
}

__device__ __noinline__ double ref_point(const PlanDev& P, const double* __restrict__ u, int64_t idx) {
    return eval_point<double, false>(P, u, idx);
}

// NX, NY: the plan has terms along axis 1, 2; KF: window of the field term (0: none).
template <int K, int KF, bool NX, bool NY, bool OW>
__global__ void __launch_bounds__(256, 4) k_rows_fx(const __grid_constant__ BfpPlan2 B,
                                                    const PlanDev* __restrict__ P, const double* __restrict__ u,
                                                    double* __restrict__ du) {
    constexpr int H = KF && (K - 1) / 2 < KF - 1 ? KF - 1 : (K - 1) / 2;
    static_assert(NX || KF == 0, "a field term comes with plain terms along its axis");
    constexpr int HX = NX ? H : 0, HY = NY ? (K - 1) / 2 : 0;
    constexpr int BX = T + 2 * HX, BY = T + 2 * HY, N = BX * BY, NLD = (N + 255) / 256, KP = K + 1;
    __shared__ Limbs s[N];
    __shared__ unsigned s_max;
    __shared__ int s_n;
    __shared__ unsigned short s_list[T * T];
    const int tx = threadIdx.x, ty = threadIdx.y, tid = ty * 32 + tx;
    const int n0 = B.n[0], n1 = B.n[1];
    const int x0 = min((int)blockIdx.x * T, n0 - T), y0 = min((int)blockIdx.y * T, n1 - T);
    if (tid == 0) {
        s_max = 0;
        s_n = 0;
    }
    double raw[NLD];
    auto load = [&] {
#pragma unroll
        for (int j = 0; j < NLD; ++j) {
            const int q = min(tid + j * 256, N - 1), r = q / BX;
            const int x = min(max(x0 + (q - r * BX) - HX, 0), n0 - 1), y = min(max(y0 + r - HY, 0), n1 - 1);
            raw[j] = __ldg(u + (int64_t)y * n0 + x);
        }
    };
    load();
    const int x = x0 + tx;
    const int64_t first = (int64_t)(y0 + ty * RY) * n0 + x;
    double c[RY];
    if constexpr (KF > 0) {
#pragma unroll
        for (int r = 0; r < RY; ++r) c[r] = __ldg(B.field + first + (int64_t)r * n0);
    }
    Limbs wx[KP];
    BfpRowMeta mx{};
    if constexpr (NX) {
        weights<KP>(B.ax[0], x, wx);
        mx = row_meta(B.ax[0], x);
    }
    __syncthreads();
    unsigned mxk = 0;
#pragma unroll
    for (int j = 0; j < NLD; ++j) mxk = max(mxk, bfp_key(raw[j]));
    mxk = __reduce_max_sync(0xffffffffu, mxk);
    if (tx == 0) atomicMax(&s_max, mxk);
    __syncthreads();
    const int E = max((int)(s_max >> 20), 64);
    const bool zero = s_max == 0, special = E >= 2047;
#pragma unroll
    for (int j = 0; j < NLD; ++j)
        if (j + 1 < NLD || tid + j * 256 < N) s[tid + j * 256] = bfp_convert<G>(raw[j], bfp_key(raw[j]), E);
    // a tile of values that are small against its largest (a fifth of a sample of them, one a thread, by more
    // than 6 binades): kept as they are, every row on the exponent of its own taps
    const bool own = __syncthreads_count(E > 64 && bfp_key(raw[NLD / 2]) < (unsigned)((E - 6) << 20)) > 256 / 5;
    if (own) {
        load();  // (the registers are others' by now)
#pragma unroll
        for (int j = 0; j < NLD; ++j)
            if (j + 1 < NLD || tid + j * 256 < N) s[tid + j * 256] = Limbs{__double2hiint(raw[j]), __double2loint(raw[j])};
        __syncthreads();
    }
    // a row's threshold: none when the whole tile is zero, out of reach for rows with a ghost's constant and
    // outside the exponent range; the sum's own (1.05 * 2^52 units of x times 2^60 of W)
    const int limit_t = special ? INT_MAX : (int)(1.05 * (1 << (52 + 60 - 51 - G - 32))) + 1;
    auto limit = [&](const BfpRowMeta& m) {
        return m.always || special || !bfp_range_ok(m.k + E) ? INT_MAX : (zero ? 0 : m.t);
    };
    const bool mine = x >= (int)blockIdx.x * T;
    const int lx = NX ? limit(mx) : 0;
    // a row's sum, rounded; its weights and window start at w, row
    auto sum = [&](auto own_exp, auto kk, const Limbs* row, int step, const auto& w, const BfpRowMeta& m, int l, bool& ok) {
        constexpr int KW = decltype(kk)::value;
        if constexpr (decltype(own_exp)::value) {
            int k20;
            const long long t = dot_own<KW>(row, step, w, m, k20, ok);
            return bfp_double(t, k20);
        } else {
            return bfp_double(dot<KW>(row, step, w, l, l == INT_MAX ? INT_MAX : limit_t, ok), (m.k + E) * (1 << 20));
        }
    };
    auto points = [&](auto own_exp) {
        using W = std::integral_constant<int, K>;
        using WF = std::integral_constant<int, KF>;
        constexpr int U = decltype(own_exp)::value ? 1 : RY;  // (more spill on own exponents)
#pragma unroll U
        for (int r = 0; r < RY; ++r) {
            const int y = y0 + ty * RY + r;
            const Limbs* row = s + (ty * RY + r + HY) * BX;
            bool ok = true;
            double v = 0.0;
            if constexpr (NX) v = sum(own_exp, W{}, row + (mx.q - x0 + HX), 1, wx, mx, lx, ok);
            if constexpr (NY) {
                Limbs wy[KP];
                weights<KP>(B.ax[1], y, wy);
                const BfpRowMeta my = row_meta(B.ax[1], y);  // the same for the warp
                const double d = sum(own_exp, W{}, s + (my.q - y0 + HY) * BX + tx + HX, BX, wy, my, limit(my), ok);
                v = NX ? v + d : d;
            }
            if constexpr (KF > 0) {
                // the sign bit alone: a zero or NaN coefficient gives the same with either variant (and it compiles
                // to no FP64 comparison)
                const double cr = U == 1 ? __ldg(B.field + first + (int64_t)r * n0) : c[r];
                const BfpRows& R = B.f[__double2hiint(cr) < 0 ? 1 : 0];
                Limbs wf[KF];
                weights<KF>(R, x, wf);
                const BfpRowMeta mf = row_meta(R, x);
                v = fma(cr, sum(own_exp, WF{}, row + (mf.q - x0 + HX), 1, wf, mf, limit(mf), ok), v);
            }
            if (mine && y >= (int)blockIdx.y * T) {
                if (ok) {
                    double* o = du + first + (int64_t)r * n0;
                    if constexpr (OW) *o = v;
                    else *o += v;
                } else {
                    s_list[atomicAdd(&s_n, 1)] = (unsigned short)((ty * RY + r) << 5 | tx);
                }
            }
        }
    };
    if (own) points(std::true_type{});
    else points(std::false_type{});
    __syncthreads();
    const int n = s_n;
    for (int i = tid; i < n; i += 256) {
        const int e = s_list[i];
        const int64_t idx = (int64_t)(y0 + (e >> 5)) * n0 + x0 + (e & 31);
        const double r = ref_point(*P, u, idx);
        if constexpr (OW) du[idx] = r;
        else du[idx] += r;
    }
}

}  // namespace rows
}  // namespace deo

using namespace deo;

template <int K, int KF, bool NX, bool NY>
static int go_rows(const BfpPlan2* B, const PlanDev* P, const void* u, void* du, int ow, cudaStream_t st) {
    const dim3 grid((unsigned)((B->n[0] + rows::T - 1) / rows::T), (unsigned)((B->n[1] + rows::T - 1) / rows::T));
    auto go = [&](auto kernel) { kernel<<<grid, dim3(32, 8), 0, st>>>(*B, P, (const double*)u, (double*)du); };
    if (ow) go(rows::k_rows_fx<K, KF, NX, NY, true>);
    else go(rows::k_rows_fx<K, KF, NX, NY, false>);
    return (int)cudaGetLastError();
}

template <int K, int KF>
static int pick_rows(const BfpPlan2* B, const PlanDev* P, const void* u, void* du, int ow, cudaStream_t st) {
    if (B->ax[0].w && B->ax[1].w) return go_rows<K, KF, true, true>(B, P, u, du, ow, st);
    if (B->ax[0].w) return go_rows<K, KF, true, false>(B, P, u, du, ow, st);
    if constexpr (KF == 0)
        if (B->ax[1].w) return go_rows<K, KF, false, true>(B, P, u, du, ow, st);
    return (int)cudaErrorNotSupported;
}

extern "C" int deo_k_rows_fx(const BfpPlan2* B, const PlanDev* d_plan, const void* u, void* du, int overwrite,
                             void* stream) {
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (B->field) switch (B->K) {
            case 3: return pick_rows<3, 4>(B, d_plan, u, du, overwrite, st);
            case 5: return pick_rows<5, 4>(B, d_plan, u, du, overwrite, st);
            case 7: return pick_rows<7, 4>(B, d_plan, u, du, overwrite, st);
            case 9: return pick_rows<9, 4>(B, d_plan, u, du, overwrite, st);
        }
    else switch (B->K) {
            case 3: return pick_rows<3, 0>(B, d_plan, u, du, overwrite, st);
            case 5: return pick_rows<5, 0>(B, d_plan, u, du, overwrite, st);
            case 7: return pick_rows<7, 0>(B, d_plan, u, du, overwrite, st);
            case 9: return pick_rows<9, 0>(B, d_plan, u, du, overwrite, st);
        }
    return (int)cudaErrorNotSupported;
}
