// deo_eval.cuh -- device-side evaluators shared by the kernels: one output
// row of one term from its row table (forward), one column of the transposed
// operator (adjoint), the multi-term point sum, and small helpers.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "deo_internal.h"

namespace deo {

template <typename T>
__device__ __forceinline__ T band_w(const RowTabDev& tb, int k);
template <>
__device__ __forceinline__ double band_w<double>(const RowTabDev& tb, int k) {
    return tb.wband[k];
}
template <>
__device__ __forceinline__ float band_w<float>(const RowTabDev& tb, int k) {
    return reinterpret_cast<const float*>(tb.wband)[k];
}

// The per-line BC record of the line starting at flat index `base`
// (multi_dim_bc_operators.jl:28-52: the BC at the line's index over the other axes).
__device__ __forceinline__ const double* line_bc(const TermDev& t, int64_t base) {
    const int64_t lo = base % t.stride, hi = base / (t.stride * (int64_t)t.len);
    return t.lbc + (lo + hi * t.stride) * (int64_t)t.lbc_stride;
}

// Ghosts from one line's own BC record: BCs[I, J] * u[I, :, J], the 1-D ghost
// fill (a periodic BC wraps around its line, bc_operators.jl:188-193).
template <typename T>
__device__ __noinline__ T ghost_line(const TermDev& t, const T* __restrict__ line, int64_t base, bool left) {
    const int64_t s = t.stride;
    const double* q = line_bc(t, base);
    if (q[0] != 0.0) return left ? line[(int64_t)(t.len - 1) * s] : line[0];
    const int m = (int)(left ? q[1] : q[2]);
    const double* a = q + 5 + (left ? 0 : t.lbc_mw);
    const int64_t o = left ? 0 : (int64_t)(t.len - m);
    T d = T(0);
    for (int j = 0; j < m; ++j) d = (j == 0) ? T(a[0]) * line[o * s] : fma(T(a[j]), line[(o + j) * s], d);
    return d + T(left ? q[3] : q[4]);
}

// LBC: the plan has per-line boundary conditions (PlanDev::has_lbc); the
// kernels are instantiated with and without that branch, so that plans
// without them carry no call to ghost_line.
template <typename T, bool LBC = false>
__device__ __forceinline__ T ghost_left(const TermDev& t, const T* __restrict__ line, int64_t base) {
    const int64_t s = t.stride;
    if (LBC && t.lbc) return ghost_line<T>(t, line, base, true);
    if (t.bc_kind == 1) return t.periodic_nd ? line[0] : line[(int64_t)(t.len - 1) * s];
    if (t.bc_kind == 2) return line[-s];  // padded input: the ghost is stored before the line
    T d = T(0);
    for (int j = 0; j < t.ml; ++j) d = (j == 0) ? T(t.al[0]) * line[0] : fma(T(t.al[j]), line[(int64_t)j * s], d);
    return d + T(t.bl);
}

template <typename T, bool LBC = false>
__device__ __forceinline__ T ghost_right(const TermDev& t, const T* __restrict__ line, int64_t base) {
    const int64_t s = t.stride;
    if (LBC && t.lbc) return ghost_line<T>(t, line, base, false);
    if (t.bc_kind == 1) return t.periodic_nd ? line[(int64_t)(t.len - 1) * s] : line[0];
    if (t.bc_kind == 2) return line[(int64_t)t.len * s];  // padded input: the ghost is stored after the line
    T d = T(0);
    const int64_t o = (int64_t)(t.len - t.mr);
    for (int j = 0; j < t.mr; ++j)
        d = (j == 0) ? T(t.ar[0]) * line[o * s] : fma(T(t.ar[j]), line[(o + j) * s], d);
    return d + T(t.br);
}

// The reference adds `!overwrite * x_temp[i]` (a strong zero) to every tap
// sum, which turns -0.0 into +0.0 and is otherwise exact.  Applied once to the
// final sum it has the same effect; done on the bits to spend no FP64 issue.
__device__ __forceinline__ double zero_fix(double x) {
    return __double_as_longlong(x) == (long long)0x8000000000000000ULL ? 0.0 : x;
}
__device__ __forceinline__ float zero_fix(float x) {
    return __float_as_uint(x) == 0x80000000u ? 0.0f : x;
}

struct RowInfo {
    int p0, nk, e;
    bool band;
};

__device__ __forceinline__ RowInfo row_info(const RowTabDev& tb, int i) {
    RowInfo r;
    r.band = (i >= tb.ilo) && (i <= tb.ihi);
    if (r.band) {
        r.p0 = i + tb.band_p0_off;
        r.nk = tb.band_nk;
        r.e = 0;
    } else {
        r.e = (i < tb.ilo) ? i - 1 : (tb.ilo - 1) + (i - tb.ihi - 1);
        r.p0 = __ldg(tb.p0 + r.e);
        r.nk = __ldg(tb.nk + r.e);
    }
    return r;
}

__device__ __forceinline__ int row_cidx(const RowTabDev& tb, int i) {
    if (i >= tb.ilo && i <= tb.ihi) return i + tb.band_cidx_off;
    const int e = (i < tb.ilo) ? i - 1 : (tb.ilo - 1) + (i - tb.ihi - 1);
    return __ldg(tb.cidx + e);
}

template <typename T>
__device__ __forceinline__ T row_w(const RowTabDev& tb, const RowInfo& r, int k) {
    return r.band ? band_w<T>(tb, k) : __ldg(reinterpret_cast<const T*>(tb.W) + (int64_t)k * tb.nexp + r.e);
}

// !(c >= 0) -- c negative (not -0) or NaN: the upwind operator's variant
// choice (convolutions.jl:134), tested on the bits so that it issues no FP64
// (Float32) comparison.
__device__ __forceinline__ bool not_nonneg(double c) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(c);
    return ((long long)b < 0 && (b << 1) != 0ULL) || (b << 1) > 0xFFE0000000000000ULL;
}
__device__ __forceinline__ bool not_nonneg(float c) {
    const unsigned b = __float_as_uint(c);
    return ((int)b < 0 && (b << 1) != 0u) || (b << 1) > 0xFF000000u;
}

// Coefficient and table variant of row i on the line starting at `base`.
template <typename T>
__device__ __forceinline__ const RowTabDev& row_variant(const TermDev& t, int64_t base, int i, T& c) {
    c = T(1);
    if (!t.has_field) return t.tab[0];
    const int ci = row_cidx(t.tab[0], i);
    c = __ldg(reinterpret_cast<const T*>(t.field) + base + (int64_t)(ci - 1) * t.stride);
    if (t.nvar == 2 && not_nonneg(c)) return t.tab[1];
    return t.tab[0];
}

// n taps in chunks of 4, 2 and 1: f(first tap, the chunk's length as a constant).
template <int N>
struct Chunk {
    __device__ constexpr operator int() const { return N; }
};
template <typename F>
__device__ __forceinline__ void tap_chunks(int n, F f) {
    int k = 0;
    for (; k + 4 <= n; k += 4) f(k, Chunk<4>{});
    if (n & 2) {
        f(k, Chunk<2>{});
        k += 2;
    }
    if (n & 1) f(k, Chunk<1>{});
}

// One term, one output row: the reference's per-point tap loop.  Float32 loads four taps
// before their products: a boundary row is a chain of latencies.
template <typename T, bool LBC = false>
__device__ __forceinline__ T eval_term(const TermDev& t, const T* __restrict__ u, int64_t idx, int i) {
    const int64_t s = t.stride;
    const int64_t base = idx - (int64_t)(i - 1) * s;
    const T* __restrict__ line = u + base;
    T c;
    const RowTabDev& tb = row_variant<T>(t, base, i, c);
    const RowInfo r = row_info(tb, i);
    const int L2 = t.len + 2;
    T gl = T(0), gr = T(0);
    if (r.p0 == 1) gl = ghost_left<T, LBC>(t, line, base);
    if (r.p0 + r.nk - 1 == L2) gr = ghost_right<T, LBC>(t, line, base);
    T acc = T(0);
    if constexpr (sizeof(T) == 4) {
        tap_chunks(r.nk, [&](int k, auto n) {
            T w[n], x[n];
#pragma unroll
            for (int m = 0; m < n; ++m) {
                const int p = r.p0 + k + m;
                const T v = __ldg(line + (int64_t)min(max(p - 2, 0), t.len - 1) * s);
                w[m] = row_w<T>(tb, r, k + m);
                x[m] = (p == 1) ? gl : (p == L2 ? gr : v);
            }
            if (t.has_field == 1) {
#pragma unroll
                for (int m = 0; m < n; ++m) acc = fma(c * w[m], x[m], acc);
            } else {
#pragma unroll
                for (int m = 0; m < n; ++m) acc = fma(w[m], x[m], acc);
            }
        });
        return t.has_field == 2 ? c * acc : acc;  // 2: DEO_PLAN_FACTOR_FIELD, c * (sum_k w_k x_k)
    }
    // Float64 in separate loops, tap by tap: a predicated-off FP64 instruction takes its
    // turn in the pipe, which is what bounds these rows (a c * w issued for every row
    // doubled their time; chunks of four cost 5 to 10 % more than they hid)
    auto tap = [&](int k) {
        const int p = r.p0 + k;
        return (p == 1) ? gl : (p == L2 ? gr : __ldg(line + (int64_t)(p - 2) * s));
    };
    if (t.has_field == 2) {
        for (int k = 0; k < r.nk; ++k) acc = fma(row_w<T>(tb, r, k), tap(k), acc);
        acc = c * acc;
    } else if (t.has_field) {
        for (int k = 0; k < r.nk; ++k) acc = fma(c * row_w<T>(tb, r, k), tap(k), acc);
    } else {
        for (int k = 0; k < r.nk; ++k) acc = fma(row_w<T>(tb, r, k), tap(k), acc);
    }
    return acc;
}

// One row of a term's table over a padded line whose ghosts are stored around
// it (bc_kind 2), so every tap is a plain load: line position p (1-based) is
// x0[(p - 1) * s], x0 pointing at the left ghost.  Same products and order as
// eval_term; no field coefficient.
template <typename T>
__device__ __forceinline__ T eval_row_padded(const RowTabDev& tb, const T* __restrict__ x0, int64_t s, int i) {
    const RowInfo r = row_info(tb, i);
    const T* __restrict__ xp = x0 + (int64_t)(r.p0 - 1) * s;
    T acc = T(0);
    for (int k = 0; k < r.nk; ++k) acc = fma(row_w<T>(tb, r, k), __ldg(xp + (int64_t)k * s), acc);
    return acc;
}

// Column p of one term's L (padded space) dotted with dbar along the line.
template <typename T>
__device__ __forceinline__ T adj_column(const TermDev& t, const T* __restrict__ d, int64_t base, int p) {
    const int64_t s = t.stride;
    const int lo = __ldg(t.rlo + (p - 1)), hi = __ldg(t.rhi + (p - 1));
    T acc = T(0);
    if (!t.has_field) {  // (no c * w multiply issued); the loads of four rows before their products
        const RowTabDev& tb = t.tab[0];
        tap_chunks(max(hi - lo + 1, 0), [&](int o, auto n) {
            T w[n], x[n];
            bool in[n];
#pragma unroll
            for (int m = 0; m < n; ++m) {
                const int i = lo + o + m;
                const RowInfo r = row_info(tb, i);
                const int k = p - r.p0;
                in[m] = k >= 0 && k < r.nk;
                w[m] = row_w<T>(tb, r, min(max(k, 0), r.nk - 1));
                x[m] = __ldg(d + base + (int64_t)(i - 1) * s);
            }
#pragma unroll
            for (int m = 0; m < n; ++m)
                if (in[m]) acc = fma(w[m], x[m], acc);
        });
        return acc;
    }
    for (int i = lo; i <= hi; ++i) {
        T c;
        const RowTabDev& tb = row_variant<T>(t, base, i, c);
        const RowInfo r = row_info(tb, i);
        const int k = p - r.p0;
        if (k < 0 || k >= r.nk) continue;
        acc = fma(c * row_w<T>(tb, r, k), __ldg(d + base + (int64_t)(i - 1) * s), acc);
    }
    return acc;
}

template <typename T, bool LBC = false>
__device__ __forceinline__ T adj_term(const TermDev& t, const T* __restrict__ d, int64_t idx, int j) {
    const int64_t base = idx - (int64_t)(j - 1) * t.stride;
    const int L = t.len;
    T w = adj_column<T>(t, d, base, j + 1);
    if (LBC && t.lbc) {  // this line's own BC
        const double* q = line_bc(t, base);
        if (q[0] != 0.0) {  // periodic line: the left ghost is u[len], the right u[1]
            if (j == L) w += adj_column<T>(t, d, base, 1);
            if (j == 1) w += adj_column<T>(t, d, base, L + 2);
        } else {
            const int ml = (int)q[1], mr = (int)q[2];
            if (j <= ml) w = fma(T(q[5 + j - 1]), adj_column<T>(t, d, base, 1), w);
            if (j > L - mr) w = fma(T(q[5 + t.lbc_mw + j - 1 - (L - mr)]), adj_column<T>(t, d, base, L + 2), w);
        }
        return w;
    }
    if (t.bc_kind == 0) {
        if (j <= t.ml) w = fma(T(t.al[j - 1]), adj_column<T>(t, d, base, 1), w);
        if (j > L - t.mr) w = fma(T(t.ar[j - 1 - (L - t.mr)]), adj_column<T>(t, d, base, L + 2), w);
    } else {
        const int jl = t.periodic_nd ? 1 : L;  // column receiving the left ghost
        const int jr = t.periodic_nd ? L : 1;
        if (j == jl) w += adj_column<T>(t, d, base, 1);
        if (j == jr) w += adj_column<T>(t, d, base, L + 2);
    }
    return w;
}

__device__ __forceinline__ uint32_t fast_div(uint32_t n, const FastDiv& d) {
    return (__umulhi(n, d.mul) + n) >> d.shr;
}

// 1-based row of flat index idx along term t's axis
__device__ __forceinline__ int term_row(const PlanDev& P, const TermDev& t, int64_t idx) {
    if (P.fastdiv) {
        const uint32_t q = fast_div((uint32_t)idx, t.div_stride);
        return (int)(q - fast_div(q, t.div_len) * (uint32_t)t.len) + 1;
    }
    return (int)((idx / t.stride) % t.len) + 1;
}

// nk taps x[m * s] in the order of the general loops: weights w[m] (REV: w[nk - 1 - m]),
// or w[m * ws], times c when SCALED.  NK > 0: unrolled, all loads before the chain of
// products; 0: any length, four loads ahead.
template <typename T, bool REV, bool ROWS, bool SCALED, int NK>
__device__ __forceinline__ T straight_nk(const T* w, int64_t ws, const T* __restrict__ x, int64_t s, T c, int nk) {
    T acc = T(0);
    auto weight = [&](int m) {
        const T v = ROWS ? __ldg(w + m * ws) : w[REV ? nk - 1 - m : m];
        return SCALED ? c * v : v;
    };
    if constexpr (NK > 0) {
        T v[NK];
#pragma unroll
        for (int m = 0; m < NK; ++m) v[m] = __ldg(x + m * s);
#pragma unroll
        for (int m = 0; m < NK; ++m) acc = fma(weight(m), v[m], acc);
    } else {
#pragma unroll 4
        for (int m = 0; m < nk; ++m) acc = fma(weight(m), __ldg(x + m * s), acc);
    }
    return acc;
}
// Which lengths are unrolled: Float32 waits on its loads (all common lengths: 2048^2,
// order 2, 45 -> 28 us), Float64 on the FP64 pipe, where the long bands lose by it what
// the short ones gain (2048^2: 3 taps 70 -> 62 us, 9 taps 158 unrolled, 156 not; the
// transposed bands 93 -> 87 at 5 taps).
template <typename T, bool REV, bool ROWS, bool SCALED>
__device__ __forceinline__ T straight(const T* w, int64_t ws, const T* __restrict__ x, int64_t s, T c, int nk) {
    if constexpr (sizeof(T) == 8 && REV && !ROWS) {
        return straight_nk<T, REV, ROWS, SCALED, 0>(w, ws, x, s, c, nk);
    } else {
        if (nk == 3) return straight_nk<T, REV, ROWS, SCALED, 3>(w, ws, x, s, c, 3);
        if (nk == 5) return straight_nk<T, REV, ROWS, SCALED, 5>(w, ws, x, s, c, 5);
        if constexpr (sizeof(T) == 4 || ROWS) {
            if (nk == 7) return straight_nk<T, REV, ROWS, SCALED, 7>(w, ws, x, s, c, 7);
            if (nk == 9) return straight_nk<T, REV, ROWS, SCALED, 9>(w, ws, x, s, c, 9);
        }
        return straight_nk<T, REV, ROWS, SCALED, 0>(w, ws, x, s, c, nk);
    }
}

// eval_term / adj_term for any row: the straight loops where TermDev's ranges allow
// them, bit for bit the same sums.  The general loops choose between band and explicit
// row, ghost and line at every tap (40 instructions a tap) and look up p0, nk and the
// touching rows at every point, also on graded lines, whose rows differ by their
// weights alone.  A warp with one row outside the range takes the general loop as a
// whole: both loops one after the other were the longest chain of the small and the
// ragged launches (graded 542 x 226 with a field 24.0 us, 20.8 so; 65 x 33 x 41, 9 taps,
// 15.4 / 15.9 and 13.8 / 14.5).  2048^2 at 5 taps, general / straight, apply and
// transposed: uniform Float64 97 -> 95 and 90 -> 86 us, Float32 49 -> 32 and 52 -> 35;
// graded Float64 107 -> 89 and 114 -> 90, Float32 78 -> 36 and 99 -> 40.
// PLAIN (k_apply): Float64 bands of 9 taps and more stay in the general loop, which keeps
// the FP64 pipe as busy there (2^22 points, order 8, 78.5 us against 82.6 straight; the
// batched kernels lose by it, 256 mixed instances 468 -> 497).
template <typename T, bool ADJ, bool LBC, bool PLAIN>
__device__ __forceinline__ T term_at(const TermDev& t, const T* __restrict__ u, int64_t idx, int i) {
    const int64_t s = t.stride;
    if constexpr (ADJ) {
        if (!__all_sync(__activemask(), i >= t.sa_lo && i <= t.sa_hi)) return adj_term<T, LBC>(t, u, idx, i);
        const int i0 = i + 2 - t.s_off[0] - t.s_nk[0];  // rows i0 + m, their taps nk - 1 - m
        const T* __restrict__ x = u + idx + (i0 - i) * s;
        if (t.s_rows) {
            const T* w = reinterpret_cast<const T*>(t.tab[0].W) + (int64_t)(t.s_nk[0] - 1) * t.tab[0].nexp + (i0 + t.s_e0[0]);
            return straight<T, true, true, false>(w, 1 - t.tab[0].nexp, x, s, T(1), t.s_nk[0]);
        }
        return straight<T, true, false, false>(reinterpret_cast<const T*>(t.tab[0].wband), 0, x, s, T(1), t.s_nk[0]);
    } else {
        if (!__all_sync(__activemask(), i >= t.sf_lo && i <= t.sf_hi)) return eval_term<T, LBC>(t, u, idx, i);
        if (!t.has_field) {
            const T* __restrict__ x = u + idx + (t.s_off[0] - 1) * s;
            if (t.s_rows)
                return straight<T, false, true, false>(reinterpret_cast<const T*>(t.tab[0].W) + (i + t.s_e0[0]),
                                                       t.tab[0].nexp, x, s, T(1), t.s_nk[0]);
            if (PLAIN && sizeof(T) == 8 && t.s_nk[0] >= 9) return eval_term<T, LBC>(t, u, idx, i);
            return straight<T, false, false, false>(reinterpret_cast<const T*>(t.tab[0].wband), 0, x, s, T(1), t.s_nk[0]);
        }
        const T c = __ldg(reinterpret_cast<const T*>(t.field) + idx + t.s_cidx * s);
        const int v = t.nvar == 2 && not_nonneg(c);
        const RowTabDev& tb = t.tab[v];
        const T* __restrict__ x = u + idx + (t.s_off[v] - 1) * s;
        const T* w = reinterpret_cast<const T*>(tb.wband);
        const int nk = t.s_nk[v];
        if (t.s_rows) {
            w = reinterpret_cast<const T*>(tb.W) + (i + t.s_e0[v]);
            if (t.has_field == 2) return c * straight_nk<T, false, true, false, 0>(w, tb.nexp, x, s, T(1), nk);
            return straight_nk<T, false, true, true, 0>(w, tb.nexp, x, s, c, nk);
        }
        if (t.has_field == 2) return c * straight_nk<T, false, false, false, 0>(w, 0, x, s, T(1), nk);
        return straight_nk<T, false, false, true, 0>(w, 0, x, s, c, nk);
    }
}

template <typename T, bool ADJ, bool LBC = false, bool PLAIN = false>
__device__ __forceinline__ T eval_point(const PlanDev& P, const T* __restrict__ u, int64_t idx) {
    if (!ADJ && P.star.n) {  // the merged star at points whose rows read no ghost along any axis
        bool in = true;
        for (int tt = 0; tt < P.nterms; ++tt) {
            const int i = term_row(P, P.t[tt], idx);
            in = in && i >= P.star.lo[tt] && i <= P.star.hi[tt];
        }
        if (in) {
            T acc = T(0);
            for (int k = 0; k < P.star.n; ++k) acc = fma(T(P.star.w[k]), __ldg(u + idx + P.star.off[k]), acc);
            return zero_fix(acc);
        }
    }
    auto term = [&](int tt) {
        const TermDev& t = P.t[tt];
        const int i = term_row(P, t, idx);
        return term_at<T, ADJ, LBC, PLAIN>(t, u, idx, i);
    };
    T acc = term(0);  // the first term as is, then the others added left to right
    for (int tt = 1; tt < P.nterms; ++tt) acc = acc + term(tt);
    return ADJ ? acc : zero_fix(acc);
}

// Out-of-line copy of the generic column evaluator (the transposed shell's
// boundary columns).
template <typename T>
__device__ __noinline__ T adj_term_cold(const TermDev& t, const T* __restrict__ d, int64_t idx, int j) {
    return adj_term<T>(t, d, idx, j);
}

// Out-of-line copy for a kernel that evaluates a few boundary points with
// the generic evaluator (the shell fallback).
template <typename T>
__device__ __noinline__ T eval_term_cold(const TermDev& t, const T* __restrict__ u, int64_t idx, int i) {
    return eval_term<T>(t, u, idx, i);
}

template <typename T>
__device__ __forceinline__ T uni_w(const UniTerm& t, int k);
template <>
__device__ __forceinline__ double uni_w<double>(const UniTerm& t, int k) { return t.w[k]; }
template <>
__device__ __forceinline__ float uni_w<float>(const UniTerm& t, int k) {
    return reinterpret_cast<const float*>(t.w)[k];
}

}  // namespace deo
