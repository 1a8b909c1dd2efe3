// deo_solve.cu -- A \ u for A = L*Q along one axis: every line of u along the
// operator's axis is solved with the same banded LU factors (partial pivoting,
// band storage as LAPACK's gbtrf leaves it), one thread per line.
//   b = u - A_b;  b <- P, L^-1 b (forward, with the row interchanges);  x = U^-1 b.
// Lines along axis 1 are contiguous, so consecutive threads own lines n
// elements apart; along the other axes consecutive threads own adjacent
// lines and every step is a coalesced access.  The lines are solved in
// Float64 (in x itself, or in a plan-owned Float64 workspace for Float32).
#include <cuda_runtime.h>
#include <stdint.h>

#include <type_traits>

#include "deo_internal.h"

namespace deo {
namespace {

template <typename T>
__global__ void __launch_bounds__(256) k_band_solve(int n, int kl, int ku, const double* __restrict__ ab,
                                                    const int* __restrict__ ipiv, const double* __restrict__ Ab,
                                                    int64_t stride, int64_t nlines, const T* u, T* x,
                                                    double* work) {
    const int64_t line = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (line >= nlines) return;
    const int64_t base = line % stride + (line / stride) * stride * n;
    double* w = work ? work + base : reinterpret_cast<double*>(x) + base;  // Float64: x itself
    const int kv = kl + ku;
    for (int i = 0; i < n; ++i) w[(int64_t)i * stride] = (double)u[base + (int64_t)i * stride] - __ldg(Ab + i);
    // forward: row interchanges and the unit lower factor
    for (int j = 0; j < n - 1; ++j) {
        const int l = __ldg(ipiv + j);
        double bj = w[(int64_t)j * stride];
        if (l != j) {
            const double t = w[(int64_t)l * stride];
            w[(int64_t)l * stride] = bj;
            bj = t;
            w[(int64_t)j * stride] = bj;
        }
        const int km = min(kl, n - 1 - j);
        for (int r = 1; r <= km; ++r) {
            double& wr = w[(int64_t)(j + r) * stride];
            wr = fma(-__ldg(ab + (int64_t)(kv + r) * n + j), bj, wr);
        }
    }
    // backward: the upper factor (kv super-diagonals)
    for (int j = n - 1; j >= 0; --j) {
        const double xj = w[(int64_t)j * stride] / __ldg(ab + (int64_t)kv * n + j);
        w[(int64_t)j * stride] = xj;
        const int i0 = max(0, j - kv);
        for (int i = i0; i < j; ++i) {
            double& wi = w[(int64_t)i * stride];
            wi = fma(-__ldg(ab + (int64_t)(kv + i - j) * n + j), xj, wi);
        }
        if (work) x[base + (int64_t)j * stride] = (T)xj;
    }
}

// The same solve with the rows in flight held in registers: the forward sweep
// keeps rows j .. j+kl (the pivot search window and the rows the current
// column updates), the backward sweep rows j-kb .. j, so every element of the
// line is read once and written once per sweep (y between the sweeps lives in
// x for Float64, in the workspace for Float32).  The pivots U[j][j] enter as
// their reciprocals rdiag (the GPU has no fast FP64 divide).  kb is the widest
// column of U that holds anything (kl + ku only where rows were interchanged),
// and meta[j] = the interchange (bits 0-7), the multipliers (8-15) and the
// entries of U above the diagonal (16-23) that column j really has.  Columns
// [plo, phi) are plain: all with FL multipliers, FU entries and the interchange P
// (0 none; 1 with the next row, as every step of a Robin line of either order
// has), and A_b is zero in the rows [alo, ahi).  Blocks of PF plain steps run
// without a condition: a predicated-off FP64 instruction takes its 16 clocks of the pipe
// all the same (with conditions in every step the tridiagonal case took 6 FP64
// slots a step instead of 3, and 290 us).  W >= max(kl, kb).
//
// What bounds it: FP64 at 2 per clock per SM, and the line's chain.  A tridiagonal
// step with its interchange is 4 FP64 instructions (6 with A_b), 107 us for 256^3
// points at the FP64 rate, beside 79 us for the four passes over memory;
// measured 247 -> 146 us (FP64 pipe 82 %), and 656 -> 195 us for 4 + 4 bands (6 a step).  64
// threads a block: 65536 lines are 1024 blocks on 152 SMs, where 256-thread
// blocks left some SMs with two and some with one.
template <typename T, int W, int FL, int FU, int P, int PF = 8>
__global__ void __launch_bounds__(64) k_band_solve_w(const BandLU b, int64_t stride, int64_t nlines, const T* u, T* x,
                                                     double* work) {
    const int64_t line = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int n = b.n, kl = b.kl, kb = b.kb;
    if (line >= nlines) return;
    const int64_t base = line % stride + (line / stride) * stride * n;
    double* y = work ? work + base : reinterpret_cast<double*>(x) + base;
    const T* ul = u + base;
    const double* diag = b.ab + (int64_t)(b.kl + b.ku) * n;  // U's diagonal; row r below: multipliers, above: U
    auto rhs = [&](int j) { return (double)ul[(int64_t)j * stride] - __ldg(b.Ab + j); };
    double f[W + 1];
#pragma unroll
    for (int r = 0; r <= W; ++r) f[r] = (r <= kl && r < n) ? rhs(r) : 0.0;
    // the next PF new rows' values are loaded one block of PF steps ahead
    double cur[PF], nxt[PF];
#pragma unroll
    for (int k = 0; k < PF; ++k) {
        const int jn = k + 1 + kl;
        cur[k] = jn < n ? rhs(jn) : 0.0;
    }
    auto forward = [&](int j, double nv, auto plain) {
        const double* l = diag + j;
        if constexpr (decltype(plain)::value) {
            if constexpr (P == 1) {
                const double t = f[0];
                f[0] = f[1];
                f[1] = t;
            }
#pragma unroll
            for (int r = 1; r <= FL; ++r) f[r] = fma(-__ldg(l + (int64_t)r * n), f[0], f[r]);
        } else {
            const int mt = __ldg(b.meta + j), p = mt & 255, nl = (mt >> 8) & 255;
#pragma unroll
            for (int r = 1; r <= W; ++r)
                if (r == p) {
                    const double t = f[0];
                    f[0] = f[r];
                    f[r] = t;
                }
#pragma unroll
            for (int r = 1; r <= W; ++r)
                if (r <= nl) f[r] = fma(-__ldg(l + (int64_t)r * n), f[0], f[r]);
        }
        y[(int64_t)j * stride] = f[0];
#pragma unroll
        for (int r = 0; r < W; ++r) f[r] = (r == kl) ? nv : f[r + 1];
        if (kl == W) f[W] = nv;
    };
    for (int jb = 0; jb < n; jb += PF) {
        const int j0 = jb + PF + 1 + kl;  // the first row loaded here
        if (j0 >= b.alo && j0 + PF <= b.ahi) {
#pragma unroll
            for (int k = 0; k < PF; ++k) nxt[k] = (double)ul[(int64_t)(j0 + k) * stride];
        } else {
#pragma unroll
            for (int k = 0; k < PF; ++k) nxt[k] = j0 + k < n ? rhs(j0 + k) : 0.0;
        }
        if (jb >= b.plo && jb + PF <= b.phi) {
#pragma unroll
            for (int k = 0; k < PF; ++k) forward(jb + k, cur[k], std::true_type{});
        } else {
#pragma unroll
            for (int k = 0; k < PF; ++k)
                if (jb + k < n) forward(jb + k, cur[k], std::false_type{});
        }
#pragma unroll
        for (int k = 0; k < PF; ++k) cur[k] = nxt[k];
    }
    // backward: g[r] = y[j - r]
    double g[W + 1];
#pragma unroll
    for (int r = 0; r <= W; ++r) g[r] = (r <= kb && n - 1 - r >= 0) ? y[(int64_t)(n - 1 - r) * stride] : 0.0;
#pragma unroll
    for (int k = 0; k < PF; ++k) {
        const int jn = n - 2 - kb - k;
        cur[k] = jn >= 0 ? y[(int64_t)jn * stride] : 0.0;
    }
    auto backward = [&](int j, double nv, auto plain) {
        const double xj = g[0] * __ldg(b.rdiag + j);  // one rounding more than a division, no FP64 divide
        if (work) x[base + (int64_t)j * stride] = (T)xj;
        else y[(int64_t)j * stride] = xj;
        const double* up = diag + j;
        if constexpr (decltype(plain)::value) {
#pragma unroll
            for (int r = 1; r <= FU; ++r) g[r] = fma(-__ldg(up - (int64_t)r * n), xj, g[r]);
        } else {
            const int nu = (__ldg(b.meta + j) >> 16) & 255;
#pragma unroll
            for (int r = 1; r <= W; ++r)
                if (r <= nu) g[r] = fma(-__ldg(up - (int64_t)r * n), xj, g[r]);
        }
#pragma unroll
        for (int r = 0; r < W; ++r) g[r] = (r == kb) ? nv : g[r + 1];
        if (kb == W) g[W] = nv;
    };
    for (int jb = n - 1; jb >= 0; jb -= PF) {
#pragma unroll
        for (int k = 0; k < PF; ++k) {
            const int jn = jb - PF - 1 - kb - k;
            nxt[k] = jn >= 0 ? y[(int64_t)jn * stride] : 0.0;
        }
        if (jb < b.phi && jb - PF + 1 >= b.plo) {
#pragma unroll
            for (int k = 0; k < PF; ++k) backward(jb - k, cur[k], std::true_type{});
        } else {
#pragma unroll
            for (int k = 0; k < PF; ++k)
                if (jb - k >= 0) backward(jb - k, cur[k], std::false_type{});
        }
#pragma unroll
        for (int k = 0; k < PF; ++k) cur[k] = nxt[k];
    }
}

}  // namespace
}  // namespace deo

extern "C" int deo_k_band_solve(const deo::BandLU* b, int64_t stride, int64_t nlines, int dtype, const void* u, void* x,
                                double* work, void* stream) {
    if (nlines <= 0) return 0;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const int wmax = b->kl > b->kb ? b->kl : b->kb;
    auto go = [&](auto w, auto pattern) {
        constexpr int W = decltype(w)::value, Q = decltype(pattern)::value, FL = Q / 100, FU = Q / 10 % 10, P = Q % 10;
        const unsigned blocks = (unsigned)((nlines + 63) / 64);
        if (dtype == 0)
            deo::k_band_solve_w<double, W, FL, FU, P><<<blocks, 64, 0, st>>>(*b, stride, nlines, (const double*)u,
                                                                             (double*)x, nullptr);
        else
            deo::k_band_solve_w<float, W, FL, FU, P><<<blocks, 64, 0, st>>>(*b, stride, nlines, (const float*)u,
                                                                            (float*)x, work);
        return (int)cudaGetLastError();
    };
    // the plain columns' pattern (multipliers, entries of U, interchange); 110 serves plans without any
    auto width = [&](auto w) {
        constexpr int W = decltype(w)::value;
        if constexpr (W >= 2) {
            if (b->plain == 121) return go(w, std::integral_constant<int, 121>{});
            if (b->plain == 220) return go(w, std::integral_constant<int, 220>{});
        }
        if constexpr (W >= 4)
            if (b->plain == 231) return go(w, std::integral_constant<int, 231>{});
        return go(w, std::integral_constant<int, 110>{});
    };
    if (wmax <= 1) return width(std::integral_constant<int, 1>{});
    if (wmax <= 2) return width(std::integral_constant<int, 2>{});
    if (wmax <= 4) return width(std::integral_constant<int, 4>{});
    if (wmax <= 8) return width(std::integral_constant<int, 8>{});
    if (wmax <= 16) return width(std::integral_constant<int, 16>{});
    const unsigned blocks = (unsigned)((nlines + 255) / 256);
    if (dtype == 0)
        deo::k_band_solve<double><<<blocks, 256, 0, st>>>(b->n, b->kl, b->ku, b->ab, b->ipiv, b->Ab, stride, nlines,
                                                          (const double*)u, (double*)x, nullptr);
    else
        deo::k_band_solve<float><<<blocks, 256, 0, st>>>(b->n, b->kl, b->ku, b->ab, b->ipiv, b->Ab, stride, nlines,
                                                         (const float*)u, (float*)x, work);
    return (int)cudaGetLastError();
}
