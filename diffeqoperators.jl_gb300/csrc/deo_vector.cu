// deo_vector.cu -- Gradient / Divergence / Curl of a padded array
// (vector_calculus_operators.jl, vector_calculus_convolutions.jl) and the
// pointwise vector algebra (vector_algebraic_operations.jl).
//
// Every derivative is one row of an axis
// operator's row table over the padded input (ghosts are the input's own
// first/last planes, bc_kind 2), so boundary rows, non-uniform stencils and
// coefficient vectors follow the same tables as the stencil-apply path; rows
// of a uniform operator's interior band take an unrolled loop with the same
// fused multiply-adds in the same order.  The reference's per-point additions
// into the output are replayed in its order (see VcDev).  Three kernels: one thread per
// output point (k_vc), per column (k_vc_march), and, for large Float64 arrays with a uniform
// band, block fixed point on tiles (k_vc_fx).
#include <cuda_runtime.h>
#include <limits.h>
#include <stdint.h>

#include <algorithm>
#include <type_traits>

#include "deo_bfp.cuh"
#include "deo_eval.cuh"
#include "deo_lap.cuh"

namespace deo {
namespace {

// 0: a BC_left row, 1: an interior row, 2: a BC_right row (0-based position o)
__device__ __forceinline__ int vc_phase(int64_t o, int64_t len, int bpc) {
    return o < bpc ? 0 : (o < len - bpc ? 1 : 2);
}

// One derivative along axis a at the point whose axis-a line passes through
// flat padded index ia (the row's centre), 0-based row oa along the axis.
// NK > 0: the row is an interior row of a uniform operator, whose NK band
// weights are the term's wband.  NK == 0: the row table gives the row (its
// first tap p0, tap count and weights: boundary rows, non-uniform stencils);
// every tap is a plain load because the input holds its own ghosts.
template <typename T, int NK>
__device__ __forceinline__ T vc_deriv(const TermDev& t, const T* __restrict__ M, int64_t ia, int64_t oa) {
    const int64_t s = t.stride;
    T acc = T(0);
    if (NK > 0) {
        const T* __restrict__ xp = M + ia - (int64_t)(NK / 2) * s;
#pragma unroll
        for (int k = 0; k < NK; ++k) acc = fma(band_w<T>(t.tab[0], k), __ldg(xp + (int64_t)k * s), acc);
        return acc;
    }
    return eval_row_padded<T>(t.tab[0], M + ia - (oa + 1) * s, s, (int)oa + 1);  // the line's left ghost
}

// One output point of the 2-D / 3-D methods (vector_calculus_convolutions.jl:174-838,
// curl :844-1067), every row from the row table (NK = 0), or an interior point
// of a uniform band of NK taps.
template <typename T, int KIND, int ND, int NK = 0>
__device__ __forceinline__ void vc_point(const VcDev& V, const T* __restrict__ M, T* __restrict__ out, int overwrite,
                                         int64_t o0, int64_t o1, int64_t o2) {
    const int64_t n = o0 + V.len[0] * (o1 + (ND == 3 ? V.len[1] : 1) * o2);
    const int64_t o[3] = {o0, o1, o2};
    // other axes at the padded index equal to the output index; +1 along the differentiated axis
    int64_t q = 0;
#pragma unroll
    for (int b = 0; b < ND; ++b) q += o[b] * V.pstride[b];
    int ph[ND];
#pragma unroll
    for (int a = 0; a < ND; ++a) ph[a] = vc_phase(o[a], V.len[a], V.bpc);
    auto D = [&](const TermDev& t, const T* x, int a) { return vc_deriv<T, NK>(t, x, q + V.pstride[a], o[a]); };
    if (KIND == DEO_VC_GRADIENT) {
#pragma unroll
        for (int a = 0; a < ND; ++a) {
            const T d = D(V.t[a], M, a);
            T* y = out + n + a * V.ovol;
            *y = overwrite ? zero_fix(d) : *y + d;
        }
    } else if (KIND == DEO_VC_DIVERGENCE) {
        T d[ND];
#pragma unroll
        for (int a = 0; a < ND; ++a) d[a] = D(V.t[a], M + a * V.pvol, a);
        T acc = overwrite ? T(0) : out[n];
        bool first = overwrite != 0;  // 0 + x is x up to the sign of zero
#pragma unroll
        for (int p = 0; p < 3; ++p)
#pragma unroll
            for (int a = 0; a < ND; ++a)
                if (ph[a] == p) {
                    acc = first ? zero_fix(d[a]) : acc + d[a];
                    first = false;
                }
        out[n] = acc;
    } else {
        // curl component c = (D_{a1} u[c1]) sign1 + (D_{a2} u[c2]) sign2, a1 < a2:
        //   x1: +D2 u3, -D3 u2;  x2: -D1 u3, +D3 u1;  x3: +D1 u2, -D2 u1
        constexpr int A1[3] = {1, 0, 0}, A2[3] = {2, 2, 1};
        constexpr int C1[3] = {2, 2, 1}, C2[3] = {1, 0, 0};
        constexpr bool N1[3] = {false, true, false}, N2[3] = {true, false, true};
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const int a1 = A1[c], a2 = A2[c];
            const T e1 = D(N1[c] ? V.tn[a1] : V.t[a1], M + C1[c] * V.pvol, a1);
            const T e2 = D(N2[c] ? V.tn[a2] : V.t[a2], M + C2[c] * V.pvol, a2);
            T* y = out + n + c * V.ovol;
            const T f = ph[a1] <= ph[a2] ? e1 : e2, g = ph[a1] <= ph[a2] ? e2 : e1;
            *y = (overwrite ? zero_fix(f) : *y + f) + g;
        }
    }
}

// The 2-D / 3-D methods point by point: blocks of 32 x 8 points of one (x, y)
// plane; blockIdx.z walks the planes.  Used where neither marching kernel
// applies (2-D Float64, operators without a uniform interior band, grids
// beyond the launch limits).
template <typename T, int KIND, int ND>
__global__ void __launch_bounds__(256) k_vc(const VcDev V, const T* __restrict__ M, T* __restrict__ out,
                                            int overwrite) {
    const int64_t n0 = V.len[0], n1 = V.len[1], n2 = ND == 3 ? V.len[2] : 1;
    const int64_t o0 = (int64_t)blockIdx.x * 32 + threadIdx.x % 32;
    if (o0 >= n0) return;
    for (int64_t o1 = (int64_t)blockIdx.y * 8 + threadIdx.x / 32; o1 < n1; o1 += (int64_t)gridDim.y * 8)
        for (int64_t o2 = blockIdx.z; o2 < n2; o2 += gridDim.z)
            vc_point<T, KIND, ND>(V, M, out, overwrite, o0, o1, o2);
}

// The same methods for operators with a uniform interior band of NK taps.
// Each thread owns one column across the axes other than the last and marches
// along the last axis (axis ND) over zb positions, keeping the taps along
// that axis in a register queue (one new load per step); taps along x are
// contiguous (compile-time offsets) and taps along y use offsets computed once
// per thread, so an interior point costs its loads and fused multiply-adds.
// A derivative along an axis on which the point is an interior row takes the
// unrolled band loop; on a boundary row, the row table.  ND = 3: blocks of
// 32 x 8 columns, blockIdx.z = the march chunk; ND = 2: 256 columns,
// blockIdx.y = the chunk.  Same fused multiply-adds in the same order as k_vc.
template <typename T, int KIND, int ND, int NK>
__global__ void __launch_bounds__(256) k_vc_march(const VcDev V, const T* __restrict__ M, T* __restrict__ out,
                                                  int overwrite, int zb) {
    constexpr int MA = ND - 1;                           // marching axis
    constexpr int NQ = KIND == DEO_VC_CURL ? 2 : 1;      // queued input components
    constexpr int MID = NK / 2;
    int64_t o[3] = {0, 0, 0};
    if (ND == 3) {
        o[0] = (int64_t)blockIdx.x * 32 + threadIdx.x % 32;
        o[1] = (int64_t)blockIdx.y * 8 + threadIdx.x / 32;
    } else {
        o[0] = (int64_t)blockIdx.x * 256 + threadIdx.x;
    }
#pragma unroll
    for (int b = 0; b < MA; ++b)
        if (o[b] >= V.len[b]) return;
    const int64_t chunk = ND == 3 ? blockIdx.z : blockIdx.y;
    const int64_t mlo = chunk * zb, mhi = min(mlo + zb, V.len[MA]);
    int ph[ND];
#pragma unroll
    for (int b = 0; b < MA; ++b) ph[b] = vc_phase(o[b], V.len[b], V.bpc);
    int64_t col = 0;  // other axes at the padded index equal to the output index
#pragma unroll
    for (int b = 0; b < MA; ++b) col += o[b] * V.pstride[b];
    const int64_t ocol = o[0] + (ND == 3 ? V.len[0] * o[1] : 0);
    const int64_t ms = V.pstride[MA], oms = ND == 3 ? V.len[0] * V.len[1] : V.len[0];
    const int64_t ys = V.pstride[1];
    // queued components: gradient M; divergence u[ND]; curl u2 (for x1 -= D3 u2) and u1 (for x2 += D3 u1)
    int64_t qoff[NQ];
    qoff[0] = KIND == DEO_VC_GRADIENT ? 0 : (KIND == DEO_VC_DIVERGENCE ? MA * V.pvol : V.pvol);
    if (NQ == 2) qoff[NQ - 1] = 0;
    T Q[NQ][NK];
    bool qvalid = false;
    for (int64_t om = mlo; om < mhi; ++om) {
        o[MA] = om;
        ph[MA] = vc_phase(om, V.len[MA], V.bpc);
        const bool mid_row = ph[MA] == 1;  // uniform over the block
        const int64_t q = col + om * ms;
        const int64_t n = ocol + om * oms;
        if (mid_row) {
            if (!qvalid) {
#pragma unroll
                for (int c = 0; c < NQ; ++c)
#pragma unroll
                    for (int k = 0; k < NK; ++k) Q[c][k] = __ldg(M + qoff[c] + q + (int64_t)(k + 1 - MID) * ms);
            } else {
#pragma unroll
                for (int c = 0; c < NQ; ++c) {
#pragma unroll
                    for (int k = 0; k < NK - 1; ++k) Q[c][k] = Q[c][k + 1];
                    Q[c][NK - 1] = __ldg(M + qoff[c] + q + (int64_t)(MID + 1) * ms);
                }
            }
        }
        qvalid = mid_row;
        // derivative along axis a of the input at component offset coff (queue qi along the marching axis)
        auto D = [&](const TermDev& t, int64_t coff, int a, int qi) -> T {
            if (ph[a] != 1) return vc_deriv<T, 0>(t, M + coff, q + V.pstride[a], o[a]);
            T acc = T(0);
            if (a == MA) {
#pragma unroll
                for (int k = 0; k < NK; ++k) acc = fma(band_w<T>(t.tab[0], k), Q[qi][k], acc);
            } else if (a == 0) {  // pstride[0] == 1
                const T* __restrict__ xp = M + coff + q + (1 - MID);
#pragma unroll
                for (int k = 0; k < NK; ++k) acc = fma(band_w<T>(t.tab[0], k), __ldg(xp + k), acc);
            } else {
                const T* __restrict__ yp = M + coff + q + (1 - MID) * ys;
#pragma unroll
                for (int k = 0; k < NK; ++k) acc = fma(band_w<T>(t.tab[0], k), __ldg(yp + k * ys), acc);
            }
            return acc;
        };
        if (KIND == DEO_VC_GRADIENT) {
#pragma unroll
            for (int a = 0; a < ND; ++a) {
                const T d = D(V.t[a], 0, a, 0);
                T* y = out + n + a * V.ovol;
                *y = overwrite ? zero_fix(d) : *y + d;
            }
        } else if (KIND == DEO_VC_DIVERGENCE) {
            T d[ND];
#pragma unroll
            for (int a = 0; a < ND; ++a) d[a] = D(V.t[a], a * V.pvol, a, 0);
            T acc = overwrite ? T(0) : out[n];
            bool first = overwrite != 0;  // 0 + x is x up to the sign of zero
#pragma unroll
            for (int p = 0; p < 3; ++p)
#pragma unroll
                for (int a = 0; a < ND; ++a)
                    if (ph[a] == p) {
                        acc = first ? zero_fix(d[a]) : acc + d[a];
                        first = false;
                    }
            out[n] = acc;
        } else {
            // x1: +D2 u3, -D3 u2 (queue 0);  x2: -D1 u3, +D3 u1 (queue 1);  x3: +D1 u2, -D2 u1
            const T x1a = D(V.t[1], 2 * V.pvol, 1, 0), x1b = D(V.tn[2], V.pvol, 2, 0);
            const T x2a = D(V.tn[0], 2 * V.pvol, 0, 0), x2b = D(V.t[2], 0, 2, NQ - 1);
            const T x3a = D(V.t[0], V.pvol, 0, 0), x3b = D(V.tn[1], 0, 1, 0);
            const T e1[3] = {x1a, x2a, x3a}, e2[3] = {x1b, x2b, x3b};
            constexpr int A1[3] = {1, 0, 0}, A2[3] = {2, 2, 1};
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                T* y = out + n + c * V.ovol;
                const bool in_order = ph[A1[c]] <= ph[A2[c]];
                const T f = in_order ? e1[c] : e2[c], g = in_order ? e2[c] : e1[c];
                *y = (overwrite ? zero_fix(f) : *y + f) + g;
            }
        }
    }
}

// The same methods for Float64 on a 3-D array whose operators share a uniform
// interior band of NK taps, in block fixed point (deo_bfp.cuh), marching along
// axis 3 as deo_march.cu does: CTA = 32 x 4 threads over 64 x 8 outputs, a
// thread 2 x 2 of them; each input component's plane (with the halo its own
// derivatives need) is converted once and read from a shared-memory ring -- NK +
// 1 planes for a component differentiated along axis 3, 2 for the others.  Points
// whose bound fails in some derivative (the larger of the two nearest taps below
// the threshold) are queued and evaluated by
// vc_point at the end of the unit; points on boundary rows are units of their own.
//
// A unit whose values are small against their block's goes on with the values themselves, each
// derivative on the largest exponent of its own taps and a quarter of the points in FP64 (see
// deo_march.cu): a Gaussian of width 0.1 / 0.05 of the box, us: k_vc / as it was without
// this / now: gradient 256^3, order 2 380 / 380 -> 411 / 619 -> 272 / 284, order 4 548 / 548 ->
// 531 / 853 -> 372 / 409, order 6 724 / 722 -> 922 / 1261 -> 580 / 607; 192^3, divergence
// order 4 242 / 243 -> 437 / 612 -> 263 / 276, order 6 316 / 316 -> 560 / 778 -> 338 / 356; curl
// order 2 322 / 323 -> 459 / 595 -> 281 / 279, order 4 466 / 466 -> 795 / 1114 -> 496 / 521 (a
// smooth field there 242 -> 191, 316 -> 254, 322 -> 207, 466 -> 353).  FP64 alone for these units:
// gradient, order 4, width 0.05, 597.
//
// What bounds it: instruction issue, 253 a gradient point (39 multiply-adds, 45 to
// load and convert 2.1 values, 39 to round and test three derivatives, the rest
// addressing and control) at 48 %.  256^3, 4th order, against the per-point
// FP64 kernel (15, 17 and 33 FP64 instructions a point at 2 per clock per SM):
// gradient 546 -> 257 us, divergence 553 -> 446, curl 1086 -> 888.  1 or 4 rows a
// thread 259 / 289 us; boundary points through the warps' queues instead of
// units of their own 376 (one warp drains a tile's whole boundary row).
template <int KIND, int NK>
struct VfCfg {
    static constexpr int NC = KIND == DEO_VC_GRADIENT ? 1 : 3;
    static constexpr int MID = NK / 2, LH = MID - 1, RH = MID + 1;  // taps o + 1 - MID .. o + 1 + MID
    static constexpr int PL = (LH + 1) / 2 * 2, PR = (RH + 1) / 2 * 2;  // x halo in whole pairs
    static constexpr int TYT = 4, RY = 2, NTHR = 32 * TYT, TY = TYT * RY;
    // does component c have a derivative along axis a
    __host__ __device__ static constexpr bool has(int c, int a) {
        return KIND == DEO_VC_GRADIENT ? true : (KIND == DEO_VC_DIVERGENCE ? c == a : c != a);
    }
    __host__ __device__ static constexpr int bx(int c) { return 64 + (has(c, 0) ? PL + PR : 0); }
    __host__ __device__ static constexpr int by(int c) { return TY + (has(c, 1) ? LH + RH : 0); }
    __host__ __device__ static constexpr int plane(int c) { return bx(c) * by(c); }
    __host__ __device__ static constexpr int nld(int c) { return (plane(c) + NTHR - 1) / NTHR; }
    __host__ __device__ static constexpr int slots(int c) { return has(c, 2) ? NK + 1 : 2; }
    __host__ __device__ static constexpr int base(int c) { return c == 0 ? 0 : base(c - 1) + slots(c - 1) * plane(c - 1); }
    static constexpr int QCAP = 1024;  // fallback points a warp can hold
    static constexpr int SMEM = base(NC) * 8 + TYT * QCAP * 2;
};

template <int C>
using Comp = std::integral_constant<int, C>;

template <int KIND, int NK, bool OW>
__global__ void __launch_bounds__(128, KIND == DEO_VC_GRADIENT ? 4 : 3)
    k_vc_fx(const __grid_constant__ VcDev V, const __grid_constant__ VcBfp B, const LapGrid g,
            const double* __restrict__ M, double* __restrict__ out) {
    using C = VfCfg<KIND, NK>;
    constexpr int MID = C::MID, RY = C::RY, NC = C::NC;
    extern __shared__ __align__(16) unsigned char smem[];
    Limbs* ring = reinterpret_cast<Limbs*>(smem);
    unsigned short* queue = reinterpret_cast<unsigned short*>(smem + C::base(NC) * 8) + threadIdx.y * C::QCAP;
    __shared__ unsigned s_max[NC][16];
    __shared__ int s_next;
    const int n0 = (int)V.len[0], n1 = (int)V.len[1], n2 = (int)V.len[2];
    const int px = n0 + 2, py = n1 + 2, bpc = V.bpc;
    const int64_t psz = (int64_t)px * py, osz = (int64_t)n0 * n1;
    const int tx = threadIdx.x, ty = threadIdx.y, tid = ty * 32 + tx;
    int nq = 0;
    __shared__ int s_nq[C::TYT];
    auto point = [&](int w, unsigned e, int x0, int y0, int z0) {  // a queued point of warp w
        vc_point<double, KIND, 3, NK>(V, M, out, OW, x0 + (int)(e & 63u), y0 + w * RY + (int)((e >> 6) & 3u),
                                      z0 + (int)(e >> 8));
    };
    auto drain = [&](int keep, int x0, int y0, int z0) {  // this warp's own, when its queue is nearly full
        while (nq > keep) {
            const int n = min(nq, 32);
            nq -= n;
            if (tx < n) point(ty, queue[nq + tx], x0, y0, z0);
            __syncwarp();
        }
    };
    // points with a boundary row: 1024 to a unit, before the others (axis 3's planes, then axis 2's rows and
    // axis 1's columns between them)
    const int iy = n1 - 2 * bpc, iz = n2 - 2 * bpc;
    const int64_t ez = (int64_t)2 * bpc * n0 * n1, ey = (int64_t)2 * bpc * n0 * iz, ex = (int64_t)2 * bpc * iy * iz;
    const int64_t etot = ez + ey + ex;
    auto out_of = [&](int i, int n) { return i < bpc ? i : n - 2 * bpc + i; };  // the i-th boundary row of n
    const int edge = (int)((etot + 1023) / 1024);
    for (int k = claim_next(g.sched, s_next); k < g.units + edge; k = claim_next(g.sched, s_next)) {
        if (k < edge) {
            for (int64_t i = (int64_t)k * 1024 + tid; i < min((int64_t)(k + 1) * 1024, etot); i += C::NTHR) {
                int64_t r = i;
                int x, y, z;
                if (r < ez) {
                    z = (int)(r / osz);
                    r -= z * osz;
                    y = (int)(r / n0);
                    x = (int)(r - (int64_t)y * n0);
                    z = out_of(z, n2);
                } else if ((r -= ez) < ey) {
                    const int64_t l = r / n0;
                    x = (int)(r - l * n0);
                    z = bpc + (int)(l / (2 * bpc));
                    y = out_of((int)(l % (2 * bpc)), n1);
                } else {
                    r -= ey;
                    const int64_t l = r / iy;
                    y = bpc + (int)(r - l * iy);
                    z = bpc + (int)(l / (2 * bpc));
                    x = out_of((int)(l % (2 * bpc)), n0);
                }
                vc_point<double, KIND, 3>(V, M, out, OW, x, y, z);
            }
            __syncthreads();  // s_next has been read by every thread
            continue;
        }
        const int unit = k - edge;
        const int txi = unit % g.tiles_x, rest = unit / g.tiles_x;
        const int tyi = rest % g.tiles_y, ci = rest / g.tiles_y;
        const int x0 = txi * 64, y0 = tyi * C::TY;
        const int z0 = bpc + ci * g.zc, z1 = min(z0 + g.zc, n2 - bpc);
        const int npl = z1 - z0 + 2 * MID;
        // the component's values this thread loads: byte offsets in a plane
        unsigned off[NC][C::nld(KIND == DEO_VC_DIVERGENCE ? 1 : NC - 1)];
        double raw[NC][C::nld(KIND == DEO_VC_DIVERGENCE ? 1 : NC - 1)];
        auto offsets = [&](auto cc) {
            constexpr int c = decltype(cc)::value, BX = C::bx(c);
#pragma unroll
            for (int j = 0; j < C::nld(c); ++j) {
                const int q = min(tid + j * C::NTHR, C::plane(c) - 1);
                const int r = q / BX, x = x0 + (q - r * BX) - (C::has(c, 0) ? C::PL : 0);
                const int y = y0 + r - (C::has(c, 1) ? C::LH : 0);
                off[c][j] = 8u * (unsigned)(min(max(y, 0), py - 1) * px + min(max(x, 0), px - 1));
            }
        };
        // the plane of component c that step p brings: o + 1 + MID for axis 3's window, else o itself
        auto load = [&](auto cc, int p) {
            constexpr int c = decltype(cc)::value;
            const char* s = reinterpret_cast<const char*>(M + c * V.pvol) +
                            (int64_t)(C::has(c, 2) ? z0 + 1 - MID + p : z0 + p - 2 * MID) * (psz * 8);
#pragma unroll
            for (int j = 0; j < C::nld(c); ++j) raw[c][j] = __ldg(reinterpret_cast<const double*>(s + off[c][j]));
        };
        int r6 = 0;  // p mod (NK + 1)
        auto slot = [&](auto cc, int p, int back) {  // of step p - back, back <= NK
            constexpr int c = decltype(cc)::value;
            const int i = C::has(c, 2) ? (r6 - back < 0 ? r6 - back + NK + 1 : r6 - back) : ((p - back) & 1);
            return ring + C::base(c) + i * C::plane(c);
        };
        unsigned probe[NC];  // keys of a value in the tile's middle rows, a plane ago
        unsigned skip = 0;   // outside the array (bit c)
        bool small = false;  // one of them is too small for its block's exponent
        auto put = [&](auto cc, int p, int back, int E) {
            constexpr int c = decltype(cc)::value;
            Limbs* w = slot(cc, p, back);
            unsigned mx = 0;
#pragma unroll
            for (int j = 0; j < C::nld(c); ++j) {
                const unsigned key = bfp_key(raw[c][j]);
                mx = max(mx, key);
                if (j == C::nld(c) / 2) {
                    small |= E > 64 && !((skip >> c) & 1u) && probe[c] < (unsigned)(max(E - B.gap, 1) << 20);  // (64: zeros)
                    probe[c] = key;
                }
                if (j + 1 < C::nld(c) || tid + j * C::NTHR < C::plane(c))
                    w[tid + j * C::NTHR] = bfp_convert(raw[c][j], key, E);
            }
            return mx;
        };
        auto each = [&](auto f) {
            f(Comp<0>{});
            if constexpr (NC == 3) {
                f(Comp<1>{});
                f(Comp<2>{});
            }
        };
        unsigned live = 0;  // own points: interior rows on both axes
#pragma unroll
        for (int b = 0; b < 2 * RY; ++b) {
            const int x = x0 + 2 * tx + (b & 1), y = y0 + ty * RY + b / 2;
            if (x >= bpc && x < n0 - bpc && y >= bpc && y < n1 - bpc) live |= 1u << b;
        }
        const bool all_live = live == (1u << (2 * RY)) - 1u;
        if (tid < 16)
#pragma unroll
            for (int c = 0; c < NC; ++c) s_max[c][tid] = 0;
        each([&](auto cc) {
            constexpr int c = decltype(cc)::value, BX = C::bx(c);
            offsets(cc);
            const int q = tid + C::nld(c) / 2 * C::NTHR, r = q / BX, x = x0 + (q - r * BX) - (C::has(c, 0) ? C::PL : 0);
            if (x < 0 || x >= px || y0 + r - (C::has(c, 1) ? C::LH : 0) >= py) skip |= 1u << c;
            if constexpr (C::has(c, 2)) load(cc, 0);
        });
        __syncthreads();
        int E[NC], low[NC], zeros[NC];
#pragma unroll
        for (int c = 0; c < NC; ++c) E[c] = 64, low[c] = 0, zeros[c] = 0, probe[c] = 0x7fffffffu;
        int crowd = 0;  // threads with a small value, over the last planes
        int p = 0;
        for (; p < npl; ++p, r6 = r6 == NK ? 0 : r6 + 1) {
            small = false;
            each([&](auto cc) {
                constexpr int c = decltype(cc)::value;
                if (C::has(c, 2) || p >= 2 * MID) {
                    const unsigned mx = __reduce_max_sync(0xffffffffu, put(cc, p, 0, E[c]));
                    if (tx == 0) atomicMax(&s_max[c][p & 15], mx);
                }
                if (p + 1 < npl && (C::has(c, 2) || p + 1 >= 2 * MID)) load(cc, p + 1);
                if (tid == 0) s_max[c][(p + 2) & 15] = 0;
            });
            crowd += __syncthreads_count(small) - crowd / 4;
            if (crowd > C::NTHR * 5 / 4) break;
            each([&](auto cc) {  // a new exponent: the planes in use again (as in deo_march.cu)
                constexpr int c = decltype(cc)::value, W = C::has(c, 2) ? NK : 1;
                if (!C::has(c, 2) && p < 2 * MID) return;
                const unsigned top = s_max[c][p & 15];
                const int ep = (int)(top >> 20);
                zeros[c] = top == 0 ? zeros[c] + 1 : 0;
                low[c] = ep < E[c] ? low[c] + 1 : 0;
                if (ep > E[c] || low[c] > W + 2) {
                    int ew = 64;
                    for (int b = 0; b < W && b <= p; ++b) ew = max(ew, (int)(s_max[c][(p - b) & 15] >> 20));
                    low[c] = 0;
                    if (ew != E[c]) {
                        E[c] = ew;
                        for (int b = min(W - 1, p); b >= 0; --b) {
                            load(cc, p - b);
                            put(cc, p, b, E[c]);
                        }
                        if (p + 1 < npl) load(cc, p + 1);
                        __syncthreads();
                    }
                }
            });
            if (p < 2 * MID) continue;
            const int z = z0 + p - 2 * MID;
            // a derivative of component c along axis a at the own points: its value and its distance
            // from its fallback
            auto taps = [&](auto cc, int a, const Limbs* t, double& d, int& far) {
                constexpr int c = decltype(cc)::value;
                BfpAcc s{0, 0, 0};
                s.cr = (long long)B.wd[a][0] * t[MID].h;
#pragma unroll
                for (int o = 1; o <= MID; ++o) {
                    bfp_mad(s, B.wh[a][o], B.wl[a][o], t[MID + o].h - t[MID - o].h, t[MID + o].l - t[MID - o].l);
                    if (NK >= 7) s.cr += (long long)B.wd[a][o] * t[MID - o].h;
                }
                d = bfp_double(bfp_total(s), (B.kbase[a] + E[c]) * (1 << 20));
                far = min(far, max(abs(t[MID - 1].h), abs(t[MID + 1].h)));
            };
            auto hl = [&](const int4& t, int w) { return w ? Limbs{t.z, t.w} : Limbs{t.x, t.y}; };
            double d[2 * RY][3 * (KIND == DEO_VC_CURL ? 2 : 1)];  // GRADIENT, DIVERGENCE: [a]; CURL: [2 c + (first, second)]
            int margin[2 * RY];  // below 0: some derivative's bound fails
#pragma unroll
            for (int b = 0; b < 2 * RY; ++b) margin[b] = INT_MAX;
            each([&](auto cc) {
                constexpr int c = decltype(cc)::value, BX = C::bx(c);
                const Limbs* pc = slot(cc, p, C::has(c, 2) ? MID + 1 : 0);
                const int own = (ty * RY + (C::has(c, 1) ? C::LH : 0)) * BX + (C::has(c, 0) ? C::PL : 0) + 2 * tx;
                bool special = E[c] >= 2047;
#pragma unroll
                for (int a = 0; a < 3; ++a) special |= C::has(c, a) && !bfp_range_ok(B.kbase[a] + E[c]);
                // none when everything in use is zero
                const int t0 = special ? INT_MAX : (zeros[c] >= (C::has(c, 2) ? NK : 1) ? 0 : B.t0);
                // where the derivative along axis a of this component goes
                auto place = [&](int a) {
                    // curl x1 = D2 u3 - D3 u2, x2 = -D1 u3 + D3 u1, x3 = D1 u2 - D2 u1
                    return KIND == DEO_VC_CURL ? (c == 2 ? (a == 1 ? 0 : 2) : (c == 1 ? (a == 2 ? 1 : 4) : (a == 2 ? 3 : 5)))
                                               : a;
                };
                int far[2 * RY];
#pragma unroll
                for (int b = 0; b < 2 * RY; ++b) far[b] = INT_MAX;
                if constexpr (C::has(c, 0)) {
#pragma unroll
                    for (int j = 0; j < RY; ++j) {
                        constexpr int NP = (C::PL + 2 + C::PR) / 2;
                        int4 xs[NP];
#pragma unroll
                        for (int m = 0; m < NP; ++m)
                            xs[m] = *reinterpret_cast<const int4*>(pc + own + j * BX - C::PL + 2 * m);
#pragma unroll
                        for (int v = 0; v < 2; ++v) {
                            Limbs t[NK];
#pragma unroll
                            for (int m = 0; m < NK; ++m) {
                                const int i = C::PL + v + 1 - MID + m;
                                t[m] = hl(xs[i >> 1], i & 1);
                            }
                            taps(cc, 0, t, d[2 * j + v][place(0)], far[2 * j + v]);
                        }
                    }
                }
                if constexpr (C::has(c, 1)) {
                    int4 yc[RY + 2 * MID];
#pragma unroll
                    for (int m = 0; m < RY + 2 * MID; ++m)
                        yc[m] = *reinterpret_cast<const int4*>(pc + own + (m + 1 - MID) * BX);
#pragma unroll
                    for (int b = 0; b < 2 * RY; ++b) {
                        Limbs t[NK];
#pragma unroll
                        for (int m = 0; m < NK; ++m) t[m] = hl(yc[b / 2 + m], b & 1);
                        taps(cc, 1, t, d[b][place(1)], far[b]);
                    }
                }
                if constexpr (C::has(c, 2)) {
#pragma unroll
                    for (int j = 0; j < RY; ++j) {
                        int4 zs[NK];
#pragma unroll
                        for (int m = 0; m < NK; ++m)
                            zs[m] = *reinterpret_cast<const int4*>(slot(cc, p, 2 * MID - m) + own + j * BX);
#pragma unroll
                        for (int v = 0; v < 2; ++v) {
                            Limbs t[NK];
#pragma unroll
                            for (int m = 0; m < NK; ++m) t[m] = hl(zs[m], v);
                            taps(cc, 2, t, d[2 * j + v][place(2)], far[2 * j + v]);
                        }
                    }
                }
#pragma unroll
                for (int b = 0; b < 2 * RY; ++b) margin[b] = min(margin[b], far[b] - t0);
            });
            const int64_t n = (int64_t)z * osz + (int64_t)(y0 + ty * RY) * n0 + x0 + 2 * tx;
            auto store = [&](int b) {
                double* y = out + n + (int64_t)(b / 2) * n0 + b % 2;
                if constexpr (KIND == DEO_VC_GRADIENT) {
#pragma unroll
                    for (int a = 0; a < 3; ++a) y[a * V.ovol] = OW ? d[b][a] : y[a * V.ovol] + d[b][a];
                } else if constexpr (KIND == DEO_VC_DIVERGENCE) {
                    *y = ((OW ? d[b][0] : *y + d[b][0]) + d[b][1]) + d[b][2];
                } else {
                    y[0] = (OW ? d[b][0] : y[0] + d[b][0]) - d[b][1];
                    y[V.ovol] = (OW ? -d[b][2] : y[V.ovol] - d[b][2]) + d[b][3];
                    y[2 * V.ovol] = (OW ? d[b][4] : y[2 * V.ovol] + d[b][4]) - d[b][5];
                }
            };
            int least = all_live ? 0 : -1;
#pragma unroll
            for (int b = 0; b < 2 * RY; ++b) least = min(least, margin[b]);
            if (__all_sync(0xffffffffu, least >= 0)) {
#pragma unroll
                for (int b = 0; b < 2 * RY; ++b) store(b);
            } else {
#pragma unroll
                for (int b = 0; b < 2 * RY; ++b) {
                    const bool on = (live >> b) & 1u, later = on && margin[b] < 0;
                    if (on && !later) store(b);
                    const unsigned bal = __ballot_sync(0xffffffffu, later);
                    if (later)
                        queue[nq + __popc(bal & ((1u << tx) - 1u))] =
                            (unsigned short)((unsigned)(p - 2 * MID) << 8 | (unsigned)(b / 2) << 6 | (unsigned)(2 * tx + b % 2));
                    nq += __popc(bal);
                }
                __syncwarp();
                if (nq > C::QCAP - 64 * RY) drain(31, x0, y0, z0);
            }
        }
        // The rest of a unit whose values are small against their block's (as in deo_march.cu), from plane
        // p on: the ring holds the values themselves, every derivative in the reference's order.
        if (p < npl) {
            auto keep = [&](auto cc, int back) {
                constexpr int c = decltype(cc)::value;
                Limbs* w = slot(cc, p, back);
#pragma unroll
                for (int j = 0; j < C::nld(c); ++j)
                    if (j + 1 < C::nld(c) || tid + j * C::NTHR < C::plane(c))
                        w[tid + j * C::NTHR] = Limbs{__double2hiint(raw[c][j]), __double2loint(raw[c][j])};
            };
            int f64 = 0;  // groups of 32 points that this warp evaluates in FP64 alone
            auto own_plane = [&] {
#pragma unroll 1
                for (int i = 0; i < 2 * RY; ++i) {  // lanes side by side in either half of the tile
                    const int cx = tx + 32 * (i & 1), cy = ty * RY + i / 2, x = x0 + cx, y = y0 + cy;
                    const bool on = x >= bpc && x < n0 - bpc && y >= bpc && y < n1 - bpc;
                    double* o = out + (int64_t)(z0 + p - 2 * MID) * osz + (int64_t)y * n0 + x;
                    auto word = [&](auto cc, auto aa, int k) {  // tap k of component c along axis a
                        constexpr int c = decltype(cc)::value, a = decltype(aa)::value, BX = C::bx(c);
                        const int at = (cy + (C::has(c, 1) ? C::LH : 0)) * BX + (C::has(c, 0) ? C::PL : 0) + cx;
                        if (a == 2) return slot(cc, p, 2 * MID - k)[at];
                        return slot(cc, p, C::has(c, 2) ? MID + 1 : 0)[at + (1 - MID + k) * (a == 0 ? 1 : BX)];
                    };
                    // a derivative in the reference's order
                    auto ref = [&](auto cc, auto aa) {
                        double acc = 0.0;
#pragma unroll
                        for (int k = 0; k < NK; ++k) {
                            const Limbs v = word(cc, aa, k);
                            acc = fma(band_w<double>(V.t[decltype(aa)::value].tab[0], k), __hiloint2double(v.h, v.l), acc);
                        }
                        return acc;
                    };
                    // and on the exponent of its own taps
                    const bool own_exp = f64 == 0 && i != ty;
                    bool ok = own_exp;
                    auto own = [&](auto cc, auto aa) {
                        constexpr int a = decltype(aa)::value;
                        Limbs t[NK];
                        unsigned mx = 0, lo = 0;
#pragma unroll
                        for (int k = 0; k < NK; ++k) {
                            t[k] = word(cc, aa, k);
                            mx = max(mx, (unsigned)t[k].h & 0x7fffffffu);
                            lo |= (unsigned)t[k].l;
                        }
                        const int e = (int)(mx >> 20), E = max(e, 64), kexp = B.kbase[a] - 1 + E;
                        BfpOwn s{0, 0, 0, 0};
                        s.lh = B.wd[a][0] * (bfp_shift(t[MID], E) >> 32);
                        int near = 0;
#pragma unroll
                        for (int d = 1; d <= MID; ++d) {
                            const long long r = bfp_shift(t[MID + d], E), l = bfp_shift(t[MID - d], E);
                            bfp_mad(s, B.wh[a][d], B.wl[a][d], r - l);
                            if (NK >= 7) s.lh += B.wd[a][d] * (l >> 32);
                            if (d == 1) near = max(abs((int)(r >> 30)), abs((int)(l >> 30)));
                        }
                        const long long sum = bfp_total(s);
                        const bool zero = (mx | lo) == 0;
                        ok = ok && (zero || (e >= 64 && e < 2047 && bfp_range_ok(kexp) &&
                                             (near >= B.t0 || abs((int)(sum >> 32)) >= BFP_OWN_LIMIT)));
                        return zero ? 0.0 : bfp_double(sum, kexp * (1 << 20));
                    };
                    using X = Comp<0>;
                    using Y = Comp<1>;
                    using Z = Comp<2>;
                    constexpr int ND = KIND == DEO_VC_CURL ? 6 : 3;
                    double d[ND] = {};  // curl: the terms of x1, x2, x3 in order, without their signs
                    auto all = [&](auto D) {
                        if constexpr (KIND == DEO_VC_CURL) {
                            d[0] = D(Z{}, Y{}), d[1] = D(Y{}, Z{}), d[2] = D(Z{}, X{});
                            d[3] = D(X{}, Z{}), d[4] = D(Y{}, X{}), d[5] = D(X{}, Y{});
                        } else if constexpr (KIND == DEO_VC_DIVERGENCE) {
                            d[0] = D(X{}, X{}), d[1] = D(Y{}, Y{}), d[2] = D(Z{}, Z{});
                        } else {
                            d[0] = D(X{}, X{}), d[1] = D(X{}, Y{}), d[2] = D(X{}, Z{});
                        }
                    };
                    if (own_exp) {
                        all(own);
                        if (__popc(__ballot_sync(0xffffffffu, !ok)) > 8) f64 = 33;
                    }
                    f64 = max(f64 - 1, 0);
                    if (!ok) all(ref);
                    if (!on) continue;
                    if constexpr (KIND == DEO_VC_GRADIENT) {
#pragma unroll
                        for (int c = 0; c < 3; ++c) o[c * V.ovol] = OW ? zero_fix(d[c]) : o[c * V.ovol] + d[c];
                    } else if constexpr (KIND == DEO_VC_DIVERGENCE) {
                        *o = ((OW ? zero_fix(d[0]) : *o + d[0]) + d[1]) + d[2];
                    } else {
#pragma unroll
                        for (int c = 0; c < 3; ++c) {
                            const double f = c == 1 ? -d[2] : d[2 * c], g = c == 1 ? d[3] : -d[2 * c + 1];
                            o[c * V.ovol] = (OW ? zero_fix(f) : o[c * V.ovol] + f) + g;
                        }
                    }
                }
            };
            auto in_use = [&](auto cc, int q) { return C::has(decltype(cc)::value, 2) || q >= 2 * MID; };
            each([&](auto cc) {
                if (in_use(cc, p))
                    for (int b = min(C::has(decltype(cc)::value, 2) ? 2 * MID : 0, p); b >= 0; --b) {
                        load(cc, p - b);
                        keep(cc, b);
                    }
                if (p + 1 < npl && in_use(cc, p + 1)) load(cc, p + 1);
            });
            while (true) {
                __syncthreads();
                if (p >= 2 * MID) own_plane();
                if (++p == npl) break;
                r6 = r6 == NK ? 0 : r6 + 1;
                each([&](auto cc) {
                    if (in_use(cc, p)) keep(cc, 0);
                    if (p + 1 < npl && in_use(cc, p + 1)) load(cc, p + 1);
                });
            }
        }
        // the queues, shared out over the CTA
        if (tx == 0) s_nq[ty] = nq;
        __syncthreads();
        nq = 0;
        for (int w = 0, i = tid; w < C::TYT; ++w) {
            for (; i < s_nq[w]; i += C::NTHR) point(w, (queue + (w - ty) * C::QCAP)[i], x0, y0, z0);
            i -= s_nq[w];
        }
        __syncthreads();  // the next unit reuses the ring, the queues and the exponents
    }
    claims_done(g.sched);
}

// The generic per-line methods (vector_calculus_convolutions.jl:1-170): any N,
// other axes read at index + 1, operators added in axis order.
template <typename T, int KIND>
__global__ void __launch_bounds__(256) k_vc_lines(const VcDev V, const T* __restrict__ M, T* __restrict__ out,
                                                  int overwrite) {
    const int64_t n = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= V.ovol) return;
    int64_t o[8];
    int64_t r = n, q = 0;
    for (int b = 0; b < V.nd; ++b) {
        o[b] = (b == V.nd - 1) ? r : r % V.len[b];
        r = (b == V.nd - 1) ? 0 : r / V.len[b];
        q += (o[b] + 1) * V.pstride[b];
    }
    if (KIND == DEO_VC_GRADIENT) {
        for (int a = 0; a < V.nd; ++a) {
            const T d = eval_term<T>(V.t[a], M, q, (int)o[a] + 1);
            T* y = out + n + a * V.ovol;
            *y = overwrite ? zero_fix(d) : *y + d;
        }
    } else {
        T acc = overwrite ? T(0) : out[n];
        for (int a = 0; a < V.nd; ++a) {
            const T d = eval_term<T>(V.t[a], M + a * V.pvol, q, (int)o[a] + 1);
            acc = (a == 0 && overwrite) ? zero_fix(d) : acc + d;
        }
        out[n] = acc;
    }
}

// L*M / mul!(x_temp, L, M; overwrite) on an already padded array M
// (derivative_operator_functions.jl:17-69, 150-163; convolutions.jl:17-22 for
// vectors): one thread per output point; its line along `axis` starts at the
// left ghost, other axes at the output index + off (1 where M is padded on that
// axis, so its edge planes are skipped; `coff` = sum of those offsets times the
// strides); the row from the operator's table (generic methods).
template <typename T>
__global__ void __launch_bounds__(256) k_padded(const VcDev V, int axis, int64_t coff, const T* __restrict__ M,
                                                T* __restrict__ out, int overwrite) {
    const int64_t n = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= V.ovol) return;
    int64_t r = n, ls = coff, oa = 0;
    for (int b = 0; b < V.nd; ++b) {
        const int64_t o = (b == V.nd - 1) ? r : r % V.len[b];
        r = (b == V.nd - 1) ? 0 : r / V.len[b];
        if (b == axis) oa = o;
        else ls += o * V.pstride[b];
    }
    const T d = eval_row_padded<T>(V.t[0].tab[0], M + ls, V.pstride[axis], (int)oa + 1);
    out[n] = overwrite ? zero_fix(d) : d + out[n];
}

// Products rounded before the sums (no contraction), as plain Julia code does.
template <typename T>
__device__ __forceinline__ T mul_rn(T a, T b);
template <>
__device__ __forceinline__ double mul_rn<double>(double a, double b) { return __dmul_rn(a, b); }
template <>
__device__ __forceinline__ float mul_rn<float>(float a, float b) { return __fmul_rn(a, b); }
template <typename T>
__device__ __forceinline__ T add_rn(T a, T b);
template <>
__device__ __forceinline__ double add_rn<double>(double a, double b) { return __dadd_rn(a, b); }
template <>
__device__ __forceinline__ float add_rn<float>(float a, float b) { return __fadd_rn(a, b); }
template <typename T>
__device__ __forceinline__ T sub_rn(T a, T b);
template <>
__device__ __forceinline__ double sub_rn<double>(double a, double b) { return __dsub_rn(a, b); }
template <>
__device__ __forceinline__ float sub_rn<float>(float a, float b) { return __fsub_rn(a, b); }

// dot_product! / square_norm! (vector_algebraic_operations.jl:11-28, :54-62)
template <typename T, bool NORM>
__global__ void __launch_bounds__(256) k_dot(int64_t npts, int ncomp, const T* __restrict__ A, const T* __restrict__ B,
                                             T* __restrict__ u) {
    const int64_t n = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= npts) return;
    T acc = T(0);
    for (int i = 0; i < ncomp; ++i) {
        const T a = A[n + i * npts];
        acc = add_rn(acc, mul_rn(a, NORM ? a : B[n + i * npts]));
    }
    u[n] = NORM ? sqrt(acc) : acc;
}

// cross_product! (vector_algebraic_operations.jl:39-52)
template <typename T>
__global__ void __launch_bounds__(256) k_cross(int64_t npts, const T* __restrict__ A, const T* __restrict__ B,
                                               T* __restrict__ u) {
    const int64_t n = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= npts) return;
    const T a1 = A[n], a2 = A[n + npts], a3 = A[n + 2 * npts];
    const T b1 = B[n], b2 = B[n + npts], b3 = B[n + 2 * npts];
    u[n] = sub_rn(mul_rn(a2, b3), mul_rn(a3, b2));
    u[n + npts] = sub_rn(mul_rn(a3, b1), mul_rn(a1, b3));
    u[n + 2 * npts] = sub_rn(mul_rn(a1, b2), mul_rn(a2, b1));
}

template <int KIND, int NK>
int resident_fx(int64_t& G) {
    using C = VfCfg<KIND, NK>;
    static PerDevice<int64_t> known;
    return occupancy_grid(known, C::NTHR, C::SMEM, G, k_vc_fx<KIND, NK, true>, k_vc_fx<KIND, NK, false>);
}

template <int KIND, int NK>
int launch_fx(const VcDev& V, const VcBfp& B, unsigned int* claims, const double* M, double* out, int ow, cudaStream_t st) {
    using C = VfCfg<KIND, NK>;
    int64_t G;
    const int e = resident_fx<KIND, NK>(G);
    if (e) return e;
    LapGrid g = march_grid(V.len[0], V.len[1], (int)V.len[2] - 2 * V.bpc, 64, C::TY, B.zc);
    g.sched = claims;
    const int grid = (int)std::min<int64_t>(G, g.units);
    auto go = [&](auto kernel) { kernel<<<grid, dim3(32, C::TYT), C::SMEM, st>>>(V, B, g, M, out); };
    if (ow) go(k_vc_fx<KIND, NK, true>);
    else go(k_vc_fx<KIND, NK, false>);
    return (int)cudaGetLastError();
}

template <int KIND>
int chunk_fx(const VcDev& V, int* zc) {
    auto find = [&](auto nk) {
        constexpr int NK = decltype(nk)::value;
        int64_t G;
        const int e = resident_fx<KIND, NK>(G);
        if (!e) *zc = march_zc(V.len[0], V.len[1], (int)V.len[2] - 2 * V.bpc, 64, VfCfg<KIND, NK>::TY, NK / 2, G);
        return e;
    };
    switch (V.band_nk) {
        case 3: return find(std::integral_constant<int, 3>{});
        case 5: return find(std::integral_constant<int, 5>{});
        case 7: return find(std::integral_constant<int, 7>{});
    }
    return 0;  // (9 taps: not this kernel)
}

template <typename T, int KIND, int ND>
int launch_tiled(const VcDev& V, const VcBfp* B, unsigned int* claims, const T* M, T* out, int ow, cudaStream_t st) {
    if constexpr (ND == 3 && std::is_same<T, double>::value)
        if (B) switch (V.band_nk) {
                case 3: return launch_fx<KIND, 3>(V, *B, claims, M, out, ow, st);
                case 5: return launch_fx<KIND, 5>(V, *B, claims, M, out, ow, st);
                case 7: return launch_fx<KIND, 7>(V, *B, claims, M, out, ow, st);
                default: break;
            }
    // marching kernel: columns x chunks of the last axis within the grid limits
    const int64_t nm = V.len[ND - 1];
    const int64_t ncol1 = ND == 3 ? (V.len[1] + 7) / 8 : 1;
    const int64_t ncols = (ND == 3 ? (V.len[0] + 31) / 32 : (V.len[0] + 255) / 256) * ncol1;
    // chunks of the march: short enough for many waves of blocks (the last wave's
    // idle SMs are the tail), long enough to amortise the queue's first fill
    int64_t zb = 4;
    while (zb < 32 && ncols * ((nm + 2 * zb - 1) / (2 * zb)) >= 8192) zb *= 2;
    while ((nm + zb - 1) / zb > 65535) zb *= 2;
    // (2-D Float64: the per-point row-table kernel keeps the FP64 pipe busier than this one)
    if (V.band_nk > 0 && ncol1 <= 65535 && !std::is_same<T, double>::value) {
        const unsigned chunks = (unsigned)((nm + zb - 1) / zb);
        const dim3 grid = ND == 3 ? dim3((unsigned)((V.len[0] + 31) / 32), (unsigned)ncol1, chunks)
                                  : dim3((unsigned)((V.len[0] + 255) / 256), chunks, 1);
        const int z = (int)zb;
        switch (V.band_nk) {
            case 3: k_vc_march<T, KIND, ND, 3><<<grid, 256, 0, st>>>(V, M, out, ow, z); return (int)cudaGetLastError();
            case 5: k_vc_march<T, KIND, ND, 5><<<grid, 256, 0, st>>>(V, M, out, ow, z); return (int)cudaGetLastError();
            case 7: k_vc_march<T, KIND, ND, 7><<<grid, 256, 0, st>>>(V, M, out, ow, z); return (int)cudaGetLastError();
            case 9: k_vc_march<T, KIND, ND, 9><<<grid, 256, 0, st>>>(V, M, out, ow, z); return (int)cudaGetLastError();
            default: break;
        }
    }
    const int64_t n2 = ND == 3 ? V.len[2] : 1;
    dim3 grid((unsigned)((V.len[0] + 31) / 32), (unsigned)std::min<int64_t>((V.len[1] + 7) / 8, 65535),
              (unsigned)std::min<int64_t>(n2, 65535));
    k_vc<T, KIND, ND><<<grid, 256, 0, st>>>(V, M, out, ow);
    return (int)cudaGetLastError();
}

template <typename T>
int launch_vc(const VcDev& V, const VcBfp* B, unsigned int* claims, const void* Mv, void* outv, int ow, cudaStream_t st) {
    const T* M = static_cast<const T*>(Mv);
    T* out = static_cast<T*>(outv);
    if (V.quirk && V.nd == 2) {
        if (V.kind == DEO_VC_GRADIENT) return launch_tiled<T, DEO_VC_GRADIENT, 2>(V, B, claims, M, out, ow, st);
        else return launch_tiled<T, DEO_VC_DIVERGENCE, 2>(V, B, claims, M, out, ow, st);
    } else if (V.quirk && V.nd == 3) {
        if (V.kind == DEO_VC_GRADIENT) return launch_tiled<T, DEO_VC_GRADIENT, 3>(V, B, claims, M, out, ow, st);
        else if (V.kind == DEO_VC_DIVERGENCE) return launch_tiled<T, DEO_VC_DIVERGENCE, 3>(V, B, claims, M, out, ow, st);
        else return launch_tiled<T, DEO_VC_CURL, 3>(V, B, claims, M, out, ow, st);
    } else {
        const unsigned blocks = (unsigned)((V.ovol + 255) / 256);
        if (V.kind == DEO_VC_GRADIENT) k_vc_lines<T, DEO_VC_GRADIENT><<<blocks, 256, 0, st>>>(V, M, out, ow);
        else k_vc_lines<T, DEO_VC_DIVERGENCE><<<blocks, 256, 0, st>>>(V, M, out, ow);
    }
    return (int)cudaGetLastError();
}

}  // namespace
}  // namespace deo

extern "C" int deo_k_vector_chunk(const deo::VcDev* V, int* zc) {
    return V->kind == DEO_VC_GRADIENT     ? deo::chunk_fx<DEO_VC_GRADIENT>(*V, zc)
           : V->kind == DEO_VC_DIVERGENCE ? deo::chunk_fx<DEO_VC_DIVERGENCE>(*V, zc)
                                          : deo::chunk_fx<DEO_VC_CURL>(*V, zc);
}

extern "C" int deo_k_vector_calculus(const deo::VcDev* V, const deo::VcBfp* B, unsigned int* claims, int dtype,
                                     const void* M, void* out, int overwrite, void* stream) {
    if (V->ovol <= 0) return 0;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    return dtype == 0 ? deo::launch_vc<double>(*V, B, claims, M, out, overwrite, st)
                      : deo::launch_vc<float>(*V, B, claims, M, out, overwrite, st);
}

extern "C" int deo_k_padded_apply(const deo::VcDev* V, int axis, int64_t coff, int dtype, const void* M, void* out,
                                  int overwrite, void* stream) {
    if (V->ovol <= 0) return 0;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const unsigned blocks = (unsigned)((V->ovol + 255) / 256);
    if (dtype == 0)
        deo::k_padded<double><<<blocks, 256, 0, st>>>(*V, axis, coff, (const double*)M, (double*)out, overwrite);
    else
        deo::k_padded<float><<<blocks, 256, 0, st>>>(*V, axis, coff, (const float*)M, (float*)out, overwrite);
    return (int)cudaGetLastError();
}

extern "C" int deo_k_vector_algebra(int op, int dtype, int64_t npts, int ncomp, const void* A, const void* B, void* u,
                                    void* stream) {
    if (npts <= 0) return 0;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const unsigned blocks = (unsigned)((npts + 255) / 256);
    if (dtype == 0) {
        const double *a = (const double*)A, *b = (const double*)B;
        if (op == 0) deo::k_dot<double, false><<<blocks, 256, 0, st>>>(npts, ncomp, a, b, (double*)u);
        else if (op == 1) deo::k_cross<double><<<blocks, 256, 0, st>>>(npts, a, b, (double*)u);
        else deo::k_dot<double, true><<<blocks, 256, 0, st>>>(npts, ncomp, a, a, (double*)u);
    } else {
        const float *a = (const float*)A, *b = (const float*)B;
        if (op == 0) deo::k_dot<float, false><<<blocks, 256, 0, st>>>(npts, ncomp, a, b, (float*)u);
        else if (op == 1) deo::k_cross<float><<<blocks, 256, 0, st>>>(npts, a, b, (float*)u);
        else deo::k_dot<float, true><<<blocks, 256, 0, st>>>(npts, ncomp, a, a, (float*)u);
    }
    return (int)cudaGetLastError();
}
