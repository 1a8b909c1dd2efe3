// deo_march.cu -- Float64 interior of a 3-D Laplacian-type plan in block fixed
// point (deo_bfp.cuh), marching along axis 3.
//
// CTA = 32 x TYT threads over a 64 x TYT*RY tile; a thread owns 2 consecutive x
// points on RY rows and marches through a chunk of planes.  Each plane of the
// tile plus its halo is loaded to registers two planes ahead (plain 8-byte
// loads, so any size and alignment; a halo position outside the array reads the
// nearest value inside, which no evaluated point uses), its largest exponent
// found on the way (one plane ahead), converted once to limbs on the block's
// exponent and put in a shared-memory ring of 2H + 2 planes, from which every
// tap is read, two points to a 16-byte load.  One barrier per plane: a slot is
// rewritten only after a barrier that follows its last reader.  When a plane
// exceeds the block's exponent, or the planes in use have all fallen two below
// it, the resident planes are converted again from global memory (rare, and
// uniform over the CTA).
//
// A point whose error bound fails (BfpMarch::Limit) is queued by its warp and
// evaluated in the reference's order, from global memory, 32 at a time at the
// end of the unit (draining as the queue passed 32 held every other warp at the
// plane's barrier: 8 us more at 256^3).  A plane with Inf/NaN, or with an exponent
// outside the range the scaled result needs, sends all its points there.
//
// Where many values are small against their block's largest (a pulse or a front of a few
// cells' width: a point below 1.7 % of the block fails its bound), every point would be
// summed twice.  Each thread compares one value of the tile's middle rows with the block's
// exponent (counted by the plane's barrier); when the count, decaying by a quarter a plane,
// passes 5/4 of the threads -- two planes of small values, or a third of the values for
// good -- the rest of the unit keeps the values themselves in the ring and evaluates each
// point on the largest exponent of its own taps, a warp's four groups of 32 points in turn
// three so and one in FP64, so that both pipes work; points that fail there too (far taps of
// a small weight alone) are evaluated in FP64 at once.  256^3, a Gaussian of width 0.1 / 0.05
// / 0.02 of the box, us: the per-point kernels before this one / as it was without this / now:
// order 2 206 / 206 / 208 -> 291 / 518 / 512 -> 180 / 192 / 211; order 4 281 / 280 / 292 ->
// 508 / 842 / 770 -> 269 / 293 / 332; order 6 610 / 610 / 676 -> 828 / 1236 / 1050 -> 445 /
// 497 / 843; three bands (256 x 240 x 200), order 4, 506 / 506 / 507 -> 461 / 708 / 622 -> 262 /
// 268 / 530.  The counting costs 2-3 % of a smooth field's time (order 4: 188 -> 194).  Evaluating
// the small units inside the plane loop cost every field 40 % (registers); all groups on own exponents 305 at
// width 0.05, order 4, half of them in FP64 361; limbs per tap, not per sum, 334; counted by
// atomics beside the largest key the kernel spilled (order 4 smooth 5-20 % more).  Positions
// outside the array are not counted: the copies of the edge filled half a narrow tile
// (73 x 93 x 221 74 -> 57 us).  Five CTAs an SM at order 2 with one band: width 0.05 211 -> 192.
//
// What bounds it (256^3, d2 a4, smooth field; start: the per-point fixed point,
// 270 us beside its shell): 164 us for the interior, 139 us of them without the 2.8 %
// of points in the reference's order.  139 instructions per point -- 20 32 x 32 ->
// 64-bit multiply-adds, about 35 to load and convert 1.6 values (halo and fill
// planes included), 16 to add neighbours and test, 12 to round -- at 45-59 % issue:
// with 12-24 warps per SM the multiply-add chains and the per-plane barrier show.
// Tiles of 64 x 16 with 4, 2 or 1 rows a thread (128, 256, 512 threads) measured
// 172-210 us, this 64 x 8 with 2 rows 164; a second rounding in integer arithmetic
// instead of the conversion and scale costs 17 us more.
#include <cuda_runtime.h>
#include <limits.h>
#include <stdint.h>

#include <algorithm>

#include "deo_bfp.cuh"
#include "deo_eval.cuh"
#include "deo_lap.cuh"

namespace deo {
namespace march {

template <int H, int TYT, int RY>
struct Cfg {
    static constexpr int TXT = 32, NTHR = TXT * TYT;
    static constexpr int TX = 64, TY = TYT * RY;
    static constexpr int HP = (H + 1) / 2 * 2;  // x halo in whole pairs (16-byte shared loads)
    static constexpr int BX = TX + 2 * HP, BY = TY + 2 * H;
    static constexpr int PLANE = BX * BY;
    static constexpr int NLD = (PLANE + NTHR - 1) / NTHR;  // values a thread loads per plane
    static constexpr int SLOTS = 2 * H + 2;
    static constexpr int QCAP = 1024 / TYT * 4;  // fallback points a warp can hold (>= 2 * 64 * RY)
    static constexpr int SLOT = PLANE;
    static constexpr int SMEM = SLOTS * SLOT * 8 + TYT * QCAP * 2;
    static_assert(RY <= 4 && QCAP >= 2 * 64 * RY, "a queued point is 8 bits of plane, 2 of row, 6 of x");
};

// One point in the reference's order, from global memory; zeros, which come in
// runs (beside a compact support), without FP64.
template <int H>
__device__ __forceinline__ double ref_point(const UniPlan& U, const double* __restrict__ u, int64_t idx, int64_t nx,
                                            int64_t sxy) {
    const int64_t st[3] = {1, nx, sxy};
    double v[3][2 * H + 1];
    unsigned any = 0;
#pragma unroll
    for (int t = 0; t < 3; ++t)
#pragma unroll
        for (int k = 0; k < 2 * H + 1; ++k) {
            v[t][k] = u[idx + (k - H) * st[t]];
            any |= bfp_key(v[t][k]);
        }
    double total = 0.0;
    if (__any_sync(__activemask(), any)) {
#pragma unroll
        for (int t = 0; t < 3; ++t) {
            double acc = 0.0;
#pragma unroll
            for (int k = 0; k < 2 * H + 1; ++k) acc = fma(U.t[t].w[k], v[t][k], acc);
            total = t == 0 ? acc : total + acc;
        }
    }
    return zero_fix(total);
}

template <int H, bool SH, bool OW, int TYT, int RY>
__global__ void __launch_bounds__(32 * TYT, H == 1 && SH ? 5 : 4) k_lap_fx(const __grid_constant__ UniPlan U,
                                                             const __grid_constant__ BfpMarch B, const LapGrid g,
                                                             const double* __restrict__ u, double* __restrict__ du, int pairs) {
    using C = Cfg<H, TYT, RY>;
    constexpr int NQ = 2 * H + 1, HL = C::HP / 2, S = C::SLOTS;
    extern __shared__ __align__(16) unsigned char smem[];
    Limbs* ring = reinterpret_cast<Limbs*>(smem);
    unsigned short* queue = reinterpret_cast<unsigned short*>(smem + S * C::SLOT * 8) + threadIdx.y * C::QCAP;
    __shared__ unsigned s_max[16];  // the largest key of plane p at p & 15
    __shared__ int s_next;
    const int nx = (int)U.n[0], ny = (int)U.n[1];
    const int64_t sxy = (int64_t)nx * ny;
    const int tx = threadIdx.x, ty = threadIdx.y, tid = ty * 32 + tx;
    const int own = (ty * RY + H) * C::BX + C::HP + 2 * tx;  // the first own row's pair inside a slot
    int nq = 0;  // this warp's queued points
    __shared__ int s_nq[TYT];
    auto point = [&](int w, unsigned e, int x0, int y0, int z0) {  // a queued point of warp w
        const int64_t idx = (int64_t)(z0 + (int)(e >> 8)) * sxy + (int64_t)(y0 + w * RY + (int)((e >> 6) & 3u)) * nx + x0 +
                            (int)(e & 63u);
        const double r = ref_point<H>(U, u, idx, nx, sxy);
        du[idx] = OW ? r : r + du[idx];
    };
    auto drain = [&](int keep, int x0, int y0, int z0) {  // this warp's own, when its queue is nearly full
        while (nq > keep) {
            const int n = min(nq, 32);
            nq -= n;
            if (tx < n) point(ty, queue[nq + tx], x0, y0, z0);
            __syncwarp();
        }
    };

    for (int unit = claim_next(g.sched, s_next); unit < g.units; unit = claim_next(g.sched, s_next)) {
        const int txi = unit % g.tiles_x, rest = unit / g.tiles_x;
        const int tyi = rest % g.tiles_y, ci = rest / g.tiles_y;
        const int x0 = txi * C::TX, y0 = tyi * C::TY;
        const int z0 = B.lo[2] + ci * g.zc, z1 = min(z0 + g.zc, B.hi[2] + 1);  // interior planes of this unit
        const int npl = z1 - z0 + 2 * H;
        unsigned off[C::NLD];  // byte offsets in a plane of the values this thread loads
#pragma unroll
        for (int j = 0; j < C::NLD; ++j) {
            const int q = min(tid + j * C::NTHR, C::PLANE - 1);
            const int r = q / C::BX, c = q - r * C::BX;
            off[j] = 8u * (unsigned)(min(max(y0 + r - H, 0), ny - 1) * nx + min(max(x0 + c - C::HP, 0), nx - 1));
        }
        unsigned live = 0;  // own points (row j, lane v: bit 2j + v) inside the box
#pragma unroll
        for (int j = 0; j < RY; ++j)
#pragma unroll
            for (int v = 0; v < 2; ++v) {
                const int x = x0 + 2 * tx + v, y = y0 + ty * RY + j;
                if (x >= B.lo[0] && x <= B.hi[0] && y >= B.lo[1] && y <= B.hi[1]) live |= 1u << (2 * j + v);
            }
        const bool all_live = live == (1u << (2 * RY)) - 1u;
        const char* up = reinterpret_cast<const char*>(u + (int64_t)(z0 - H) * sxy);
        char* dp = reinterpret_cast<char*>(du + (int64_t)(z0 - 2 * H) * sxy);  // plane p finishes plane p of this
        const unsigned dof = 8u * (unsigned)((y0 + ty * RY) * nx + x0 + 2 * tx);
        double raw[C::NLD];
        auto load = [&](int p) {
            const char* s = up + (int64_t)p * (sxy * 8);
#pragma unroll
            for (int j = 0; j < C::NLD; ++j) raw[j] = __ldg(reinterpret_cast<const double*>(s + off[j]));
        };
        unsigned probe = 0x7fffffffu;  // the key of this thread's value in the tile's middle rows, a plane ago
        const int pr = (tid + C::NLD / 2 * C::NTHR) / C::BX, pcol = x0 + tid + C::NLD / 2 * C::NTHR - pr * C::BX - C::HP;
        const int gap = pcol < 0 || pcol >= nx || y0 + pr - H >= ny ? 4096 : B.limit.gap;  // (none outside the array)
        bool small = false;            // that is too small for the block's exponent
        // the loaded plane on exponent E into a slot; its largest key
        auto put = [&](Limbs* w, int E) {
            unsigned mx = 0;
#pragma unroll
            for (int j = 0; j < C::NLD; ++j) {
                const unsigned key = bfp_key(raw[j]);
                mx = max(mx, key);
                if (j == C::NLD / 2) {
                    small = probe < (unsigned)(max(E - gap, 0) << 20);
                    probe = key;
                }
                if (j + 1 < C::NLD || tid + j * C::NTHR < C::PLANE) w[tid + j * C::NTHR] = bfp_convert(raw[j], key, E);
            }
            return mx;
        };
        if (tid < 16) s_max[tid] = 0;
        load(0);
        __syncthreads();
        int E = 64;
        int low = 0;           // planes since one last reached E
        int zeros = 0;         // planes since one last held anything but zeros
        int crowd = 0;         // small values of the last planes
        int sl = 0;            // ring slot of plane p
        int p = 0;
        for (; p < npl; ++p) {
            {
                const unsigned mx = __reduce_max_sync(0xffffffffu, put(ring + sl * C::SLOT, E));
                if (p + 1 < npl) load(p + 1);
                if (tx == 0) atomicMax(&s_max[p & 15], mx);
                if (tid == 0) s_max[(p + 2) & 15] = 0;
            }
            crowd += __syncthreads_count(small) - crowd / 4;
            const unsigned top = s_max[p & 15];
            const int ep = (int)(top >> 20);
            zeros = top == 0 ? zeros + 1 : 0;
            low = ep < E ? low + 1 : 0;
            if (top == 0) crowd = 0;
            if (crowd > C::NTHR * 5 / 4) break;
            if (ep > E || low > NQ + 2) {
                // a new exponent: the planes in use (this one included) again
                int ew = 64;
                for (int b = 0; b < NQ && b <= p; ++b) ew = max(ew, (int)(s_max[(p - b) & 15] >> 20));
                low = 0;
                if (ew != E) {
                    E = ew;
                    for (int b = min(NQ - 1, p); b >= 0; --b) {
                        load(p - b);
                        put(ring + (sl - b < 0 ? sl - b + S : sl - b) * C::SLOT, E);
                    }
                    if (p + 1 < npl) load(p + 1);
                    __syncthreads();
                }
            }
            const int cur = sl;
            sl = sl + 1 == S ? 0 : sl + 1;
            if (p < 2 * H) continue;
            const int kexp = B.kbase + E;
            // the threshold of this plane: none when everything in use is zero, out of reach when the exponent
            // rules fixed point out
            const bool special = E >= 2047 || !bfp_range_ok(kexp);
            const int t0 = special ? INT_MAX : (zeros >= NQ ? 0 : B.limit.t);
            const double scale = special ? 1.0 : bfp_pow2(kexp);
            const int4* pl[NQ];  // own pair of the first row in the planes z - H .. z + H
#pragma unroll
            for (int m = 0; m < NQ; ++m) {
                const int i = cur - (NQ - 1 - m);
                pl[m] = reinterpret_cast<const int4*>(ring + (i < 0 ? i + S : i) * C::SLOT + own);
            }
            int4 yc[RY + 2 * H];  // the centre plane's pair at rows -H .. RY - 1 + H
#pragma unroll
            for (int m = 0; m < RY + 2 * H; ++m) yc[m] = pl[H][(m - H) * (C::BX / 2)];
            char* dz = dp + (int64_t)p * (sxy * 8);
            double r[RY][2];
            int far[RY][2];  // distance of each point from its fallback, against t0
#pragma unroll
            for (int j = 0; j < RY; ++j) {
                int4 xs[2 * HL + 1], zs[NQ];
#pragma unroll
                for (int m = 0; m < 2 * HL + 1; ++m) xs[m] = m == HL ? yc[H + j] : pl[H][j * (C::BX / 2) + m - HL];
#pragma unroll
                for (int m = 0; m < NQ; ++m) zs[m] = m == H ? yc[H + j] : pl[m][j * (C::BX / 2)];
#pragma unroll
                for (int v = 0; v < 2; ++v) {
                    auto hl = [&](const int4& t, int w) { return w ? Limbs{t.z, t.w} : Limbs{t.x, t.y}; };
                    const Limbs c = hl(yc[H + j], v);
                    BfpAcc a{0, 0, 0};
                    bfp_mad(a, B.c0h, B.c0l, c.h, c.l);
                    int n1 = 0;  // the neighbours at +1
#pragma unroll
                    for (int o = 1; o <= H; ++o)
#pragma unroll
                        for (int sd = 0; sd < 2; ++sd) {
                            const int so = sd ? o : -o, xi = 2 * HL + v + so;
                            const Limbs X = hl(xs[xi >> 1], xi & 1), Y = hl(yc[H + j + so], v), Z = hl(zs[H + so], v);
                            if constexpr (SH) {
                                const int sh = X.h + Y.h + Z.h, sl3 = X.l + Y.l + Z.l;
                                bfp_mad(a, B.wh[0][H + so], B.wl[0][H + so], sh, sl3);
                                if (so == 1) n1 = sh;
                            } else {
                                bfp_mad(a, B.wh[0][H + so], B.wl[0][H + so], X.h, X.l);
                                bfp_mad(a, B.wh[1][H + so], B.wl[1][H + so], Y.h, Y.l);
                                bfp_mad(a, B.wh[2][H + so], B.wl[2][H + so], Z.h, Z.l);
                                if (so == 1) n1 = X.h;
                            }
                        }
                    r[j][v] = bfp_double(bfp_total(a), scale);
                    far[j][v] = max(abs(c.h) >> B.limit.sh0, abs(n1) >> B.limit.sh1);
                }
            }
            int nearest = INT_MAX;
#pragma unroll
            for (int j = 0; j < RY; ++j) nearest = min(nearest, min(far[j][0], far[j][1]));
            if (__all_sync(0xffffffffu, all_live && nearest >= t0)) {
#pragma unroll
                for (int j = 0; j < RY; ++j) {
                    double* d = reinterpret_cast<double*>(dz + (dof + 8u * (unsigned)(j * nx)));
                    if (pairs) {
                        double2* d2 = reinterpret_cast<double2*>(d);
                        if constexpr (OW) *d2 = make_double2(r[j][0], r[j][1]);
                        else *d2 = make_double2(r[j][0] + d2->x, r[j][1] + d2->y);
                    } else {
                        d[0] = OW ? r[j][0] : r[j][0] + d[0];
                        d[1] = OW ? r[j][1] : r[j][1] + d[1];
                    }
                }
            } else {
#pragma unroll
                for (int b = 0; b < 2 * RY; ++b) {
                    const bool on = (live >> b) & 1u, ok = far[b / 2][b % 2] >= t0;
                    if (on && ok) {
                        double* d = reinterpret_cast<double*>(dz + (dof + 8u * (unsigned)((b / 2) * nx + b % 2)));
                        *d = OW ? r[b / 2][b % 2] : r[b / 2][b % 2] + *d;
                    }
                    const unsigned bal = __ballot_sync(0xffffffffu, on && !ok);
                    if (on && !ok)
                        queue[nq + __popc(bal & ((1u << tx) - 1u))] =
                            (unsigned short)((unsigned)(p - 2 * H) << 8 | (unsigned)(b / 2) << 6 | (unsigned)(2 * tx + b % 2));
                    nq += __popc(bal);
                }
                __syncwarp();
                if (nq > C::QCAP - 64 * RY) drain(31, x0, y0, z0);
            }
        }
        int f64 = 0;  // groups of 32 points that this warp evaluates in FP64 alone
        auto own_plane = [&](int p) {
            constexpr int G = BFP_OWN[H];
            const Limbs* pl[NQ];  // the tile's origin in the planes z - H .. z + H
#pragma unroll
            for (int m = 0; m < NQ; ++m) pl[m] = ring + (p - 2 * H + m) % S * C::SLOT + H * C::BX + C::HP;
            double* dz = du + (int64_t)(z0 + p - 2 * H) * sxy;
#pragma unroll 1
            for (int i = 0; i < 2 * RY; ++i) {  // rows ty * RY + i / 2, lanes side by side in either half of the tile
                const int cx = tx + 32 * (i & 1), cy = ty * RY + i / 2, at = cy * C::BX + cx;
                auto word = [&](int a, int k) { return a == 0 ? pl[H][at + k - H] : (a == 1 ? pl[H][at + (k - H) * C::BX] : pl[k][at]); };
                auto value = [&](int a, int k) {
                    const Limbs b = word(a, k);
                    return __hiloint2double(b.h, b.l);
                };
                // (19 taps are read once more for the sum; kept in registers they spill)
                unsigned mx = 0;
                auto taps = [&](auto f) {
#pragma unroll
                    for (int a = 0; a < 3; ++a)
#pragma unroll
                        for (int k = 0; k < NQ; ++k)
                            if (a == 0 || k != H) f(word(a, k));
                };
                taps([&](Limbs b) { mx = max(mx, (unsigned)b.h & 0x7fffffffu); });
                if constexpr (H == 3) asm volatile("" ::: "memory");
                double r = 0.0;
                bool ok = false;
                if (__any_sync(0xffffffffu, mx == 0)) {  // zeros alone?
                    unsigned lo = 0;
                    taps([&](Limbs b) { lo |= (unsigned)b.l; });
                    ok = (mx | lo) == 0;
                }
                if (f64 == 0 && i != ty) {
                    const int e = (int)(mx >> 20), E = max(e, 64), kexp = B.kbase - 1 + E;
                    long long sum;
                    int cen = 0, near = 0;  // the centre and the neighbours at +1, in 2^30 units of limit's scale
                    if constexpr (SH) {
                        BfpOwn s{0, 0, 0, 0};
                        const long long c = bfp_shift(word(0, H), E);
                        bfp_mad(s, B.c0h, B.c0l, c);
                        cen = (int)(c >> 30);
#pragma unroll
                        for (int k = 0; k < NQ; ++k) {
                            if (k == H) continue;
                            const long long n = bfp_shift(word(0, k), E) + bfp_shift(word(1, k), E) + bfp_shift(word(2, k), E);
                            bfp_mad(s, B.wh[0][k], B.wl[0][k], n);
                            if (k == H + 1) near = (int)(n >> 32);
                        }
                        sum = bfp_total(s);
                    } else {
                        const Limbs c = bfp_nearest<G>(value(0, H), E);
                        BfpAcc s{0, 0, 0};
                        bfp_mad(s, B.c0h, B.c0l, c.h, c.l);
                        cen = c.h;
#pragma unroll
                        for (int a = 0; a < 3; ++a)
#pragma unroll
                            for (int k = 0; k < NQ; ++k) {
                                if (k == H) continue;
                                const Limbs x = bfp_nearest<G>(value(a, k), E);
                                bfp_mad(s, B.wh[a][k], B.wl[a][k], x.h, x.l);
                                if (a == 0 && k == H + 1) near = x.h;
                            }
                        sum = bfp_total_own<G>(s);
                    }
                    r = ok ? 0.0 : bfp_double(sum, kexp * (1 << 20));
                    ok = ok || (e >= 64 && e < 2047 && bfp_range_ok(kexp) &&
                                (B.own_any || max(abs(cen) >> B.limit.sh0, abs(near) >> B.limit.sh1) >= B.limit.t ||
                                 abs((int)(sum >> 32)) >= (SH ? BFP_OWN_LIMIT : bfp_own_limit(G))));
                    if (__popc(__ballot_sync(0xffffffffu, !ok)) > 8) f64 = 32;
                } else {
                    f64 = max(f64 - 1, 0);
                }
                if (__any_sync(0xffffffffu, !ok)) {  // the reference's order
                    double v = 0.0;
#pragma unroll
                    for (int a = 0; a < 3; ++a) {
                        double acc = 0.0;
#pragma unroll
                        for (int k = 0; k < NQ; ++k) acc = fma(U.t[a].w[k], value(a, k), acc);
                        v = a == 0 ? acc : v + acc;
                    }
                    if (!ok) r = zero_fix(v);
                }
                const int x = x0 + cx, y = y0 + cy;
                if (x >= B.lo[0] && x <= B.hi[0] && y >= B.lo[1] && y <= B.hi[1]) {
                    double* d = dz + (int64_t)y * nx + x;
                    *d = OW ? r : r + *d;
                }
            }
        };
        // The rest of a unit whose values are small against their block's, from plane p on: the
        // ring holds the values themselves, and every point is evaluated on its own exponent.
        if (p < npl) {
            auto keep = [&](int q) {
                Limbs* w = ring + q % S * C::SLOT;
#pragma unroll
                for (int j = 0; j < C::NLD; ++j)
                    if (j + 1 < C::NLD || tid + j * C::NTHR < C::PLANE)
                        w[tid + j * C::NTHR] = Limbs{__double2hiint(raw[j]), __double2loint(raw[j])};
            };
            for (int b = min(2 * H, p); b > 0; --b) {
                load(p - b);
                keep(p - b);
            }
            load(p);
            for (; p < npl; ++p) {
                keep(p);
                if (p + 1 < npl) load(p + 1);
                __syncthreads();
                if (p < 2 * H) continue;
                own_plane(p);
            }
        }
        // the queues, shared out over the CTA
        if (tx == 0) s_nq[ty] = nq;
        __syncthreads();
        nq = 0;
        for (int w = 0, i = tid; w < TYT; ++w) {
            for (; i < s_nq[w]; i += C::NTHR) point(w, (queue + (w - ty) * C::QCAP)[i], x0, y0, z0);
            i -= s_nq[w];
        }
        __syncthreads();  // the next unit reuses the ring, the queues and the exponents
    }
    claims_done(g.sched);
}

}  // namespace march
}  // namespace deo

using namespace deo;

namespace {

template <int H, bool SH, int TYT = 4, int RY = 2>
struct Kernel {
    using C = march::Cfg<H, TYT, RY>;
    static int resident(int64_t& G) {
        static PerDevice<int64_t> known;
        return occupancy_grid(known, C::NTHR, C::SMEM, G, march::k_lap_fx<H, SH, true, TYT, RY>,
                              march::k_lap_fx<H, SH, false, TYT, RY>);
    }
    static int chunk(const UniPlan* up, int planes, int* zc) {
        int64_t G;
        const int e = resident(G);
        if (!e) *zc = march_zc(up->n[0], up->n[1], planes, C::TX, C::TY, H, G);
        return e;
    }
    static int launch(const UniPlan* up, const BfpMarch* B, unsigned int* sched, const void* u, void* du, int ow,
                      cudaStream_t st) {
        int64_t G;
        const int e = resident(G);
        if (e) return e;
        LapGrid g = march_grid(up->n[0], up->n[1], B->hi[2] - B->lo[2] + 1, C::TX, C::TY, B->zc);
        g.sched = sched;
        const int grid = (int)std::min<int64_t>(G, g.units);
        const int pairs = up->n[0] % 2 == 0 && (uintptr_t)du % 16 == 0;  // 16-byte stores
        auto go = [&](auto kernel) {
            kernel<<<grid, dim3(32, TYT), C::SMEM, st>>>(*up, *B, g, (const double*)u, (double*)du, pairs);
        };
        if (ow) go(march::k_lap_fx<H, SH, true, TYT, RY>);
        else go(march::k_lap_fx<H, SH, false, TYT, RY>);
        return (int)cudaGetLastError();
    }
};

// f(the kernel of a plan's radius and bands)
template <typename F>
int pick(const UniPlan* up, const BfpMarch* B, F f) {
    switch (up->radius) {
        case 1: return B->shared ? f(Kernel<1, true>{}) : f(Kernel<1, false>{});
        case 2: return B->shared ? f(Kernel<2, true>{}) : f(Kernel<2, false>{});
        case 3: return B->shared ? f(Kernel<3, true>{}) : f(Kernel<3, false>{});
    }
    return (int)cudaErrorNotSupported;
}

}  // namespace

extern "C" int deo_k_march_chunk(const UniPlan* up, const BfpMarch* B, int planes, int* zc) {
    return planes < 1 ? 0 : pick(up, B, [&](auto k) { return k.chunk(up, planes, zc); });
}

extern "C" int deo_k_apply_march(const UniPlan* up, const BfpMarch* B, unsigned int* sched, const void* u, void* du,
                                 int overwrite, void* stream) {
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    for (int a = 0; a < 3; ++a)
        if (B->lo[a] > B->hi[a]) return 0;  // no interior point
    return pick(up, B, [&](auto k) { return k.launch(up, B, sched, u, du, overwrite, st); });
}
