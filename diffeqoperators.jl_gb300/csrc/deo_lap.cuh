// deo_lap.cuh -- the work units of the TMA-fed Laplacian-type kernels
// (deo_tma.cu, deo_vec.cu): a persistent grid walks units of (tile x, tile y,
// z chunk), claimed from a device counter; the host picks the z chunk and
// the grid size.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "deo_internal.h"
#include "deo_once.h"

namespace deo {

// Work unit u = (tile x, tile y, z chunk); a persistent grid of G CTAs takes
// units b, b + G, b + 2G, ... (static, so one plan may run on several streams
// at once).  Planes stream through the ring with a running count, so slot and
// mbarrier phase carry over from one unit to the next.
struct LapGrid {
    int tiles_x, tiles_y, chunks, zc;
    int units;
    int perm;  // coprime with units: unit k of the round-robin is (k * perm) % units,
               // so one CTA's units are spread over tile columns and z chunks
    unsigned int* sched;  // null: static round-robin; else a zeroed device counter the CTAs claim units from
};

// The next unit of a CTA: with g.sched claimed from the counter (dynamic, so
// CTAs that share their SM with other work take fewer units), else k_static.
// Every thread of the CTA calls it (it contains a barrier).
__device__ __forceinline__ int claim_unit(const LapGrid& g, int& s_next, int k_static) {
    if (!g.sched) return k_static;
    if (threadIdx.x == 0 && threadIdx.y == 0) s_next = (int)atomicAdd(g.sched, 1u);
    __syncthreads();
    return s_next;
}

// The marching and batched kernels' claims: counter[0] the next unit, counter[1] the CTAs
// that have left; the last to leave zeroes both, so a launch needs no memset before it
// (a memset node costs about 2 us of a short apply).  It zeroes the other pair of its
// block of four words too, whose turn comes half a rotation later (ClaimSlots): launches
// that overlapped on one pair, against the rules, leave no pair wrong for good.
__device__ __forceinline__ int claim_next(unsigned int* counter, int& s_next) {
    if (threadIdx.x == 0 && threadIdx.y == 0) s_next = (int)atomicAdd(counter, 1u);
    __syncthreads();
    return s_next;
}
__device__ __forceinline__ void claims_done(unsigned int* counter) {
    if (threadIdx.x == 0 && threadIdx.y == 0) {
        __threadfence();
        if (atomicAdd(counter + 1, 1u) == gridDim.x - 1) {  // every CTA has made its last claim
            *reinterpret_cast<uint2*>(counter) = make_uint2(0u, 0u);
            *reinterpret_cast<uint2*>(reinterpret_cast<uintptr_t>(counter) ^ 8) = make_uint2(0u, 0u);
        }
    }
}

// Units and z chunk for a persistent grid of G CTAs (see LapGrid).
static inline LapGrid make_grid(const UniPlan* up, int tx, int ty, int H, int nt, int64_t G) {
    const int64_t nx = up->n[0], ny = up->n[1], nz = up->n[2];
    LapGrid g;
    g.tiles_x = (int)((nx + tx - 1) / tx);
    g.tiles_y = (int)((ny + ty - 1) / ty);
    const int64_t tiles = (int64_t)g.tiles_x * g.tiles_y;
    g.zc = (int)nz;
    if (nt == 3) {
        double best = -1.0;
        const int zmin = (int)std::min<int64_t>(nz, 12);
        for (int zc = zmin; zc <= nz; ++zc) {
            const int64_t chunks = (nz + zc - 1) / zc;
            const int64_t units = tiles * chunks;
            const int64_t rounds = (units + G - 1) / G;
            const double eff = (double)units / (double)(rounds * G) * (double)zc / (double)(zc + 2 * H) *
                               ((double)nz / (double)(chunks * zc));
            if (eff > best + 1e-9) {
                best = eff;
                g.zc = zc;
            }
        }
    }
    g.chunks = (int)((nz + g.zc - 1) / g.zc);
    g.units = (int)(tiles * g.chunks);
    g.sched = nullptr;
    g.perm = 1;
    for (int cand : {7919, 6007, 4099, 2053, 1031, 521, 263, 131, 67, 37, 17}) {
        int a = cand, b = g.units;
        while (b) {
            const int t = a % b;
            a = b;
            b = t;
        }
        if (a == 1 && cand < g.units) {
            g.perm = cand;
            break;
        }
    }
    return g;
}

// The chunk of nz planes of the marching block fixed-point kernels, whose units of (tile,
// chunk) G resident CTAs share out.  A unit of zc planes costs about
// zc + 0.4 * 2H + 3 planes (the planes that only fill the ring are converted, not
// evaluated), and the last round leaves about a third of a unit idle.  A queued
// point holds its plane in 8 bits, so zc <= 256.  Searched once, when a plan is made.
static inline int march_zc(int64_t nx, int64_t ny, int nz, int tx, int ty, int H, int64_t G) {
    const int64_t tiles = ((nx + tx - 1) / tx) * ((ny + ty - 1) / ty);
    int found = 1;
    double best = 1e300;
    for (int c = (nz + 255) / 256, zc; c <= nz; c = (nz + zc - 2) / (zc - 1)) {  // (the next shorter chunk)
        zc = (nz + c - 1) / c;
        const double rounds = std::max(1.0, (double)(tiles * ((nz + zc - 1) / zc)) / (double)G + 0.35);
        const double t = rounds * (zc + 0.8 * H + 3.0);
        if (t < best) {
            best = t;
            found = zc;
        }
        if (zc <= 4) break;
    }
    return found;
}
static inline LapGrid march_grid(int64_t nx, int64_t ny, int nz, int tx, int ty, int zc) {
    LapGrid g{};
    g.tiles_x = (int)((nx + tx - 1) / tx);
    g.tiles_y = (int)((ny + ty - 1) / ty);
    g.zc = zc;
    g.chunks = (nz + zc - 1) / zc;
    g.units = (int)((int64_t)g.tiles_x * g.tiles_y * g.chunks);
    g.perm = 1;
    return g;
}

// The resident grid of a kernel's instantiations, which run with one grid (that of the
// last), found once per device: `known` is a static of the launcher.
template <typename... K>
static inline int occupancy_grid(PerDevice<int64_t>& known, int threads, int smem, int64_t& G, K... kernels) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return (int)e;
    return known.get(dev, G, [&](int64_t& grid) {
        auto one = [&](auto kernel) {
            int sms = 0, per_sm = 0;
            cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
            cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
            // the largest shared-memory carveout: an SM configured for the interior's CTAs alone would leave
            // no room for the boundary-shell CTAs that run beside them
            if (e == cudaSuccess)
                e = cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout,
                                         (int)cudaSharedmemCarveoutMaxShared);
            if (e != cudaSuccess) return (int)e;
            e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem);
            if (e != cudaSuccess || per_sm < 1) per_sm = 1;
            grid = (int64_t)sms * per_sm;
            return 0;
        };
        int err = 0;
        ((err = err ? err : one(kernels)), ...);
        return err;
    });
}


}  // namespace deo
