// deo_kernels.cu -- sm_103a kernels of the stencil-apply path.
//
// The forward evaluator computes, for output point `idx` and each term t,
//     r_t = sum_k W_i[k] * x[p0_i + k]      (row table, see deo_internal.h)
// with the ghost values x[1], x[len+2] produced in-kernel from the boundary
// condition's affine map; then du = ((r_0 + r_1) + r_2) ... as the
// reference's `sum(op -> op*u, ops)` does.  Nothing is materialised: the
// ghost fill, the boundary rows and the interior stencil are one pass.
//
// The adjoint evaluator computes ubar = A_l^T dbar by gathering, for every
// padded column p, the rows whose window covers p (deterministic, no atomics),
// then folding the ghost columns back through the affine map.
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

#include <algorithm>

#include "deo_eval.cuh"
#include "deo_lap.cuh"

namespace deo {

// The forward evaluator without per-line BCs is held to the 32 registers of a full
// SM (eight CTAs, 64 warps) with a few hundred bytes of spills: its chains wait on
// loads and, in Float64, on the FP64 pipe, and the extra warps cover that.  2048^2,
// order 2: Float64 62 us against 66 with five CTAs and 72 with four; Float32 27
// against 31 (six) and 39 (four).
template <typename T, bool ADJ, bool LBC>
__global__ void __launch_bounds__(256, !ADJ && !LBC ? 8 : 0)
    k_apply(const __grid_constant__ PlanDev P, const T* __restrict__ u, T* __restrict__ du, int overwrite) {
    const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= P.total) return;
    const T r = eval_point<T, ADJ, LBC, true>(P, u, idx);
    du[idx] = overwrite ? r : r + du[idx];
}

// Persistent batched kernel: CTAs pull work items from a global counter until
// the list is exhausted (no waiting on other CTAs, so no spin loops).
// The instance's plan is staged into shared memory when a work item belongs to
// a different instance than the previous one (items are instance-contiguous
// within a size class, so consecutive pulls usually share it): the header, the
// plan's own terms and, when it has one, its star, not the whole 8-term struct.
// The next item is claimed while the current one is evaluated (its atomic's
// latency is covered), one barrier pair per item.  The counters are those of
// claims_done (deo_lap.cuh).  Each work item is claimed in
// 1 << lsplit parts of a multiple of 256 points (split_for).
struct PlanCache {
    static_assert(sizeof(PlanDev) % 8 == 0 && offsetof(PlanDev, t) % 8 == 0 && sizeof(TermDev) % 8 == 0 &&
                      offsetof(PlanDev, star) % 8 == 0,
                  "PlanDev copied in 8-byte words");
    unsigned long long words[sizeof(PlanDev) / 8];
};

__device__ __forceinline__ void stage_words(PlanCache& c, const PlanDev* p, size_t from, size_t to) {
    const unsigned long long* s = reinterpret_cast<const unsigned long long*>(p);
    for (int q = (int)(from / 8) + threadIdx.x; q < (int)(to / 8); q += blockDim.x) c.words[q] = s[q];
}

__device__ __forceinline__ void stage_plan(PlanCache& c, const PlanDev* p) {
    const int nt = p->nterms;  // uniform
    stage_words(c, p, 0, offsetof(PlanDev, t) + nt * sizeof(TermDev));
    stage_words(c, p, offsetof(PlanDev, star), p->star.n ? sizeof(PlanDev) : offsetof(PlanDev, star) + 8);
}

// The work-list walk shared by k_batch and k_stage: plan_of(w) names the plan
// of work item w, body(w, plan, q0, q1) evaluates its points q0 .. q1 - 1.
template <typename PlanOf, typename Body>
__device__ __forceinline__ void walk_items(const WorkItem* __restrict__ items, int64_t n_items, int lsplit,
                                           unsigned int* counter, PlanOf plan_of, Body body) {
    __shared__ unsigned int s_item[2];
    __shared__ __align__(16) PlanCache cache;
    if (threadIdx.x == 0) s_item[0] = atomicAdd(counter, 1u);
    __syncthreads();
    const PlanDev* cur = nullptr;
    int ph = 0;
    for (;;) {
        const int64_t it = s_item[ph];
        if (it >= n_items << lsplit) break;
        if (threadIdx.x == 0) s_item[ph ^ 1] = atomicAdd(counter, 1u);
        const WorkItem w = items[it >> lsplit];
        const int part = ((w.count - 1) >> (lsplit + 8)) * 256 + 256;  // ceil(count / split) to a multiple of 256
        const int q0 = ((int)it & ((1 << lsplit) - 1)) * part;
        const PlanDev* p = plan_of(w);
        if (p != cur) {  // uniform across the CTA
            stage_plan(cache, p);
            cur = p;
            __syncthreads();
        }
        body(w, *reinterpret_cast<const PlanDev*>(cache.words), q0, min(q0 + part, w.count));
        __syncthreads();  // every thread is done with the plan and has seen this item; the next claim is visible
        ph ^= 1;
    }
    claims_done(counter);
}

template <typename T, bool ADJ, bool LBC>
__global__ void __launch_bounds__(256) k_batch(const InstDev* __restrict__ inst, const WorkItem* __restrict__ items,
                                               int64_t n_items, int lsplit, unsigned int* counter) {
    walk_items(
        items, n_items, lsplit, counter, [&](const WorkItem& w) { return inst[w.inst].plan; },
        [&](const WorkItem& w, const PlanDev& P, int q0, int q1) {
            const InstDev in = inst[w.inst];
            const T* __restrict__ u = reinterpret_cast<const T*>(in.u);
            T* __restrict__ du = reinterpret_cast<T*>(in.du);
            for (int q = q0 + threadIdx.x; q < q1; q += blockDim.x) {
                const int64_t idx = w.start + q;
                du[idx] = eval_point<T, ADJ, LBC>(P, u, idx);
            }
        });
}

// Batched Runge-Kutta stage: same work-list scheme; each instance may run
// the forward operator or its adjoint (uniform per work item).
template <typename T, bool LBC>
__global__ void __launch_bounds__(256) k_stage(const StageDev* __restrict__ st, const WorkItem* __restrict__ items,
                                               int64_t n_items, int lsplit, unsigned int* counter) {
    walk_items(
        items, n_items, lsplit, counter, [&](const WorkItem& w) { return st[w.inst].plan; },
        [&](const WorkItem& w, const PlanDev& P, int q0, int q1) {
            const StageDev S = st[w.inst];
            const T* a = reinterpret_cast<const T*>(S.a);  // may alias out
            const T* b = reinterpret_cast<const T*>(S.b);
            const T* __restrict__ c = reinterpret_cast<const T*>(S.c);
            T* out = reinterpret_cast<T*>(S.out);
            const T al = T(S.alpha), be = T(S.beta), ga = T(S.gamma), dt = T(S.dt);
            for (int q = q0 + threadIdx.x; q < q1; q += blockDim.x) {
                const int64_t idx = w.start + q;
                const T f = S.adjoint ? eval_point<T, true, LBC>(P, c, idx) : eval_point<T, false, LBC>(P, c, idx);
                const T t = fma(dt, f, c[idx]);
                T acc = a ? al * a[idx] : T(0);
                if (b) acc = fma(be, b[idx], acc);
                out[idx] = fma(ga, t, acc);
            }
        });
}

// A stage of a single instance: the plan in the launch's parameters and a plain grid,
// two points a thread, five CTAs a SM.  The work-list kernel spends a third of such a
// stage on the claim, the list and the staged plan, each a trip to L2 before the first
// point, and its 64 registers leave half of the warps that hide the points' own
// loads.  768 x 500 Float64, 3 terms: 26 -> 16 us a stage; 100 x 50: 9 -> 6.7.
// (One point a thread with six CTAs the same; four CTAs 22.)
constexpr int STAGE_PT = 2;
template <typename T, bool ADJ, bool LBC>
__global__ void __launch_bounds__(256, 5)
    k_stage_one(const __grid_constant__ PlanDev P, const __grid_constant__ StageDev S) {
    const T* a = reinterpret_cast<const T*>(S.a);  // may alias out
    const T* b = reinterpret_cast<const T*>(S.b);
    const T* __restrict__ c = reinterpret_cast<const T*>(S.c);
    T* out = reinterpret_cast<T*>(S.out);
    const T al = T(S.alpha), be = T(S.beta), ga = T(S.gamma), dt = T(S.dt);
#pragma unroll 1
    for (int m = 0; m < STAGE_PT; ++m) {
        const int64_t idx = ((int64_t)blockIdx.x * STAGE_PT + m) * 256 + threadIdx.x;
        if (idx >= P.total) return;
        const T f = eval_point<T, ADJ, LBC>(P, c, idx);
        const T t = fma(dt, f, c[idx]);
        T acc = a ? al * a[idx] : T(0);
        if (b) acc = fma(be, b[idx], acc);
        out[idx] = fma(ga, t, acc);
    }
}

}  // namespace deo

using namespace deo;

// nonlinear_diffusion!{N}(du, n, m, approx, p, q, dx, len) on padded vectors
// (derivative_operator.jl:34-66): with D_k the order-k centred operator (plan
// term k-1) applied to a padded vector by the generic method,
//   du = (D_m q) .* (D_n p)            (m > 0)   or   q[2:len+1] .* (D_n p)   (m == 0)
//   du = du .+ binomial(n, l) * (D_{l+m} q) .* (D_{n-l} p),   l = 1 .. n-1
//   du = du .+ (D_{m+n} q) .* p[2:len+1]
// each broadcast in the reference's operation order, one thread per point.
template <typename T>
__global__ void __launch_bounds__(256) k_nld(const PlanDev P, int len, int n, int m, const T* __restrict__ p,
                                             const T* __restrict__ q, T* __restrict__ du) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= len) return;
    // the vectors hold their own ghosts: row i + 1 of D_k over x[0 .. len + 1]
    auto D = [&](int k, const T* x) { return eval_row_padded<T>(P.t[k - 1].tab[0], x, 1, i + 1); };
    T acc = (m > 0 ? D(m, q) : q[i + 1]) * D(n, p);
    long long b = 1;  // binomial(n, l)
    for (int l = 1; l <= n - 1; ++l) {
        b = b * (n - l + 1) / l;
        acc = acc + (T(b) * D(l + m, q)) * D(n - l, p);
    }
    acc = acc + D(m + n, q) * p[i + 1];
    du[i] = acc;
}

extern "C" int deo_k_nonlinear_diffusion(const PlanDev* plan, int len, int n, int m, int dtype, const void* p,
                                         const void* q, void* du, void* stream) {
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const unsigned blocks = (unsigned)((len + 255) / 256);
    if (dtype == 0)
        k_nld<double><<<blocks, 256, 0, st>>>(*plan, len, n, m, (const double*)p, (const double*)q, (double*)du);
    else
        k_nld<float><<<blocks, 256, 0, st>>>(*plan, len, n, m, (const float*)p, (const float*)q, (float*)du);
    return (int)cudaGetLastError();
}

extern "C" int deo_k_num_sms(void);

template <typename T>
__global__ void __launch_bounds__(256) k_scale(T* __restrict__ x, int64_t n, T f) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        x[i] = f * x[i];
}

// x *= f over n points of the dtype (the adjoint seed 2 u(T) of ||u(T)||^2).
extern "C" int deo_k_scale(void* x, int64_t n, int dtype, double f, void* stream) {
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const int sms = deo_k_num_sms();
    const int64_t want = (n + 255) / 256;
    const unsigned blocks = (unsigned)std::max<int64_t>(1, std::min<int64_t>(want, (int64_t)sms * 8));
    if (dtype == 0) k_scale<double><<<blocks, 256, 0, st>>>((double*)x, n, f);
    else k_scale<float><<<blocks, 256, 0, st>>>((float*)x, n, (float)f);
    return (int)cudaGetLastError();
}

// log2 of the parts per work item: the persistent grid balances to within one part, so a
// list with few items is claimed in parts until there are 8 for each resident
// CTA, of 256 points (one per thread) at the least for the default 8192-point
// items.  256 mixed instances (1100 items), forward + transposed 705 -> 565 us (456 with
// the straight loops of deo_eval.cuh).
static int split_for(int64_t n_items, int64_t ctas) {
    int lsplit = 0;
    while (lsplit < 5 && (n_items << lsplit) < 8 * ctas) ++lsplit;
    return lsplit;
}

extern "C" int deo_k_stage_batch(const StageDev* st, const WorkItem* items, int64_t n_items, unsigned int* counter,
                                 int lbc,
                                 int dtype, int ctas_per_sm, int threads, void* stream) {
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const int sms = deo_k_num_sms();
    int64_t grid = (int64_t)sms * (ctas_per_sm > 0 ? ctas_per_sm : 4);
    const int lsplit = split_for(n_items, grid);
    if (grid > n_items << lsplit) grid = n_items << lsplit;
    if (grid <= 0) return 0;
    auto go = [&](auto kernel) { kernel<<<(unsigned)grid, threads, 0, s>>>(st, items, n_items, lsplit, counter); };
    if (dtype == 0) lbc ? go(k_stage<double, true>) : go(k_stage<double, false>);
    else lbc ? go(k_stage<float, true>) : go(k_stage<float, false>);
    return (int)cudaGetLastError();
}

extern "C" int deo_k_stage_one(const PlanDev* p, const StageDev* S, void* stream) {
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const int64_t blocks = (p->total + 256 * STAGE_PT - 1) / (256 * STAGE_PT);
    if (blocks == 0) return 0;
    auto go = [&](auto kernel) { kernel<<<(unsigned)blocks, 256, 0, st>>>(*p, *S); };
    if (p->dtype == 0) {
        if (p->has_lbc) S->adjoint ? go(k_stage_one<double, true, true>) : go(k_stage_one<double, false, true>);
        else S->adjoint ? go(k_stage_one<double, true, false>) : go(k_stage_one<double, false, false>);
    } else {
        if (p->has_lbc) S->adjoint ? go(k_stage_one<float, true, true>) : go(k_stage_one<float, false, true>);
        else S->adjoint ? go(k_stage_one<float, true, false>) : go(k_stage_one<float, false, false>);
    }
    return (int)cudaGetLastError();
}

extern "C" int deo_k_apply(const PlanDev* p, const void* u, void* du, int overwrite, int adjoint, void* stream) {
    const int threads = 256;
    const int64_t blocks = (p->total + threads - 1) / threads;
    if (blocks == 0) return 0;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    auto go = [&](auto kernel, const auto* in, auto* out) {
        kernel<<<(unsigned)blocks, threads, 0, st>>>(*p, in, out, overwrite);
    };
    const double* ud = (const double*)u;
    const float* uf = (const float*)u;
    if (p->dtype == 0) {
        if (p->has_lbc) adjoint ? go(k_apply<double, true, true>, ud, (double*)du) : go(k_apply<double, false, true>, ud, (double*)du);
        else adjoint ? go(k_apply<double, true, false>, ud, (double*)du) : go(k_apply<double, false, false>, ud, (double*)du);
    } else {
        if (p->has_lbc) adjoint ? go(k_apply<float, true, true>, uf, (float*)du) : go(k_apply<float, false, true>, uf, (float*)du);
        else adjoint ? go(k_apply<float, true, false>, uf, (float*)du) : go(k_apply<float, false, false>, uf, (float*)du);
    }
    return (int)cudaGetLastError();
}

extern "C" int deo_k_num_sms(void) {
    int dev = 0, n = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 0;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 0;
    return n;
}

// Loads the k_batch instantiations onto the current device and runs each
// once over an empty work-list (one CTA; it leaves the counters zero), so that the
// module image and the resources a launch of them takes are committed now:
// with lazy module loading (the CUDA default) that would otherwise happen at
// their first real launch.
extern "C" int deo_k_batch_prepare(unsigned int* counter, void* stream) {
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    cudaFuncAttributes a;
    cudaError_t e = cudaSuccess;
    auto prep = [&](auto kernel) {
        if (e == cudaSuccess) e = cudaFuncGetAttributes(&a, kernel);
        if (e == cudaSuccess) kernel<<<1, 256, 0, st>>>(nullptr, nullptr, 0, 0, counter);
    };
    prep(k_batch<double, false, false>);
    prep(k_batch<double, true, false>);
    prep(k_batch<float, false, false>);
    prep(k_batch<float, true, false>);
    prep(k_batch<double, false, true>);
    prep(k_batch<double, true, true>);
    prep(k_batch<float, false, true>);
    prep(k_batch<float, true, true>);
    if (e != cudaSuccess) return (int)e;
    return (int)cudaGetLastError();
}

extern "C" int deo_k_batch(const InstDev* inst, const WorkItem* items, int64_t n_items, unsigned int* counter,
                           int dtype, int adjoint, int lbc, int ctas_per_sm, int threads, void* stream) {
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const int sms = deo_k_num_sms();
    int64_t grid = (int64_t)sms * (ctas_per_sm > 0 ? ctas_per_sm : 4);
    const int lsplit = split_for(n_items, grid);
    if (grid > n_items << lsplit) grid = n_items << lsplit;
    if (grid <= 0) return 0;
    auto go = [&](auto kernel) { kernel<<<(unsigned)grid, threads, 0, st>>>(inst, items, n_items, lsplit, counter); };
    if (dtype == 0) {
        if (lbc) adjoint ? go(k_batch<double, true, true>) : go(k_batch<double, false, true>);
        else adjoint ? go(k_batch<double, true, false>) : go(k_batch<double, false, false>);
    } else {
        if (lbc) adjoint ? go(k_batch<float, true, true>) : go(k_batch<float, false, true>);
        else adjoint ? go(k_batch<float, true, false>) : go(k_batch<float, false, false>);
    }
    return (int)cudaGetLastError();
}
