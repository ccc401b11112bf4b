// Edge-list sweeps: the reference-shaped entry points (device edge lists,
// one query per call) answered without building a CSR.
//
//   bfs_wrapper            algorithm/bfs/gpu/bfs.cu:43-81
//   bfs() of the SCC step  algorithm/scc/gpu/forward_backward.cu:139-170
//   bellman_ford_wrapper   algorithm/sssp/gpu/bellman_ford.cu:103-144
//
// One query on an edge list reads every edge a few times; sorting the edges
// into a CSR first reads and writes them about thirty times.  So one
// cooperative launch checks the edges and then sweeps over them until a sweep
// changes nothing, as the reference does, with the decision on the device.
// What bounds a sweep is the stream of edge ends: the state that every edge
// looks up is one bit per vertex, copied into shared memory by every CTA
// before the sweep while it fits (1.6 M vertices; larger graphs read the
// bitmap through L1 / L2), and an edge's other fields are only loaded when its
// bit says that they matter.
//
// Measured, whole calls on a B200: bfs_wrapper on RMAT scale 20, edge factor 16
// 27.8 -> 0.29 ms; init + bellman_ford_wrapper on 300,007 vertices, 4.8 M edges
// 22-28 -> 0.48 ms (before: CSR build, then bfs_persistent / sssp_persistent).
//
// A graph whose answer needs many sweeps (long paths) is better served by the
// CSR kernels, whose steps touch the frontier only: after kMaxSweeps sweeps
// the launch gives up and the caller builds the CSR (see capi.cu).
#include <cfloat>
#include <cstddef>

#include "trav_internal.cuh"

namespace trav {
namespace {

constexpr unsigned kAll = 0xffffffffu;
constexpr unsigned kFltMaxBits = 0x7f7fffffu;
constexpr int kSweepThreads = 1024;
// Edges one CTA takes before another joins: two 16-byte loads of each array
// per thread.  Below that a second CTA only adds the barrier.
constexpr int kCtaEdges = 8 * kSweepThreads;
// Sweeps before the CSR path takes over.  A sweep reads 4-12 bytes an edge and
// copies the bitmaps to every CTA, a fixed 5-30 us on sparse graphs; 64 of them
// cost at most about what the build and the query that they hoped to save do.
// Measured, whole calls, with the sweeps first and without them:
//   reachability    paths side by side, 1.6 M vertices and edges, 80 / 200 / 1,000 levels: 2.03, 2.28, 4.1 ms and
//                   0.97, 1.24, 3.1; grids 100 x 100, 1100 x 911, 3000 x 3000: 1.48, 9.3, 42 ms and 1.18, 8.0, 36
//   masked          780,000 vertices, 60 levels: 0.88 ms and 0.75
//   Bellman-Ford    the same paths 1.33, 1.89, 5.6 ms and 1.17, 1.68, 5.2; grids 1.72, 19.0, 156 ms and 1.63, 18.8, 154
// and where the sweeps are enough: 60 levels 0.29 ms and 0.89, 100 levels of 160,000 vertices each 2.3 and 8.2.
constexpr int kMaxSweeps = 64;
constexpr int kSmemMax = 200 * 1024;  // bytes of bitmap a CTA copies

constexpr int kBadId = 1, kBadNegative = 2, kBadInfinite = 4;

struct SweepCtl {
    unsigned long long bar;  // grid-barrier arrivals
    int err;                 // kErrTimeout
    int err_phase;
    int bad;                 // kBad* of the edge check
    int converged;
    int changed[4];          // ring: sweep k changed something
};

struct SweepArgs {
    const int32_t *src, *dst;
    const float *w;
    int32_t V, W;
    int64_t E;
    int vec;                 // the edge arrays are 16-byte aligned
    int32_t source;
    const int32_t *trees;    // reach: only vertices of tree `want` (nullptr: all)
    int32_t want;
    unsigned char *visited;  // reach: V result bytes
    unsigned *d;             // Bellman-Ford: V distance bits, relaxed in place
    unsigned *bits[3];       // bitmaps of W words
    SweepCtl *ctl;
    unsigned long long timeout_ns;
};

__device__ __forceinline__ unsigned long long now_ns()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Grid barrier with a bounded wait (the scheme of grid_sync in traverse.cu).
__device__ bool sweep_sync(const SweepArgs &a, int phase)
{
    __shared__ int s_ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        int ok = 1;
        unsigned long long old;
        asm volatile("atom.add.acq_rel.gpu.global.u64 %0, [%1], 1;" : "=l"(old) : "l"(&a.ctl->bar) : "memory");
        const unsigned long long nb = gridDim.x, target = (old / nb + 1) * nb;
        if (old + 1 != target) {
            const unsigned long long t0 = now_ns();
            while (true) {
                unsigned long long c;
                asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(c) : "l"(&a.ctl->bar) : "memory");
                if (c >= target) break;
                if (*reinterpret_cast<volatile int *>(&a.ctl->err) != 0) { ok = 0; break; }
                __nanosleep(32);
                if (now_ns() - t0 > a.timeout_ns) {
                    if (atomicCAS(&a.ctl->err, 0, kErrTimeout) == 0) atomicExch(&a.ctl->err_phase, phase);
                    ok = 0;
                    break;
                }
            }
        }
        s_ok = ok;
    }
    __syncthreads();
    return s_ok != 0;
}

// The four edges at e (e % 4 == 0) of an array; entries at or past E read as
// `fill`.  kAgain: the next sweep reads them again, so they may stay in L2
// (the others are marked to leave first).  The targets of a reachability sweep,
// RMAT scale 20: 302 -> 289 us a call; all of a Bellman-Ford sweep's, 300,007
// vertices, 4.8 M edges: 548 -> 483 us.
template <bool kAgain = false>
__device__ __forceinline__ int4 edge4(const int32_t *p, unsigned e, unsigned E, int vec, int fill)
{
    if (vec && e + 4 <= E) {
        const int4 *q = reinterpret_cast<const int4 *>(p + e);
        return kAgain ? __ldg(q) : __ldcs(q);
    }
    int4 r;
    r.x = e < E ? __ldcs(p + e) : fill;
    r.y = e + 1 < E ? __ldcs(p + e + 1) : fill;
    r.z = e + 2 < E ? __ldcs(p + e + 2) : fill;
    r.w = e + 3 < E ? __ldcs(p + e + 3) : fill;
    return r;
}

__device__ __forceinline__ bool test(const unsigned *b, int v) { return (b[v >> 5] >> (v & 31)) & 1u; }

__device__ __forceinline__ int check_ids(const int4 &x, int32_t V)
{
    return (unsigned)x.x >= (unsigned)V || (unsigned)x.y >= (unsigned)V || (unsigned)x.z >= (unsigned)V ||
                   (unsigned)x.w >= (unsigned)V ? kBadId : 0;
}

__device__ __forceinline__ int check_weight(int bits)
{
    const float x = __int_as_float(bits);
    return (x < 0.0f ? kBadNegative : 0) | (!isfinite(x) ? kBadInfinite : 0);
}

// Phase 0 of a query: every edge checked before anything is looked up by it.
__device__ __forceinline__ void check_edges(const SweepArgs &a)
{
    const unsigned E = (unsigned)a.E, step = gridDim.x * kSweepThreads * 4;  // E < 2^31: e + 4 steps fit 32 bits
    int flag = 0;
    for (unsigned e = (blockIdx.x * kSweepThreads + threadIdx.x) * 4; e < E; e += step) {
        flag |= check_ids(edge4(a.src, e, E, a.vec, 0), a.V) | check_ids(edge4(a.dst, e, E, a.vec, 0), a.V);
        if (a.w) {
            const int4 w = edge4(reinterpret_cast<const int32_t *>(a.w), e, E, a.vec, 0);
            flag |= check_weight(w.x) | check_weight(w.y) | check_weight(w.z) | check_weight(w.w);
        }
    }
    flag = __reduce_or_sync(kAll, flag);
    if (flag && (threadIdx.x & 31) == 0) atomicOr(&a.ctl->bad, flag);
}

// The same for reachability with the bitmap in shared memory, as a sweep: an
// edge whose ends are in range and whose source is reached marks its target.
// It reads both ends of every edge, as the first sweep would again (RMAT scale
// 20: 337 -> 302 us a call).
__device__ __forceinline__ bool check_and_mark(const SweepArgs &a, unsigned *reached)
{
    const unsigned E = (unsigned)a.E, V = (unsigned)a.V, step = gridDim.x * kSweepThreads * 4;
    int flag = 0;
    bool marked = false;
    for (unsigned e = (blockIdx.x * kSweepThreads + threadIdx.x) * 4; e < E; e += step) {
        const int4 f = edge4(a.src, e, E, a.vec, 0), t = edge4(a.dst, e, E, a.vec, 0);
        flag |= check_ids(f, a.V) | check_ids(t, a.V);
        const int fv[4] = {f.x, f.y, f.z, f.w}, tv[4] = {t.x, t.y, t.z, t.w};
#pragma unroll
        for (int j = 0; j < 4; j++) {
            if (e + j >= E || (unsigned)fv[j] >= V || (unsigned)tv[j] >= V || !test(reached, fv[j])) continue;
            atomicOr(&reached[tv[j] >> 5], 1u << (tv[j] & 31));
            marked = true;
        }
    }
    flag = __reduce_or_sync(kAll, flag);
    if (flag && (threadIdx.x & 31) == 0) atomicOr(&a.ctl->bad, flag);
    return marked;
}

// Result of sweep k once its barrier has passed: 0 = nothing changed.  Entry
// k + 2 of the ring was last read after sweep k - 2's barrier.
__device__ __forceinline__ bool publish(const SweepArgs &a, int k, bool changed)
{
    const int any = __syncthreads_or(changed);
    if (threadIdx.x == 0) {
        if (any) *reinterpret_cast<volatile int *>(&a.ctl->changed[k & 3]) = 1;
        if (blockIdx.x == 0) *reinterpret_cast<volatile int *>(&a.ctl->changed[(k + 2) & 3]) = 0;
    }
    return any;
}

// Add a CTA's copy of a bitmap to the one in memory.
__device__ __forceinline__ void merge_bits(unsigned *g, const unsigned *copy, int W)
{
    for (int w = threadIdx.x; w < W; w += kSweepThreads) {
        const unsigned x = copy[w] & ~__ldcg(&g[w]);
        if (x) atomicOr(&g[w], x);
    }
}

__device__ __forceinline__ int changed_in(const SweepArgs &a, int k)
{
    return *reinterpret_cast<volatile int *>(&a.ctl->changed[k & 3]);
}

// Reachability.  bits[0] (clear at first): vertices reached; bits[1] (kMask only): vertices
// reached or outside the tree, which no edge may reach.  An edge matters when
// its target is still open and its source is reached; late sweeps find almost
// every target closed and read 4 bytes an edge.
//
// With the bitmaps in shared memory a CTA marks what it finds there, and takes
// its copy to memory once a sweep, a word an atomic and 32 consecutive words a
// warp.  (A global atomic for every vertex that a CTA finds was up to one per
// edge in the sweep that reaches most vertices, each waited for.)  RMAT scale 20,
// edge factor 16, whole call: 0.39 -> 0.34 ms.
template <bool kMask, bool kSmem>
__global__ void __launch_bounds__(kSweepThreads, 1) el_reach_kernel(SweepArgs a)
{
    extern __shared__ unsigned sm[];
    const int gtid = blockIdx.x * kSweepThreads + threadIdx.x, nth = gridDim.x * kSweepThreads;
    unsigned *const gr = a.bits[0], *const gc = kMask ? a.bits[1] : a.bits[0];
    unsigned *const r = kSmem ? sm : gr, *const c = kMask ? (kSmem ? sm + a.W : gc) : r;
    const int s = a.source;
    if (!kMask && kSmem) {
        // gr is clear
        for (int w = threadIdx.x; w < a.W; w += kSweepThreads) sm[w] = w == (s >> 5) ? 1u << (s & 31) : 0u;
        __syncthreads();
        const bool marked = check_and_mark(a, sm);
        if (__syncthreads_or(marked) || blockIdx.x == 0) merge_bits(gr, sm, a.W);
    } else {
        check_edges(a);
    }
    if (kMask) {
        for (int w = gtid >> 5; w < a.W; w += nth >> 5) {
            const int v = w * 32 + (int)(threadIdx.x & 31);
            const unsigned m = __ballot_sync(kAll, v < a.V && (v == s || a.trees[v] != a.want));
            if ((threadIdx.x & 31) == 0) {
                gr[w] = w == (s >> 5) ? 1u << (s & 31) : 0u;
                gc[w] = m;
            }
        }
    } else if (!kSmem) {
        for (int w = gtid; w < a.W; w += nth) gr[w] = w == (s >> 5) ? 1u << (s & 31) : 0u;
    }
    int phase = 0;
    if (!sweep_sync(a, phase++)) return;
    if (*reinterpret_cast<volatile int *>(&a.ctl->bad)) return;  // the same answer in every CTA

    constexpr int kU = kMask ? 2 : 3;  // 16-byte loads of a thread in flight (more spill)
    const unsigned E = (unsigned)a.E, step = (unsigned)nth * 4;
    bool done = false;
    for (int k = 0; k < kMaxSweeps && !done; k++) {
        if (kSmem) {
            for (int w = threadIdx.x; w < a.W; w += kSweepThreads) {
                sm[w] = __ldcg(&gr[w]);
                if (kMask) sm[a.W + w] = __ldcg(&gc[w]);
            }
            __syncthreads();
        }
        bool changed = false;
        for (unsigned e0 = (unsigned)gtid * 4; e0 < E; e0 += kU * step) {
            int4 t[kU];
            unsigned open[kU];
#pragma unroll
            for (int u = 0; u < kU; u++) {
                const unsigned e = e0 + u * step;
                t[u] = e < E ? edge4<true>(a.dst, e, E, a.vec, s) : make_int4(s, s, s, s);  // the source is closed
            }
#pragma unroll
            for (int u = 0; u < kU; u++)
                open[u] = (test(c, t[u].x) ? 0u : 1u) | (test(c, t[u].y) ? 0u : 2u) | (test(c, t[u].z) ? 0u : 4u) |
                          (test(c, t[u].w) ? 0u : 8u);
#pragma unroll
            for (int u = 0; u < kU; u++) {
                if (!open[u]) continue;
                const int4 f = edge4(a.src, e0 + u * step, E, a.vec, 0);
                const int tv[4] = {t[u].x, t[u].y, t[u].z, t[u].w}, fv[4] = {f.x, f.y, f.z, f.w};
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    if (!((open[u] >> j) & 1u) || !test(r, fv[j])) continue;
                    const unsigned bit = 1u << (tv[j] & 31);
                    // in the CTA's own copy (merge_bits takes it to memory)
                    const unsigned old = atomicOr(&r[tv[j] >> 5], bit);
                    if (kMask) atomicOr(&c[tv[j] >> 5], bit);
                    if (!(old & bit)) changed = true;
                }
            }
        }
        if (publish(a, k, changed) && kSmem) {
            merge_bits(gr, r, a.W);
            if (kMask) merge_bits(gc, c, a.W);
        }
        if (!sweep_sync(a, phase++)) return;
        done = !changed_in(a, k);
    }
    if (!done) return;  // converged stays 0: the caller takes the CSR path
    for (unsigned v = (unsigned)gtid; v < (unsigned)a.V; v += (unsigned)nth)  // (V may be near 2^31)
        a.visited[v] = (__ldcg(&gr[v >> 5]) >> (v & 31u)) & 1u;
    if (gtid == 0) a.ctl->converged = 1;
}

// Bellman-Ford to the fixpoint of whatever d holds.  bits[k % 3]: vertices
// lowered in sweep k - 1 (at first, every vertex below FLT_MAX); an edge
// matters when its source is one of them, so a sweep streams the sources and
// reads targets, weights and distances of those edges only.  d is lowered in
// place (float bits >= 0 order like unsigned integers), so a distance travels
// several edges in one sweep; the fixpoint does not depend on the order.
//
// Distances are read through L1: on a skewed graph most of them are those of a
// few vertices, whose lines would keep single L2 slices busy.  One in L1 is at
// most a sweep old (the barrier's acquire invalidates L1), so it is too high if
// anything: an edge out of a vertex lowered meanwhile is looked at again in the
// next sweep, and atomicMin decides about the target.  300,007 vertices, 4.8 M
// edges, whole call: 0.93 -> 0.54 ms (0.87 with the targets' distances alone).
__device__ __forceinline__ float dist_l1(const unsigned *p)
{
    float d;
    asm volatile("ld.global.ca.f32 %0, [%1];" : "=f"(d) : "l"(p));
    return d;
}

template <bool kSmem>
__global__ void __launch_bounds__(kSweepThreads, 1) el_bellman_ford_kernel(SweepArgs a)
{
    extern __shared__ unsigned sm[];
    const int gtid = blockIdx.x * kSweepThreads + threadIdx.x, nth = gridDim.x * kSweepThreads;
    check_edges(a);
    for (int w = gtid >> 5; w < a.W; w += nth >> 5) {
        const int v = w * 32 + (int)(threadIdx.x & 31);
        const unsigned m = __ballot_sync(kAll, v < a.V && __ldcg(&a.d[v < a.V ? v : 0]) < kFltMaxBits);
        if ((threadIdx.x & 31) == 0) {
            a.bits[0][w] = m;
            a.bits[1][w] = 0u;
        }
    }
    int phase = 0;
    if (!sweep_sync(a, phase++)) return;
    if (*reinterpret_cast<volatile int *>(&a.ctl->bad)) return;

    constexpr int kU = 2;  // 4 spill
    const unsigned E = (unsigned)a.E, step = (unsigned)nth * 4;
    bool done = false;
    unsigned *cur = a.bits[0], *next = a.bits[1], *later = a.bits[2];
    for (int k = 0; k < kMaxSweeps && !done; k++) {
        for (int w = gtid; w < a.W; w += nth) later[w] = 0u;  // it was read in sweep k - 1
        const unsigned *act = kSmem ? sm : cur;
        if (kSmem) {
            for (int w = threadIdx.x; w < a.W; w += kSweepThreads) sm[w] = __ldcg(&cur[w]);
            __syncthreads();
        }
        bool changed = false;
        for (unsigned e0 = (unsigned)gtid * 4; e0 < E; e0 += kU * step) {
            int4 f[kU];
            unsigned on[kU];
#pragma unroll
            for (int u = 0; u < kU; u++) {
                const unsigned e = e0 + u * step;
                f[u] = e < E ? edge4<true>(a.src, e, E, a.vec, -1) : make_int4(-1, -1, -1, -1);
            }
#pragma unroll
            for (int u = 0; u < kU; u++)
                on[u] = (f[u].x >= 0 && test(act, f[u].x) ? 1u : 0u) | (f[u].y >= 0 && test(act, f[u].y) ? 2u : 0u) |
                        (f[u].z >= 0 && test(act, f[u].z) ? 4u : 0u) | (f[u].w >= 0 && test(act, f[u].w) ? 8u : 0u);
#pragma unroll
            for (int u = 0; u < kU; u++) {
                if (!on[u]) continue;
                const unsigned e = e0 + u * step;
                const int4 t = edge4<true>(a.dst, e, E, a.vec, 0);
                const int4 wt = edge4<true>(reinterpret_cast<const int32_t *>(a.w), e, E, a.vec, 0);
                const int fv[4] = {f[u].x, f[u].y, f[u].z, f[u].w}, tv[4] = {t.x, t.y, t.z, t.w};
                const int wv[4] = {wt.x, wt.y, wt.z, wt.w};
                float nd[4], od[4];
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const bool ok = (on[u] >> j) & 1u;
                    nd[j] = ok ? dist_l1(a.d + fv[j]) : 0.0f;
                    od[j] = ok ? dist_l1(a.d + tv[j]) : 0.0f;
                }
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    nd[j] = __fadd_rn(nd[j], __int_as_float(wv[j]));  // one rounded add, as sssp.hpp:56
                    if (!((on[u] >> j) & 1u) || !(nd[j] < od[j])) continue;
                    const float old = __uint_as_float(atomicMin(&a.d[tv[j]], __float_as_uint(nd[j])));
                    if (!(nd[j] < old)) continue;
                    changed = true;
                    const unsigned bit = 1u << (tv[j] & 31);
                    if (!(__ldcg(&next[tv[j] >> 5]) & bit)) atomicOr(&next[tv[j] >> 5], bit);
                }
            }
        }
        publish(a, k, changed);
        if (!sweep_sync(a, phase++)) return;
        done = !changed_in(a, k);
        unsigned *const x = cur;
        cur = next;
        next = later;
        later = x;
    }
    if (done && gtid == 0) a.ctl->converged = 1;
}

#define TRY_CUDA(expr)                                      \
    do {                                                    \
        cudaError_t _e = (expr);                            \
        if (_e != cudaSuccess) return cuda_fail(_e, #expr); \
    } while (0)

struct Scratch {
    void *p = nullptr;
    cudaStream_t st;
    explicit Scratch(cudaStream_t s) : st(s) {}
    ~Scratch() { dev_free(p, st); }
};

bool aligned16(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

// Launch one sweep query with `maps` bitmaps (`copied` of them copied into
// shared memory when they fit) and wait for it.
int run_sweeps(SweepArgs a, int maps, int copied, const void *fn_smem, const void *fn_global, const char *what,
               cudaStream_t st, bool *done)
{
    *done = false;
    a.W = (int32_t)(((int64_t)a.V + 31) / 32);
    a.vec = aligned16(a.src) && aligned16(a.dst) && aligned16(a.w);
    a.timeout_ns = kDefaultTimeoutNs;
    const size_t map_bytes = (sizeof(unsigned) * (size_t)a.W + 255) & ~(size_t)255;
    Scratch mem(st);
    TRY_CUDA(dev_malloc(&mem.p, 256 + map_bytes * (size_t)maps));
    unsigned char *m = static_cast<unsigned char *>(mem.p);
    a.ctl = reinterpret_cast<SweepCtl *>(m);
    for (int i = 0; i < maps; i++) a.bits[i] = reinterpret_cast<unsigned *>(m + 256 + map_bytes * (size_t)i);
    const size_t smem = sizeof(unsigned) * (size_t)a.W * (size_t)copied;
    const bool fits = smem <= (size_t)kSmemMax;
    const void *fn = fits ? fn_smem : fn_global;
    int dev = 0, sms = 0;
    TRY_CUDA(cudaGetDevice(&dev));
    TRY_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    if (fits) TRY_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemMax));
    int64_t ctas = (a.E + kCtaEdges - 1) / kCtaEdges;
    if (ctas < 1) ctas = 1;
    if (ctas > sms) ctas = sms;  // one CTA of 1024 threads per SM
    TRY_CUDA(cudaMemsetAsync(mem.p, 0, 256 + map_bytes, st));  // ctl and the first bitmap
    void *params[] = {&a};
    TRY_CUDA(cudaLaunchCooperativeKernel(fn, dim3((unsigned)ctas), dim3(kSweepThreads), params, fits ? smem : 0, st));
    SweepCtl h;
    TRY_CUDA(cudaMemcpyAsync(&h, a.ctl, sizeof(h), cudaMemcpyDeviceToHost, st));
    TRY_CUDA(cudaStreamSynchronize(st));
    if (h.err == kErrTimeout) {
        set_error(std::string(what) + ": a bounded grid-barrier wait timed out (phase " + std::to_string(h.err_phase) + ")");
        return TRAV_ERR_TIMEOUT;
    }
    if (h.bad & kBadId) { set_error("edge list holds a vertex id outside [0, V)"); return TRAV_ERR_BAD_ARG; }
    if (h.bad & kBadNegative) { set_error("edge list holds a negative weight (only weights >= 0 are supported)"); return TRAV_ERR_BAD_ARG; }
    if (h.bad & kBadInfinite) { set_error("edge list holds a NaN or infinite weight (weights must be finite)"); return TRAV_ERR_BAD_ARG; }
    *done = h.converged != 0;
    return TRAV_OK;
}

}  // namespace

int el_reach_sweeps(const int32_t *src, const int32_t *dst, int32_t V, int64_t E, int32_t source, const int32_t *trees,
                    int32_t want, uint8_t *visited, cudaStream_t st, bool *done)
{
    SweepArgs a{};
    a.src = src;
    a.dst = dst;
    a.V = V;
    a.E = E;
    a.source = source;
    a.trees = trees;
    a.want = want;
    a.visited = visited;
    if (trees)
        return run_sweeps(a, 2, 2, (const void *)el_reach_kernel<true, true>, (const void *)el_reach_kernel<true, false>,
                          "trav_reach_el_masked", st, done);
    return run_sweeps(a, 1, 1, (const void *)el_reach_kernel<false, true>, (const void *)el_reach_kernel<false, false>,
                      "bfs_wrapper", st, done);
}

int el_bellman_ford_sweeps(const int32_t *src, const int32_t *dst, const float *w, int32_t V, int64_t E, float *d,
                           cudaStream_t st, bool *done)
{
    SweepArgs a{};
    a.src = src;
    a.dst = dst;
    a.w = w;
    a.V = V;
    a.E = E;
    a.d = reinterpret_cast<unsigned *>(d);
    return run_sweeps(a, 3, 1, (const void *)el_bellman_ford_kernel<true>, (const void *)el_bellman_ford_kernel<false>,
                      "bellman_ford_wrapper", st, done);
}

}  // namespace trav
