// Graph optimisation pass on a device edge list, and the memory-transaction
// count of an edge-per-thread sweep: the GPU forms of GraphOptimizationAPI
// (include/test/optimization/graph_optimization_API.hpp).
//
//   reorder_edges_in_adjacency_list_format :14-55   sort by (src, dst, weight)
//   remove_loops_and_multiple_arcs          :60-117  drop loops and repeated arcs (the lightest arc stays)
//   reorder_edges_for_cache                 :122-166 group by (src / segment, dst / segment)
//   check_gpu_memory_transactions_count     :229-266 distinct 128-byte segments per warp of 32 edges
//
// The sorts are stable radix sorts (weight bits, then the (src, dst)
// key, then the segment key), so the order inside a segment pair -- which the
// reference's std::sort leaves unspecified -- is the (src, dst, weight) order.
#include <cuda_runtime.h>
#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_select.cuh>

#include <algorithm>
#include <cstdint>

#include "trav_internal.cuh"

namespace trav {
namespace {

#define TRY_CUDA(expr)                                      \
    do {                                                    \
        cudaError_t _e = (expr);                            \
        if (_e != cudaSuccess) return cuda_fail(_e, #expr); \
    } while (0)

template <class T>
struct Buf {
    T *p = nullptr;
    cudaStream_t st;
    explicit Buf(cudaStream_t s) : st(s) {}
    cudaError_t alloc(int64_t n) { return dev_malloc((void **)&p, sizeof(T) * (size_t)(n > 0 ? n : 1)); }
    ~Buf() { dev_free(p, st); }
};

int grid_of(int64_t n) { return (int)std::min<int64_t>((n + 255) / 256, 65535); }

// weight bits with -0.0 read as +0.0 (non-negative floats order like their bits), and the identity permutation
__global__ void weight_keys_kernel(int64_t E, const float *__restrict__ w, unsigned *__restrict__ key,
                                   int32_t *__restrict__ idx)
{
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < E; i += (int64_t)gridDim.x * blockDim.x) {
        const float x = w[i];
        key[i] = x == 0.0f ? 0u : __float_as_uint(x);
        idx[i] = (int32_t)i;
    }
}

// Keys are packed to the bits that ids can have (ids are in [0, V)), since every
// eight bits are a pass of the sort: 5 instead of 8 passes of 0.1 ms for the
// pairs of 2^19 vertices, 1 instead of 8 of 0.07 ms for 4 x 4 segments, 8.4 M
// edges; the whole pass 1.86 ms instead of 2.67.
int bits_of(int32_t ids)
{
    int b = 1;
    while (b < 31 && (ids - 1) >> b) b++;
    return b;
}

// (src, dst) of the permuted edges as one key, dst in the low `bits`
__global__ void pair_keys_kernel(int64_t E, const int32_t *__restrict__ src, const int32_t *__restrict__ dst,
                                 const int32_t *__restrict__ idx, int bits, unsigned long long *__restrict__ key)
{
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < E; i += (int64_t)gridDim.x * blockDim.x) {
        const int32_t e = idx[i];
        key[i] = ((unsigned long long)(unsigned)src[e] << bits) | (unsigned)dst[e];
    }
}

// (src / segment, dst / segment) as one key in the same way, identity permutation
__global__ void segment_keys_kernel(int64_t E, const int32_t *__restrict__ src, const int32_t *__restrict__ dst,
                                    int32_t segment, int bits, unsigned long long *__restrict__ key,
                                    int32_t *__restrict__ idx)
{
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < E; i += (int64_t)gridDim.x * blockDim.x) {
        key[i] = ((unsigned long long)(unsigned)(src[i] / segment) << bits) | (unsigned)(dst[i] / segment);
        idx[i] = (int32_t)i;
    }
}

__global__ void gather_kernel(int64_t E, const int32_t *__restrict__ idx, const int32_t *__restrict__ src,
                              const int32_t *__restrict__ dst, const float *__restrict__ w, int32_t *__restrict__ os,
                              int32_t *__restrict__ od, float *__restrict__ ow)
{
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < E; i += (int64_t)gridDim.x * blockDim.x) {
        const int32_t e = idx[i];
        os[i] = src[e];
        od[i] = dst[e];
        const float x = w[e];
        ow[i] = x == 0.0f ? 0.0f : x;
    }
}

// keep an edge unless it is a loop or repeats the previous sorted edge's (src, dst)
__global__ void keep_kernel(int64_t E, const int32_t *__restrict__ s, const int32_t *__restrict__ d,
                            unsigned char *__restrict__ keep)
{
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < E; i += (int64_t)gridDim.x * blockDim.x) {
        bool k = s[i] != d[i];
        if (k && i > 0 && s[i] == s[i - 1] && d[i] == d[i - 1]) k = false;
        keep[i] = k ? 1 : 0;
    }
}

// One warp per 32 consecutive edges of the counted warps: the distinct
// 128-byte segments among the warp's src * elem and among its dst * elem.
__global__ void transactions_kernel(int64_t warps, const int32_t *__restrict__ src, const int32_t *__restrict__ dst,
                                    int32_t elem, unsigned long long *__restrict__ total)
{
    const unsigned lane = threadIdx.x & 31;
    unsigned long long acc = 0;
    for (int64_t k = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; k < warps;
         k += ((int64_t)gridDim.x * blockDim.x) >> 5) {
        const int64_t i = 32 * k + lane;
        const unsigned long long a = (unsigned long long)((int64_t)src[i] * elem / 128);
        const unsigned long long b = (unsigned long long)((int64_t)dst[i] * elem / 128);
        const unsigned ma = __match_any_sync(0xffffffffu, a), mb = __match_any_sync(0xffffffffu, b);
        // a lane leads its group when no lower lane holds the same segment
        const unsigned lower = (1u << lane) - 1u;
        acc += ((ma & lower) == 0u ? 1u : 0u) + ((mb & lower) == 0u ? 1u : 0u);
    }
    for (int o = 16; o; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
    if (lane == 0 && acc) atomicAdd(total, acc);
}

}  // namespace

int el_optimize_device(int32_t *src, int32_t *dst, float *w, int32_t V, int64_t E, int32_t segment, int64_t *E_out,
                       cudaStream_t st)
{
    *E_out = 0;
    if (E == 0) return TRAV_OK;
    DevSlab mem(st);
    unsigned *wkey, *wkey2;
    int32_t *idx, *idx2, *s2, *d2;
    unsigned long long *key, *key2;
    float *w2;
    unsigned char *keep, *temp;
    int64_t *nsel;
    mem.add(&wkey, E);
    mem.add(&wkey2, E);
    mem.add(&idx, E);
    mem.add(&idx2, E);
    mem.add(&key, E);
    mem.add(&key2, E);
    mem.add(&s2, E);
    mem.add(&d2, E);
    mem.add(&w2, E);
    mem.add(&keep, E);
    mem.add(&nsel, 1);
    // (with one segment the edges are in order already)
    const int32_t segments = segment > 0 ? (V - 1) / segment + 1 : 0;
    const int n = (int)E, bits = bits_of(V), sbits = bits_of(segments);
    size_t tb = 0, t1 = 0;
    TRY_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, t1, wkey, wkey2, idx, idx2, n, 0, 32, st));
    tb = t1;
    TRY_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, t1, key, key2, idx2, idx, n, 0, 2 * bits, st));
    tb = std::max(tb, t1);
    TRY_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, t1, key, key2, idx, idx2, n, 0, 2 * sbits, st));
    tb = std::max(tb, t1);
    TRY_CUDA(cub::DeviceSelect::Flagged(nullptr, t1, s2, keep, src, nsel, n, st));
    tb = std::max(tb, t1);
    mem.add(&temp, (int64_t)tb);
    TRY_CUDA(mem.commit());

    // (src, dst, weight) order: weight first, then a stable sort by (src, dst)
    weight_keys_kernel<<<grid_of(E), 256, 0, st>>>(E, w, wkey, idx);
    TRY_CUDA(cub::DeviceRadixSort::SortPairs(temp, tb, wkey, wkey2, idx, idx2, n, 0, 32, st));
    pair_keys_kernel<<<grid_of(E), 256, 0, st>>>(E, src, dst, idx2, bits, key);
    TRY_CUDA(cub::DeviceRadixSort::SortPairs(temp, tb, key, key2, idx2, idx, n, 0, 2 * bits, st));
    gather_kernel<<<grid_of(E), 256, 0, st>>>(E, idx, src, dst, w, s2, d2, w2);
    keep_kernel<<<grid_of(E), 256, 0, st>>>(E, s2, d2, keep);
    TRY_CUDA(cudaGetLastError());
    TRY_CUDA(cub::DeviceSelect::Flagged(temp, tb, s2, keep, src, nsel, n, st));
    TRY_CUDA(cub::DeviceSelect::Flagged(temp, tb, d2, keep, dst, nsel, n, st));
    TRY_CUDA(cub::DeviceSelect::Flagged(temp, tb, w2, keep, w, nsel, n, st));
    int64_t kept = 0;
    TRY_CUDA(cudaMemcpyAsync(&kept, nsel, sizeof(int64_t), cudaMemcpyDeviceToHost, st));
    TRY_CUDA(cudaStreamSynchronize(st));
    if (segments > 1 && kept > 0) {
        segment_keys_kernel<<<grid_of(kept), 256, 0, st>>>(kept, src, dst, segment, sbits, key, idx);
        TRY_CUDA(cub::DeviceRadixSort::SortPairs(temp, tb, key, key2, idx, idx2, (int)kept, 0, 2 * sbits, st));
        gather_kernel<<<grid_of(kept), 256, 0, st>>>(kept, idx2, src, dst, w, s2, d2, w2);
        TRY_CUDA(cudaGetLastError());
        TRY_CUDA(cudaMemcpyAsync(src, s2, sizeof(int32_t) * (size_t)kept, cudaMemcpyDeviceToDevice, st));
        TRY_CUDA(cudaMemcpyAsync(dst, d2, sizeof(int32_t) * (size_t)kept, cudaMemcpyDeviceToDevice, st));
        TRY_CUDA(cudaMemcpyAsync(w, w2, sizeof(float) * (size_t)kept, cudaMemcpyDeviceToDevice, st));
        TRY_CUDA(cudaStreamSynchronize(st));
    }
    *E_out = kept;
    return TRAV_OK;
}

int el_transactions_device(const int32_t *src, const int32_t *dst, int64_t E, int32_t elem, int64_t *count,
                           cudaStream_t st)
{
    const int64_t warps = E > 0 ? (E - 1) / 32 : 0;  // the warp holding the last edge is not counted
    Buf<unsigned long long> tot(st);
    TRY_CUDA(tot.alloc(1));
    TRY_CUDA(cudaMemsetAsync(tot.p, 0, sizeof(unsigned long long), st));
    if (warps > 0) {
        transactions_kernel<<<(int)std::min<int64_t>((warps + 7) / 8, 65535), 256, 0, st>>>(warps, src, dst, elem,
                                                                                             tot.p);
        TRY_CUDA(cudaGetLastError());
    }
    unsigned long long h = 0;
    TRY_CUDA(cudaMemcpyAsync(&h, tot.p, sizeof(h), cudaMemcpyDeviceToHost, st));
    TRY_CUDA(cudaStreamSynchronize(st));
    *count = (int64_t)h;
    return TRAV_OK;
}

}  // namespace trav
