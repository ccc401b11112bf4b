// Device memory and streams of the library.
//
// cudaMalloc and cudaFree of a few megabytes take 0.3 ms each on a B200, a
// stream 0.1 ms; a call that builds a graph handle for one query, as the
// reference's callers do, made some 35 allocations and spent 20 of its 27 ms
// there.  Arrays that live together share one allocation (DevSlab), and freed
// blocks stay here for the next allocation of about their size, up to kKeepBytes
// per device (0.6% of the memory); the oldest go first when the bound is
// reached, and all of them when an allocation fails.
// Measured: a graph built from 4.2 M host edges, one BFS and one SSSP, 31 -> 6.0
// ms; the optimisation pass on 8.4 M edges 10.9 -> 2.7 ms (8.4 and 5.0 ms with a
// bound of 256 MB, which the blocks of these two calls exceed).
// Blocks larger than the bound come from cudaMalloc and go back to it.
//
// A block is idle before it is kept (dev_free waits for the stream of its last
// work), so its next owner may use it on any stream.  A wait for the whole device
// would do the same, but CUDA refuses one while any of its streams is captured,
// and the capture, another thread's perhaps, is lost.
#include <cuda_runtime.h>

#include <atomic>
#include <list>
#include <mutex>
#include <unordered_map>
#include <vector>

#include "trav_internal.cuh"

namespace trav {
namespace {

constexpr size_t kKeepBytes = size_t(1024) << 20;
constexpr size_t kKeepStreams = 8;

struct Block {
    void *p;
    size_t bytes;
    int device;
};

// never destroyed: handles may be freed while the process exits
std::mutex &g_mu = *new std::mutex;
std::unordered_map<void *, Block> &g_live = *new std::unordered_map<void *, Block>;  // blocks handed out
std::list<Block> &g_kept = *new std::list<Block>;                                    // idle blocks, oldest first
std::vector<std::pair<int, cudaStream_t>> &g_streams = *new std::vector<std::pair<int, cudaStream_t>>;  // idle streams

// Allocations left before the injected failure (-1: none armed).
std::atomic<int64_t> g_fail_after{-1};

int current_device()
{
    int d = 0;
    cudaGetDevice(&d);
    return d;
}

// Take idle blocks of `device` out of the list, oldest first, until those left hold at most `keep` bytes.
std::vector<void *> take_over(int device, size_t keep)
{
    size_t held = 0;
    for (const Block &b : g_kept) held += b.device == device ? b.bytes : 0;
    std::vector<void *> out;
    for (auto it = g_kept.begin(); it != g_kept.end() && held > keep;) {
        if (it->device != device) {
            ++it;
            continue;
        }
        held -= it->bytes;
        out.push_back(it->p);
        it = g_kept.erase(it);
    }
    return out;
}

}  // namespace

void arm_alloc_failure(int32_t after) { g_fail_after.store(after); }

bool alloc_failure_due()
{
    int64_t left = g_fail_after.load();
    while (left >= 0)
        if (g_fail_after.compare_exchange_weak(left, left - 1)) return left == 0;  // fires once, then disarmed
    return false;
}

cudaError_t dev_malloc_bytes(void **p, size_t bytes)
{
    *p = nullptr;
    if (alloc_failure_due()) return cudaErrorMemoryAllocation;
    const int dev = current_device();
    bytes = (bytes + 511) & ~(size_t)511;
    if (bytes == 0) bytes = 512;
    {
        std::lock_guard<std::mutex> lock(g_mu);
        auto best = g_kept.end();
        for (auto it = g_kept.begin(); it != g_kept.end(); ++it)
            if (it->device == dev && it->bytes >= bytes && it->bytes <= bytes + bytes / 4 + 4096 &&
                (best == g_kept.end() || it->bytes < best->bytes))
                best = it;
        if (best != g_kept.end()) {
            *p = best->p;
            g_live[best->p] = *best;
            g_kept.erase(best);
            return cudaSuccess;
        }
    }
    cudaError_t e = cudaMalloc(p, bytes);
    if (e == cudaErrorMemoryAllocation && dev_trim() > 0) {
        cudaGetLastError();
        e = cudaMalloc(p, bytes);
    }
    if (e != cudaSuccess) {
        *p = nullptr;
        return e;
    }
    std::lock_guard<std::mutex> lock(g_mu);
    g_live[*p] = Block{*p, bytes, dev};
    return cudaSuccess;
}

size_t dev_trim()
{
    const int dev = current_device();
    size_t bytes = 0;
    std::vector<void *> out;
    {
        std::lock_guard<std::mutex> lock(g_mu);
        for (const Block &b : g_kept) bytes += b.device == dev ? b.bytes : 0;
        out = take_over(dev, 0);
    }
    for (void *q : out) cudaFree(q);
    return bytes;
}

cudaError_t dev_free_bytes(size_t want, size_t *bytes)
{
    size_t total = 0;
    cudaError_t e = cudaMemGetInfo(bytes, &total);
    if (e == cudaSuccess && *bytes < want && dev_trim() > 0) e = cudaMemGetInfo(bytes, &total);
    return e;
}

void dev_free(void *p, cudaStream_t st)
{
    if (!p) return;
    Block b{p, 0, -1};
    {
        std::lock_guard<std::mutex> lock(g_mu);
        auto it = g_live.find(p);
        if (it != g_live.end()) {
            b = it->second;
            g_live.erase(it);
        }
    }
    if (b.device < 0 || b.bytes > kKeepBytes) {
        cudaFree(p);
        return;
    }
    // nothing may still read or write the block when it is handed on
    const int cur = current_device();
    if (cur != b.device) cudaSetDevice(b.device);
    const cudaError_t e = cudaStreamSynchronize(st);
    if (cur != b.device) cudaSetDevice(cur);
    if (e != cudaSuccess) {
        cudaGetLastError();  // not the caller's next launch's
        cudaFree(p);
        return;
    }
    std::vector<void *> out;
    {
        std::lock_guard<std::mutex> lock(g_mu);
        out = take_over(b.device, kKeepBytes - b.bytes);
        g_kept.push_back(b);
    }
    for (void *q : out) cudaFree(q);
}

cudaError_t stream_get(cudaStream_t *st)
{
    const int dev = current_device();
    {
        std::lock_guard<std::mutex> lock(g_mu);
        for (auto it = g_streams.begin(); it != g_streams.end(); ++it)
            if (it->first == dev) {
                *st = it->second;
                g_streams.erase(it);
                return cudaSuccess;
            }
    }
    return cudaStreamCreateWithFlags(st, cudaStreamNonBlocking);
}

void stream_put(cudaStream_t st)
{
    if (!st) return;
    if (cudaStreamSynchronize(st) == cudaSuccess) {
        std::lock_guard<std::mutex> lock(g_mu);
        if (g_streams.size() < kKeepStreams) {
            g_streams.emplace_back(current_device(), st);
            return;
        }
    }
    cudaStreamDestroy(st);
}

}  // namespace trav
