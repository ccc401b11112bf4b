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
//
// Host memory can run out too: an allocation then fails as one of the device's
// does, and freeing allocates nothing (the list nodes move), since it happens in
// destructors.
//
// Blocks and streams belong to the context they were made in, and are gone when
// it ends (cudaDeviceReset).  So they are kept by context, and each context's
// keeps hold a mark: an allocation whose buffer id, which no other allocation of
// the process ever has, is asked for before anything is handed out.
#include <cuda.h>
#include <cuda_runtime.h>

#include <atomic>
#include <list>
#include <mutex>
#include <new>
#include <unordered_map>
#include <vector>

#include "trav_internal.cuh"

namespace trav {
namespace {

constexpr size_t kKeepBytes = size_t(1024) << 20;
constexpr size_t kKeepStreams = 8;
constexpr size_t kMarkBytes = 512;

struct Block {
    void *p;
    size_t bytes;
    int device;
    unsigned long long epoch;  // of its context (0: unknown)
};

// What is kept of one context.
struct Context {
    CUcontext handle;
    unsigned long long epoch;  // no other context of the process has it, a later one at the same address neither
    void *mark;
    unsigned long long mark_id;
    std::list<Block> kept;     // idle blocks, oldest first
    std::vector<cudaStream_t> streams;  // idle streams
};

// never destroyed: handles may be freed while the process exits
std::mutex &g_mu = *new std::mutex;
std::list<Block> &g_live = *new std::list<Block>;  // blocks handed out, and where to find them
std::unordered_map<void *, std::list<Block>::iterator> &g_live_at = *new std::unordered_map<void *, std::list<Block>::iterator>;
std::unordered_map<cudaStream_t, unsigned long long> &g_live_streams =
    *new std::unordered_map<cudaStream_t, unsigned long long>;  // streams handed out, and their contexts' epochs
std::list<Context> &g_contexts = *new std::list<Context>;
unsigned long long g_epochs = 0;

// Allocations left before the injected failure (-1: none armed).
std::atomic<int64_t> g_fail_after{-1};

int current_device()
{
    int d = 0;
    cudaGetDevice(&d);
    return d;
}

// The two driver calls that know about contexts (the runtime has none, and the
// library does not link the driver, which a machine without a GPU lacks).
struct Driver {
    CUresult (*current)(CUcontext *) = nullptr;
    CUresult (*attribute)(void *, CUpointer_attribute, CUdeviceptr) = nullptr;
    Driver()
    {
        cudaDriverEntryPointQueryResult r;
        if (cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", (void **)&current, 12000, cudaEnableDefault, &r) != cudaSuccess ||
            cudaGetDriverEntryPointByVersion("cuPointerGetAttribute", (void **)&attribute, 12000, cudaEnableDefault, &r) != cudaSuccess) {
            cudaGetLastError();
            current = nullptr;
        }
    }
    CUcontext context() const
    {
        CUcontext c = nullptr;
        return current(&c) == CUDA_SUCCESS ? c : nullptr;
    }
    unsigned long long buffer_id(void *p) const  // 0: no allocation
    {
        unsigned long long id = 0;
        return attribute(&id, CU_POINTER_ATTRIBUTE_BUFFER_ID, (CUdeviceptr)p) == CUDA_SUCCESS ? id : 0;
    }
};

const Driver &the_driver()
{
    static const Driver d;
    return d;
}

// The keeps of the current context (g_mu held); nullptr: nothing can be kept.
Context *context_here()
{
    const Driver &driver = the_driver();
    if (!driver.current || !driver.attribute) return nullptr;
    CUcontext c = driver.context();
    if (!c) {
        // a thread's first call: the runtime makes the device's context current
        if (cudaFree(nullptr) != cudaSuccess) cudaGetLastError();
        c = driver.context();
    }
    for (auto it = g_contexts.begin(); c && it != g_contexts.end(); ++it) {
        if (it->handle != c) continue;
        if (driver.buffer_id(it->mark) == it->mark_id) return &*it;
        // that context has ended, and its blocks and streams with it
        g_contexts.erase(it);
        break;
    }
    Context n{nullptr, 0, nullptr, 0, {}, {}};
    if (cudaMalloc(&n.mark, kMarkBytes) != cudaSuccess) {
        cudaGetLastError();
        return nullptr;
    }
    n.handle = driver.context();
    n.mark_id = driver.buffer_id(n.mark);
    if (!n.handle || !n.mark_id) {
        cudaFree(n.mark);
        return nullptr;
    }
    n.epoch = ++g_epochs;
    try {
        g_contexts.push_back(n);
        g_contexts.back().streams.reserve(kKeepStreams);
    } catch (const std::bad_alloc &) {
        while (!g_contexts.empty() && g_contexts.back().epoch == n.epoch) g_contexts.pop_back();
        cudaFree(n.mark);
        return nullptr;
    }
    return &g_contexts.back();
}

// Whether the context of this epoch is not known to have ended (g_mu held).
bool lives(unsigned long long epoch)
{
    if (epoch == 0) return true;
    for (auto it = g_contexts.begin(); it != g_contexts.end(); ++it) {
        if (it->epoch != epoch) continue;
        if (the_driver().buffer_id(it->mark) == it->mark_id) return true;
        g_contexts.erase(it);
        break;
    }
    return false;
}

// Take idle blocks of a context out of its list, oldest first, until those left hold at most `keep` bytes.
std::list<Block> take_over(Context *c, size_t keep)
{
    size_t held = 0;
    for (const Block &b : c->kept) held += b.bytes;
    std::list<Block> out;
    while (!c->kept.empty() && held > keep) {
        held -= c->kept.front().bytes;
        out.splice(out.end(), c->kept, c->kept.begin());
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

unsigned long long context_epoch()
{
    std::lock_guard<std::mutex> lock(g_mu);
    const Context *c = context_here();
    return c ? c->epoch : 0;
}

cudaError_t dev_malloc_bytes(void **p, size_t bytes)
{
    *p = nullptr;
    if (alloc_failure_due()) return cudaErrorMemoryAllocation;
    bytes = (bytes + 511) & ~(size_t)511;
    if (bytes == 0) bytes = 512;
    unsigned long long epoch = 0;
    {
        std::lock_guard<std::mutex> lock(g_mu);
        if (Context *c = context_here()) {
            epoch = c->epoch;
            auto best = c->kept.end();
            for (auto it = c->kept.begin(); it != c->kept.end(); ++it)
                if (it->bytes >= bytes && it->bytes <= bytes + bytes / 4 + 4096 &&
                    (best == c->kept.end() || it->bytes < best->bytes))
                    best = it;
            if (best != c->kept.end()) {
                try {
                    g_live_at.emplace(best->p, best);
                } catch (const std::bad_alloc &) {
                    return cudaErrorMemoryAllocation;
                }
                g_live.splice(g_live.end(), c->kept, best);
                *p = best->p;
                return cudaSuccess;
            }
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
    std::list<Block> node;
    std::lock_guard<std::mutex> lock(g_mu);
    try {
        node.push_back(Block{*p, bytes, current_device(), epoch});
        g_live_at[*p] = node.begin();
    } catch (const std::bad_alloc &) {
        cudaFree(*p);
        *p = nullptr;
        return cudaErrorMemoryAllocation;
    }
    g_live.splice(g_live.end(), node);
    return cudaSuccess;
}

size_t dev_trim()
{
    size_t bytes = 0;
    std::list<Block> out;
    {
        std::lock_guard<std::mutex> lock(g_mu);
        if (Context *c = context_here()) out = take_over(c, 0);
    }
    for (const Block &b : out) {
        bytes += b.bytes;
        cudaFree(b.p);
    }
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
    std::list<Block> node;
    {
        std::lock_guard<std::mutex> lock(g_mu);
        auto it = g_live_at.find(p);
        if (it != g_live_at.end()) {
            node.splice(node.end(), g_live, it->second);
            g_live_at.erase(it);
        }
    }
    if (node.empty()) {
        cudaFree(p);
        return;
    }
    const Block b = node.front();
    const int cur = current_device();
    if (cur != b.device) cudaSetDevice(b.device);
    // nothing may still read or write the block when it is handed on
    const cudaError_t e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) cudaGetLastError();  // not the caller's next launch's
    std::list<Block> out;
    {
        std::lock_guard<std::mutex> lock(g_mu);
        Context *c = context_here();
        if (e == cudaSuccess && c && c->epoch == b.epoch && b.bytes <= kKeepBytes) {
            out = take_over(c, kKeepBytes - b.bytes);
            c->kept.splice(c->kept.end(), node);
        } else if (lives(b.epoch)) {
            out.splice(out.end(), node);
        }
    }
    for (const Block &x : out) cudaFree(x.p);
    if (cur != b.device) cudaSetDevice(cur);
}

cudaError_t stream_get(cudaStream_t *st)
{
    std::lock_guard<std::mutex> lock(g_mu);
    Context *c = context_here();
    if (c && !c->streams.empty()) {
        *st = c->streams.back();
        c->streams.pop_back();
    } else {
        const cudaError_t e = cudaStreamCreateWithFlags(st, cudaStreamNonBlocking);
        if (e != cudaSuccess) return e;
    }
    try {
        g_live_streams[*st] = c ? c->epoch : 0;
    } catch (const std::bad_alloc &) {
        cudaStreamDestroy(*st);
        *st = nullptr;
        return cudaErrorMemoryAllocation;
    }
    return cudaSuccess;
}

void stream_put(cudaStream_t st)
{
    if (!st) return;
    unsigned long long epoch = 0;
    {
        std::lock_guard<std::mutex> lock(g_mu);
        auto it = g_live_streams.find(st);
        if (it != g_live_streams.end()) {
            epoch = it->second;
            g_live_streams.erase(it);
        }
        context_here();
        if (!lives(epoch)) return;
    }
    if (cudaStreamSynchronize(st) == cudaSuccess) {
        std::lock_guard<std::mutex> lock(g_mu);
        Context *c = context_here();
        if (c && c->epoch == epoch && c->streams.size() < kKeepStreams) {
            c->streams.push_back(st);
            return;
        }
    }
    cudaStreamDestroy(st);
}

}  // namespace trav
