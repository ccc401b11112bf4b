// A CUDA runtime of the host for tests of the library's memory management: allocations, streams, captures and
// contexts are records that the test looks at, and calls follow the documented rules (a device-wide wait is
// refused while any stream is captured, memory of an ended context is gone, and so on).  Compiled into the test
// program together with csrc/device_memory.cu; no device is needed.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>

#include <cstring>

#include <map>
#include <mutex>
#include <string>
#include <vector>

static const uint3 blockIdx{}, threadIdx{};

namespace fake {

struct Alloc {
    size_t bytes;
    unsigned long long id;
    int context;
};
struct Stream {
    bool busy = false;
    bool captured = false;
    int context = 0;
};

inline std::mutex mu;
inline thread_local int inside = 0;  // calls of this runtime on the thread's stack
struct Entry {
    std::lock_guard<std::mutex> lock{mu};
    Entry() { inside++; }
    ~Entry() { inside--; }
};
inline std::map<void *, Alloc> allocs;
inline std::map<cudaStream_t, Stream> streams;  // key 0: the legacy stream
inline std::vector<std::string> log;
inline size_t capacity = size_t(180) << 30, used = 0;
inline unsigned long long next_id = 1;
inline unsigned char *const first_at = reinterpret_cast<unsigned char *>(0x700000000000ull), *next_at = first_at;
inline int context = 1;       // the context that lives now
inline bool current = false;  // and whether it is current yet (in any thread: there is one)
inline CUcontext handle = reinterpret_cast<CUcontext>(0x10);  // where the driver keeps it
inline bool driver = true;    // the driver's entry points can be found
inline cudaError_t last = cudaSuccess;

inline cudaError_t fail(cudaError_t e) { return last = e; }
inline size_t count(const std::string &what)
{
    size_t n = 0;
    for (const std::string &s : log) n += s == what;
    return n;
}
// What cudaDeviceReset leaves: no allocation, no stream, and another context at the next call, which the driver may
// keep where the old one was and whose memory may begin where the old one's did.
inline void reset(CUcontext at, bool same_addresses)
{
    handle = at;
    if (same_addresses) next_at = first_at;
    current = false;
    allocs.clear();
    streams.clear();
    used = 0;
    context++;
}

}  // namespace fake

extern "C" {

cudaError_t cudaMalloc(void **p, size_t bytes)
{
    fake::Entry entry;
    using namespace fake;
    log.push_back("malloc");
    current = true;
    if (used + bytes > capacity) return fail(cudaErrorMemoryAllocation);
    *p = next_at;
    next_at += (bytes + 511) & ~size_t(511);
    allocs[*p] = Alloc{bytes, next_id++, context};
    used += bytes;
    return cudaSuccess;
}
cudaError_t cudaFree(void *p)
{
    fake::Entry entry;
    using namespace fake;
    current = true;
    if (!p) return cudaSuccess;
    log.push_back("free");
    auto it = allocs.find(p);
    if (it == allocs.end()) return fail(cudaErrorInvalidValue);
    used -= it->second.bytes;
    allocs.erase(it);
    return cudaSuccess;
}
cudaError_t cudaMemGetInfo(size_t *f, size_t *t)
{
    fake::Entry entry;
    *f = fake::capacity - fake::used;
    *t = fake::capacity;
    return cudaSuccess;
}
cudaError_t cudaGetDevice(int *d) { return *d = 0, cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetLastError()
{
    fake::Entry entry;
    const cudaError_t e = fake::last;
    fake::last = cudaSuccess;
    return e;
}
cudaError_t cudaDeviceSynchronize()
{
    fake::Entry entry;
    using namespace fake;
    log.push_back("device wait");
    for (auto &s : streams)
        if (s.second.captured) return fail(cudaErrorStreamCaptureUnsupported);
    for (auto &s : streams) s.second.busy = false;
    return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *st, unsigned)
{
    fake::Entry entry;
    using namespace fake;
    static unsigned long long at = 0x1000;
    log.push_back("stream create");
    *st = reinterpret_cast<cudaStream_t>(at += 16);
    streams[*st] = Stream{false, false, context};
    return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t st)
{
    fake::Entry entry;
    using namespace fake;
    log.push_back("stream destroy");
    if (!streams.erase(st)) log.push_back("destroyed a stream that is gone");
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t st)
{
    fake::Entry entry;
    using namespace fake;
    if (st && !streams.count(st)) {
        log.push_back("waited for a stream that is gone");
        return fail(cudaErrorInvalidResourceHandle);
    }
    if (streams[st].captured) return fail(cudaErrorStreamCaptureUnsupported);
    streams[st].busy = false;
    return cudaSuccess;
}

CUresult fake_cuCtxGetCurrent(CUcontext *c)
{
    *c = fake::current ? fake::handle : nullptr;
    return CUDA_SUCCESS;
}
CUresult fake_cuPointerGetAttribute(void *out, CUpointer_attribute what, CUdeviceptr p)
{
    fake::Entry entry;
    auto it = fake::allocs.find(reinterpret_cast<void *>(p));
    if (what != CU_POINTER_ATTRIBUTE_BUFFER_ID || it == fake::allocs.end()) return CUDA_ERROR_INVALID_VALUE;
    *static_cast<unsigned long long *>(out) = it->second.id;
    return CUDA_SUCCESS;
}
cudaError_t cudaGetDriverEntryPointByVersion(const char *name, void **fn, unsigned, unsigned long long,
                                             cudaDriverEntryPointQueryResult *r)
{
    *fn = nullptr;
    *r = cudaDriverEntryPointSymbolNotFound;
    if (!fake::driver) return fake::fail(cudaErrorInsufficientDriver);
    if (!std::strcmp(name, "cuCtxGetCurrent")) *fn = reinterpret_cast<void *>(fake_cuCtxGetCurrent);
    if (!std::strcmp(name, "cuPointerGetAttribute")) *fn = reinterpret_cast<void *>(fake_cuPointerGetAttribute);
    *r = cudaDriverEntryPointSuccess;
    return cudaSuccess;
}

}  // extern "C"
