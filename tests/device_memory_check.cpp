// The library's device-memory management (csrc/device_memory.cu) on a CUDA runtime of the host: one scenario a run.
#include "fake_cudart.hpp"

#include "../parallel-task1_b200/csrc/device_memory.cu"

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>
#include <thread>

using namespace trav;

// The library's host allocations that still succeed (-1: all).
static std::atomic<int> g_host_left{-1};
void *operator new(size_t n)
{
    if (!fake::inside && g_host_left >= 0 && g_host_left-- == 0) {
        g_host_left = 0;
        throw std::bad_alloc();
    }
    if (void *p = std::malloc(n ? n : 1)) return p;
    throw std::bad_alloc();
}
void operator delete(void *p) noexcept { std::free(p); }
void operator delete(void *p, size_t) noexcept { std::free(p); }

static int g_bad = 0;
#define CHECK(x)                                                      \
    do {                                                              \
        if (!(x)) {                                                   \
            std::printf("line %d: not so: %s\n", __LINE__, #x);       \
            g_bad = 1;                                                \
        }                                                             \
    } while (0)

static const size_t MB = size_t(1) << 20;

static void *get(size_t bytes)
{
    void *p = nullptr;
    CHECK(dev_malloc_bytes(&p, bytes) == cudaSuccess && p);
    return p;
}
// Bytes allocated, but for the mark of the context.
static size_t in_use() { return fake::used - 512; }
static cudaStream_t stream()
{
    cudaStream_t st = nullptr;
    CHECK(stream_get(&st) == cudaSuccess && st);
    return st;
}

// A freed block goes to the next owner of about its size, once the stream of its last work has been waited for.
static void reuse()
{
    cudaStream_t a = stream();
    void *p = get(10 * MB);
    fake::streams[a].busy = true;
    dev_free(p, a);
    CHECK(!fake::streams[a].busy);
    CHECK(get(20 * MB) != p);
    CHECK(get(10 * MB - 100) == p);  // on whatever stream
    CHECK(get(10 * MB) != p);
    CHECK(fake::count("free") == 0);
}

// Another stream is being captured: no wait for the device, no error left behind, and the block is kept.
static void capture()
{
    cudaStream_t a = stream(), b = stream();
    fake::streams[b].captured = true;
    void *p = get(10 * MB);
    dev_free(p, a);
    CHECK(cudaGetLastError() == cudaSuccess);
    CHECK(fake::count("device wait") == 0);
    CHECK(get(10 * MB) == p);
    // a wait that fails leaves no error for the caller's next launch, and the block is not kept
    dev_free(p, b);
    CHECK(cudaGetLastError() == cudaSuccess);
    CHECK(fake::count("free") == 1);
}

// What is kept stays below the bound: the oldest blocks go, and a block above the bound is not kept at all.
static void bound()
{
    cudaStream_t a = stream();
    void *big = get(1025 * MB);
    dev_free(big, a);
    CHECK(in_use() == 0);
    std::vector<void *> p;
    for (int i = 0; i < 12; i++) p.push_back(get(100 * MB));
    for (void *x : p) {
        dev_free(x, a);
    }
    CHECK(in_use() == 1000 * MB);
    CHECK(!fake::allocs.count(p[0]) && !fake::allocs.count(p[1]) && fake::allocs.count(p[2]));
}

// An allocation that does not fit beside the kept blocks gets their memory; one that cannot fit fails.
static void give_back()
{
    cudaStream_t a = stream();
    fake::capacity = 1000 * MB;
    void *p = get(600 * MB);
    dev_free(p, a);
    void *q = get(900 * MB);
    CHECK(in_use() == 900 * MB);
    void *r = nullptr;
    CHECK(dev_malloc_bytes(&r, 200 * MB) == cudaErrorMemoryAllocation && !r);
    dev_free(q, a);
    CHECK(get(999 * MB) != nullptr);
    arm_alloc_failure(0);
    CHECK(dev_malloc_bytes(&r, 1) == cudaErrorMemoryAllocation && !r);
}

// What is kept counts as free where the free memory decides what is asked for.
static void counts_as_free()
{
    cudaStream_t a = stream();
    fake::capacity = 1000 * MB;
    get(300 * MB);
    dev_free(get(200 * MB), a);
    size_t bytes = 0;
    CHECK(dev_free_bytes(400 * MB, &bytes) == cudaSuccess && bytes / MB == 499);
    CHECK(fake::count("free") == 0);  // enough: the block stays
    CHECK(dev_free_bytes(600 * MB, &bytes) == cudaSuccess && bytes / MB == 699);
    CHECK(fake::count("free") == 1 && dev_trim() == 0);
    CHECK(dev_free_bytes(900 * MB, &bytes) == cudaSuccess && bytes / MB == 699);
}

// The context ends and another begins, where the old one was or elsewhere: nothing of the old one is handed out,
// freed or waited for.
static void contexts(CUcontext at, bool same_addresses)
{
    cudaStream_t a = stream(), b = stream();
    void *p = get(10 * MB), *late = get(30 * MB);
    dev_free(p, a);
    stream_put(b);
    const unsigned long long epoch = context_epoch();
    CHECK(epoch != 0 && context_epoch() == epoch);
    fake::reset(at, same_addresses);
    fake::log.clear();
    CHECK(context_epoch() != epoch && context_epoch() != 0);
    cudaStream_t c = stream();
    CHECK(c != b && fake::streams.count(c));
    void *q = get(10 * MB), *r = get(30 * MB);
    CHECK(fake::allocs.count(q) && fake::allocs.count(r) && in_use() == 40 * MB);
    dev_free(r, c);
    CHECK(get(30 * MB) == r);  // kept and handed out again
    CHECK(dev_trim() == 0);
    if (late != q && late != r) dev_free(late, nullptr);  // of the old one: there is nothing to free
    CHECK(fake::count("free") == 0 && fake::count("waited for a stream that is gone") == 0);
    stream_put(a);
    CHECK(fake::count("destroyed a stream that is gone") == 0);
}
static void context_in_place() { contexts(fake::handle, true); }
static void context_elsewhere() { contexts(reinterpret_cast<CUcontext>(0x20), false); }

// A driver without the entry points: nothing is kept.
static void no_driver()
{
    fake::driver = false;
    cudaStream_t a = stream();
    dev_free(get(10 * MB), a);
    CHECK(fake::count("free") == 1 && fake::used == 0 && context_epoch() == 0);
    stream_put(a);
    CHECK(fake::count("stream destroy") == 1 && cudaGetLastError() == cudaSuccess);
}

// No host memory: allocations fail without a leak, and freeing needs none.
static void host_memory()
{
    cudaStream_t a = stream(), b = nullptr;
    void *p = get(10 * MB), *q = get(20 * MB), *r = nullptr;
    dev_free(q, a);
    for (int left = 0; left < 4; left++) {
        const size_t used = fake::used;
        g_host_left = left;
        const cudaError_t e = dev_malloc_bytes(&r, 30 * MB);
        g_host_left = -1;
        CHECK(e == cudaSuccess ? r != nullptr : e == cudaErrorMemoryAllocation && !r && fake::used == used);
        dev_free(r, a);
        dev_trim();
    }
    dev_free(get(20 * MB), a);
    g_host_left = 0;
    CHECK(dev_malloc_bytes(&r, 20 * MB) == cudaErrorMemoryAllocation && !r);  // a kept block stays where it is
    CHECK(stream_get(&b) == cudaErrorMemoryAllocation && !b);
    dev_free(p, a);
    stream_put(a);
    g_host_left = -1;
    CHECK(get(10 * MB) == p);
    CHECK(stream() == a);
    DevSlab s(a);
    int *x[25];
    for (int **i = x; i < x + 24; i++) s.add(i, 100);
    CHECK(s.commit() == cudaSuccess && x[23] == x[0] + 23 * 128);
    DevSlab t(a);
    for (int *&i : x) t.add(&i, 100);
    CHECK(t.commit() == cudaErrorInvalidValue && !x[24]);
}

// Several threads: no block has two owners.
static void threads()
{
    std::mutex mu;
    std::map<void *, int> owner;
    std::vector<std::thread> ts;
    for (int t = 0; t < 8; t++)
        ts.emplace_back([&, t] {
            std::mt19937 rng(t);
            cudaStream_t st = nullptr;
            CHECK(stream_get(&st) == cudaSuccess);
            std::vector<void *> mine;
            for (int k = 0; k < 4000; k++) {
                if (mine.empty() || rng() % 2) {
                    void *p = nullptr;
                    CHECK(dev_malloc_bytes(&p, (1 + rng() % 40) * MB) == cudaSuccess);
                    std::lock_guard<std::mutex> lock(mu);
                    CHECK(owner.emplace(p, t).second);
                    mine.push_back(p);
                } else {
                    std::swap(mine[rng() % mine.size()], mine.back());
                    {
                        std::lock_guard<std::mutex> lock(mu);
                        CHECK(owner[mine.back()] == t);
                        owner.erase(mine.back());
                    }
                    dev_free(mine.back(), st);
                    mine.pop_back();
                }
            }
            for (void *p : mine) {
                {
                    std::lock_guard<std::mutex> lock(mu);
                    owner.erase(p);
                }
                dev_free(p, st);
            }
            stream_put(st);
        });
    for (auto &t : ts) t.join();
    CHECK(in_use() <= 1024 * MB);
    CHECK(fake::count("waited for a stream that is gone") == 0);
}

int main(int argc, char **argv)
{
    const struct {
        const char *name;
        void (*run)();
    } all[] = {{"reuse", reuse}, {"capture", capture}, {"bound", bound}, {"give_back", give_back},
                {"counts_as_free", counts_as_free}, {"context_in_place", context_in_place},
                {"context_elsewhere", context_elsewhere}, {"no_driver", no_driver}, {"host_memory", host_memory},
                {"threads", threads}};
    for (const auto &s : all)
        if (argc == 2 && !std::strcmp(argv[1], s.name)) {
            s.run();
            return g_bad;
        }
    std::printf("unknown scenario\n");
    return 2;
}
