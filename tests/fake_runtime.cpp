// csrc/memory.cu on a CUDA runtime of the host: copies wait in one queue and are carried out when something waits for them (or now and
// then when an event is asked for), device memory is host memory with a limit. A staging buffer that is used again too early, a
// block that is not given back, an exception in a destructor all show. Argument: the part to run.
#include <omp.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include <atomic>
#include <deque>
#include <map>
#include <mutex>
#include <new>
#include <random>
#include <set>
#include <string>
#include <thread>
#include <vector>

#include "../alphasparse_b200/csrc/host/crew.cpp"
#include "../alphasparse_b200/csrc/host/hostmem.cpp"
#include "../alphasparse_b200/csrc/memory.cu"

static std::atomic<long> countdown{-1}, refused{0};
static thread_local bool in_runtime = false; // (the queue below is no part of what is tested)
void *operator new(size_t n)
{
    const bool no = !in_runtime && countdown >= 0 && countdown-- == 0;
    if (no) refused++;
    void *p = no ? nullptr : malloc(n ? n : 1);
    if (!p) throw std::bad_alloc();
    return p;
}
void operator delete(void *p) noexcept { free(p); }
void operator delete(void *p, size_t) noexcept { free(p); }

static void need(bool ok, const char *what)
{
    if (ok) return;
    printf("failed: %s\n", what);
    fflush(stdout);
    _Exit(4);
}

namespace fake
{
struct Op
{
    void *dst;
    const void *src;
    size_t n;
    cudaEvent_t event;
};
std::recursive_mutex lock;
std::deque<Op> queue;
std::map<cudaEvent_t, int> pending; // records of an event that are still in the queue
std::map<void *, size_t> blocks;
std::vector<std::pair<const char *, size_t>> page_locked;
bool read_only = false;
size_t in_use = 0, limit = ~0ull;
std::mt19937 rng(1);
long next_event = 1;

void step()
{
    Op o = queue.front();
    queue.pop_front();
    if (o.event) pending[o.event]--;
    else memcpy(o.dst, o.src, o.n);
}
} // namespace fake
struct InRuntime
{
    const bool was = in_runtime;
    InRuntime() { in_runtime = true; }
    ~InRuntime() { in_runtime = was; }
};
#define LOCKED std::lock_guard<std::recursive_mutex> g(fake::lock); InRuntime in

extern "C" {
cudaError_t cudaGetDevice(int *d) { return *d = 0, cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaMalloc(void **p, size_t n)
{
    LOCKED;
    if (fake::in_use + n > fake::limit) return cudaErrorMemoryAllocation;
    *p = malloc(n);
    fake::blocks[*p] = n;
    fake::in_use += n;
    return cudaSuccess;
}
cudaError_t cudaFree(void *p)
{
    LOCKED;
    if (!p) return cudaSuccess;
    need(fake::blocks.count(p) == 1, "freed a block that is none");
    fake::in_use -= fake::blocks[p];
    fake::blocks.erase(p);
    free(p);
    return cudaSuccess;
}
cudaError_t cudaMemGetInfo(size_t *f, size_t *all) { return *all = fake::limit, *f = fake::limit - fake::in_use, cudaSuccess; }
cudaError_t cudaDeviceSynchronize()
{
    LOCKED;
    while (!fake::queue.empty()) fake::step();
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaDeviceSynchronize(); }
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) { return *p = malloc(n), cudaSuccess; }
cudaError_t cudaFreeHost(void *p) { return free(p), cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned)
{
    LOCKED;
    return *e = (cudaEvent_t)(fake::next_event++), cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t)
{
    LOCKED;
    fake::pending[e]++;
    fake::queue.push_back({nullptr, nullptr, 0, e});
    return cudaSuccess;
}
cudaError_t cudaEventQuery(cudaEvent_t e)
{
    LOCKED;
    for (unsigned k = fake::rng() % 3; k > 0 && !fake::queue.empty(); k--) fake::step();
    return fake::pending[e] ? cudaErrorNotReady : cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t e)
{
    LOCKED;
    while (fake::pending[e]) fake::step();
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *dst, const void *src, size_t n, cudaMemcpyKind kind, cudaStream_t)
{
    LOCKED;
    if (n < (64u << 10) && kind == cudaMemcpyHostToDevice)
    {
        // pageable memory (or a small piece): taken when the call returns, written in order
        void *copy = malloc(n);
        memcpy(copy, src, n);
        fake::queue.push_back({dst, copy, n, nullptr});
    }
    else
        fake::queue.push_back({dst, src, n, nullptr});
    return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *a, const void *p)
{
    *a = {};
    a->type = cudaMemoryTypeUnregistered;
    for (auto &r : fake::page_locked)
        if ((const char *)p >= r.first && (const char *)p < r.first + r.second) a->type = cudaMemoryTypeHost, a->hostPointer = a->devicePointer = (void *)p;
    return cudaSuccess;
}
static CUresult pointer_attribute(void *out, CUpointer_attribute what, CUdeviceptr p)
{
    for (auto &r : fake::page_locked)
        if ((const char *)p >= r.first && (const char *)p < r.first + r.second)
        {
            if (what == CU_POINTER_ATTRIBUTE_RANGE_START_ADDR) *(CUdeviceptr *)out = (CUdeviceptr)r.first;
            else if (what == CU_POINTER_ATTRIBUTE_RANGE_SIZE) *(size_t *)out = r.second;
            else if (what == CU_POINTER_ATTRIBUTE_ACCESS_FLAGS) *(int *)out = fake::read_only ? CU_POINTER_ATTRIBUTE_ACCESS_FLAG_READ : CU_POINTER_ATTRIBUTE_ACCESS_FLAG_READWRITE;
            else return CUDA_ERROR_INVALID_VALUE;
            return CUDA_SUCCESS;
        }
    return CUDA_ERROR_INVALID_VALUE;
}
cudaError_t cudaGetDriverEntryPoint(const char *name, void **f, unsigned long long, cudaDriverEntryPointQueryResult *found)
{
    need(std::string(name) == "cuPointerGetAttribute", "an unknown call of the driver");
    return *f = (void *)pointer_attribute, *found = cudaDriverEntryPointSuccess, cudaSuccess;
}
}

typedef std::vector<unsigned char> Bytes;
static Bytes random_bytes(size_t n, unsigned seed)
{
    Bytes b(n);
    std::mt19937 r(seed);
    for (size_t i = 0; i + 4 <= n; i += 4) *(unsigned *)&b[i] = r();
    for (size_t i = n & ~3ull; i < n; i++) b[i] = (unsigned char)r();
    return b;
}

// uploads whose source changes as soon as the call is back, downloads, in turn, from changing places of the ring
static void ring(asp::Stager &s, unsigned seed, int rounds)
{
    std::mt19937 r(seed);
    const size_t sizes[] = {1, 65535, 65536, 196609, 262143, 262144, 262145, 1 << 20, (1 << 20) + 1, (5 << 20) + 12345, (17 << 20) + 1, (40 << 20) + 4097};
    for (int i = 0; i < rounds; i++)
    {
        const size_t n = sizes[(i + seed) % 12];
        Bytes src = random_bytes(n, seed * 1000 + i), keep = src, dev(n, 1), back(n, 2);
        if (r() % 2) need(s.to_device(dev.data(), src.data(), n, nullptr) == cudaSuccess, "to_device");
        else
        {
            std::vector<asp::Stager::Segment> seg;
            for (size_t at = 0; at < n;)
            {
                const size_t len = std::min<size_t>(n - at, 1 + r() % (1 << 21));
                seg.push_back({at, src.data() + at, len});
                at += len;
            }
            need(s.to_device(dev.data(), seg, nullptr) == cudaSuccess, "to_device of segments");
        }
        memset(src.data(), 0x55, n);
        need(s.to_host(back.data(), dev.data(), n, nullptr) == cudaSuccess, "to_host");
        need(back == keep, "an upload or a download is damaged");
    }
}

int main(int, char **argv)
{
    const std::string part = argv[1];
    omp_set_num_threads(4);
    asp::device_pool_retain(0);
    if (part == "ring")
    {
        asp::Stager s;
        ring(s, 1, 36);
        s.release();
    }
    if (part == "threads")
    {
        // two threads, one context's ring (a program that makes plans in the background)
        asp::Stager s;
        std::thread a([&] { omp_set_num_threads(2); ring(s, 2, 36); }), b([&] { omp_set_num_threads(2); ring(s, 7, 36); });
        a.join();
        b.join();
        s.release();
    }
    if (part == "no memory")
    {
        // blocks that come back, and an upload, while nothing can be allocated
        asp::Stager s;
        void *p = nullptr;
        size_t got = 0;
        need(asp::device_alloc(0, 1 << 20, &p, &got) == cudaSuccess, "device_alloc");
        std::shared_ptr<void> big = asp::host::big_buffer(8 << 20);
        Bytes src = random_bytes(9 << 20, 3), dev(src.size()), back(src.size());
        need(s.to_device(dev.data(), src.data(), 1 << 20, nullptr) == cudaSuccess, "first upload"); // (makes the ring)
        countdown = 0;
        asp::device_free(0, p, got);
        need(refused == 1, "the pool noted the block without memory");
        countdown = 0;
        big.reset();
        need(refused == 2, "the host pool noted the block without memory");
        for (long n = 0; n < 8; n++)
        {
            memset(dev.data(), 0, dev.size());
            countdown = n;
            need(s.to_device(dev.data(), src.data(), src.size(), nullptr) == cudaSuccess, "an upload without memory for its tables");
            countdown = -1;
            cudaDeviceSynchronize();
            need(dev == src, "the upload is damaged");
        }
        s.release();
    }
    if (part == "full device")
    {
        // idle blocks fill the device: allocations of every kind get them, and a trim call gives them back
        void *p[3], *q = nullptr;
        size_t got[3];
        fake::limit = 100u << 20;
        for (int i = 0; i < 3; i++) need(asp::device_alloc(0, (30u << 20) + i * (2u << 20), &p[i], &got[i]) == cudaSuccess, "device_alloc");
        for (int i = 0; i < 3; i++) asp::device_free(0, p[i], got[i]);
        need(fake::in_use > (90u << 20), "the pool keeps nothing");
        need(asp::device_has_room(0, 100u << 20) && !asp::device_has_room(0, 101u << 20), "idle blocks count as room");
        need(asp::device_malloc(0, 60u << 20, &q) == cudaSuccess, "an allocation beside the pool");
        size_t size = 0;
        void *r = nullptr;
        need(asp::device_alloc(0, 30u << 20, &r, &size, 11u << 20) == cudaErrorMemoryAllocation, "an allocation that leaves too little");
        need(asp::device_alloc(0, 30u << 20, &r, &size, 10u << 20) == cudaSuccess, "one that leaves enough");
        asp::device_free(0, r, size);
        need(asp::device_alloc(0, 30u << 20, &r, &size, 11u << 20) == cudaSuccess, "one from the pool");
        asp::device_free(0, r, size);
        need(asp::device_has_room(0, 40u << 20) && !asp::device_has_room(0, 41u << 20), "what is in use is none");
        cudaFree(q);
        for (int i = 0; i < 3; i++) need(asp::device_alloc(0, 30u << 20, &p[i], &got[i]) == cudaSuccess, "device_alloc");
        for (int i = 0; i < 3; i++) asp::device_free(0, p[i], got[i]);
        need(fake::in_use > 0, "the pool keeps nothing");
        asp::device_trim(0);
        need(fake::in_use == 0, "idle blocks after a trim");
    }
    if (part == "views")
    {
        // a buffer is seen by the device only where all of it is page-locked, in one range
        Bytes b(1 << 20);
        char *p = (char *)b.data();
        fake::page_locked = {{p + 4096, 8192}, {p + 12288, 4096}, {p + 40960, 4096}};
        need(asp::device_view(p + 4096, 8192) == p + 4096 && asp::device_view(p + 4104, 8184) == p + 4104 && asp::device_view(p + 12287, 1) == p + 12287, "page-locked buffers");
        need(!asp::device_view(p, 4096) && !asp::device_view(p + 4095, 8192), "a buffer that begins before its range");
        need(!asp::device_view(p + 4096, 8193) && !asp::device_view(p + 40968, 4096), "a buffer that ends behind its range");
        need(!asp::device_view(p + 4096, 12288), "a buffer over two ranges");
        need(!asp::device_view(p + 12288, 32768), "a buffer whose ends are page-locked");
        fake::read_only = true;
        need(!asp::device_view(p + 4096, 8192), "a buffer that is registered for reading");
    }
    asp::device_pool_release(0);
    need(fake::blocks.empty(), "device memory is left");
    printf("%s: ok\n", part.c_str());
    return 0;
}
