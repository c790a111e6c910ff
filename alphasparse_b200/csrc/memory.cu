#include "memory.h"

#include <stdint.h>
#include <string.h>
#if defined(__SSE2__)
#include <emmintrin.h>
#endif

#include <atomic>

#include <algorithm>
#include <map>
#include <mutex>

#include "host/hostmem.hpp"

namespace asp
{
namespace
{
const size_t kMostBlock = 256u << 20, kMostCached = 1u << 30;

struct Pool
{
    std::mutex lock;
    std::multimap<size_t, void *> idle; // by size
    size_t cached = 0;
    int contexts = 0;
};
const int kMaxDevices = 64;
// (never destroyed: plans may be freed while the process ends)
Pool &pool(int device)
{
    static Pool *p = new Pool[kMaxDevices];
    return p[device < 0 || device >= kMaxDevices ? 0 : device];
}

struct OnDevice
{
    int prev = -1;
    explicit OnDevice(int device)
    {
        if (cudaGetDevice(&prev) != cudaSuccess || prev == device) prev = -1;
        else cudaSetDevice(device);
    }
    ~OnDevice()
    {
        if (prev >= 0) cudaSetDevice(prev);
    }
};

std::vector<void *> take_all(Pool &p)
{
    std::vector<void *> out;
    for (auto &b : p.idle) out.push_back(b.second);
    p.idle.clear();
    p.cached = 0;
    return out;
}

// Into pinned memory that the copy engine reads next: past the caches, where it would have to snoop every line out of another
// core's (8 MB filled and sent: 284 us with memcpy, 208 us so).
#if defined(__SSE2__) && !defined(__CUDA_ARCH__)
void stream_copy(unsigned char *dst, const unsigned char *src, size_t n)
{
    if (((uintptr_t)dst & 15) != 0) return (void)memcpy(dst, src, n);
    const size_t body = n / 64 * 64;
    for (size_t i = 0; i < body; i += 64)
        for (int k = 0; k < 64; k += 16) _mm_stream_si128((__m128i *)(dst + i + k), _mm_loadu_si128((const __m128i *)(src + i + k)));
    memcpy(dst + body, src + body, n - body);
    _mm_sfence();
}
#else
void stream_copy(unsigned char *dst, const unsigned char *src, size_t n) { memcpy(dst, src, n); }
#endif

// dst[0, n) from the segments, dst standing for offset `at` of their block
void gather(unsigned char *dst, size_t at, size_t n, const std::vector<Stager::Segment> &seg)
{
    size_t i = (size_t)(std::upper_bound(seg.begin(), seg.end(), at, [](size_t o, const Stager::Segment &s) { return o < s.off; }) - seg.begin());
    if (i > 0) i--;
    for (; i < seg.size() && seg[i].off < at + n; i++)
    {
        const size_t lo = std::max(at, seg[i].off), hi = std::min(at + n, seg[i].off + seg[i].bytes);
        if (lo < hi) stream_copy(dst + (lo - at), (const unsigned char *)seg[i].host + (lo - seg[i].off), hi - lo);
    }
}

const size_t kPart = 64u << 10; // what one thread copies at a time
// a copy of fewer parts is over before the threads are awake
template <class F>
void parts(size_t n, F &&f)
{
    const long long k = (long long)((n + kPart - 1) / kPart);
#pragma omp parallel for schedule(static) if (k > 3)
    for (long long i = 0; i < k; i++) f((size_t)i * kPart, std::min(kPart, n - (size_t)i * kPart));
}
} // namespace

cudaError_t device_alloc(int device, size_t bytes, void **out, size_t *got)
{
    const size_t unit = bytes < (1u << 20) ? (64u << 10) : (2u << 20);
    const size_t want = (std::max<size_t>(bytes, 1) + unit - 1) / unit * unit;
    Pool &p = pool(device);
    {
        std::lock_guard<std::mutex> g(p.lock);
        auto it = p.idle.lower_bound(want);
        if (it != p.idle.end() && it->first <= want + want / 4 + unit)
        {
            *out = it->second;
            *got = it->first;
            p.cached -= it->first;
            p.idle.erase(it);
            return cudaSuccess;
        }
    }
    OnDevice on(device);
    cudaError_t e = cudaMalloc(out, want);
    if (e == cudaErrorMemoryAllocation)
    {
        cudaGetLastError();
        std::vector<void *> idle;
        {
            std::lock_guard<std::mutex> g(p.lock);
            idle = take_all(p);
        }
        for (void *q : idle) cudaFree(q);
        e = cudaMalloc(out, want);
    }
    *got = want;
    return e;
}

void device_free(int device, void *ptr, size_t got)
{
    if (!ptr) return;
    OnDevice on(device);
    Pool &p = pool(device);
    if (got <= kMostBlock && cudaDeviceSynchronize() == cudaSuccess)
    {
        std::lock_guard<std::mutex> g(p.lock);
        if (p.contexts > 0 && p.cached + got <= kMostCached)
        {
            p.idle.insert({got, ptr});
            p.cached += got;
            return;
        }
    }
    cudaFree(ptr);
}

void device_pool_retain(int device)
{
    Pool &p = pool(device);
    std::lock_guard<std::mutex> g(p.lock);
    p.contexts++;
}

void device_pool_release(int device)
{
    Pool &p = pool(device);
    std::vector<void *> idle;
    {
        std::lock_guard<std::mutex> g(p.lock);
        if (--p.contexts > 0) return;
        idle = take_all(p);
    }
    OnDevice on(device);
    for (void *q : idle) cudaFree(q);
    host::host_pool_trim();
}

bool Stager::ready()
{
    if (ring) return true;
    if (off) return false;
    off = true;
    void *p = nullptr;
    if (cudaHostAlloc(&p, kPiece * kPieces, cudaHostAllocDefault) != cudaSuccess)
    {
        cudaGetLastError();
        return false;
    }
    for (int i = 0; i < kPieces; i++)
        if (cudaEventCreateWithFlags(&done[i], cudaEventDisableTiming) != cudaSuccess)
        {
            cudaGetLastError();
            for (int j = 0; j < i; j++) cudaEventDestroy(done[j]);
            cudaFreeHost(p);
            return false;
        }
    ring = (unsigned char *)p;
    off = false;
    return true;
}

void Stager::release()
{
    if (!ring) return;
    for (int i = 0; i < kPieces; i++) cudaEventDestroy(done[i]);
    cudaFreeHost(ring);
    ring = nullptr;
}

bool Stager::pinned(const void *host)
{
    cudaPointerAttributes at;
    if (cudaPointerGetAttributes(&at, host) != cudaSuccess)
    {
        cudaGetLastError();
        return true; // whatever it is, the runtime's own copy knows best
    }
    return at.type != cudaMemoryTypeUnregistered;
}

cudaError_t Stager::slot(unsigned char **p, int *i)
{
    *i = next;
    next = (next + 1) % kPieces;
    *p = ring + (size_t)*i * kPiece;
    return cudaEventSynchronize(done[*i]); // (an event that was never recorded counts as done)
}

cudaError_t Stager::to_device(void *dev, const void *host, size_t bytes, cudaStream_t st)
{
    if (bytes < (64u << 10) || pinned(host)) return cudaMemcpyAsync(dev, host, bytes, cudaMemcpyHostToDevice, st);
    return to_device(dev, std::vector<Segment>(1, Segment{0, host, bytes}), st);
}

cudaError_t Stager::to_device(void *dev, const std::vector<Segment> &seg, cudaStream_t st)
{
    if (seg.empty()) return cudaSuccess;
    if (!ready())
    {
        for (const Segment &s : seg)
        {
            const cudaError_t e = cudaMemcpyAsync((unsigned char *)dev + s.off, s.host, s.bytes, cudaMemcpyHostToDevice, st);
            if (e != cudaSuccess) return e;
        }
        return cudaSuccess;
    }
    const size_t end = seg.back().off + seg.back().bytes;
    // the first piece's filling and the last one's copy are all that does not overlap; a piece costs 3 us and more by itself
    const size_t piece = std::min(kPiece, std::max<size_t>(512u << 10, (end / 4 + kPart - 1) / kPart * kPart));
    const size_t begin = seg.front().off, total = end - begin;
    const long long n_pieces = (long long)((total + piece - 1) / piece), per = (long long)(piece / kPart), n_parts = (long long)((total + kPart - 1) / kPart);
    if (n_parts <= 3)
    {
        // (over before other threads are awake)
        unsigned char *p;
        int i;
        cudaError_t e = slot(&p, &i);
        if (e != cudaSuccess) return e;
        gather(p, begin, total, seg);
        e = cudaMemcpyAsync((unsigned char *)dev + begin, p, total, cudaMemcpyHostToDevice, st);
        return e == cudaSuccess ? cudaEventRecord(done[i], st) : e;
    }
    // The threads take parts in order; the calling one also sends every piece whose parts are in. A piece is opened (its slot of
    // the ring free again) before its parts may be filled.
    unsigned char *where[kPieces];
    int used[kPieces];
    std::atomic<long long> next_part(0), open_pieces(0);
    std::atomic<int> filled[kPieces];
    for (auto &f : filled) f.store(0);
    std::atomic<bool> stop(false);
    cudaError_t e = cudaSuccess;
    auto open = [&](long long k) { // by the calling thread only
        e = slot(&where[k % kPieces], &used[k % kPieces]);
        filled[k % kPieces].store(0);
        if (e != cudaSuccess) stop.store(true);
        else open_pieces.store(k + 1);
    };
    auto fill_one = [&]() -> bool { // false: no part to be had now
        long long q = next_part.load();
        do
        {
            if (q >= n_parts || q / per >= open_pieces.load()) return false;
        } while (!next_part.compare_exchange_weak(q, q + 1));
        const long long k = q / per;
        const size_t at = (size_t)(q - k * per) * kPart, o = (size_t)k * piece + at;
        gather(where[k % kPieces] + at, begin + o, std::min(kPart, total - o), seg);
        filled[k % kPieces].fetch_add(1);
        return true;
    };
    for (long long k = 0; k < n_pieces && k < kPieces && e == cudaSuccess; k++) open(k);
#pragma omp parallel
    {
        bool mine = false;
#pragma omp master
        mine = true;
        if (mine)
        {
            for (long long k = 0; k < n_pieces && e == cudaSuccess; k++)
            {
                const long long parts_of = std::min(per, n_parts - k * per);
                while (filled[k % kPieces].load() < parts_of) fill_one();
                const size_t o = (size_t)k * piece, n = std::min(piece, total - o);
                e = cudaMemcpyAsync((unsigned char *)dev + begin + o, where[k % kPieces], n, cudaMemcpyHostToDevice, st);
                if (e == cudaSuccess) e = cudaEventRecord(done[used[k % kPieces]], st);
                if (e == cudaSuccess && k + kPieces < n_pieces) open(k + kPieces);
            }
            stop.store(true);
        }
        else
            while (!stop.load() && next_part.load() < n_parts) fill_one();
    }
    return e;
}

cudaError_t Stager::to_host(void *host, const void *dev, size_t bytes, cudaStream_t st)
{
    if (bytes < (256u << 10) || pinned(host) || !ready())
    {
        const cudaError_t e = cudaMemcpyAsync(host, dev, bytes, cudaMemcpyDeviceToHost, st);
        return e == cudaSuccess ? cudaStreamSynchronize(st) : e;
    }
    const size_t piece = std::min(kPiece, std::max<size_t>(256u << 10, (bytes / 8 + kPart - 1) / kPart * kPart)), n_pieces = (bytes + piece - 1) / piece;
    cudaError_t e = cudaSuccess;
    int at[kPieces];
    auto send = [&](size_t k) {
        unsigned char *p;
        e = slot(&p, &at[k % kPieces]);
        const size_t o = k * piece;
        if (e == cudaSuccess) e = cudaMemcpyAsync(p, (const unsigned char *)dev + o, std::min(piece, bytes - o), cudaMemcpyDeviceToHost, st);
        if (e == cudaSuccess) e = cudaEventRecord(done[at[k % kPieces]], st);
    };
    for (size_t k = 0; k < n_pieces && k < (size_t)kPieces && e == cudaSuccess; k++) send(k);
    for (size_t k = 0; k < n_pieces && e == cudaSuccess; k++)
    {
        const int i = at[k % kPieces];
        e = cudaEventSynchronize(done[i]);
        if (e != cudaSuccess) break;
        const size_t o = k * piece;
        const unsigned char *p = ring + (size_t)i * kPiece;
        parts(std::min(piece, bytes - o), [&](size_t a, size_t n) { memcpy((unsigned char *)host + o + a, p + a, n); });
        if (k + kPieces < n_pieces) send(k + kPieces);
    }
    if (e != cudaSuccess) cudaStreamSynchronize(st);
    return e;
}
} // namespace asp
