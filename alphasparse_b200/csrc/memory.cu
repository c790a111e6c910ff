#include "memory.h"

#include <cuda.h>
#include <stdint.h>
#include <string.h>
#if defined(__SSE2__)
#include <emmintrin.h>
#endif

#include <atomic>

#include <algorithm>
#include <memory>
#include <mutex>
#include <vector>

#include "host/hostmem.hpp"

namespace asp
{
namespace
{
const size_t kMostBlock = 256u << 20, kMostCached = 1u << 30;

struct Pool
{
    std::mutex lock;
    host::IdleBlocks idle;
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
void gather(unsigned char *dst, size_t at, size_t n, const Stager::Segment *seg, size_t count)
{
    size_t i = (size_t)(std::upper_bound(seg, seg + count, at, [](size_t o, const Stager::Segment &s) { return o < s.off; }) - seg);
    if (i > 0) i--;
    for (; i < count && seg[i].off < at + n; i++)
    {
        const size_t lo = std::max(at, seg[i].off), hi = std::min(at + n, seg[i].off + seg[i].bytes);
        if (lo < hi) stream_copy(dst + (lo - at), (const unsigned char *)seg[i].host + (lo - seg[i].off), hi - lo);
    }
}

const size_t kPart = 64u << 10; // what one thread copies at a time
const long long kFirstParts = 16, kMostParts = 64; // of the pieces of an upload: first pieces of 512 KB cost 8 us more with 1.3 MB of x, longest ones of 2 MB 5 us more with 8 MB
// a copy of fewer parts is over before the threads are awake
template <class F>
void parts(size_t n, F &&f)
{
    const long long k = (long long)((n + kPart - 1) / kPart);
    host::for_each((uint64_t)k, k > 3, [&](uint64_t i) { f((size_t)i * kPart, std::min(kPart, n - (size_t)i * kPart)); });
}
} // namespace

namespace
{
// frees the longest idle blocks until no more than `most` bytes are left (the device is current)
void shrink(Pool &p, size_t most)
{
    for (;;)
    {
        void *q;
        {
            std::lock_guard<std::mutex> g(p.lock);
            q = p.idle.beyond(most);
        }
        if (!q) return;
        cudaFree(q);
    }
}
} // namespace

cudaError_t device_alloc(int device, size_t bytes, void **out, size_t *got, size_t spare)
{
    const size_t unit = bytes < (1u << 20) ? (64u << 10) : (2u << 20);
    const size_t want = (std::max<size_t>(bytes, 1) + unit - 1) / unit * unit;
    Pool &p = pool(device);
    {
        std::lock_guard<std::mutex> g(p.lock);
        *out = p.idle.take(want, unit, got);
        if (*out) return cudaSuccess;
    }
    // (asking costs 0.1 to 0.2 ms, a tenth of what cudaMalloc does)
    if (spare > 0 && !device_has_room(device, want + spare)) return cudaErrorMemoryAllocation;
    *got = want;
    return device_malloc(device, want, out);
}

cudaError_t device_malloc(int device, size_t bytes, void **out)
{
    OnDevice on(device);
    cudaError_t e = cudaMalloc(out, bytes);
    if (e == cudaErrorMemoryAllocation)
    {
        cudaGetLastError();
        shrink(pool(device), 0);
        e = cudaMalloc(out, bytes);
    }
    return e;
}

bool device_has_room(int device, size_t bytes)
{
    OnDevice on(device);
    size_t idle, free_now = 0, all = 0;
    {
        std::lock_guard<std::mutex> g(pool(device).lock);
        idle = pool(device).idle.total();
    }
    if (cudaMemGetInfo(&free_now, &all) != cudaSuccess)
    {
        cudaGetLastError();
        return false;
    }
    return free_now + idle >= bytes;
}

void device_trim(int device)
{
    OnDevice on(device);
    shrink(pool(device), 0);
}

// (a destructor calls it: nothing may be thrown)
void device_free(int device, void *ptr, size_t got) noexcept
{
    if (!ptr) return;
    OnDevice on(device);
    Pool &p = pool(device);
    bool kept = got <= kMostBlock && cudaDeviceSynchronize() == cudaSuccess;
    if (kept)
    {
        std::lock_guard<std::mutex> g(p.lock);
        kept = p.contexts > 0 && p.idle.put(ptr, got);
    }
    if (!kept) cudaFree(ptr);
    shrink(p, kMostCached);
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
    {
        std::lock_guard<std::mutex> g(p.lock);
        if (--p.contexts > 0) return;
    }
    OnDevice on(device);
    shrink(p, 0);
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
    for (int i = 0; i < kPieces; i++) owner[i] = i;
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

void *device_view(const void *p, size_t bytes)
{
    typedef CUresult (*Query)(void *, CUpointer_attribute, CUdeviceptr);
    static const Query query = []() -> Query {
        void *f = nullptr;
        cudaDriverEntryPointQueryResult found = cudaDriverEntryPointSymbolNotFound;
        const cudaError_t e = cudaGetDriverEntryPoint("cuPointerGetAttribute", &f, cudaEnableDefault, &found);
        if (e != cudaSuccess) cudaGetLastError();
        return e == cudaSuccess && found == cudaDriverEntryPointSuccess ? (Query)f : nullptr;
    }();
    cudaPointerAttributes at;
    if (cudaPointerGetAttributes(&at, p) != cudaSuccess)
    {
        cudaGetLastError();
        return nullptr;
    }
    if (at.type != cudaMemoryTypeHost || !at.devicePointer || !query) return nullptr;
    const CUdeviceptr d = (CUdeviceptr)at.devicePointer;
    CUdeviceptr start = 0;
    size_t size = 0;
    int access = 0;
    if (query(&start, CU_POINTER_ATTRIBUTE_RANGE_START_ADDR, d) != CUDA_SUCCESS || query(&size, CU_POINTER_ATTRIBUTE_RANGE_SIZE, d) != CUDA_SUCCESS) return nullptr;
    if (query(&access, CU_POINTER_ATTRIBUTE_ACCESS_FLAGS, d) != CUDA_SUCCESS || access != CU_POINTER_ATTRIBUTE_ACCESS_FLAG_READWRITE) return nullptr;
    return d >= start && d - start <= size && bytes <= size - (d - start) ? at.devicePointer : nullptr;
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

// (an event that was never recorded counts as done)
bool Stager::free_now(int slots) const
{
    const int first = next + slots > kPieces ? 0 : next;
    for (int i = first; i < first + slots; i++)
        if (cudaEventQuery(done[owner[i]]) != cudaSuccess)
        {
            cudaGetLastError(); // not ready is no error
            return false;
        }
    return true;
}

cudaError_t Stager::take(int slots, unsigned char **p, int *event)
{
    const int first = next + slots > kPieces ? 0 : next, last = first + slots - 1;
    for (int i = first; i <= last; i++)
    {
        const cudaError_t e = cudaEventSynchronize(done[owner[i]]);
        if (e != cudaSuccess) return e;
    }
    // (slots outside that still name this event belong to a piece that is over: the last slot was its, too)
    for (int i = first; i <= last; i++) owner[i] = last;
    next = (last + 1) % kPieces;
    *p = ring + (size_t)first * kPiece;
    *event = last;
    return cudaSuccess;
}

cudaError_t Stager::to_device(void *dev, const void *host, size_t bytes, cudaStream_t st)
{
    if (bytes < (64u << 10) || pinned(host)) return cudaMemcpyAsync(dev, host, bytes, cudaMemcpyHostToDevice, st);
    const Segment whole = {0, host, bytes};
    return to_device(dev, &whole, 1, st);
}

cudaError_t Stager::to_device(void *dev, const void *host, size_t bytes, cudaStream_t st, size_t piece, const Sent &sent)
{
    if (bytes >= (64u << 10) && !pinned(host))
    {
        const Segment whole = {0, host, bytes};
        return to_device(dev, &whole, 1, st, piece, &sent);
    }
    cudaError_t e = cudaSuccess;
    for (size_t o = 0; o < bytes && e == cudaSuccess;)
    {
        const size_t n = bytes - o < piece + piece / 2 ? bytes - o : piece;
        e = cudaMemcpyAsync((unsigned char *)dev + o, (const unsigned char *)host + o, n, cudaMemcpyHostToDevice, st);
        o += n;
        if (e == cudaSuccess) e = sent.f(sent.with, o);
    }
    return e;
}

cudaError_t Stager::to_device(void *dev, const std::vector<Segment> &seg, cudaStream_t st) { return to_device(dev, seg.data(), seg.size(), st); }

cudaError_t Stager::to_device(void *dev, const Segment *seg, size_t count, cudaStream_t st, size_t piece, const Sent *sent)
{
    if (count == 0) return cudaSuccess;
    const size_t begin = seg[0].off, total = seg[count - 1].off + seg[count - 1].bytes - begin;
    auto plain = [&]() {
        for (size_t i = 0; i < count; i++)
        {
            const cudaError_t e = cudaMemcpyAsync((unsigned char *)dev + seg[i].off, seg[i].host, seg[i].bytes, cudaMemcpyHostToDevice, st);
            if (e != cudaSuccess) return e;
        }
        return sent ? sent->f(sent->with, total) : cudaSuccess;
    };
    std::lock_guard<std::mutex> turn(one);
    if (!ready()) return plain();
    const long long n_parts = (long long)((total + kPart - 1) / kPart);
    if (n_parts <= 3)
    {
        // (over before other threads are awake)
        unsigned char *p;
        int i;
        cudaError_t e = take(1, &p, &i);
        if (e != cudaSuccess) return e;
        gather(p, begin, total, seg, count);
        e = cudaMemcpyAsync((unsigned char *)dev + begin, p, total, cudaMemcpyHostToDevice, st);
        if (e == cudaSuccess) e = cudaEventRecord(done[i], st);
        return e == cudaSuccess && sent ? sent->f(sent->with, total) : e;
    }
    // Pieces that double: the filling of the first is all that does not overlap with a copy, and a copy costs 3.5 us by itself
    // (8 MB on this link: 161 us in one copy, 187 in eight). The ring is filled faster than the link empties it. `piece`: of that size
    // instead, if the ring can hold three.
    const long long even = (long long)(std::min(piece, kPiece * (kPieces / 4)) / kPart);
    struct Piece
    {
        long long part, end; // parts of 64 KB
        int slots, event = 0;
        long long at = 0; // slots that the call had taken before, those left free at the ring's end included
        unsigned char *p = nullptr;
    };
    const long long slot_parts = (long long)(kPiece / kPart);
    std::vector<Piece> pieces;
    std::vector<int> piece_of;
    // The threads take parts in order; the calling one also sends every piece whose parts are in. A piece is opened (its slots of
    // the ring free again) before its parts may be filled.
    std::unique_ptr<std::atomic<int>[]> filled;
    try
    {
        piece_of.resize((size_t)n_parts);
        for (long long q = 0, n = even > 0 ? even : kFirstParts; q < n_parts; n = even > 0 ? even : std::min(2 * n, kMostParts))
        {
            const long long e = n_parts - q <= n + n / 4 ? n_parts : q + n;
            std::fill(piece_of.begin() + q, piece_of.begin() + e, (int)pieces.size());
            pieces.push_back({q, e, (int)((e - q + slot_parts - 1) / slot_parts)});
            q = e;
        }
        filled.reset(new std::atomic<int>[pieces.size()]);
    }
    catch (const std::bad_alloc &)
    {
        return plain();
    }
    for (size_t k = 0; k < pieces.size(); k++) filled[k].store(0);
    std::atomic<long long> next_part(0), open_parts(0);
    std::atomic<bool> stop(false);
    cudaError_t e = cudaSuccess;
    size_t opened = 0;
    long long taken = 0;
    auto open_from = [&](size_t unsent) { // by the calling thread only
        while (opened < pieces.size() && e == cudaSuccess)
        {
            Piece &k = pieces[opened];
            const long long at = taken + (next + k.slots > kPieces ? kPieces - next : 0);
            if (opened > unsent && (at + k.slots - pieces[unsent].at > kPieces || !free_now(k.slots))) return;
            e = take(k.slots, &k.p, &k.event);
            if (e != cudaSuccess) return;
            k.at = at;
            taken = at + k.slots;
            opened++;
            open_parts.store(k.end);
        }
    };
    auto fill_one = [&]() { // one part, if there is one to be had now
        long long q = next_part.load();
        do
        {
            if (q >= open_parts.load()) return;
        } while (!next_part.compare_exchange_weak(q, q + 1));
        const Piece &k = pieces[piece_of[(size_t)q]];
        const size_t o = (size_t)q * kPart;
        gather(k.p + (size_t)(q - k.part) * kPart, begin + o, std::min(kPart, total - o), seg, count);
        filled[piece_of[(size_t)q]].fetch_add(1);
    };
    open_from(0);
    // (everybody else's piece begins and ends whenever, the caller is not kept waiting for them)
    const unsigned width = std::min(host::crew_width(), host::kMostPieces);
    host::share_pieces(width, width, [&](unsigned piece, unsigned) {
        if (piece == 0) // the caller's
        {
            for (size_t k = 0; k < pieces.size() && e == cudaSuccess; k++)
            {
                const Piece &q = pieces[k];
                while (filled[k].load() < q.end - q.part) fill_one();
                const size_t o = (size_t)q.part * kPart, n = std::min((size_t)(q.end - q.part) * kPart, total - o);
                e = cudaMemcpyAsync((unsigned char *)dev + begin + o, q.p, n, cudaMemcpyHostToDevice, st);
                if (e == cudaSuccess) e = cudaEventRecord(done[q.event], st);
                if (e == cudaSuccess && sent) e = sent->f(sent->with, o + n);
                open_from(k + 1);
            }
            stop.store(true);
        }
        else
            while (!stop.load() && next_part.load() < n_parts) fill_one();
    }, host::kCallAll);
    return e;
}

cudaError_t Stager::to_host(void *host, const void *dev, size_t bytes, cudaStream_t st)
{
    auto plain = [&]() {
        const cudaError_t e = cudaMemcpyAsync(host, dev, bytes, cudaMemcpyDeviceToHost, st);
        return e == cudaSuccess ? cudaStreamSynchronize(st) : e;
    };
    if (bytes < (256u << 10) || pinned(host)) return plain();
    std::lock_guard<std::mutex> turn(one);
    if (!ready()) return plain();
    const size_t piece = std::min(kPiece, std::max<size_t>(256u << 10, (bytes / 8 + kPart - 1) / kPart * kPart)), n_pieces = (bytes + piece - 1) / piece;
    cudaError_t e = cudaSuccess;
    int at[kPieces];
    auto send = [&](size_t k) {
        unsigned char *p;
        e = take(1, &p, &at[k % kPieces]);
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
