// Arrays of the host operators: shared, copy-free views of large buffers.
//
// A matrix passes through several objects on its way to a plan (asp_matrix -> compressed matrix -> format), and its
// non-zeros only change in a few operators. An Arr is a view of a reference-counted buffer, so those hand-overs copy
// nothing; who writes makes a buffer of its own first. Buffers are not initialised (the loops that fill them run on all
// cores and are the first to touch the pages) and large ones ask for huge pages: with 4 KB pages the faults of a fresh
// buffer cost more than filling it.
#ifndef ASP_HOSTMEM_HPP
#define ASP_HOSTMEM_HPP

#include <stdint.h>
#include <stdlib.h>
#include <string.h>

#include <map>
#include <memory>
#include <new>
#include <vector>

#include "crew.hpp"

namespace asp
{
namespace host
{
// Blocks that nobody uses, kept for a later request of about their size. The caller locks.
class IdleBlocks
{
    struct Block
    {
        void *p;
        uint64_t since;
    };
    std::multimap<size_t, Block> by_size;
    size_t bytes = 0;
    uint64_t clock = 0;

  public:
    size_t total() const { return bytes; }
    // the smallest block of want to 1.25 want + unit bytes, or NULL
    void *take(size_t want, size_t unit, size_t *size)
    {
        auto it = by_size.lower_bound(want);
        if (it == by_size.end() || it->first > want + want / 4 + unit) return nullptr;
        void *p = it->second.p;
        *size = it->first;
        bytes -= it->first;
        by_size.erase(it);
        return p;
    }
    // keeps the block; false (it stays the caller's) when there is no memory to note it
    bool put(void *p, size_t size) noexcept
    {
        try
        {
            by_size.insert({size, {p, clock++}});
        }
        catch (const std::bad_alloc &)
        {
            return false;
        }
        bytes += size;
        return true;
    }
    // the longest idle block, no longer kept, while there are more than `most` bytes in all, else NULL: without that, blocks of
    // sizes that are not asked for again would fill the pool for good
    void *beyond(size_t most)
    {
        if (bytes <= most) return nullptr;
        auto old = by_size.begin();
        for (auto it = by_size.begin(); it != by_size.end(); ++it)
            if (it->second.since < old->second.since) old = it;
        void *p = old->second.p;
        bytes -= old->first;
        by_size.erase(old);
        return p;
    }
};

// Large buffers come from a pool (hostmem.cpp): a fresh one costs a page fault per 2 MB, zeroed by the kernel at 5 to 20 GB/s, which
// is several times what the operators do with it. Idle buffers are bounded (256 MB in all, the longest idle ones go first) and given back with host_pool_trim().
std::shared_ptr<void> big_buffer(size_t bytes);
void host_pool_trim();

// Below these a loop runs on the calling thread alone: sharing one costs 1 to 5 us. (The limits were 4 MB, 2^18 rows and 2^19 non-zeros
// while loops were OpenMP's; crew.hpp has the figures of both.)
const size_t kParallelBytes = 1u << 18;
const uint64_t kParallelRows = 1u << 13, kParallelNnz = 1u << 14;
inline void par_copy(void *dst, const void *src, size_t bytes)
{
    const size_t line = 64, most = 1u << 16;
    share_ranges((bytes + line - 1) / line, bytes > kParallelBytes, [=](uint64_t i, uint64_t e) {
        const size_t end = std::min<size_t>(bytes, e * line);
        for (size_t o = i * line; o < end; o += most) memcpy((char *)dst + o, (const char *)src + o, std::min(most, end - o));
    });
}

inline void par_zero(void *dst, size_t bytes)
{
    share_ranges((bytes + 63) / 64, bytes > kParallelBytes, [=](uint64_t i, uint64_t e) { memset((char *)dst + i * 64, 0, std::min<size_t>(bytes, e * 64) - i * 64); });
}

template <class T>
class Arr
{
    template <class>
    friend class Arr;
    std::shared_ptr<void> s;
    T *p = nullptr;
    uint64_t n = 0;

  public:
    uint64_t size() const { return n; }
    bool empty() const { return n == 0; }
    const T *data() const { return p; }
    T *mut() { return p; } // for a buffer that make() gave to this array and nobody else has seen
    const T &operator[](uint64_t i) const { return p[i]; }
    const T &back() const { return p[n - 1]; }
    const T *begin() const { return p; }
    const T *end() const { return p + n; }
    void clear() { s.reset(), p = nullptr, n = 0; }
    void swap(Arr &o) { std::swap(s, o.s), std::swap(p, o.p), std::swap(n, o.n); }
    // a fresh buffer of this array alone, to be filled through the pointer that is returned
    T *make(uint64_t count)
    {
        s = big_buffer(count * sizeof(T));
        p = (T *)s.get();
        n = count;
        return p;
    }
    T *make_zero(uint64_t count)
    {
        make(count);
        par_zero(p, count * sizeof(T));
        return p;
    }
    void assign(const T *src, uint64_t count)
    {
        make(count);
        par_copy(p, src, count * sizeof(T));
    }
    // somebody else's memory, which has to stay as it is while this array or a view of it lives
    void borrow(const T *src, uint64_t count)
    {
        s = std::shared_ptr<void>();
        p = const_cast<T *>(src); // (never written: who writes makes a buffer of its own first)
        n = count;
    }
    Arr view(uint64_t off, uint64_t count) const
    {
        Arr a;
        a.s = s;
        a.p = p + off;
        a.n = count;
        return a;
    }
    // the same buffer as bytes
    Arr<uint8_t> bytes() const
    {
        Arr<uint8_t> a;
        a.s = s;
        a.p = (uint8_t *)p;
        a.n = n * sizeof(T);
        return a;
    }
    // `count` entries of which the first keep their values and the others are zero; returns them for writing
    T *grow(uint64_t count)
    {
        Arr a;
        a.make(count);
        const uint64_t keep = count < n ? count : n;
        par_copy(a.p, p, keep * sizeof(T));
        par_zero(a.p + keep, (count - keep) * sizeof(T));
        swap(a);
        return p;
    }
};
} // namespace host
} // namespace asp
#endif
