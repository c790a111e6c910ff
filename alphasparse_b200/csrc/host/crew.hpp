// Loops that the calling thread shares with helpers.
//
// A parallel region of OpenMP ends when every thread of the team has come to its end. Where other programs keep the cores busy that is a
// thread that is not running: with a spinning process on each of 8 cores, formats of 28,800 to 400,000 non-zeros took 16 to 168 ms with
// OpenMP's regions around loops of this size, 0.2 to 23 ms without any. And a forked process waits for threads that it does not have.
// Here the caller publishes a loop as pieces, begins with the first, and goes on taking pieces until there are none left; helpers that are
// awake take pieces, too. The caller waits for pieces that somebody has begun, never for somebody to begin. us a build, rows of 8
// non-zeros, 8 cores (OpenMP from 2^19 non-zeros on / OpenMP from 2^14 on / this):
//                                  28,800 non-zeros       96,000                  400,000
//   nothing else runs   ELL-like   365 / 195 / 251        802 / 273 / 296         5693 / 908 / 985
//                       CSR5-like  253 / 114 / 115        780 / 193 / 207         2994 / 779 / 737
//                       2 x 2      873 / 208 / 206        3485 / 647 / 648        16812 / 3184 / 2535
//   all cores busy      ELL-like   331 / 24003 / 336      715 / 167998 / 1055     4751 / 163997 / 6079
//                       2 x 2      1412 / 32051 / 1324    5213 / 56010 / 4212     24382 / 64007 / 14053
//   4 callers at once   ELL-like   81 / 167 / 108         226 / 506 / 238         1261 / 1450 / 1225
//   8 callers at once   ELL-like   86 / 140 / 123         121 / 236 / 195         637 / 828 / 748
#ifndef ASP_HOST_CREW_HPP
#define ASP_HOST_CREW_HPP

#include <stdint.h>

#include <algorithm>
#include <atomic>

// for the body of a loop, called where its range is known: what it holds by value then is in registers. As calls, with the values read from
// the closure after every store, 3 x 3 blocks took half as long again (3.2 million non-zeros, 8 threads: 7.2 instead of 4.8 ms).
#define ASP_INLINE __attribute__((always_inline))

namespace asp
{
namespace host
{
// threads that a loop of this thread may have, itself included: as many as an OpenMP region would (omp_get_max_threads), one inside
// of a piece or of such a region
unsigned crew_width();
// whether this thread is in a piece of a loop that is shared
bool in_piece();
// A thread that has loops to share, one after the other. Several of them leave the helpers fewer cores, so that the threads are
// never more than one caller's would be.
class Caller
{
  public:
    Caller();
    ~Caller();
    Caller(const Caller &) = delete;
    Caller &operator=(const Caller &) = delete;
};
const unsigned kMostPieces = 256;
// run(arg, piece, who) for every piece of [0, pieces), pieces <= kMostPieces, who < width one thread's own number: the caller is 0 and
// takes piece 0. Nothing may be thrown in a piece.
// `call`: helpers that the caller wakes at once; those that come call others.
const unsigned kCallSome = 2, kCallAll = 255;
void crew_run(unsigned pieces, unsigned width, unsigned call, void (*run)(void *, unsigned, unsigned), void *arg) noexcept;

// f(piece, who)
template <class F>
void share_pieces(unsigned pieces, unsigned width, F &&f, unsigned call = kCallSome)
{
    if (pieces <= 1 || width <= 1)
    {
        for (unsigned p = 0; p < pieces; p++) f(p, 0u);
        return;
    }
    typedef typename std::remove_reference<F>::type Fn;
    crew_run(pieces, width, call, [](void *a, unsigned p, unsigned who) { (*(Fn *)a)(p, who); }, (void *)&f);
}

// f(begin, end) over ranges of [0, n) in as many pieces as suit the threads. A thread takes its own pieces first, so that successive loops
// over the same rows find them in its cache.
template <class F>
void share_ranges(uint64_t n, bool share, F &&f)
{
    const unsigned width = share ? crew_width() : 1;
    if (width <= 1)
    {
        if (n > 0) f((uint64_t)0, n);
        return;
    }
    const unsigned pieces = (unsigned)std::min<uint64_t>(n, std::min<uint64_t>(kMostPieces, width * std::max<uint64_t>(2, std::min<uint64_t>(8, n / 512 / width))));
    share_pieces(pieces, width, [&](unsigned p, unsigned) { f(n * p / pieces, n * (p + 1) / pieces); });
}

// f(i) for i in [0, n): in ranges as above
template <class F>
void for_each(uint64_t n, bool share, F &&f)
{
    share_ranges(n, share, [&](uint64_t i, uint64_t e) {
        for (; i < e; i++) f(i);
    });
}

// f(begin, end, who) over runs of `step` in [0, n), the next one to whoever is free: where rows differ
template <class F>
void share_steps(uint64_t n, uint64_t step, unsigned width, F &&f)
{
    std::atomic<uint64_t> next(0);
    share_pieces(std::min(width, kMostPieces), width, [&](unsigned, unsigned who) {
        for (;;)
        {
            const uint64_t i = next.fetch_add(step, std::memory_order_relaxed);
            if (i >= n) return;
            f(i, std::min(n, i + step), who);
        }
    });
}

template <class T>
void raise(std::atomic<T> &to, T v)
{
    for (T old = to.load(std::memory_order_relaxed); old < v && !to.compare_exchange_weak(old, v, std::memory_order_relaxed);) {}
}
template <class T>
void lower(std::atomic<T> &to, T v)
{
    for (T old = to.load(std::memory_order_relaxed); v < old && !to.compare_exchange_weak(old, v, std::memory_order_relaxed);) {}
}
} // namespace host
} // namespace asp
#endif
