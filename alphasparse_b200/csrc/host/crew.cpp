// The helpers of crew.hpp.
#include "crew.hpp"

#include <linux/futex.h>
#include <omp.h>
#include <pthread.h>
#include <sched.h>
#include <signal.h>
#include <sys/syscall.h>
#include <time.h>
#include <unistd.h>

#include <mutex>
#include <new>

namespace asp
{
namespace host
{
namespace
{
const unsigned kMostHelpers = 255, kSlots = 8;

// A loop that is under way. `word` names it: generation, width, pieces (0: none). A piece belongs to whoever replaces an older generation in
// `taken` by that of the loop. Generations only grow, and a loop ends when all of its pieces are taken and done, so that nobody who comes
// late takes a piece of a loop that has ended: `run` and `arg` are read by those who hold a piece.
struct Slot
{
    alignas(64) std::atomic<bool> used{false};
    std::atomic<uint64_t> word{0};
    void (*run)(void *, unsigned, unsigned) = nullptr;
    void *arg = nullptr;
    alignas(64) std::atomic<unsigned> done{0};
    alignas(64) std::atomic<uint64_t> taken[kMostPieces];
    Slot()
    {
        for (auto &t : taken) t.store(0, std::memory_order_relaxed);
    }
};

struct Crew
{
    Slot slots[kSlots];
    alignas(64) std::atomic<uint32_t> epoch{0}; // changes with every loop that begins
    alignas(64) std::atomic<int> asleep{0};
    // Helpers have been kept from running with pieces in their hands: until then (ns) no core is free for them. The time doubles from
    // one such piece to the next, and halves again with every 32 loops without one: a piece may also be late by itself (pages that
    // it is the first to write).
    std::atomic<int64_t> alone_until{0};
    std::atomic<int> late{0}, in_time{0};
    std::atomic<int> helpers{0};
    std::mutex growing;
    const int cores = omp_get_num_procs();
};

std::atomic<Crew *> g_crew{nullptr}; // (never freed: helpers look at it until the process ends)
std::atomic<int> g_callers{0};       // threads between Caller() and ~Caller()
thread_local bool t_in_piece = false;
thread_local int t_caller = 0;
// callers and helpers that are awake, less the cores
int too_many(const Crew &c) { return g_callers.load(std::memory_order_relaxed) + c.helpers.load(std::memory_order_relaxed) - c.asleep.load(std::memory_order_relaxed) - c.cores; }

uint64_t make_word(uint64_t gen, unsigned width, unsigned pieces) { return gen << 24 | (uint64_t)width << 12 | pieces; }
uint64_t gen_of(uint64_t word) { return word >> 24; }
unsigned width_of(uint64_t word) { return (unsigned)(word >> 12) & 4095; }
unsigned pieces_of(uint64_t word) { return (unsigned)word & 4095; }

void relax()
{
#if defined(__x86_64__)
    __builtin_ia32_pause();
#endif
}
int64_t now()
{
    timespec t;
    clock_gettime(CLOCK_MONOTONIC, &t);
    return t.tv_sec * 1000000000ll + t.tv_nsec;
}
void wake(Crew &c, int n) { syscall(SYS_futex, &c.epoch, FUTEX_WAKE_PRIVATE, n, nullptr, nullptr, 0); }

bool take(Slot &s, uint64_t gen, unsigned p)
{
    uint64_t old = s.taken[p].load(std::memory_order_relaxed);
    return old < gen && s.taken[p].compare_exchange_strong(old, gen, std::memory_order_acq_rel, std::memory_order_relaxed);
}

// Runs pieces of the loop until none is left, this thread's own share first: the next loop over the same rows finds them in its cache.
// Returns how long the longest of them took (ns), 0: there was none. came(): when the first one has been taken.
template <class T>
int64_t work(Slot &s, uint64_t word, unsigned who, T &&came)
{
    const uint64_t gen = gen_of(word);
    const unsigned n = pieces_of(word), first = n * who / width_of(word);
    int64_t longest = 0;
    for (unsigned k = 0; k < n; k++)
    {
        const unsigned p = first + k < n ? first + k : first + k - n;
        if (!take(s, gen, p)) continue;
        if (longest == 0) came();
        const int64_t begin = now();
        s.run(s.arg, p, who);
        longest = std::max<int64_t>({1, longest, now() - begin});
        s.done.fetch_add(1, std::memory_order_release);
    }
    return longest;
}

struct Start
{
    Crew *crew;
    unsigned who;
};

void *helper(void *p)
{
    Crew &c = *((Start *)p)->crew;
    const unsigned who = ((Start *)p)->who;
    delete (Start *)p;
    t_in_piece = true;
    uint64_t seen[kSlots] = {0}; // loops of which nothing was left
    for (;;)
    {
        const uint32_t epoch = c.epoch.load(std::memory_order_seq_cst);
        bool any = false;
        for (unsigned i = 0; i < kSlots; i++)
        {
            Slot &s = c.slots[i];
            const uint64_t word = s.word.load(std::memory_order_acquire);
            if (word == seen[i] || who >= width_of(word)) continue;
            // whoever comes in time calls two others: the caller pays for two
            any |= work(s, word, who, [&]() {
                if (c.asleep.load(std::memory_order_relaxed) > 0 && too_many(c) < 0) wake(c, 2);
            }) > 0;
            seen[i] = word;
        }
        // The next loop of the same call comes within microseconds, that of the next call within a millisecond where calls follow one another
        // (with 0.2 ms a host-to-host product took 414 instead of 405 us). Who came too late waits, too, if not as long.
        const int64_t end = now() + (any ? 1000000 : 50000);
        do
            for (int i = 0; i < 64 && c.epoch.load(std::memory_order_relaxed) == epoch; i++) relax();
        while (c.epoch.load(std::memory_order_relaxed) == epoch && too_many(c) <= 0 && now() < end);
        if (c.epoch.load(std::memory_order_seq_cst) != epoch) continue;
        c.asleep.fetch_add(1, std::memory_order_seq_cst);
        syscall(SYS_futex, &c.epoch, FUTEX_WAIT_PRIVATE, epoch, nullptr, nullptr, 0);
        c.asleep.fetch_sub(1, std::memory_order_seq_cst);
    }
    return nullptr;
}

// a forked process makes a crew of its own: the threads stayed with its parent
const int g_at_fork = pthread_atfork(nullptr, nullptr, [] {
    g_crew.store(nullptr, std::memory_order_relaxed);
    g_callers.store(t_caller > 0 ? 1 : 0, std::memory_order_relaxed);
});

// a crew with `want` helpers, or as many as there can be
Crew *crew(unsigned want)
{
    Crew *c = g_crew.load(std::memory_order_acquire);
    if (!c)
    {
        Crew *made = new (std::nothrow) Crew();
        if (!made) return nullptr;
        if (g_crew.compare_exchange_strong(c, made, std::memory_order_acq_rel)) c = made;
        else delete made;
    }
    if (c->helpers.load(std::memory_order_relaxed) >= (int)want) return c;
    std::unique_lock<std::mutex> lock(c->growing, std::try_to_lock);
    if (!lock.owns_lock()) return c;
    pthread_attr_t attr;
    pthread_attr_init(&attr);
    pthread_attr_setdetachstate(&attr, PTHREAD_CREATE_DETACHED);
    sigset_t all, old;
    sigfillset(&all);
    pthread_sigmask(SIG_SETMASK, &all, &old); // (signals are the program's threads')
    for (unsigned n = (unsigned)c->helpers.load(std::memory_order_relaxed); n < want; n++)
    {
        Start *s = new (std::nothrow) Start{c, n + 1};
        pthread_t t;
        if (!s || pthread_create(&t, &attr, helper, s) != 0)
        {
            delete s;
            break;
        }
        c->helpers.store((int)n + 1, std::memory_order_relaxed);
    }
    pthread_sigmask(SIG_SETMASK, &old, nullptr);
    pthread_attr_destroy(&attr);
    return c;
}
} // namespace

bool in_piece() { return t_in_piece; }

Caller::Caller()
{
    if (t_caller++ == 0) g_callers.fetch_add(1, std::memory_order_relaxed);
}
Caller::~Caller()
{
    if (--t_caller == 0) g_callers.fetch_sub(1, std::memory_order_relaxed);
}

unsigned crew_width()
{
    if (t_in_piece || omp_in_parallel()) return 1;
    return (unsigned)std::max(1, std::min<int>(omp_get_max_threads(), (int)kMostHelpers));
}

void crew_run(unsigned pieces, unsigned width, unsigned call, void (*run)(void *, unsigned, unsigned), void *arg) noexcept
{
    const Caller caller;
    Crew *c = t_in_piece || width <= 1 ? nullptr : crew(std::min(width, kMostHelpers) - 1);
    // (as many callers as cores: a helper would only take a core from one of them, with a piece in its hands)
    const int callers = g_callers.load(std::memory_order_relaxed);
    if (c && callers > 1 && 2 * callers > c->cores) c = nullptr;
    unsigned alone = 0; // pieces that have been done alone
    while (c && alone < pieces && now() < c->alone_until.load(std::memory_order_relaxed)) run(arg, alone++, 0);
    Slot *s = nullptr;
    for (unsigned i = 0; c && i < kSlots && alone < pieces && !s; i++)
        if (!c->slots[i].used.exchange(true, std::memory_order_acquire)) s = &c->slots[i];
    if (!s)
    {
        while (alone < pieces) run(arg, alone++, 0);
        return;
    }
    const int64_t begin = now();
    const uint64_t gen = gen_of(s->word.load(std::memory_order_relaxed)) + 1, word = make_word(gen, std::min(width, kMostHelpers), pieces);
    s->run = run;
    s->arg = arg;
    s->done.store(alone, std::memory_order_relaxed);
    for (unsigned p = 0; p < std::max(1u, alone); p++) s->taken[p].store(gen, std::memory_order_relaxed);
    s->word.store(word, std::memory_order_release);
    c->epoch.fetch_add(1, std::memory_order_seq_cst);
    if (c->asleep.load(std::memory_order_seq_cst) > 0 && too_many(*c) < 0) wake(*c, c->helpers.load(std::memory_order_relaxed) >= (int)width ? (int)kCallAll : (int)call);
    t_in_piece = true;
    if (alone == 0)
    {
        run(arg, 0, 0);
        s->done.fetch_add(1, std::memory_order_release);
    }
    const int64_t first = now() - begin, longest = std::max(first, work(*s, word, 0, [] {}));
    t_in_piece = false;
    // what others have begun. A piece that takes four times as long as any of this thread's is somebody's who has been kept from running
    const int64_t idle = now();
    if (s->done.load(std::memory_order_acquire) != pieces)
    {
        for (unsigned i = 0; s->done.load(std::memory_order_acquire) != pieces; i++)
            if (i < 1024) relax();
            else sched_yield();
        const int64_t end = now();
        if (end - idle > std::max<int64_t>(400000, 4 * longest))
        {
            const int times = std::min(c->late.fetch_add(1, std::memory_order_relaxed), 5);
            c->alone_until.store(end + ((end - idle) << times), std::memory_order_relaxed);
            c->in_time.store(0, std::memory_order_relaxed);
        }
        else if (c->late.load(std::memory_order_relaxed) > 0 && c->in_time.fetch_add(1, std::memory_order_relaxed) >= 32)
        {
            c->in_time.store(0, std::memory_order_relaxed);
            c->late.store(std::min(c->late.load(std::memory_order_relaxed) - 1, 5), std::memory_order_relaxed);
        }
    }
    s->word.store(make_word(gen, 0, 0), std::memory_order_relaxed);
    s->used.store(false, std::memory_order_release);
}
} // namespace host
} // namespace asp
