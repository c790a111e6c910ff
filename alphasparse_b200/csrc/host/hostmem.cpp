#include "hostmem.hpp"

#include <sys/mman.h>

#include <mutex>

namespace asp
{
namespace host
{
namespace
{
const size_t kHuge = 2u << 20, kMostIdle = 256u << 20;

struct Pool
{
    std::mutex lock;
    IdleBlocks idle;
};
Pool &pool()
{
    static Pool *p = new Pool(); // (never destroyed: buffers may come back while the process ends)
    return *p;
}

// frees the longest idle buffers until no more than `most` bytes are left
void shrink(size_t most)
{
    Pool &q = pool();
    for (;;)
    {
        void *p;
        {
            std::lock_guard<std::mutex> g(q.lock);
            p = q.idle.beyond(most);
        }
        if (!p) return;
        free(p);
    }
}

// (the deleter of a shared buffer: nothing may be thrown)
void give_back(void *p, size_t size) noexcept
{
    Pool &q = pool();
    bool kept = size <= kMostIdle;
    if (kept)
    {
        std::lock_guard<std::mutex> g(q.lock);
        kept = q.idle.put(p, size);
    }
    if (!kept) free(p);
    shrink(kMostIdle);
}
} // namespace

void host_pool_trim() { shrink(0); }

std::shared_ptr<void> big_buffer(size_t bytes)
{
    if (bytes < kHuge / 2)
    {
        void *p = malloc(bytes ? bytes : 1);
        if (!p) throw std::bad_alloc();
        return std::shared_ptr<void>(p, free);
    }
    const size_t want = (bytes + kHuge - 1) / kHuge * kHuge;
    void *p = nullptr;
    size_t size = want;
    {
        Pool &q = pool();
        std::lock_guard<std::mutex> g(q.lock);
        p = q.idle.take(want, kHuge, &size);
    }
    if (!p && posix_memalign(&p, kHuge, want) != 0)
    {
        host_pool_trim();
        if (posix_memalign(&p, kHuge, want) != 0) throw std::bad_alloc();
    }
    madvise(p, size, MADV_HUGEPAGE); // (advice only: without huge pages everything still works)
    return std::shared_ptr<void>(p, [size](void *q) { give_back(q, size); });
}
} // namespace host
} // namespace asp
