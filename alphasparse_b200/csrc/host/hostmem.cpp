#include "hostmem.hpp"

#include <sys/mman.h>

#include <mutex>
#include <vector>

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

void give_back(void *p, size_t size)
{
    Pool &q = pool();
    std::vector<void *> out;
    {
        std::lock_guard<std::mutex> g(q.lock);
        q.idle.put(p, size, kMostIdle, out);
    }
    for (void *o : out) free(o);
}
} // namespace

void host_pool_trim()
{
    Pool &q = pool();
    std::vector<void *> idle;
    {
        std::lock_guard<std::mutex> g(q.lock);
        q.idle.take_all(idle);
    }
    for (void *p : idle) free(p);
}

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
