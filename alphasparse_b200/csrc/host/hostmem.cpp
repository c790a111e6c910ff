#include "hostmem.hpp"

#include <sys/mman.h>

#include <map>
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
    std::multimap<size_t, void *> idle; // by size
    size_t bytes = 0;
};
Pool &pool()
{
    static Pool *p = new Pool(); // (never destroyed: buffers may come back while the process ends)
    return *p;
}

void give_back(void *p, size_t size)
{
    Pool &q = pool();
    {
        std::lock_guard<std::mutex> g(q.lock);
        if (q.bytes + size <= kMostIdle)
        {
            q.idle.insert({size, p});
            q.bytes += size;
            return;
        }
    }
    free(p);
}
} // namespace

void host_pool_trim()
{
    Pool &q = pool();
    std::multimap<size_t, void *> idle;
    {
        std::lock_guard<std::mutex> g(q.lock);
        idle.swap(q.idle);
        q.bytes = 0;
    }
    for (auto &b : idle) free(b.second);
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
        auto it = q.idle.lower_bound(want);
        if (it != q.idle.end() && it->first <= want + want / 4 + kHuge)
        {
            size = it->first;
            p = it->second;
            q.bytes -= size;
            q.idle.erase(it);
        }
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
