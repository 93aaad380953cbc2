// The pool of page-locked blocks against a fake device: what is kept, reused,
// unlocked and forgotten, over device resets and with several threads.
#include <cstdio>
#include <cstdlib>
#include <set>
#include <thread>
#include <vector>

#include "staging.hpp"

using namespace rbps_gpu;

static std::mutex g_lock;
static std::set<void *> g_locked; // the fake driver's page-locked blocks
static uint64_t g_context[2] = {1, 2}, g_next = 3;
static thread_local int g_device = 0;
static bool g_fail = false;

struct Fake
{
    static uint64_t context() { return g_context[g_device]; }
    static void *lock(size_t n)
    {
        std::lock_guard<std::mutex> l(g_lock);
        if (g_fail)
            return nullptr;
        void *p = std::malloc(n);
        g_locked.insert(p);
        return p;
    }
    static void unlock(void *p)
    {
        std::lock_guard<std::mutex> l(g_lock);
        if (!g_locked.erase(p))
        {
            std::printf("unlock of a block that is not locked\n");
            std::exit(1);
        }
        std::free(p);
    }
};

static void reset(int device) // every block of the context is unlocked with it
{
    g_context[device] = g_next++;
    g_locked.clear();
}

#define CHECK(x)                                        \
    if (!(x))                                           \
    {                                                   \
        std::printf("line %d: %s\n", __LINE__, #x);     \
        return 1;                                       \
    }

int main()
{
    StagingPool<Fake> pool(64);
    // one batch after another: one block, locked once, kept
    void *first = nullptr;
    for (int k = 0; k < 3; ++k)
    {
        pool.begin();
        StagingBlock b = pool.take(0);
        CHECK(b.p && (k == 0 || b.p == first));
        first = b.p;
        pool.end(b);
        CHECK(pool.kept() == 1 && g_locked.size() == 1);
    }
    // a reset: the kept pointer is neither handed out nor unlocked
    reset(0);
    pool.begin();
    StagingBlock a = pool.take(0);
    CHECK(a.p && g_locked.count(a.p) && pool.kept() == 0);
    // a reset under a living batch, which ends after it
    reset(0);
    pool.end(a);
    CHECK(pool.kept() == 0);
    // many batches: at most as many blocks as batches are left, one at the end
    std::vector<StagingBlock> held;
    for (int k = 0; k < 20; ++k)
    {
        pool.begin();
        held.push_back(pool.take(0));
    }
    CHECK(g_locked.size() == 20);
    for (int k = 0; k < 20; ++k)
    {
        const int left = 19 - k;
        pool.end(held[k]);
        const int limit = left < 1 ? 1 : left < pool.kKeep ? left : pool.kKeep;
        CHECK(pool.kept() <= limit && g_locked.size() == (size_t)(left + pool.kept()));
    }
    CHECK(pool.kept() == 1);
    // another device's block is not handed out
    g_device = 1;
    pool.begin();
    StagingBlock d = pool.take(1);
    CHECK(d.device == 1 && d.context == g_context[1] && pool.kept() == 1);
    pool.end(d);
    // a batch that never read, and a lock that fails
    g_device = 0;
    pool.begin();
    pool.end(StagingBlock());
    reset(0);
    g_fail = true;
    pool.begin();
    CHECK(!pool.take(0).p);
    pool.end(StagingBlock());
    g_fail = false;
    // threads
    std::vector<std::thread> t;
    for (int k = 0; k < 8; ++k)
        t.emplace_back([&] {
            for (int i = 0; i < 2000; ++i)
            {
                pool.begin();
                StagingBlock b = pool.take(0);
                *(volatile char *)b.p = 1;
                pool.end(b);
            }
        });
    for (auto &x : t)
        x.join();
    CHECK(pool.kept() >= 1 && g_locked.size() <= 2);
    std::printf("ok\n");
    return 0;
}
