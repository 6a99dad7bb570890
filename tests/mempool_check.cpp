// The handles' memory (cism_b200/csrc/mempool.h) on a driver of the host's own.
#include <atomic>
#include <chrono>
#include <condition_variable>
#include <cstdio>
#include <cstdlib>
#include <set>
#include <thread>

#include "mempool.h"

using namespace cismgpu;

#define EXPECT(c)                                                      \
    do {                                                               \
        if (!(c)) {                                                    \
            std::printf("%s:%d: %s\n", __FILE__, __LINE__, #c);        \
            std::exit(1);                                              \
        }                                                              \
    } while (0)

static std::mutex g_mu;
static std::condition_variable g_cv;
static std::set<void *> g_dev, g_host;  // what the driver has handed out
static size_t g_allocs = 0;
static int g_device = 0, g_fail = 0;    // g_fail: allocations that still fail
static bool g_hold = false, g_held = false, g_go = false;

struct Drv {
    static int device(int *d) { *d = g_device; return 0; }
    static int alloc(void **p, size_t n) {
        std::lock_guard<std::mutex> lk(g_mu);
        ++g_allocs;
        if (g_fail > 0) { --g_fail; return 2; }
        *p = std::malloc(1);
        (void)n;
        g_dev.insert(*p);
        return 0;
    }
    static void release(void *p) {
        std::unique_lock<std::mutex> lk(g_mu);
        EXPECT(g_dev.erase(p) == 1);
        if (g_hold) {  // a free that waits for the device, until the other thread has been served
            g_held = true;
            g_cv.notify_all();
            EXPECT(g_cv.wait_for(lk, std::chrono::seconds(20), [] { return g_go; }));
        }
    }
    static int alloc_host(void **p, size_t) {
        std::lock_guard<std::mutex> lk(g_mu);
        *p = std::malloc(1);
        g_host.insert(*p);
        return 0;
    }
    static void release_host(void *p) {
        std::lock_guard<std::mutex> lk(g_mu);
        EXPECT(g_host.erase(p) == 1);
    }
    static bool out_of_memory(int e) { return e == 2; }
};

int main() {
    const size_t MB = 1u << 20, GB = 1u << 30;
    void *a, *b, *c;
    {  // kept and reused; a block that wastes more than a quarter, or of another device, is not
        MemPool<Drv> P;
        P.join();
        EXPECT(!P.take(&a, 10 * MB));
        P.give(a, true);
        EXPECT(!P.take(&b, 9 * MB) && b == a);
        P.give(b, true);
        EXPECT(!P.take(&b, 7 * MB) && b != a);
        g_device = 1;
        EXPECT(!P.take(&c, 10 * MB) && c != a);
        g_device = 0;
        P.give(b, false);  // not idle: freed
        P.give(c, false);
        EXPECT(g_dev.size() == 1 && g_dev.count(a));
        P.leave();  // the last user: all of it goes back
        EXPECT(g_dev.empty());
    }
    {  // without a user nothing is kept
        MemPool<Drv> P;
        EXPECT(!P.take(&a, MB) && !P.take_host(&b));
        P.give(a, true);
        P.give_host(b, true);
        EXPECT(g_dev.empty() && g_host.empty());
    }
    {  // the bound: the oldest make room
        MemPool<Drv> P;
        P.join();
        void *p[6];
        for (auto &q : p) EXPECT(!P.take(&q, GB));
        for (auto &q : p) P.give(q, true);
        EXPECT(g_dev.size() == 4 && !g_dev.count(p[0]) && !g_dev.count(p[1]));
        EXPECT(!P.take(&a, 5 * GB));
        P.give(a, true);  // larger than the bound
        EXPECT(g_dev.size() == 4);
        EXPECT(P.shrink(2 * GB) && g_dev.size() == 2 && g_dev.count(p[5]));
        EXPECT(!P.shrink(2 * GB));
        P.leave();
        EXPECT(g_dev.empty());
    }
    {  // out of memory: what is kept goes back first, then the call is tried again, and fails for good
        MemPool<Drv> P;
        P.join();
        EXPECT(!P.take(&a, GB));
        P.give(a, true);
        g_fail = 1;
        EXPECT(!P.take(&b, 3 * GB) && g_dev.size() == 1 && g_dev.count(b));
        g_fail = 1;
        EXPECT(P.take(&c, MB) == 2 && c == nullptr);
        P.give(b, true);
        P.leave();
        EXPECT(g_dev.empty());
    }
    {  // a free that waits does not hold up a request that the kept blocks satisfy
        MemPool<Drv> P;
        P.join();
        EXPECT(!P.take(&a, MB) && !P.take(&b, 8 * MB));
        P.give(a, true);
        g_hold = true;
        std::thread t([&] { P.give(b, false); });
        {
            std::unique_lock<std::mutex> lk(g_mu);
            EXPECT(g_cv.wait_for(lk, std::chrono::seconds(20), [] { return g_held; }));
        }
        EXPECT(!P.take(&c, MB) && c == a);
        {
            std::lock_guard<std::mutex> lk(g_mu);
            g_go = true;
            g_cv.notify_all();
        }
        t.join();
        g_hold = false;
        P.give(c, true);
        P.leave();
    }
    {  // threads: every block handed out once, nothing lost
        MemPool<Drv> P;
        P.join();
        std::atomic<bool> bad{false};
        std::mutex mu;
        std::set<void *> out;
        std::vector<std::thread> ts;
        for (int t = 0; t < 4; ++t)
            ts.emplace_back([&, t] {
                for (int k = 0; k < 2000; ++k) {
                    void *p = nullptr, *h = nullptr;
                    if (P.take(&p, (1 + (k * 7 + t) % 5) * MB) || P.take_host(&h)) bad = true;
                    {
                        std::lock_guard<std::mutex> lk(mu);
                        if (!out.insert(p).second || !out.insert(h).second) bad = true;
                    }
                    {
                        std::lock_guard<std::mutex> lk(mu);
                        out.erase(p);
                        out.erase(h);
                    }
                    P.give(p, k % 3 != 0);
                    P.give_host(h, true);
                    if (k % 500 == 0) P.shrink(0);
                }
            });
        for (auto &t : ts) t.join();
        EXPECT(!bad);
        P.leave();
        EXPECT(g_dev.empty() && g_host.empty());
    }
    std::puts("ok");
}
