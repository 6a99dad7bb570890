// mempool.h -- freed memory of the handles, kept for the next one.
//
// Systems come and go with the same sizes (served requests, the members of an ensemble), and cudaMalloc
// and cudaFree of their blocks cost milliseconds per handle; so freed blocks are kept, up to kPoolBytes
// of device memory and kPoolHost pinned blocks in the process, and given to the next handle that fits
// them.  All of it goes back to the driver when the last handle or server is gone (the one-shot
// calls' cached solver does not count), and when an allocation of the library runs out of memory.
// Only a block whose owner has waited for its last use (idle) is kept; any other is freed by cudaFree,
// which waits for the device itself.
//
// The lock covers the bookkeeping alone.  An allocation or a free of the driver can wait for a long
// launch, and another handle's request that the kept blocks satisfy must not wait with it.
//
// Drv: the driver's calls (int codes, 0: success), so that the pool is tested without a device.
// out_of_memory also clears the error, which the caller reports or has dealt with.
#pragma once

#include <algorithm>
#include <cstddef>
#include <map>
#include <mutex>
#include <vector>

namespace cismgpu {

constexpr size_t kPoolBytes = 4ull << 30;
constexpr size_t kPoolHostBlock = 4096, kPoolHost = 64;

template <class Drv>
class MemPool {
public:
    int take(void **p, size_t bytes) {
        *p = nullptr;
        const size_t unit = bytes >= (1u << 20) ? (1u << 20) : 512;
        const size_t n = std::max(unit, (bytes + unit - 1) / unit * unit);
        int dev = 0, e = Drv::device(&dev);
        if (e) return e;
        Blk b{nullptr, n, dev};
        {
            std::lock_guard<std::mutex> lk(mu);
            size_t best = idle.size();
            for (size_t k = 0; k < idle.size(); ++k)  // the smallest that fits without wasting a quarter
                if (idle[k].dev == dev && idle[k].n >= n && idle[k].n - n <= n / 4 &&
                    (best == idle.size() || idle[k].n < idle[best].n))
                    best = k;
            if (best < idle.size()) {
                b = idle[best];
                idle.erase(idle.begin() + best);
                held -= b.n;
                live[b.p] = b;
                *p = b.p;
                return 0;
            }
        }
        e = Drv::alloc(&b.p, n);
        if (e && Drv::out_of_memory(e) && shrink(0)) {
            e = Drv::alloc(&b.p, n);
            if (e) (void)Drv::out_of_memory(e);
        }
        if (e) return e;
        std::lock_guard<std::mutex> lk(mu);
        live[b.p] = b;
        *p = b.p;
        return 0;
    }

    void give(void *p, bool idle_block) {
        if (!p) return;
        std::vector<Blk> out;
        {
            std::lock_guard<std::mutex> lk(mu);
            auto it = live.find(p);
            if (it == live.end()) return;
            const Blk b = it->second;
            live.erase(it);
            if (!idle_block || b.n > kPoolBytes || users == 0) {
                out.push_back(b);
            } else {
                evict(kPoolBytes - b.n, out);
                idle.push_back(b);
                held += b.n;
            }
        }
        for (const Blk &b : out) Drv::release(b.p);
    }

    int take_host(void **p) {
        {
            std::lock_guard<std::mutex> lk(mu);
            if (!host.empty()) {
                *p = host.back();
                host.pop_back();
                return 0;
            }
        }
        return Drv::alloc_host(p, kPoolHostBlock);
    }

    void give_host(void *p, bool idle_block) {
        if (!p) return;
        {
            std::lock_guard<std::mutex> lk(mu);
            if (idle_block && host.size() < kPoolHost && users > 0) {
                host.push_back(p);
                return;
            }
        }
        Drv::release_host(p);
    }

    // Frees the oldest kept blocks until at most `bytes` are held; whether any was freed.
    bool shrink(size_t bytes) {
        std::vector<Blk> out;
        {
            std::lock_guard<std::mutex> lk(mu);
            evict(bytes, out);
        }
        for (const Blk &b : out) Drv::release(b.p);
        return !out.empty();
    }

    void join() {
        std::lock_guard<std::mutex> lk(mu);
        ++users;
    }

    void leave() {
        std::vector<Blk> out;
        std::vector<void *> out_host;
        {
            std::lock_guard<std::mutex> lk(mu);
            if (--users > 0) return;
            evict(0, out);
            out_host.swap(host);
        }
        for (const Blk &b : out) Drv::release(b.p);
        for (void *h : out_host) Drv::release_host(h);
    }

private:
    struct Blk {
        void *p;
        size_t n;
        int dev;
    };
    std::mutex mu;
    std::vector<Blk> idle;      // freed device blocks, oldest first
    size_t held = 0;            // their bytes
    std::map<void *, Blk> live; // blocks handed out
    std::vector<void *> host;   // freed pinned blocks of kPoolHostBlock bytes
    int users = 0;

    void evict(size_t bytes, std::vector<Blk> &out) {  // caller holds mu and frees out after it
        size_t k = 0;
        for (; k < idle.size() && held > bytes; ++k) {
            held -= idle[k].n;
            out.push_back(idle[k]);
        }
        idle.erase(idle.begin(), idle.begin() + k);
    }
};

}  // namespace cismgpu
