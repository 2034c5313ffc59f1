// A process-wide pool of page-locked host blocks that results are fetched into.
//
// A device-to-host copy into fresh pageable memory ran at 2.2 GB/s (the driver stages it through a
// small buffer on one thread, and that thread takes every page fault of the destination); into
// page-locked memory the same copy runs at 55 GB/s, the bus's rate.  cudaHostAlloc costs 0.38 ms a
// megabyte, so a block is made of huge pages touched by several threads and then registered
// (256 MB: 16 ms, against 97 ms by cudaHostAlloc and 121 ms for one pageable copy of that size):
// even a block used once pays for itself.  Blocks that come back are kept for the next result.
//
// Bounds: blocks in use and kept together stay below an eighth of the machine's memory (at most
// 16 GB; xlb_host_alloc then gives nothing and the caller uses memory of its own), kept ones below
// 1 GB; what is kept is given back when the last context of the process closes.  One lock guards the
// lists; a block has one owner at a time and no device work refers to it once it is handed back
// (xlb_rel_to_host returns when its copies are done).
#include <sys/mman.h>
#include <unistd.h>

#include <algorithm>
#include <list>
#include <mutex>
#include <system_error>
#include <thread>
#include <unordered_map>
#include <vector>

#include "xlb_error.h"
#include "xlb_host.h"

namespace {

constexpr uint64_t HUGE_PAGE = 2ull << 20, IDLE_MAX = 1ull << 30, LIVE_MAX = 16ull << 30;

struct HostPool {
    std::mutex mu;
    std::unordered_map<void*, uint64_t> used;         // blocks handed out
    std::list<std::pair<void*, uint64_t>> idle;       // blocks kept, the one kept longest first
    uint64_t used_bytes = 0, idle_bytes = 0, limit = 0;
    int contexts = 0;

    static void destroy(void* p, uint64_t size) {
        CUDA_QUIET(cudaHostUnregister(p));
        munmap(p, size);
    }
    static void* create(uint64_t size) {
        char* raw = (char*)mmap(nullptr, size + HUGE_PAGE, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
        if (raw == (char*)MAP_FAILED) return nullptr;
        char* p = (char*)(((uintptr_t)raw + HUGE_PAGE - 1) & ~(uintptr_t)(HUGE_PAGE - 1));
        if (p != raw) munmap(raw, p - raw);
        if (const uint64_t tail = HUGE_PAGE - (p - raw)) munmap(p + size, tail);
        madvise(p, size, MADV_HUGEPAGE);
        auto touch = [](char* at, uint64_t n) {
            for (uint64_t o = 0; o < n; o += 4096) at[o] = 0;
        };
        const unsigned cores = std::max(1u, std::thread::hardware_concurrency());
        const uint64_t pages = size / HUGE_PAGE, parts = std::min<uint64_t>({8, cores, (pages + 3) / 4});
        std::vector<std::thread> helpers;
        const uint64_t per = (pages + parts - 1) / parts * HUGE_PAGE;
        for (uint64_t at = per; at < size; at += per) {
            try {
                helpers.emplace_back(touch, p + at, std::min(per, size - at));
            } catch (const std::system_error&) {  // no thread to be had: registering touches the pages then
                break;
            }
        }
        touch(p, std::min(per, size));
        for (auto& t : helpers) t.join();
        if (cuda_take(cudaHostRegister(p, size, cudaHostRegisterPortable)) != cudaSuccess) {
            munmap(p, size);
            return nullptr;
        }
        return p;
    }
    void trim(uint64_t keep) {
        while (idle_bytes > keep) {
            auto b = idle.front();
            idle.pop_front();
            idle_bytes -= b.second;
            destroy(b.first, b.second);
        }
    }
    void* take(uint64_t bytes) {
        const uint64_t size = (bytes + HUGE_PAGE - 1) / HUGE_PAGE * HUGE_PAGE;
        std::lock_guard<std::mutex> g(mu);
        if (!limit) limit = std::min<uint64_t>(LIVE_MAX, (uint64_t)sysconf(_SC_PHYS_PAGES) * (uint64_t)sysconf(_SC_PAGESIZE) / 8);
        auto best = idle.end();  // the smallest kept block that fits without wasting more than a quarter
        for (auto it = idle.begin(); it != idle.end(); ++it)
            if (it->second >= size && it->second <= size + size / 4 + HUGE_PAGE && (best == idle.end() || it->second < best->second)) best = it;
        if (best != idle.end()) {
            auto b = *best;
            idle.erase(best);
            idle_bytes -= b.second;
            used[b.first] = b.second;
            used_bytes += b.second;
            return b.first;
        }
        if (used_bytes + size > limit) return nullptr;
        if (used_bytes + idle_bytes + size > limit) trim(limit - used_bytes - size);
        void* p = create(size);
        if (!p) return nullptr;
        used[p] = size;
        used_bytes += size;
        return p;
    }
    void give(void* p) {
        std::lock_guard<std::mutex> g(mu);
        auto it = used.find(p);
        if (it == used.end()) return;
        const uint64_t size = it->second;
        used.erase(it);
        used_bytes -= size;
        idle.emplace_back(p, size);
        idle_bytes += size;
        trim(contexts > 0 ? IDLE_MAX : 0);
    }
};
HostPool& pool() {
    static HostPool* p = new HostPool;  // never destroyed: results may outlive everything else in the process
    return *p;
}

}  // namespace

void host_pool_context_opened() {
    std::lock_guard<std::mutex> g(pool().mu);
    ++pool().contexts;
}
void host_pool_context_closed() {
    std::lock_guard<std::mutex> g(pool().mu);
    if (--pool().contexts == 0) pool().trim(0);
}

extern "C" xlb_status xlb_host_alloc(uint64_t bytes, void** out) {
    if (!out || !bytes) return XLB_ERR_INVALID;
    try {
        void* p = pool().take(bytes);
        if (!p) return XLB_ERR_RESOURCE_EXHAUSTED;
        *out = p;
    } catch (const std::bad_alloc&) {
        return XLB_ERR_RESOURCE_EXHAUSTED;
    }
    return XLB_OK;
}

extern "C" void xlb_host_free(void* p) {
    if (p) pool().give(p);
}
