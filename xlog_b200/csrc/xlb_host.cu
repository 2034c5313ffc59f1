// A process-wide pool of page-locked host blocks that results are fetched into.
//
// A device-to-host copy into fresh pageable memory ran at 2.2 GB/s (the driver stages it through a
// small buffer on one thread, and that thread takes every page fault of the destination); into
// page-locked memory the same copy runs at 55 GB/s, the bus's rate.  cudaHostAlloc costs 0.38 ms a
// megabyte, so a block is made of huge pages touched by several threads and then registered
// (256 MB: 16 ms, against 97 ms by cudaHostAlloc and 121 ms for one pageable copy of that size):
// even a block used once pays for itself.  Blocks that come back are kept for the next result.
//
// Bounds: blocks in use and kept together stay below this process's share of an eighth of the
// machine's memory (at most 16 GB; xlb_host_alloc then gives nothing and the caller uses memory of its
// own), kept ones below 1 GB.  Ranks on one machine share the eighth: their number is LOCAL_WORLD_SIZE
// where the launcher says so, else that of the communicator; what is kept is given back when the last context of the process closes.  One lock guards the
// lists, and is not held while a block is made or given back; a block has one owner at a time and no device work refers to it once it is handed back
// (xlb_rel_to_host returns when its copies are done).  Blocks are registered on the device of an open
// context, whatever thread asks for them, and usable by all (cudaHostRegisterPortable).
#include <sys/mman.h>
#include <unistd.h>

#include <algorithm>
#include <cstdlib>
#include <exception>
#include <fstream>
#include <list>
#include <mutex>
#include <new>
#include <string>
#include <thread>
#include <unordered_map>
#include <vector>

#include "xlb_error.h"
#include "xlb_host.h"

namespace {

constexpr uint64_t HUGE_PAGE = 2ull << 20, IDLE_MAX = 1ull << 30, LIVE_MAX = 16ull << 30;

struct Block {
    void* p;
    uint64_t size;
    int device;  // that it was registered on, -1: the one its first user's thread had (no context was open)
};
using Blocks = std::list<Block>;
struct HostPool {
    std::mutex mu;
    Blocks used, idle;                                     // handed out; kept, the one kept longest first
    std::unordered_map<void*, Blocks::iterator> used_at;
    uint64_t used_bytes = 0, idle_bytes = 0;               // (used: with what is being made)
    uint64_t leaving_bytes = 0;                            // no longer kept, not yet given back
    unsigned ranks = 1;                                    // of the communicators made in this process, the most
    std::vector<int> devices;                              // of the open contexts

    // `f` with `device` current: on this thread where it is already, else on one of its own.  (The caller's
    // current device stays what it is, and a device that no context is open on is not set up by a
    // thread that never chose one.)  False: there is no thread to be had.
    template <class F>
    static bool with_device(int device, F f) {
        int current = -1;
        if (device < 0 || (cuda_take(cudaGetDevice(&current)) == cudaSuccess && current == device)) {
            f();
            return true;
        }
        try {
            std::thread([&] {
                if (cuda_take(cudaSetDevice(device)) == cudaSuccess) f();
            }).join();
        } catch (const std::exception&) {
            return false;
        }
        return true;
    }
    static void destroy(const Block& b) {
        bool done = false;
        const auto unregister = [&] { done = cuda_take(cudaHostUnregister(b.p)) == cudaSuccess; };
        if (!with_device(b.device, unregister)) unregister();
        if (done) munmap(b.p, b.size);  // (else the device still knows the pages: not for anybody else)
    }
    static void* create(uint64_t size, int device) {
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
        const uint64_t per = (pages + parts - 1) / parts * HUGE_PAGE;
        std::vector<std::thread> helpers;
        try {
            helpers.reserve(parts);
            for (uint64_t at = per; at < size; at += per) helpers.emplace_back(touch, p + at, std::min(per, size - at));
        } catch (const std::exception&) {  // no thread (or memory for one) to be had: registering touches the pages then
        }
        touch(p, std::min(per, size));
        for (auto& t : helpers) t.join();
        bool registered = false;
        with_device(device, [&] { registered = cuda_take(cudaHostRegister(p, size, cudaHostRegisterPortable)) == cudaSuccess; });
        if (!registered) {
            munmap(p, size);
            return nullptr;
        }
        return p;
    }
    // Kept blocks to be given back until `enough` holds.  (Lock held; what comes out goes to give_back without it.)
    template <class F>
    Blocks pick(F enough) {
        Blocks out;
        while (!idle.empty() && !enough()) {
            idle_bytes -= idle.front().size;
            leaving_bytes += idle.front().size;
            out.splice(out.end(), idle, idle.begin());
        }
        return out;
    }
    void give_back(const Blocks& blocks) {
        uint64_t bytes = 0;
        for (const Block& b : blocks) {
            destroy(b);
            bytes += b.size;
        }
        if (!bytes) return;
        std::lock_guard<std::mutex> g(mu);
        leaving_bytes -= bytes;
    }
    unsigned long sharers() const {
        const char* local = getenv("LOCAL_WORLD_SIZE");
        const unsigned long said = local ? strtoul(local, nullptr, 10) : 0;
        return said ? said : ranks;
    }
    uint64_t most() const {
        const uint64_t memory = (uint64_t)sysconf(_SC_PHYS_PAGES) * (uint64_t)sysconf(_SC_PAGESIZE);
        return std::min<uint64_t>(LIVE_MAX, memory / 8 / sharers());
    }
    void* take(uint64_t bytes) {
        if (bytes > LIVE_MAX) return nullptr;
        const uint64_t size = (bytes + HUGE_PAGE - 1) / HUGE_PAGE * HUGE_PAGE;
        Blocks one, out;
        {
            std::lock_guard<std::mutex> g(mu);
            auto best = idle.end();  // the smallest kept block that fits without wasting more than a quarter
            for (auto it = idle.begin(); it != idle.end(); ++it)
                if (it->size >= size && it->size <= size + size / 4 + HUGE_PAGE && (best == idle.end() || it->size < best->size)) best = it;
            if (best != idle.end()) {
                used_at.emplace(best->p, best);
                idle_bytes -= best->size;
                used_bytes += best->size;
                used.splice(used.end(), idle, best);
                return best->p;
            }
            const uint64_t limit = most();
            if (used_bytes + leaving_bytes + size > limit) return nullptr;
            one.push_back(Block{nullptr, size, devices.empty() ? -1 : devices.back()});
            const uint64_t gone = leaving_bytes;  // by other threads; what is picked here is gone before the new block is made
            out = pick([&] { return used_bytes + idle_bytes + gone + size <= limit; });
            used_bytes += size;
        }
        // Making a block takes milliseconds: without the lock.
        give_back(out);
        one.front().p = create(size, one.front().device);
        std::unique_lock<std::mutex> g(mu);
        if (one.front().p) {
            try {
                used_at.emplace(one.front().p, one.begin());
                used.splice(used.end(), one);
                return used.back().p;
            } catch (const std::bad_alloc&) {
            }
        }
        used_bytes -= size;
        g.unlock();
        if (one.front().p) destroy(one.front());
        return nullptr;
    }
    void give(void* p) {
        Blocks out;
        {
            std::lock_guard<std::mutex> g(mu);
            const auto at = used_at.find(p);
            if (at == used_at.end()) return;
            const auto it = at->second;
            used_at.erase(at);
            used_bytes -= it->size;
            idle_bytes += it->size;
            idle.splice(idle.end(), used, it);
            const uint64_t keep = devices.empty() ? 0 : IDLE_MAX;
            out = pick([&] { return idle_bytes <= keep; });
        }
        give_back(out);
    }
    void closed(int device) {
        Blocks out;
        {
            std::lock_guard<std::mutex> g(mu);
            const auto it = std::find(devices.begin(), devices.end(), device);
            if (it != devices.end()) devices.erase(it);
            if (devices.empty()) out = pick([] { return false; });
        }
        give_back(out);
    }
};
HostPool& pool() {
    static HostPool* p = new HostPool;  // never destroyed: results may outlive everything else in the process
    return *p;
}

}  // namespace

void host_pool_context_opened(int device) {
    std::lock_guard<std::mutex> g(pool().mu);
    pool().devices.push_back(device);
}
void host_pool_context_closed(int device) { pool().closed(device); }
void host_pool_ranks(unsigned ranks) {
    std::lock_guard<std::mutex> g(pool().mu);
    pool().ranks = std::max(pool().ranks, ranks);
}
uint64_t host_pool_most() {
    std::lock_guard<std::mutex> g(pool().mu);
    return pool().most();
}

// What the control groups of this process, and those above them, allow it of the cores (0: no bound is set).  `groups` is
// /proc/self/cgroup, `mount` where the groups' files are; version 2 has one tree, version 1 one for the processor.
unsigned host_cores_quota(const char* groups, const char* mount) {
    double least = 0;
    std::ifstream lines(groups);
    for (std::string line; std::getline(lines, line);) {
        const size_t a = line.find(':'), b = a == std::string::npos ? a : line.find(':', a + 1);
        if (b == std::string::npos) continue;
        const std::string kinds = "," + line.substr(a + 1, b - a - 1) + ",";
        const bool v2 = kinds == ",,";
        if (!v2 && kinds.find(",cpu,") == std::string::npos) continue;
        for (std::string path = line.substr(b + 1);; path.erase(path.find_last_of('/'))) {
            if (path == "/") path.clear();
            double quota = 0, period = 0;
            const std::string at = std::string(mount) + (v2 ? "" : "/cpu") + path;
            if (v2) std::ifstream(at + "/cpu.max") >> quota >> period;  // ("max": no number, none set)
            else {
                std::ifstream(at + "/cpu.cfs_quota_us") >> quota;  // (-1: none set)
                std::ifstream(at + "/cpu.cfs_period_us") >> period;
            }
            if (quota > 0 && period > 0 && (least == 0 || quota / period < least)) least = quota / period;
            if (path.empty() || path.find('/') == std::string::npos) break;
        }
    }
    return least > 0 ? std::max(1u, (unsigned)std::min(least, 1e6)) : 0;
}

unsigned host_pool_cores() {
    static const unsigned quota = host_cores_quota("/proc/self/cgroup", "/sys/fs/cgroup");
    const unsigned cores = std::thread::hardware_concurrency();
    std::lock_guard<std::mutex> g(pool().mu);
    return (quota ? std::min(quota, cores) : cores) / (unsigned)pool().sharers();
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
