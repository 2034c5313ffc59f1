// Shared host-side plumbing: status handling, the context, the stream-ordered device arena.
#pragma once
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <chrono>
#include <cstring>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <map>
#include <memory>
#include <string>
#include <vector>

#include "xlb_error.h"

struct Comm;  // NCCL exchange layer (xlb_comm.cu)

// Device-side status word, after the reference's ResidentTerminalStatus convention
// (crates/xlog-cuda/kernels/resident_relational.cu:22-31): kernels never trap; the first failure
// publishes (code, detail) and the host reads it at the next phase boundary.
struct DevStatus {
    unsigned int code;   // xlb_status
    unsigned int where;  // kernel-specific site id
    unsigned long long detail;
};

// Driver entry points of the virtual-memory API, looked up through the runtime so that the
// library does not link against the driver library (it must load on a machine without one).
struct VmmApi {
    PFN_cuMemAddressReserve reserve = nullptr;
    PFN_cuMemAddressFree addr_free = nullptr;
    PFN_cuMemCreate create = nullptr;
    PFN_cuMemRelease release = nullptr;
    PFN_cuMemMap map = nullptr;
    PFN_cuMemUnmap unmap = nullptr;
    PFN_cuMemSetAccess set_access = nullptr;
    PFN_cuMemGetAllocationGranularity granularity = nullptr;
    bool ok = false;
    static const VmmApi& get() {
        static const VmmApi api = load();
        return api;
    }
    static VmmApi load() {
        VmmApi a;
        auto sym = [](const char* name, void** fn) {
            cudaDriverEntryPointQueryResult q = cudaDriverEntryPointSymbolNotFound;
            return cuda_take(cudaGetDriverEntryPoint(name, fn, cudaEnableDefault, &q)) == cudaSuccess && q == cudaDriverEntryPointSuccess && *fn != nullptr;
        };
        a.ok = sym("cuMemAddressReserve", (void**)&a.reserve) && sym("cuMemAddressFree", (void**)&a.addr_free) && sym("cuMemCreate", (void**)&a.create) &&
               sym("cuMemRelease", (void**)&a.release) && sym("cuMemMap", (void**)&a.map) && sym("cuMemUnmap", (void**)&a.unmap) &&
               sym("cuMemSetAccess", (void**)&a.set_access) && sym("cuMemGetAllocationGranularity", (void**)&a.granularity);
        return a;
    }
};

// Device memory arena.  Every buffer of a context is used on the context's one stream, so a block
// that the host has freed can be handed out again at once: the work that used it was enqueued
// earlier on the same stream.  That makes a plain host-side free list enough, and keeps the CUDA
// allocator off the hot path: a fixpoint allocates and frees a few hundred temporaries, and the
// driver's stream-ordered pool was measured to spend milliseconds remapping its reserve in one
// step out of three for the first twenty steps of a repeated workload.
//
// Backing store: one reserved virtual address range as large as the device's memory, with physical
// memory mapped at its front chunk by chunk (the driver's virtual-memory API).  The arena is then
// one contiguous block that grows at its end, free neighbours always coalesce, and a request that
// does not fit extends the last free block by the missing part only.  With separate cudaMalloc
// slabs instead, a repeated workload with 128 MB buffers was seen to need a new 1 GB slab (a 4 to
// 11 ms stall) in its eighth repetition with 380 MB free in six pieces.  Slabs remain as the
// fallback where the virtual-memory API is unavailable (or XLB_ARENA_SLABS is set).
struct Arena {
    struct Slab {
        char* base;
        uint64_t size;
    };
    struct Chunk {
        CUmemGenericAllocationHandle handle;
        uint64_t size;
    };
    std::vector<Slab> slabs;    // fallback backing
    std::vector<Chunk> chunks;  // virtual-memory backing: mapped back to back from va_base
    char* va_base = nullptr;
    uint64_t va_size = 0, mapped = 0, gran = 0;
    int device = 0;
    bool vmm = false, vmm_tried = false;
    std::map<char*, uint64_t> free_by_addr;
    std::multimap<uint64_t, char*> free_by_size;
    uint64_t reserved = 0;
    bool trace = getenv("XLB_ARENA_TRACE") != nullptr;  // report every time the arena has to grow
    static constexpr uint64_t ALIGN = 512, MIN_SLAB = 256ull << 20, MAX_GROW = 8ull << 30;
    static constexpr uint64_t VMM_MIN_STEP = 64ull << 20, VMM_MAX_STEP = 2ull << 30;

    static uint64_t round_up(uint64_t n) { return (n + ALIGN - 1) / ALIGN * ALIGN; }
    void insert_free(char* p, uint64_t n) {
        free_by_addr[p] = n;
        free_by_size.emplace(n, p);
    }
    void erase_free(char* p, uint64_t n) {
        free_by_addr.erase(p);
        auto r = free_by_size.equal_range(n);
        for (auto it = r.first; it != r.second; ++it)
            if (it->second == p) {
                free_by_size.erase(it);
                break;
            }
    }
    CUmemAllocationProp vmm_prop() const {
        CUmemAllocationProp prop;
        memset(&prop, 0, sizeof prop);
        prop.type = CU_MEM_ALLOCATION_TYPE_PINNED;
        prop.location.type = CU_MEM_LOCATION_TYPE_DEVICE;
        prop.location.id = device;
        return prop;
    }
    // Reserve the address range (once).  False: use slabs.
    bool vmm_start() {
        if (vmm_tried) return vmm;
        vmm_tried = true;
        if (getenv("XLB_ARENA_SLABS")) return false;
        const VmmApi& api = VmmApi::get();
        int supported = 0;
        if (!api.ok || cuda_take(cudaDeviceGetAttribute(&supported, cudaDevAttrMemoryPoolsSupported, device)) != cudaSuccess || !supported) return false;
        CUmemAllocationProp prop = vmm_prop();
        size_t g = 0;
        if (api.granularity(&g, &prop, CU_MEM_ALLOC_GRANULARITY_RECOMMENDED) != CUDA_SUCCESS || g == 0) return false;
        size_t free_b = 0, total_b = 0;
        if (cuda_take(cudaMemGetInfo(&free_b, &total_b)) != cudaSuccess) return false;
        gran = g;
        va_size = (total_b + gran - 1) / gran * gran;
        CUdeviceptr base = 0;
        if (api.reserve(&base, va_size, 0, 0, 0) != CUDA_SUCCESS) return false;
        va_base = (char*)base;
        vmm = true;
        return true;
    }
    // Map `step` more bytes at the end of the mapped part and hand them to the free list.
    bool vmm_map(uint64_t step) {
        const VmmApi& api = VmmApi::get();
        if (mapped + step > va_size) return false;
        CUmemAllocationProp prop = vmm_prop();
        CUmemGenericAllocationHandle h;
        if (api.create(&h, step, &prop, 0) != CUDA_SUCCESS) return false;
        CUdeviceptr at = (CUdeviceptr)(va_base + mapped);
        if (api.map(at, step, 0, h, 0) != CUDA_SUCCESS) {
            api.release(h);
            return false;
        }
        CUmemAccessDesc acc;
        memset(&acc, 0, sizeof acc);
        acc.location.type = CU_MEM_LOCATION_TYPE_DEVICE;
        acc.location.id = device;
        acc.flags = CU_MEM_ACCESS_FLAGS_PROT_READWRITE;
        if (api.set_access(at, step, &acc, 1) != CUDA_SUCCESS) {
            api.unmap(at, step);
            api.release(h);
            return false;
        }
        chunks.push_back({h, step});
        char* p = va_base + mapped;
        mapped += step;
        reserved += step;
        release(p, step);  // coalesces with a free block that ended at the old end
        return true;
    }
    // size of the free block that ends where the mapped part ends (0: none)
    uint64_t vmm_tail_free() const {
        if (free_by_addr.empty()) return 0;
        auto last = std::prev(free_by_addr.end());
        return last->first + last->second == va_base + mapped ? last->second : 0;
    }
    bool vmm_grow(uint64_t n) {
        const uint64_t tail = vmm_tail_free();
        const uint64_t need = ((n > tail ? n - tail : 0) + gran - 1) / gran * gran;
        if (need == 0) return true;
        // grow by half of what is mapped, within [64 MB, 2 GB], or by the request if that is more
        uint64_t step = std::max<uint64_t>(need, std::min<uint64_t>(std::max<uint64_t>(mapped / 2, VMM_MIN_STEP), VMM_MAX_STEP));
        step = (step + gran - 1) / gran * gran;
        return vmm_map(step) || (step > need && vmm_map(need));
    }
    // Unmap whole chunks at the end that are entirely free (after the stream has drained).
    void vmm_trim() {
        const VmmApi& api = VmmApi::get();
        while (!chunks.empty()) {
            const uint64_t tail = vmm_tail_free(), sz = chunks.back().size;
            if (tail < sz) break;
            char* tail_at = va_base + mapped - tail;
            erase_free(tail_at, tail);
            if (tail > sz) insert_free(tail_at, tail - sz);
            api.unmap((CUdeviceptr)(va_base + mapped - sz), sz);
            api.release(chunks.back().handle);
            chunks.pop_back();
            mapped -= sz;
            reserved -= sz;
        }
    }
    bool add_slab(uint64_t size) {
        void* p = nullptr;
        if (cuda_take(cudaMalloc(&p, size)) != cudaSuccess) return false;
        slabs.push_back({(char*)p, size});
        reserved += size;
        insert_free((char*)p, size);
        return true;
    }
    // Give back every part of the backing store that is entirely free (after the stream has drained).
    void trim(cudaStream_t stream) {
        CUDA_QUIET(cudaStreamSynchronize(stream));
        if (vmm) {
            vmm_trim();
            return;
        }
        for (size_t i = 0; i < slabs.size();) {
            auto it = free_by_addr.find(slabs[i].base);
            if (it != free_by_addr.end() && it->second == slabs[i].size) {
                erase_free(slabs[i].base, slabs[i].size);
                CUDA_QUIET(cudaFree(slabs[i].base));
                reserved -= slabs[i].size;
                slabs.erase(slabs.begin() + i);
            } else ++i;
        }
    }
    void* alloc(uint64_t n, cudaStream_t stream) {
        n = round_up(n);
        for (int attempt = 0; attempt < 3; ++attempt) {
            auto it = free_by_size.lower_bound(n);  // best fit
            if (it != free_by_size.end()) {
                char* p = it->second;
                uint64_t have = it->first;
                erase_free(p, have);
                if (have > n) insert_free(p + n, have - n);
                return p;
            }
            if (trace) {
                uint64_t free_total = 0;
                for (auto& f : free_by_size) free_total += f.first;
                fprintf(stderr, "[xlb arena] attempt %d: no block of %llu bytes; reserved %llu in %zu pieces, free %llu in %zu blocks, largest %llu\n", attempt,
                        (unsigned long long)n, (unsigned long long)reserved, vmm ? chunks.size() : slabs.size(), (unsigned long long)free_total, free_by_size.size(),
                        (unsigned long long)(free_by_size.empty() ? 0 : free_by_size.rbegin()->first));
            }
            if (vmm_start()) {
                if (attempt == 0 && vmm_grow(n)) continue;
                return nullptr;  // the device (or the address range) is full: trimming this arena cannot help it
            }
            if (attempt == 0) {
                uint64_t grow = std::max<uint64_t>(MIN_SLAB, std::min<uint64_t>(reserved, MAX_GROW));
                if (add_slab(std::max(n, grow)) || (grow > n && add_slab(n))) continue;
            } else if (attempt == 1) {
                trim(stream);
                if (add_slab(n)) continue;
            }
        }
        return nullptr;
    }
    void release(void* ptr, uint64_t n) {
        char* p = (char*)ptr;
        n = round_up(n);
        auto next = free_by_addr.lower_bound(p);
        // coalesce with the free block after and before, unless a slab boundary lies between
        if (next != free_by_addr.end() && next->first == p + n && !is_slab_base(next->first)) {
            uint64_t m = next->second;
            erase_free(next->first, m);
            n += m;
        }
        auto prev = free_by_addr.lower_bound(p);
        if (prev != free_by_addr.begin()) {
            --prev;
            if (prev->first + prev->second == p && !is_slab_base(p)) {
                char* q = prev->first;
                uint64_t m = prev->second;
                erase_free(q, m);
                p = q;
                n += m;
            }
        }
        insert_free(p, n);
    }
    bool is_slab_base(char* p) const {
        for (auto& s : slabs)
            if (s.base == p) return true;
        return false;
    }
    void destroy() {
        for (auto& s : slabs) CUDA_QUIET(cudaFree(s.base));
        slabs.clear();
        if (vmm) {
            const VmmApi& api = VmmApi::get();
            uint64_t at = mapped;
            for (size_t i = chunks.size(); i-- > 0;) {
                at -= chunks[i].size;
                api.unmap((CUdeviceptr)(va_base + at), chunks[i].size);
                api.release(chunks[i].handle);
            }
            chunks.clear();
            api.addr_free((CUdeviceptr)va_base, va_size);
            va_base = nullptr;
            va_size = mapped = 0;
            vmm = vmm_tried = false;
        }
        free_by_addr.clear();
        free_by_size.clear();
        reserved = 0;
    }
};

struct xlb_ctx {
    int device = 0;
    cudaStream_t stream = nullptr;
    Arena arena;
    uint64_t budget = 0, allocated = 0, peak = 0;
    uint64_t max_iterations = 1000000;
    uint64_t join_chunk = 0;
    uint32_t flags = 0;
    uint64_t launches = 0;
    uint64_t syncs = 0;       // host waits on the stream (count read-backs)
    double ms_sync_wait = 0;  // wall time spent inside those waits
    double ms_alloc = 0;      // wall time spent in the device allocator (allocate + free calls)
    std::string last_error;
    // pinned scratch for scalar read-backs
    unsigned long long* h_scalar = nullptr;  // SCALAR_WORDS words; read_words uses those from READ_WORDS_AT on
    unsigned long long* h_scalar_dev = nullptr;  // the same words as the device sees them (mapped): a kernel can leave counts there
    unsigned long long publish_seq = 0;          // number of the last set of counts a kernel was asked to leave there
    char* h_stage = nullptr;      // page-locked staging of small results and of the runs of large ones (made on first use) ...
    char* h_stage_dev = nullptr;  // ... as the device sees it
    DevStatus* d_status = nullptr;
    unsigned read_seq = 0;      // number of the last read-back (read_words)
    unsigned status_code = 0;   // device status as the last read-back found it ...
    bool drained = false;       // ... and nothing was enqueued since: all of it has done its work and the code is current
    bool leaving = false;       // the last kernel enqueued leaves the status itself (Publish), which nobody has read yet
    unsigned* arrived = nullptr;  // its blocks that are done: zero between kernels
    cudaEvent_t plan_e0 = nullptr, plan_e1 = nullptr;  // around a plan (made on first use)
    cudaStream_t copy_stream = nullptr;                // copies of a large result, beside the stream (made on first use)
    cudaEvent_t copy_behind = nullptr;
    int sm_count = 148;
    // executor state
    std::map<uint32_t, std::string> rel_names;
    std::map<std::string, xlb_rel*> store;
    std::map<std::string, uint64_t> versions;
    struct IndexCache* indexes = nullptr;
    Comm* comm = nullptr;
    // `world` / `rank` are what the executor plans by; while a strongly connected component runs
    // on replicated relations they read 1 / 0 although the communicator has comm_world ranks.
    uint32_t rank = 0, world = 1;
    uint32_t comm_rank = 0, comm_world = 1;
    void (*wait_hook)(xlb_ctx*) = nullptr;  // set with a communicator: host waits then watch it as well
    // bounded look-back of the one-sweep sort: polls before a tile gives up (XLB_ERR_TIMEOUT), and
    // the number the first tile takes (0; a test makes tile 0 never run so that the wait runs out)
    unsigned lb_spin_limit = 1u << 22, lb_first_tile = 0;
    unsigned delta_spin_limit = 1u << 26;  // polls (tens of seconds) for which a block of the delta loop waits without seeing anything go on
    bool frontier_attr_set = false, frontier_many_attr_set = false, frontier_large_attr_set = false;  // the same for the frontier kernels
    bool index_attr_set = false;  // the same for direct_small_k
    bool delta_wide_attr_set = false;  // the same for the kernel by rows of the head
    bool query_attr_set = false;  // the same for the one-block joins and group-bys
    bool delta_attr_set = false;  // the same for the delta loop's kernel
    bool sort_attr_set = false;  // the scatter kernels' shared-memory opt-in was made on this context's device
    // per-kernel event timing (xlb_profile_enable)
    struct ProfEntry {
        uint64_t launches = 0, bytes = 0;
        double ms = 0;
        std::vector<std::pair<cudaEvent_t, cudaEvent_t>> pending;
    };
    std::map<std::string, ProfEntry> prof;
    std::string prof_filter;  // "" = off, "*" = every kernel, else kernel names separated by commas
    ProfEntry* prof_open = nullptr;
    cudaEvent_t prof_e0 = nullptr;
    cudaError_t error_before = cudaSuccess;  // what was on the thread when the operation at hand began (nothing, if every call is checked)
    // host timeline of one plan execution (XLB_TRACE_HOST=1): every launch and every wait with its
    // wall-clock interval, printed to stderr when the plan is done
    struct TraceNote {
        double t0, t1;
        const char* what;
    };
    bool trace_on = false;
    std::vector<TraceNote> trace;
};

constexpr uint64_t STAGE_BYTES = 256ull << 10;  // of h_stage
constexpr int SCALAR_WORDS = 128, READ_WORDS_AT = 64, READ_WORDS_MAX = 16;

// Counts a kernel leaves in pinned memory for the host: low 40 bits the count, top 24 the number
// of the launch that wrote it.
constexpr int PUBLISH_COUNT_BITS = 40;
constexpr unsigned long long PUBLISH_TAG_MASK = 0xFFFFFFull;

inline double trace_now() { return std::chrono::duration<double, std::micro>(std::chrono::steady_clock::now().time_since_epoch()).count(); }
inline void trace_note(xlb_ctx* c, const char* what, double t0) {
    if (c->trace_on) c->trace.push_back({t0, trace_now(), what});
}

// Bracket one launch with CUDA events on the launching stream when its kernel is profiled.
inline void prof_begin(xlb_ctx* c, const char* name, uint64_t bytes) {
    if (c->trace_on) trace_note(c, name, trace_now());
    if (c->prof_filter.empty()) return;
    if (c->prof_filter != "*") {  // a kernel name, or several separated by commas
        const std::string& f = c->prof_filter;
        const size_t len = strlen(name);
        bool hit = false;
        for (size_t at = f.find(name); at != std::string::npos && !hit; at = f.find(name, at + 1))
            hit = (at == 0 || f[at - 1] == ',') && (at + len == f.size() || f[at + len] == ',');
        if (!hit) return;
    }
    auto& e = c->prof[name];
    e.launches++;
    e.bytes += bytes;
    CUDA_OK(cudaEventCreate(&c->prof_e0));
    CUDA_OK(cudaEventRecord(c->prof_e0, c->stream));
    c->prof_open = &e;
}

// Bytes of a launch that the host learns only later (a count read back after the launch).
inline void prof_add_bytes(xlb_ctx* c, const char* name, uint64_t bytes) {
    if (c->prof_filter.empty()) return;
    auto it = c->prof.find(name);
    if (it != c->prof.end()) it->second.bytes += bytes;
}

// A device allocation charged to the context's budget (GpuMemoryManager::alloc with a
// MemoryBudget, crates/xlog-cuda/src/memory.rs:57-1350).  Freed stream-ordered.
struct DevBuf {
    xlb_ctx* ctx;
    void* p = nullptr;
    uint64_t bytes = 0;
    DevBuf(xlb_ctx* c, uint64_t n) : ctx(c), bytes(n) {
        if (n == 0) return;
        if (c->budget && c->allocated + n > c->budget)
            xlb_fail(XLB_ERR_RESOURCE_EXHAUSTED, "device memory budget exceeded: %llu + %llu > %llu bytes",
                     (unsigned long long)c->allocated, (unsigned long long)n, (unsigned long long)c->budget);
        auto t0 = std::chrono::steady_clock::now();
        p = c->arena.alloc(n, c->stream);
        c->ms_alloc += std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
        if (!p)
            xlb_fail(XLB_ERR_RESOURCE_EXHAUSTED, "device memory exhausted: %llu bytes requested with %llu allocated and %llu reserved",
                     (unsigned long long)n, (unsigned long long)c->allocated, (unsigned long long)c->arena.reserved);
        c->allocated += n;
        if (c->allocated > c->peak) c->peak = c->allocated;
    }
    ~DevBuf() {
        if (p) {
            ctx->arena.release(p, bytes);
            ctx->allocated -= bytes;
        }
    }
    DevBuf(const DevBuf&) = delete;
    DevBuf& operator=(const DevBuf&) = delete;
    // Only the first n bytes are kept; the others are free for later work on the stream.
    void keep(uint64_t n) {
        if (!p || n >= bytes) return;
        const uint64_t held = Arena::round_up(n);
        if (held < bytes) ctx->arena.release((char*)p + held, bytes - held);
        ctx->allocated -= bytes - n;
        bytes = n;
        if (!n) p = nullptr;
    }
    template <class T>
    T* as() const { return (T*)p; }
};
using Buf = std::shared_ptr<DevBuf>;
inline Buf make_buf(xlb_ctx* c, uint64_t bytes) { return std::make_shared<DevBuf>(c, bytes); }
// Whether the budget leaves room for `bytes` more.  A route that wants more than the result and has another
// route behind it asks first.
inline bool within_budget(const xlb_ctx* c, uint64_t bytes) { return !c->budget || (c->allocated <= c->budget && bytes <= c->budget - c->allocated); }

inline void check_launch(xlb_ctx* c, const char* what) {
    const cudaError_t launched = cudaGetLastError();  // (before anything else takes it)
    c->launches++;
    c->drained = c->leaving = false;
    if (c->prof_open) {
        cudaEvent_t e1;
        CUDA_OK(cudaEventCreate(&e1));
        CUDA_OK(cudaEventRecord(e1, c->stream));
        c->prof_open->pending.emplace_back(c->prof_e0, e1);
        c->prof_open = nullptr;
    }
    if (launched == cudaSuccess) return;
    if (c->error_before != cudaSuccess) xlb_fail(XLB_ERR_CUDA, "an error from before the operation, found at the launch of %s: %s", what, cudaGetErrorString(c->error_before));
    xlb_fail(XLB_ERR_CUDA, "launch of %s failed: %s", what, cudaGetErrorString(launched));
}

// Copies and fills enqueued on the context's stream.
inline cudaError_t copy_async(xlb_ctx* c, void* dst, const void* src, size_t n, cudaMemcpyKind kind) {
    c->drained = c->leaving = false;
    return cudaMemcpyAsync(dst, src, n, kind, c->stream);
}
inline cudaError_t set_async(xlb_ctx* c, void* dst, int value, size_t n) {
    c->drained = c->leaving = false;
    return cudaMemsetAsync(dst, value, n, c->stream);
}

// Wait for everything enqueued on the stream.
inline void stream_wait(xlb_ctx* c) {
    const double tr0 = c->trace_on ? trace_now() : 0;
    if (c->wait_hook) {  // several ranks: never block for good on a stream a late peer may be holding up
        c->wait_hook(c);
        trace_note(c, "wait (communicator watched)", tr0);
        return;
    }
    auto t0 = std::chrono::steady_clock::now();
    static const bool spin = getenv("XLB_BLOCKING_WAIT") == nullptr;
    bool done = false;
    if (spin) {  // poll first: a fixpoint waits for a row count many times, and a blocked thread's wake-up
                 // costs milliseconds on a busy host; after 5 ms fall back to a blocking wait
        for (;;) {
            const cudaError_t q = cuda_take(cudaStreamQuery(c->stream));
            if (q == cudaSuccess) {
                done = true;
                break;
            }
            if (q != cudaErrorNotReady) xlb_fail(XLB_ERR_CUDA, "waiting for the stream: %s", cudaGetErrorString(q));
            if (std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count() > 5.0) break;
        }
    }
    if (!done) CUDA_OK(cudaStreamSynchronize(c->stream));
    c->ms_sync_wait += std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
    c->syncs++;
    trace_note(c, "wait", tr0);
}

// A read-back of a few words and of the device status.  A kernel writes them into mapped pinned
// memory and the host polls for them: 7 us from launch to value, where a copy and a wait for the
// stream took 16.  A word goes out as two halves, each with the read-back's number beside it, so
// the host knows that a half has arrived whatever order the writes cross the bus in, and no fence
// towards the host is needed.
static __global__ void publish_words_k(const unsigned long long* __restrict__ src, int n, const DevStatus* st, unsigned long long* dst, unsigned seq) {
    const int i = threadIdx.x;
    if (i > 2 * n) return;
    unsigned half = i == 2 * n ? st->code : (unsigned)(src[i >> 1] >> ((i & 1) * 32));
    *(volatile unsigned long long*)(dst + i) = ((unsigned long long)seq << 32) | half;
}

// The same by the kernel that computes the words: its last block to finish sends them, which saves the
// launch of another (4 us).  For kernels of few blocks, which all pass publish_last at their end (the
// arrivals queue on one counter); or publish_now, by one block that knows all others are done.
struct Publish {
    unsigned long long* dst = nullptr;  // null: not asked to
    const unsigned long long* src = nullptr;
    const DevStatus* st = nullptr;
    unsigned* arrived = nullptr;
    int n = 0;
    unsigned seq = 0;
};
constexpr unsigned PUBLISH_BLOCKS_MAX = 1184;
__device__ __forceinline__ void publish_now(const Publish& p) {  // all threads of a block
    if (!p.dst) return;
    __syncthreads();
    for (int i = threadIdx.x; i <= 2 * p.n; i += blockDim.x) {
        const unsigned half = i == 2 * p.n ? __ldcg(&p.st->code) : (unsigned)(__ldcg(&p.src[i >> 1]) >> ((i & 1) * 32));
        *(volatile unsigned long long*)(p.dst + i) = ((unsigned long long)p.seq << 32) | half;
    }
}
__device__ __forceinline__ void publish_last(const Publish& p) {  // all threads of all blocks
    if (!p.dst) return;
    __shared__ bool last_s;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        last_s = atomicAdd(p.arrived, 1u) == gridDim.x - 1;
        if (last_s) {
            *(volatile unsigned*)p.arrived = 0;
            __threadfence();
        }
    }
    __syncthreads();
    if (last_s) publish_now(p);
}
inline bool publish_ok(xlb_ctx* c, int n) {
    static const bool spin = getenv("XLB_BLOCKING_WAIT") == nullptr;
    return !c->wait_hook && spin && n <= READ_WORDS_MAX;
}
// What a kernel of `blocks` blocks gets so that it leaves `n` words from `dptr` (none: the status alone).
inline Publish publish_by(xlb_ctx* c, uint64_t blocks, const void* dptr = nullptr, int n = 0) {
    Publish p;
    c->leaving = false;
    if (blocks > PUBLISH_BLOCKS_MAX || !publish_ok(c, n)) return p;
    if (++c->read_seq == 0) ++c->read_seq;  // 0 is what untouched words carry
    p.dst = c->h_scalar_dev + READ_WORDS_AT;
    p.src = (const unsigned long long*)dptr;
    p.st = c->d_status;
    p.arrived = c->arrived;
    p.n = n;
    p.seq = c->read_seq;
    return p;
}
inline void poll_words(xlb_ctx* c, int n, unsigned long long* out) {
    const double tr0 = c->trace_on ? trace_now() : 0;
    auto t0 = std::chrono::steady_clock::now();
    const volatile unsigned long long* w = c->h_scalar + READ_WORDS_AT;
    uint64_t polls = 0;
    bool waited = false;
    for (int i = 0; i <= 2 * n; ++i)
        while ((unsigned)(w[i] >> 32) != c->read_seq) {
            if ((++polls & 1023) || std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count() < 5.0) continue;
            if (waited) xlb_fail(XLB_ERR_CUDA, "internal: a read-back finished without leaving its words");
            CUDA_OK(cudaStreamSynchronize(c->stream));  // long work, or a failure: let the driver say which
            waited = true;
        }
    std::atomic_thread_fence(std::memory_order_acquire);
    for (int i = 0; i < n; ++i) out[i] = (w[2 * i] & 0xFFFFFFFFull) | (w[2 * i + 1] << 32);
    c->status_code = (unsigned)w[2 * n];
    c->drained = true;
    c->leaving = false;
    c->ms_sync_wait += std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
    c->syncs++;
    trace_note(c, "wait (words)", tr0);
}

// Fails with the status that the last read-back brought, and clears it.
[[noreturn]] inline void fail_with_status(xlb_ctx* c);
// What a kernel reported ends an operation at its next read-back: what such a kernel left (a list that is not
// sorted, counts that do not fit) is nothing to size buffers by or to search in.  (Not with several ranks: the others
// are in the same exchanges, and hear of it when the plan is done.)
inline void stop_on_status(xlb_ctx* c) {
    if (c->status_code && !c->wait_hook) fail_with_status(c);
}
inline void read_words_only(xlb_ctx* c, const void* dptr, int n, unsigned long long* out) {
    if (!publish_ok(c, n)) {
        if (n) CUDA_OK(copy_async(c, c->h_scalar, dptr, (size_t)n * 8, cudaMemcpyDeviceToHost));
        CUDA_OK(copy_async(c, c->h_scalar + READ_WORDS_AT, c->d_status, 8, cudaMemcpyDeviceToHost));
        stream_wait(c);
        for (int i = 0; i < n; ++i) out[i] = c->h_scalar[i];
        c->status_code = (unsigned)c->h_scalar[READ_WORDS_AT];
        c->drained = true;
        return;
    }
    if (++c->read_seq == 0) ++c->read_seq;
    publish_words_k<<<1, 64, 0, c->stream>>>((const unsigned long long*)dptr, n, c->d_status, c->h_scalar_dev + READ_WORDS_AT, c->read_seq);
    CUDA_OK(cudaGetLastError());
    poll_words(c, n, out);
}
// Read `n` 64-bit words from device memory (everything enqueued before has run when this returns).
inline void read_words(xlb_ctx* c, const void* dptr, int n, unsigned long long* out) {
    read_words_only(c, dptr, n, out);
    stop_on_status(c);
}
// After the launch of a kernel that got `p`: its words (by a read-back of their own where it was not asked).
inline void read_published(xlb_ctx* c, const Publish& p, const void* dptr, int n, unsigned long long* out) {
    if (p.dst) poll_words(c, n, out);
    else read_words_only(c, dptr, n, out);
    stop_on_status(c);
}
// The same for a kernel that may be the last of an operation: its status is read when one is asked for.
inline void status_published(xlb_ctx* c, const Publish& p) { c->leaving = p.dst != nullptr; }

// Fails with what a kernel reported, if one did; everything enqueued has run when this returns.
inline void check_dev_status(xlb_ctx* c) {
    if (!c->drained) {
        if (c->leaving) poll_words(c, 0, nullptr);
        else read_words_only(c, nullptr, 0, nullptr);
    }
    if (c->status_code) fail_with_status(c);
}
inline void fail_with_status(xlb_ctx* c) {
    DevStatus s;
    CUDA_OK(copy_async(c, c->h_scalar, c->d_status, sizeof s, cudaMemcpyDeviceToHost));
    stream_wait(c);
    memcpy(&s, c->h_scalar, sizeof s);
    CUDA_OK(set_async(c, c->d_status, 0, sizeof s));
    c->status_code = 0;
    xlb_fail((xlb_status)s.code, "device kernel reported status %u at site %u (detail %llu)", s.code, s.where, s.detail);
}

// The relation handle.  Either representation may be present; both describe the same rows.
//   cols   : column-major, one allocation per column (the ABI's layout);
//   packed : arity <= 2 and 32-bit columns only: one u64 per row, (c0 << 32) | c1 for arity 2,
//            c0 for arity 1, so ascending u64 order is the lexicographic column order.
struct xlb_rel {
    xlb_ctx* ctx = nullptr;
    xlb_schema schema{};
    uint64_t rows = 0;
    mutable Buf cols[XLB_MAX_ARITY];
    mutable Buf packed;
    mutable uint64_t or_bound = ~0ull;  // host-known upper bound of the OR of the packed rows (~0: unknown)
    uint64_t firsts = ~0ull;  // host-known bound of how many different values the first column has (~0: unknown)
    bool canonical = false;
};

inline uint32_t type_width(uint8_t t) {
    switch (t) {
        case XLB_U32: case XLB_I32: case XLB_F32: case XLB_SYMBOL: return 4;
        case XLB_U64: case XLB_I64: case XLB_F64: return 8;
        default: return 1;
    }
}
inline bool type_built(uint8_t t) { return t <= XLB_SYMBOL; }
inline bool type_unsigned(uint8_t t) { return t == XLB_U32 || t == XLB_SYMBOL || t == XLB_U64; }
inline bool rel_packable(const xlb_schema& s) {
    if (s.arity < 1 || s.arity > 2) return false;
    for (uint32_t i = 0; i < s.arity; ++i)
        if (s.types[i] != XLB_U32 && s.types[i] != XLB_SYMBOL) return false;
    return true;
}
