// Results of some size, fetched into page-locked host memory.
//
// What bounds a large result is the bus (55 GB/s against the 6.5 TB/s at which the device wrote it), and
// the first column of a sorted relation is runs of equal values: it crosses the bus as (first row,
// value) pairs and is written out by host threads while the other columns are copied.  Two columns of 26.8 M
// rows took 4.1 ms, now 2.0; of 3.9 M rows 570 us, now 330; of 2.2 M rows 320, now 190.
//   One core writes 19 GB/s around the cache, four 73 (host of a B200, 16 cores).  Four are enough for a column
// to be there before the next one; more only slow the copies beside them (four 2.0 ms, six 2.1, eight 2.2),
// and ordinary stores, which read what they overwrite, took 2.6.
//   The column is read twice on the device (heads counted per tile, then written in order), while the copy of
// the next column runs on a stream of its own.
#include <algorithm>
#include <optional>

#include "xlb_common.cuh"
#include "xlb_fill.h"
#include "xlb_host.h"
#include "xlb_kernels.cuh"
#include "xlb_ops.h"

using namespace xk;

namespace {

constexpr uint64_t RUNS_TILE = 4096;                     // rows a block looks at, 512 a warp
constexpr uint64_t RUNS_MIN_BYTES = 6ull << 20;          // below, the 60 us until the runs are there and 11 us a thread are hardly made up for (4 MB: 73 us of bus)
constexpr unsigned RUNS_THREADS_MAX = 4, RUNS_CORES_MIN = 4;
constexpr uint64_t RUNS_RUN_BYTES = 400;                 // a run has to have on average: it is 10 to 15 ns of its own, whatever its rows' width (16 384 runs of 4-byte rows: of 96 rows 244 us copied, 249 to 269 as runs; of 104 263, 237; of 112 281, 233; of 128 318, 255; 16 000 of 8-byte rows: of 50 rows 460, 315; of 80 526, 315)

template <class T>
__device__ __forceinline__ unsigned warp_heads(const T* __restrict__ col, uint64_t n, uint64_t base, int k) {
    const uint64_t i = base + k * 32 + lane_id();
    return __ballot_sync(FULL, i < n && (i == 0 || col[i] != col[i - 1]));
}
// counts[t]: runs that begin in tile t
template <class T>
__global__ void __launch_bounds__(BLOCK) runs_count_k(const T* __restrict__ col, uint64_t n, unsigned* __restrict__ counts) {
    __shared__ unsigned warp_s[BLOCK / 32];
    const uint64_t base = blockIdx.x * RUNS_TILE + (threadIdx.x >> 5) * 512;
    unsigned c = 0;
#pragma unroll
    for (int k = 0; k < 16; ++k) c += __popc(warp_heads(col, n, base, k));
    if (lane_id() == 0) warp_s[threadIdx.x >> 5] = c;
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned total = 0;
        for (int w = 0; w < BLOCK / 32; ++w) total += warp_s[w];
        counts[blockIdx.x] = total;
    }
}
// The runs in order, into mapped host memory; none when there are more than `cap`.  `total` gets their number.
template <class T>
__global__ void __launch_bounds__(BLOCK) runs_write_k(const T* __restrict__ col, uint64_t n, const unsigned* __restrict__ counts, Run<T>* out, uint64_t cap, unsigned long long* total) {
    __shared__ unsigned long long before_s[BLOCK / 32], all_s[BLOCK / 32];
    __shared__ unsigned warp_s[BLOCK / 32];
    const unsigned lane = lane_id(), warp = threadIdx.x >> 5, mine = counts[blockIdx.x];
    if (!mine && blockIdx.x) return;
    unsigned long long before = 0, all = 0;
    for (unsigned t = threadIdx.x; t < gridDim.x; t += BLOCK) {
        const unsigned v = counts[t];
        all += v;
        if (t < blockIdx.x) before += v;
    }
#pragma unroll
    for (int d = 16; d; d >>= 1) {
        before += __shfl_xor_sync(FULL, before, d);
        all += __shfl_xor_sync(FULL, all, d);
    }
    const uint64_t base = blockIdx.x * RUNS_TILE + warp * 512;
    unsigned heads[16], c = 0;
#pragma unroll
    for (int k = 0; k < 16; ++k) {
        heads[k] = warp_heads(col, n, base, k);
        c += __popc(heads[k]);
    }
    if (lane == 0) {
        before_s[warp] = before;
        all_s[warp] = all;
        warp_s[warp] = c;
    }
    __syncthreads();
    before = all = 0;
    for (int w = 0; w < BLOCK / 32; ++w) {
        before += before_s[w];
        all += all_s[w];
        if (w < (int)warp) before += warp_s[w];
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) *total = all;
    if (all > cap) return;
#pragma unroll
    for (int k = 0; k < 16; ++k) {
        const uint64_t i = base + k * 32 + lane;
        if ((heads[k] >> lane) & 1u) out[before + __popc(heads[k] & lanemask_lt())] = {(T)i, col[i]};
        before += __popc(heads[k]);
    }
}

// Copies that run beside the context's stream, behind what is on it now.  However the operation ends, they are
// over before it returns: the memory they write is the caller's.
struct SideCopies {
    xlb_ctx* c;
    explicit SideCopies(xlb_ctx* ctx) : c(ctx) {
        if (!c->copy_stream) CUDA_OK(cudaStreamCreateWithFlags(&c->copy_stream, cudaStreamNonBlocking));
        if (!c->copy_behind) CUDA_OK(cudaEventCreateWithFlags(&c->copy_behind, cudaEventDisableTiming));
        CUDA_OK(cudaEventRecord(c->copy_behind, c->stream));
        CUDA_OK(cudaStreamWaitEvent(c->copy_stream, c->copy_behind, 0));
    }
    void add(void* to, const void* from, uint64_t bytes) { CUDA_OK(cudaMemcpyAsync(to, from, bytes, cudaMemcpyDeviceToHost, c->copy_stream)); }
    void wait() { CUDA_OK(cudaStreamSynchronize(c->copy_stream)); }
    ~SideCopies() { CUDA_QUIET(cudaStreamSynchronize(c->copy_stream)); }
};

bool page_locked(const void* p) {
    cudaPointerAttributes a{};
    return cuda_take(cudaPointerGetAttributes(&a, p)) == cudaSuccess && a.type == cudaMemoryTypeHost;
}

template <class T>
constexpr uint64_t runs_room() { return (STAGE_BYTES - 16) / sizeof(Run<T>); }
// False: what it needs is not to be had (device memory within the budget, the staging, a stream); nothing was done.
template <class T>
bool fetch_with_runs(xlb_ctx* c, const xlb_rel* r, void* const* cols, uint64_t n, unsigned threads) {
    const uint64_t tiles = (n + RUNS_TILE - 1) / RUNS_TILE, cap = runs_room<T>();
    char* stage;
    Buf counts;
    std::optional<SideCopies> side;
    try {
        stage = stage_buffer(c);
        counts = make_buf(c, tiles * 4);
        side.emplace(c);
    } catch (const XlbError&) {
        return false;
    }
    unsigned long long* total = reinterpret_cast<unsigned long long*>(stage);
    const Run<T>* runs = reinterpret_cast<const Run<T>*>(stage + 16);
    const T* col = r->cols[0]->as<T>();
    prof_begin(c, "to_host", n * sizeof(T));
    runs_count_k<T><<<(unsigned)tiles, BLOCK, 0, c->stream>>>(col, n, counts->as<unsigned>());
    check_launch(c, "to_host");
    prof_begin(c, "to_host", n * sizeof(T));
    runs_write_k<T><<<(unsigned)tiles, BLOCK, 0, c->stream>>>(col, n, counts->as<unsigned>(), reinterpret_cast<Run<T>*>(c->h_stage_dev + 16), cap, reinterpret_cast<unsigned long long*>(c->h_stage_dev));
    check_launch(c, "to_host");
    for (uint32_t i = 1; i < r->schema.arity; ++i) side->add(cols[i], r->cols[i]->p, n * type_width(r->schema.types[i]));
    {
        Filler<T> filler(threads);
        stream_wait(c);
        if (*total <= cap) filler.fill(static_cast<T*>(cols[0]), runs, *total, n);
        else side->add(cols[0], col, n * sizeof(T));  // (more values than were announced)
    }
    side->wait();
    return true;
}

}  // namespace

void ops_fetch_columns(xlb_ctx* c, const xlb_rel* r, void* const* cols, uint64_t n) {
    ops_rel_columns(c, r);
    const uint32_t arity = r->schema.arity, width = type_width(r->schema.types[0]);
    // Only of a set, which is in order, whose first values are known to be few (looking for runs where there are none took
    // 11 us of a sort's 1500 and 15 of 790 of a union over 2^18 first values); not with several ranks (whose waits watch the
    // communicator), and not into memory that the driver copies to by itself: such a copy does not run beside anything.
    const uint64_t bound = rel_packable(r->schema) && r->or_bound != ~0ull ? (r->or_bound >> 32) + 1 : ~0ull, firsts = std::min(bound, r->firsts);
    if (r->canonical && arity >= 2 && firsts <= std::min(n * width / RUNS_RUN_BYTES, width == 4 ? runs_room<uint32_t>() : runs_room<unsigned long long>()) && width >= 4 && n * width >= RUNS_MIN_BYTES &&
        n < 1ull << 32 && !c->wait_hook) {
        const unsigned cores = host_pool_cores();
        bool locked = cores >= RUNS_CORES_MIN;
        for (uint32_t i = 0; i < arity; ++i) locked = locked && page_locked(cols[i]) && (uintptr_t)cols[i] % width == 0;
        const unsigned threads = std::min(RUNS_THREADS_MAX, cores / 2);  // (two or more)
        if (locked && (width == 4 ? fetch_with_runs<uint32_t>(c, r, cols, n, threads) : fetch_with_runs<unsigned long long>(c, r, cols, n, threads))) return;
    }
    for (uint32_t i = 0; i < arity; ++i) CUDA_OK(copy_async(c, cols[i], r->cols[i]->p, n * type_width(r->schema.types[i]), cudaMemcpyDeviceToHost));
    CUDA_OK(cudaStreamSynchronize(c->stream));
}
