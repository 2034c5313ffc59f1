// Whole frontier fixpoints in one launch, for relations of up to two million rows.
//
//   r(V) :- e(..) with a column equal to a constant.     r(V) :- r(K), e(K, ..).
//
// Launch by launch such a query was a sweep for the bounds, five kernels for the seed, two per
// iteration, two for the sorted list and a read-back after most of them: 180 us on a graph of 16 K edges
// whose rows fit one SM's reach, 230 us on one of a million.  Here one kernel sweeps, seeds, iterates and
// writes the sorted result; the host reads four words.  Every iteration streams over all rows
// (they are in the L2), so it is for few iterations or few rows: beyond FM_ITERATIONS the many-block
// kernel gives up, and the frontier loop, which drops rows that are of no more use and changes over
// to an index, starts from the beginning.
#include <algorithm>

#include "xlb_kernels.cuh"
#include "xlb_ops.h"

using namespace xk;

namespace {

constexpr int F_THREADS = 1024;
constexpr uint64_t F1_ROWS = 1ull << 15;       // up to here one block
constexpr int F1_BITS = 19;                    // three bitmaps of 64 KB in shared memory
constexpr uint64_t FM_ROWS = 1ull << 21;
constexpr int FM_BITS = 19, FM_ITERATIONS = 48;  // two bitmaps of 64 KB in every block's shared memory
constexpr unsigned F_SPIN_LIMIT = 1u << 24;

struct Args {
    const uint32_t *key, *value;  // join column, and the column the head takes
    const uint32_t *c0, *c1;      // both columns, for the bound
    uint64_t n;
    FrontierSeed seed[FRONTIER_SEEDS];
    int seeds;
    uint64_t max_iterations;
    uint32_t* out;                // room for n values
    unsigned long long* words;    // [0] rows, [1] iterations, [2] candidates, [3] 1: a fixpoint, 2: not for this kernel
    // many blocks
    unsigned int* sync;           // [0] blocks arrived at the barriers so far, [1] OR of the columns, [2] a block gave up
    unsigned int* marks;          // three bitmaps
    DevStatus* st;
};

// One block: bitmaps in shared memory.
__global__ void __launch_bounds__(F_THREADS, 1) frontier_one_k(const __grid_constant__ Args a) {
    extern __shared__ unsigned bm[];
    __shared__ unsigned or_s, fresh_s[3], cand_s;
    __shared__ unsigned sm[33];
    const unsigned n = (unsigned)a.n;
    if (threadIdx.x == 0) {
        or_s = 0;
        fresh_s[0] = fresh_s[1] = fresh_s[2] = 0;
        cand_s = 0;
    }
    __syncthreads();
    unsigned o = 0;
    for (unsigned i = threadIdx.x; i < n; i += F_THREADS) o |= a.c0[i] | a.c1[i];
    o = __reduce_or_sync(FULL, o);
    if (lane_id() == 0 && o) atomicOr(&or_s, o);
    __syncthreads();
    const int bits = or_s ? 32 - __clz(or_s) : 1;
    if (bits > F1_BITS) {
        if (threadIdx.x == 0) a.words[3] = 2;
        return;
    }
    const unsigned words = ((1u << bits) + 31) / 32;
    unsigned *seen = bm, *front = bm + words, *marks = front + words;
    for (unsigned w = threadIdx.x; w < 3 * words; w += F_THREADS) bm[w] = 0;
    __syncthreads();
    unsigned cand = 0;
    for (int q = 0; q < a.seeds; ++q)
        for (unsigned i = threadIdx.x; i < n; i += F_THREADS)
            if (a.seed[q].filter[i] == a.seed[q].constant) {
                const uint32_t v = a.seed[q].take[i];
                atomicOr(&front[v >> 5], 1u << (v & 31));
                ++cand;
            }
    __syncthreads();
    for (unsigned w = threadIdx.x; w < words; w += F_THREADS) seen[w] = front[w];
    __syncthreads();
    uint64_t it = 0;
    bool fix = false;
    for (unsigned turn = 0; it < a.max_iterations && !fix; turn = turn == 2 ? 0 : turn + 1) {
        if (threadIdx.x == 0) fresh_s[turn == 2 ? 0 : turn + 1] = 0;  // (read last two barriers ago)
        for (unsigned i = threadIdx.x; i < n; i += F_THREADS) {
            const uint32_t k = a.key[i];
            if (!((front[k >> 5] >> (k & 31)) & 1u)) continue;
            ++cand;
            const uint32_t v = a.value[i];
            const unsigned bit = 1u << (v & 31);
            if (!((seen[v >> 5] | marks[v >> 5]) & bit)) atomicOr(&marks[v >> 5], bit);
        }
        __syncthreads();
        unsigned fresh = 0;
        for (unsigned w = threadIdx.x; w < words; w += F_THREADS) {
            const unsigned m = marks[w];
            front[w] = m;
            if (m) {
                seen[w] |= m;
                marks[w] = 0;
                fresh = 1;
            }
        }
        if (fresh) fresh_s[turn] = 1;
        __syncthreads();
        ++it;
        fix = fresh_s[turn] == 0;
    }
    cand = __reduce_add_sync(FULL, cand);
    if (lane_id() == 0) atomicAdd(&cand_s, cand);  // (a key is in the frontier once: every row counts once, and once as a seed)
    const unsigned per = (words + F_THREADS - 1) / F_THREADS, lo = min(threadIdx.x * per, words), hi = min(lo + per, words);
    unsigned rows = 0, total;
    for (unsigned w = lo; w < hi; ++w) rows += __popc(seen[w]);
    unsigned pos = block_exclusive_scan<unsigned>(rows, &total, sm);
    for (unsigned w = lo; w < hi; ++w)
        for (unsigned m = seen[w]; m; m &= m - 1) a.out[pos++] = (w << 5) | (__ffs(m) - 1);
    if (threadIdx.x == 0) {
        a.words[0] = total;
        a.words[1] = it;
        a.words[2] = cand_s;
        a.words[3] = fix ? 1 : 0;
    }
}

// Many blocks, resident together.  Every block keeps the whole head and the frontier as bitmaps in its
// shared memory, marks a value there first and in global memory only if it was not marked there yet
// (a byte or bit per value in global memory alone made a hub's neighbours a queue in the L2: 100 us of
// the 150 an evaluation over a million rows took), and reads what all blocks marked after the
// iteration's one barrier.
__global__ void __launch_bounds__(F_THREADS, 1) frontier_many_k(const __grid_constant__ Args a) {
    extern __shared__ unsigned bm[];
    __shared__ unsigned go_s, or_s;
    __shared__ unsigned sm[33];
    unsigned passed = 0;
    auto barrier = [&]() {
        __syncthreads();
        if (threadIdx.x == 0) {
            passed += gridDim.x;
            go_s = 1;
            asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(&a.sync[0]) : "memory");
            unsigned arrived = 0;
            for (unsigned polls = 0;; ++polls) {
                asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(arrived) : "l"(&a.sync[0]) : "memory");
                if ((int)(arrived - passed) >= 0) break;
                if (polls > F_SPIN_LIMIT || *(volatile unsigned*)&a.sync[2]) {
                    *(volatile unsigned*)&a.sync[2] = 1;
                    set_status(a.st, XLB_ERR_TIMEOUT, 21, passed);
                    go_s = 0;
                    break;
                }
            }
        }
        __syncthreads();
        return go_s != 0;
    };
    const uint64_t first = (uint64_t)blockIdx.x * F_THREADS + threadIdx.x, step = (uint64_t)gridDim.x * F_THREADS;
    if (threadIdx.x == 0) or_s = 0;
    __syncthreads();
    unsigned o = 0;
    for (uint64_t i = first; i < a.n; i += step) o |= a.c0[i] | a.c1[i];
    o = __reduce_or_sync(FULL, o);
    if (lane_id() == 0 && o) atomicOr(&or_s, o);
    __syncthreads();
    if (threadIdx.x == 0 && (*(volatile unsigned*)&a.sync[1] & or_s) != or_s) atomicOr(&a.sync[1], or_s);
    if (!barrier()) return;
    const unsigned all = *(volatile unsigned*)&a.sync[1];
    const int bits = all ? 32 - __clz(all) : 1;
    if (bits > FM_BITS) {
        if (first == 0) a.words[3] = 2;
        return;
    }
    const unsigned words = ((1u << bits) + 31) / 32;
    unsigned *seen = bm, *front = bm + words;
    for (unsigned w = threadIdx.x; w < 2 * words; w += F_THREADS) bm[w] = 0;
    __syncthreads();
    auto mark = [&](unsigned* to, uint32_t v) {
        const unsigned bit = 1u << (v & 31);
        if (!(seen[v >> 5] & bit) && !(atomicOr(&seen[v >> 5], bit) & bit)) atomicOr(&to[v >> 5], bit);
    };
    unsigned long long cand = 0;
    for (int q = 0; q < a.seeds; ++q)
        for (uint64_t i = first; i < a.n; i += step)
            if (a.seed[q].filter[i] == a.seed[q].constant) {
                mark(a.marks, a.seed[q].take[i]);
                ++cand;
            }
    uint64_t it = 0;
    bool fix = false;
    const uint64_t limit = a.max_iterations < FM_ITERATIONS ? a.max_iterations : FM_ITERATIONS;
    unsigned turn = 0;  // marks are kept in three bitmaps used in turn: one is read, one written, one cleared
    for (;;) {
        if (!barrier()) return;
        unsigned fresh = 0;
        const unsigned* marks = a.marks + turn * (1u << (FM_BITS - 5));
        turn = turn == 2 ? 0 : turn + 1;
        unsigned *to = a.marks + turn * (1u << (FM_BITS - 5)), *clear = a.marks + (turn == 2 ? 0 : turn + 1) * (1u << (FM_BITS - 5));
        for (unsigned w = threadIdx.x; w < words; w += F_THREADS) {
            const unsigned m = __ldcg(&marks[w]);
            front[w] = m;
            seen[w] |= m;
            fresh |= m;
        }
        const int any = __syncthreads_or(fresh != 0);
        if (it > 0 && !any) {
            fix = true;
            break;
        }
        if (it == limit) break;
        for (unsigned w = (unsigned)first; w < words; w += (unsigned)step) clear[w] = 0;  // (read by everybody before the barrier just passed)
        constexpr int V = 4;
        for (uint64_t i0 = first; i0 < a.n; i0 += V * step) {
            uint32_t k[V], v[V];
#pragma unroll
            for (int u = 0; u < V; ++u) {
                const uint64_t i = min(i0 + u * step, a.n - 1);
                k[u] = a.key[i];
                v[u] = a.value[i];
            }
#pragma unroll
            for (int u = 0; u < V; ++u) {
                if (i0 + u * step >= a.n || !((front[k[u] >> 5] >> (k[u] & 31)) & 1u)) continue;
                ++cand;
                mark(to, v[u]);
            }
        }
        ++it;
    }
#pragma unroll
    for (int d = 16; d; d >>= 1) cand += __shfl_xor_sync(FULL, cand, d);
    if (lane_id() == 0 && cand) atomicAdd(&a.words[2], cand);
    // the sorted list: every block knows the whole head, counts what lies before its stretch and writes that
    const unsigned stretch = (words + gridDim.x - 1) / gridDim.x, lo = min(blockIdx.x * stretch, words), hi = min(lo + stretch, words);
    unsigned before = 0, every = 0;
    for (unsigned w = threadIdx.x; w < words; w += F_THREADS) {
        const unsigned p = __popc(seen[w]);
        every += p;
        if (w < lo) before += p;
    }
    block_exclusive_scan<unsigned>(before, &before, sm);
    block_exclusive_scan<unsigned>(every, &every, sm);
    for (unsigned base = lo; base < hi; base += F_THREADS) {
        const unsigned w = base + threadIdx.x;
        unsigned m = w < hi ? seen[w] : 0, count;
        unsigned at = before + block_exclusive_scan<unsigned>(__popc(m), &count, sm);
        for (; m; m &= m - 1) a.out[at++] = (w << 5) | (__ffs(m) - 1);
        before += count;
    }
    if (first == 0) {
        a.words[0] = every;
        a.words[1] = it;
        a.words[3] = fix ? 1 : (it >= a.max_iterations ? 0 : 2);
    }
}

}  // namespace

bool ops_frontier_whole(xlb_ctx* c, const xlb_rel* rel, int key_col, int value_col, const std::vector<FrontierConst>& seeds, uint64_t max_iterations, FrontierWhole* out) {
    const uint64_t n = rel->rows;
    if (n == 0 || n > FM_ROWS || seeds.size() > FRONTIER_SEEDS || !rel->cols[0] || !rel->cols[1]) return false;
    const bool one = n <= F1_ROWS;
    if (one) max_iterations = std::min<uint64_t>(max_iterations, 1u << 17);
    Args a{};
    a.c0 = rel->cols[0]->as<uint32_t>();
    a.c1 = rel->cols[1]->as<uint32_t>();
    a.key = key_col == 0 ? a.c0 : a.c1;
    a.value = value_col == 0 ? a.c0 : a.c1;
    a.n = n;
    a.seeds = (int)seeds.size();
    for (size_t q = 0; q < seeds.size(); ++q)
        a.seed[q] = FrontierSeed{seeds[q].filter_col == 0 ? a.c0 : a.c1, seeds[q].take_col == 0 ? a.c0 : a.c1, seeds[q].constant};
    a.max_iterations = max_iterations;
    Buf values = make_buf(c, n * 4);
    a.out = values->as<uint32_t>();
    a.st = c->d_status;
    Buf work = make_buf(c, one ? 32 : 64 + (3ull << (FM_BITS - 3)));
    a.words = work->as<unsigned long long>();
    prof_begin(c, "dense_mark", n * 8ull);
    if (one) {
        const int smem = 3 << (F1_BITS - 3);
        if (!c->frontier_attr_set) CUDA_OK(cudaFuncSetAttribute(frontier_one_k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
        c->frontier_attr_set = true;
        frontier_one_k<<<1, F_THREADS, smem, c->stream>>>(a);
    } else {
        a.sync = (unsigned*)((char*)work->p + 32);
        a.marks = a.sync + 8;
        CUDA_OK(set_async(c, work->p, 0, 64 + (2ull << (FM_BITS - 3))));  // (the third is cleared on the way)
        const int smem = 2 << (FM_BITS - 3);
        if (!c->frontier_many_attr_set) CUDA_OK(cudaFuncSetAttribute(frontier_many_k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
        c->frontier_many_attr_set = true;
        const unsigned grid = (unsigned)std::min<uint64_t>({(uint64_t)c->sm_count, (n + 4 * F_THREADS - 1) / (4 * F_THREADS)});
        void* args[] = {&a};
        CUDA_OK(cudaLaunchCooperativeKernel((const void*)frontier_many_k, dim3(grid), dim3(F_THREADS), args, smem, c->stream));
    }
    check_launch(c, "dense_mark");
    unsigned long long w[4];
    read_words(c, work->p, 4, w);
    if (c->status_code) check_dev_status(c);
    if (w[3] == 2 || (w[3] == 0 && one && max_iterations == 1u << 17)) return false;
    out->rows = w[0];
    out->iterations = w[1];
    out->candidates = w[2];
    out->fix = w[3] == 1;
    out->values = values;
    if (n > (1u << 16) && w[0] * 2 < n) {  // give the large buffer back
        out->values = make_buf(c, w[0] * 4);
        if (w[0]) CUDA_OK(copy_async(c, out->values->p, values->p, w[0] * 4, cudaMemcpyDeviceToDevice));
    }
    return true;
}
