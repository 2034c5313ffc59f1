// Whole frontier fixpoints in one launch.
//
//   r(V) :- e(..) with a column equal to a constant.     r(V) :- r(K), e(K, ..).
//
// Launch by launch such a query was a sweep for the bounds, five kernels for the seed, two per
// iteration, two for the sorted list and a read-back after most of them: 180 us on a graph of 16 K edges
// whose rows fit one SM's reach, 230 us on one of a million.  Here one kernel sweeps, seeds, iterates and
// writes the sorted result; the host reads a few words.  Up to two million rows every iteration streams
// over all of them (they are in the L2), above over those that are still of use.  Where there are more than
// 48 iterations the kernels of many blocks give up, and the frontier loop, which changes over to an
// index, starts from the beginning.
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
    unsigned long long* words;    // [0] rows, [1] iterations, [2] candidates, [3] 1: a fixpoint, 2: not for this kernel, [4] rows streamed over and written (large)
    // many blocks
    unsigned int* sync;           // [0] blocks arrived at the barriers so far, [1] OR of the columns, [2] a block gave up
    unsigned int* marks;          // three bitmaps
    uint64_t* list[2];            // large relations: room for the rows still of use, twice
    DevStatus* st;
};

// One block: bitmaps in shared memory.
__device__ __forceinline__ void frontier_one(const Args& a) {
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

// Arrive at the barrier that `passed` arrivals end, and wait for the others (one thread per block).
__device__ __forceinline__ unsigned grid_arrive_and_wait(const Args& a, unsigned passed) {
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(&a.sync[0]) : "memory");
    unsigned arrived = 0;
    for (unsigned polls = 0;; ++polls) {
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(arrived) : "l"(&a.sync[0]) : "memory");
        if ((int)(arrived - passed) >= 0) return 1;
        if (polls > F_SPIN_LIMIT || *(volatile unsigned*)&a.sync[2]) {
            *(volatile unsigned*)&a.sync[2] = 1;
            set_status(a.st, XLB_ERR_TIMEOUT, 21, passed);
            return 0;
        }
    }
}
// The sorted list off the bitmap that every block holds: a block counts what lies before its stretch of
// the words and writes that stretch.
__device__ __forceinline__ void write_sorted(const unsigned* seen, unsigned words, uint32_t* out, unsigned* sm, unsigned long long* rows) {
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
        for (; m; m &= m - 1) out[at++] = (w << 5) | (__ffs(m) - 1);
        before += count;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) *rows = every;
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
            go_s = grid_arrive_and_wait(a, passed);
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
    write_sorted(seen, words, a.out, sm, a.words);
    if (first == 0) {
        a.words[1] = it;
        a.words[3] = fix ? 1 : (it >= a.max_iterations ? 0 : 2);
    }
}

// ---- large relations: values of up to 20 bits
// One bitmap of the head (128 KB) fits a block's shared memory.  A key is in the frontier once, so a row
// whose key the head holds is done with after this iteration: every block keeps the rows of its own
// stretch of the relation that are still of use in a list of its own (no counter is shared, nobody
// else reads it), and the next iteration streams over those.  What an iteration marks goes to a bitmap
// in global memory, past what the head holds and past a small cache of what the block marked
// lately.  Looked up in the L1 (one line a cycle), the bitmaps and not the stream were what the
// launch-by-launch loop paid for: 16 M edges took it 190 us in six scans and 350 us in all, and take
// this kernel 178 us from launch to end (160 to 190 from process to process; 4 more with the L2 flushed).  Of that, by the clock inside it, 19 the seed, 76 the first stream, 21
// the second, 4 each iteration after; the rest is the launch, the barriers and the list written off.  (Looking
// at what all blocks have marked before sending an atomic evens the blocks out but costs as much.)
constexpr int FL_BITS = 20, FL_CACHE = 1 << 14, FL_ITERATIONS = 48;
constexpr unsigned FL_WORDS = 1u << (FL_BITS - 5);
constexpr size_t FL_SMEM = FL_WORDS * 4 + FL_CACHE * 4;

__global__ void __launch_bounds__(F_THREADS, 1) frontier_large_k(const __grid_constant__ Args a) {
    extern __shared__ __align__(16) unsigned bm[];
    __shared__ unsigned go_s, kept_s, used_s;
    __shared__ unsigned sm[33];
    unsigned *seen = bm, *cache = bm + FL_WORDS;
    const unsigned lane = lane_id();
    unsigned passed = 0;
    auto barrier = [&]() {
        __syncthreads();
        if (threadIdx.x == 0) {
            passed += gridDim.x;
            go_s = grid_arrive_and_wait(a, passed);
        }
        __syncthreads();
        return go_s != 0;
    };
    for (unsigned w = threadIdx.x; w < FL_WORDS; w += F_THREADS) seen[w] = 0;
    for (unsigned w = threadIdx.x; w < FL_CACHE; w += F_THREADS) cache[w] = 0xFFFFFFFFu;
    __syncthreads();
    bool outside = false;
    auto mark = [&](unsigned* to, uint32_t v) {
        if (v >> FL_BITS) {
            outside = true;
            return;
        }
        if ((seen[v >> 5] >> (v & 31)) & 1u) return;
        if (cache[v & (FL_CACHE - 1)] == v) return;
        cache[v & (FL_CACHE - 1)] = v;
        atomicOr(&to[v >> 5], 1u << (v & 31));
    };
    // Four rows a thread, those with a bit in `keep` appended to the block's list (all threads of the warp)
    auto append = [&](uint64_t* list, const uint64_t (&row)[4], unsigned keep) {
        unsigned b[4], total = 0, at = 0;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            b[j] = __ballot_sync(FULL, (keep >> j) & 1u);
            total += __popc(b[j]);
        }
        if (!total) return;
        if (lane == 0) at = atomicAdd(&kept_s, total);
        at = __shfl_sync(FULL, at, 0);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            if ((keep >> j) & 1u) list[at + __popc(b[j] & lanemask_lt())] = row[j];
            at += __popc(b[j]);
        }
    };
    // this block's stretch of the relation (starts are multiples of four rows: 16-byte loads)
    const uint64_t stretch = ((a.n + gridDim.x - 1) / gridDim.x + 3) & ~3ull;
    const uint64_t lo = min(blockIdx.x * stretch, a.n), hi = min(lo + stretch, a.n);
    const uint64_t steps = (hi - lo + 4 * F_THREADS - 1) / (4 * F_THREADS);
    unsigned long long cand = 0, streamed = 0;
    for (int q = 0; q < a.seeds; ++q) {
        const uint32_t* f = a.seed[q].filter;
        const uint32_t constant = a.seed[q].constant;
        constexpr int V = 4;
        for (uint64_t i0 = lo + 4 * threadIdx.x; i0 < hi; i0 += V * 4 * F_THREADS) {
            uint4 x[V];
#pragma unroll
            for (int u = 0; u < V; ++u) {
                const uint64_t i = i0 + u * (4 * F_THREADS);
                if (i + 4 <= hi) x[u] = *reinterpret_cast<const uint4*>(f + i);
                else {
                    x[u].x = i < hi ? f[i] : ~constant, x[u].y = i + 1 < hi ? f[i + 1] : ~constant;
                    x[u].z = i + 2 < hi ? f[i + 2] : ~constant, x[u].w = ~constant;
                }
            }
#pragma unroll
            for (int u = 0; u < V; ++u) {
                if (x[u].x != constant && x[u].y != constant && x[u].z != constant && x[u].w != constant) continue;
                const uint64_t i = i0 + u * (4 * F_THREADS);
                const uint32_t k[4] = {x[u].x, x[u].y, x[u].z, x[u].w};
                for (int j = 0; j < 4; ++j)
                    if (k[j] == constant) {
                        mark(a.marks, a.seed[q].take[i + j]);
                        ++cand;
                    }
            }
        }
        streamed += (hi - lo) / 2;
    }
    uint64_t it = 0;
    bool fix = false;
    const uint64_t limit = a.max_iterations < FL_ITERATIONS ? a.max_iterations : FL_ITERATIONS;
    unsigned turn = 0, rows = 0;
    bool many_used = true;
    int at_list = -1;  // which list holds the rows (-1: the relation itself)
    for (;;) {
        if (outside) *(volatile unsigned*)&a.sync[1] = 1;
        if (!barrier()) return;
        if (*(volatile unsigned*)&a.sync[1]) {
            if (blockIdx.x == 0 && threadIdx.x == 0) a.words[3] = 2;
            return;
        }
        const unsigned* marks = a.marks + turn * FL_WORDS;
        turn = turn == 2 ? 0 : turn + 1;
        unsigned *to = a.marks + turn * FL_WORDS, *clear = a.marks + (turn == 2 ? 0 : turn + 1) * FL_WORDS;
        unsigned fresh = 0;
        for (unsigned w = 4 * threadIdx.x; w < FL_WORDS; w += 4 * F_THREADS) {
            const uint4 m = __ldcg(reinterpret_cast<const uint4*>(marks + w));
            const unsigned any = m.x | m.y | m.z | m.w;
            if (any) {
                uint4 s = *reinterpret_cast<uint4*>(seen + w);
                s.x |= m.x, s.y |= m.y, s.z |= m.z, s.w |= m.w;
                *reinterpret_cast<uint4*>(seen + w) = s;
            }
            fresh |= any;
        }
        if (threadIdx.x == 0) kept_s = used_s = 0;
        const int any = __syncthreads_or(fresh != 0);
        if (it > 0 && !any) {
            fix = true;
            break;
        }
        if (it == limit) break;
        for (unsigned w = blockIdx.x * F_THREADS + threadIdx.x; w < FL_WORDS; w += gridDim.x * F_THREADS) clear[w] = 0;  // (read by everybody before the barrier just passed)
        if (at_list < 0) {
            // (the next rows are loaded while these are looked up)
            auto load = [&](uint64_t s, uint4& x, uint4& y) {
                const uint64_t i = lo + s * (4 * F_THREADS) + 4 * threadIdx.x;
                if (i + 4 <= hi) {
                    x = *reinterpret_cast<const uint4*>(a.key + i);
                    y = *reinterpret_cast<const uint4*>(a.value + i);
                } else {
                    x.x = i < hi ? a.key[i] : 0xFFFFFFFFu, y.x = i < hi ? a.value[i] : 0u;
                    x.y = i + 1 < hi ? a.key[i + 1] : 0xFFFFFFFFu, y.y = i + 1 < hi ? a.value[i + 1] : 0u;
                    x.z = i + 2 < hi ? a.key[i + 2] : 0xFFFFFFFFu, y.z = i + 2 < hi ? a.value[i + 2] : 0u;
                    x.w = 0xFFFFFFFFu, y.w = 0u;
                }
            };
            uint4 x, y, nx, ny;
            load(0, x, y);
            for (uint64_t s = 0; s < steps; ++s, x = nx, y = ny) {
                load(s + 1, nx, ny);
                const uint32_t k[4] = {x.x, x.y, x.z, x.w}, v[4] = {y.x, y.y, y.z, y.w};
                uint64_t row[4];
                unsigned keep = 0;
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    row[j] = ((uint64_t)k[j] << 32) | v[j];
                    if (k[j] >> FL_BITS) continue;  // never derived, or the relation is not for this kernel
                    if ((seen[k[j] >> 5] >> (k[j] & 31)) & 1u) {
                        ++cand;
                        mark(to, v[j]);
                    } else keep |= 1u << j;
                }
                append(a.list[0] + lo, row, keep);
            }
            streamed += hi - lo;
            __syncthreads();
            rows = kept_s;
            streamed += rows;
            at_list = 0;
        } else {
            // Where the last iteration used up an eighth of the rows the rest moves on to the other list;
            // else the rows used now are struck out where they are (a long path uses one an iteration).
            uint64_t* from = a.list[at_list] + lo;
            const bool move = many_used;
            unsigned mine = 0;
            for (unsigned base = 0; base < rows; base += 4 * F_THREADS) {
                uint64_t row[4];
                unsigned keep = 0;
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const unsigned i = base + j * F_THREADS + threadIdx.x;
                    row[j] = i < rows ? from[i] : ~0ull;
                }
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const uint32_t k = (uint32_t)(row[j] >> 32);
                    if (k == 0xFFFFFFFFu) continue;  // past the end, or struck out
                    if ((seen[k >> 5] >> (k & 31)) & 1u) {
                        ++mine;
                        mark(to, (uint32_t)row[j]);
                        if (!move) from[base + j * F_THREADS + threadIdx.x] = ~0ull;
                    } else keep |= 1u << j;
                }
                if (move) append(a.list[at_list ^ 1] + lo, row, keep);
            }
            cand += mine;
            mine = __reduce_add_sync(FULL, mine);
            if (lane == 0 && mine) atomicAdd(&used_s, mine);
            __syncthreads();
            streamed += rows;
            many_used = used_s * 8 >= rows;
            if (move) {
                rows = kept_s;
                streamed += rows;
                at_list ^= 1;
            }
        }
        __syncthreads();
        ++it;
    }
#pragma unroll
    for (int d = 16; d; d >>= 1) cand += __shfl_xor_sync(FULL, cand, d);
    if (lane == 0 && cand) atomicAdd(&a.words[2], cand);
    if (threadIdx.x == 0) atomicAdd(&a.words[4], streamed);
    write_sorted(seen, FL_WORDS, a.out, sm, a.words);
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        a.words[1] = it;
        a.words[3] = fix ? 1 : (it >= a.max_iterations ? 0 : 2);
    }
}

__global__ void __launch_bounds__(F_THREADS, 1) frontier_one_k(const __grid_constant__ Args a, const Publish pub) {
    frontier_one(a);
    publish_now(pub);
}

}  // namespace

bool ops_frontier_whole(xlb_ctx* c, const xlb_rel* rel, int key_col, int value_col, const std::vector<FrontierConst>& seeds, uint64_t max_iterations, FrontierWhole* out) {
    const uint64_t n = rel->rows;
    if (n == 0 || n >= (1ull << 32) || seeds.size() > FRONTIER_SEEDS || !rel->cols[0] || !rel->cols[1]) return false;
    const bool one = n <= F1_ROWS, large = n > FM_ROWS;
    if (one) max_iterations = std::min<uint64_t>(max_iterations, 1u << 17);
    if (large && ((((uintptr_t)rel->cols[0]->p | (uintptr_t)rel->cols[1]->p) & 15) != 0 || (c->budget && c->allocated + 18 * n > c->budget))) return false;
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
    const uint64_t most = std::min<uint64_t>(n, 1ull << (large ? FL_BITS : one ? F1_BITS : FM_BITS));  // values that can come out
    Buf values = make_buf(c, most * 4);
    a.out = values->as<uint32_t>();
    a.st = c->d_status;
    const uint64_t bitmap = 1ull << ((large ? FL_BITS : FM_BITS) - 3);
    Buf work = make_buf(c, 64 + (one ? 0 : 32 + 3 * bitmap)), lists[2];
    a.words = work->as<unsigned long long>();
    const char* name = large ? "scan_join_mark" : "dense_mark";
    const unsigned grid = one ? 1u : (unsigned)std::min<uint64_t>({(uint64_t)c->sm_count, (n + 4 * F_THREADS - 1) / (4 * F_THREADS)});
    Publish pub;
    prof_begin(c, name, large ? 0 : n * 8ull);
    if (one) {
        const int smem = 3 << (F1_BITS - 3);
        if (!c->frontier_attr_set) CUDA_OK(cudaFuncSetAttribute(frontier_one_k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
        c->frontier_attr_set = true;
        pub = publish_by(c, grid, work->p, 5);
        frontier_one_k<<<grid, F_THREADS, smem, c->stream>>>(a, pub);
    } else {
        a.sync = (unsigned*)((char*)work->p + 64);
        a.marks = a.sync + 8;
        CUDA_OK(set_async(c, work->p, 0, 96 + 2 * bitmap));  // (the third is cleared on the way)
        const int smem = large ? (int)FL_SMEM : 2 << (FM_BITS - 3);
        const void* kernel = large ? (const void*)frontier_large_k : (const void*)frontier_many_k;
        bool& set = large ? c->frontier_large_attr_set : c->frontier_many_attr_set;
        if (!set) CUDA_OK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
        set = true;
        if (large)
            for (int k = 0; k < 2; ++k) {
                lists[k] = make_buf(c, n * 8);
                a.list[k] = lists[k]->as<uint64_t>();
            }
        void* args[] = {&a};  // (the words left by these two kernels themselves: 80 -> 89 us at 80 K rows)
        CUDA_OK(cudaLaunchCooperativeKernel(kernel, dim3(grid), dim3(F_THREADS), args, smem, c->stream));
    }
    check_launch(c, name);
    unsigned long long w[5];
    read_published(c, pub, work->p, 5, w);
    if (large) prof_add_bytes(c, name, w[4] * 8ull);
    if (w[3] == 2 || (w[3] == 0 && one && max_iterations == 1u << 17)) return false;
    out->rows = w[0];
    out->iterations = w[1];
    out->candidates = w[2];
    out->fix = w[3] == 1;
    out->values = values;
    if (most > (1u << 16) && w[0] * 2 < most) {  // give the large buffer back
        out->values = make_buf(c, w[0] * 4);
        if (w[0]) CUDA_OK(copy_async(c, out->values->p, values->p, w[0] * 4, cudaMemcpyDeviceToDevice));
    }
    return true;
}
