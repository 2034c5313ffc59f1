// The delta loop: a recursive component whose rules join one recursive atom with stored relations
// (closure, same generation, copies along assignments), evaluated to its fixpoint by one kernel.
//
// Evaluated launch by launch, an iteration of such a component was a probe, two prefix-sum kernels,
// a marking expansion, a count, an emission and a read-back of the row count: 47 us on a chain of
// 1500 nodes, whose iterations hold next to nothing, and as many passes over bitmaps and offset
// arrays where they hold much.  Here a candidate is new exactly when the atomic OR that sets its bit in the
// head's bitmap finds it clear; it then goes straight to the log of derived tuples, whose tail is the
// next iteration's delta.  Blocks stay resident (one per SM) and meet at a grid barrier between
// iterations; while an iteration is small, block 0 runs on alone and the others wait.
#include <algorithm>

#include "xlb_kernels.cuh"
#include "xlb_ops.h"

using namespace xk;

namespace {

constexpr int DL_THREADS = 1024, DL_WARPS = DL_THREADS / 32;
constexpr int DL_UNROLL = 4, DL_STEP = 32 * DL_UNROLL;   // outputs a warp has in flight
constexpr int DL_STAGE = 256;                            // new tuples a warp collects before it reserves room in the log
constexpr unsigned DL_HEAVY = 1024;                      // a row with more outputs than this is shared by a block ...
constexpr unsigned DL_PIECE = 16384;                     // ... in pieces of this many outputs
constexpr unsigned DL_HEAVY_MAX = 1u << 16;              // pieces an iteration can list (rows beyond stay with their warp)
constexpr uint64_t DL_SOLO_ROWS = 1024, DL_SOLO_OUTPUTS = 4096;  // iterations of at most this size run on one block
constexpr unsigned DL_SPIN_LIMIT = 1u << 26;             // polls of a barrier before a block gives up (tens of seconds)

struct Ix {
    const unsigned long long* cursor;  // direct form: ends of the groups in `pay`, for keys below `domain`
    uint64_t domain;
    const ulonglong2* table;           // hash form
    uint64_t mask;
    const uint64_t* S;
    const uint32_t* pay;
};
struct Rule {
    Ix ix[2];
    int key_src[2];  // which half of the delta row is the key: 0 high, 1 low
    int joins;       // 1 or 2
    int hi_src, lo_src;  // output halves: 0 / 1 the delta row's, 2 / 3 the joined rows' other column, 4 zero
};
constexpr int DL_RULES = 4;
struct Rules {
    Rule r[DL_RULES];
    int n;
};
// Rules with two recursive atoms (`square` components).  The partner of the delta is the head itself as
// the iteration found it, kept as a bitmap and its transpose: a row of either is the partner's side of
// the join, 32 candidates a word, and what the head holds already is masked out of it word by word
// before any single candidate is looked at.
constexpr int SQ_VARIANTS = 8, SQ_AUX = 2, SQ_UNROLL = 4;
struct Variant {
    Ix a;              // list step on a stored relation, keyed on a delta half (a_key), or none (a_key < 0)
    int a_key;
    const unsigned int* rows;   // bit rows joined with: the head, its transpose, or a composite
    int row_key;       // the row: 0 / 1 the delta's high / low half, 2 the list step's value
    int fixed;         // the output half that does not come from the bit row: 0 / 1 / 2 likewise
    int bits_are_hi;   // the bit row's value is the output's high half
    const unsigned long long* counts;  // composite: candidates a row stands for (its bits are a set, the join a bag)
};
// Composite of the head with a stored relation joined on the head's column that the output drops:
// rows[key] = values of the stored rows joined with the head rows of that key.  Kept up to date by
// the delta's rows.
struct Composite {
    Ix ix;
    int list_key, row_key;  // halves of a head row: 0 high, 1 low
    unsigned int* rows;
    unsigned long long* counts;
};
struct Square {
    Variant v[SQ_VARIANTS];
    Composite aux[SQ_AUX];
    int n, n_aux;
    unsigned int *known_t, *full, *full_t;  // transpose of the head's bitmap; the head and its transpose as the iteration found them
    int bits;                               // of a value
};
enum Phase { PH_ROWS = 0, PH_HEAVY = 1, PH_SOLO = 2, PH_DONE = 3, PH_FULL = 4 };
struct Ctl {
    unsigned long long tail;        // tuples appended to the log so far (may pass its capacity: see overflow)
    unsigned long long start, end;  // the delta at hand: log[start, end)
    unsigned long long iterations, candidates, fix, overflow;
    unsigned long long cand_before; // candidates when the iteration began
    unsigned arrived;               // grid barrier: blocks that wait ...
    unsigned sync;                  // ... for this word to change: (generation << 3) | phase, always written as one
    unsigned next_chunk;            // rows are taken in chunks
    unsigned heavy_n, next_heavy;
    unsigned abort;
};
struct Heavy {
    uint64_t row;
    unsigned rule, piece;
};

__device__ __forceinline__ void find(const Ix& ix, uint32_t key, uint32_t& start, uint32_t& len) {
    start = len = 0;
    if (ix.cursor) {
        if (key < ix.domain) {
            const uint64_t e = __ldg(&ix.cursor[key]), s = key ? __ldg(&ix.cursor[key - 1]) : 0;
            start = (uint32_t)s;
            len = (uint32_t)(e - s);
        }
        return;
    }
    uint64_t h = mix64(key) & ix.mask;
    for (uint64_t probe = 0; probe <= ix.mask; ++probe) {  // bounded by the table size
        const ulonglong2 s = __ldg(&ix.table[h]);
        if (s.y == 0) return;
        if (s.x == key) {
            start = (uint32_t)(s.y >> 32);
            len = (uint32_t)s.y;
            return;
        }
        h = (h + 1) & ix.mask;
    }
}
__device__ __forceinline__ uint32_t other_of(const Ix& ix, uint32_t at) { return ix.pay ? __ldg(&ix.pay[at]) : (uint32_t)__ldg(&ix.S[at]); }
__device__ __forceinline__ uint32_t pick(int src, uint64_t row, uint32_t m1, uint32_t m2) {
    return src == 0 ? (uint32_t)(row >> 32) : src == 1 ? (uint32_t)row : src == 2 ? m1 : src == 3 ? m2 : 0u;
}

struct Out {
    unsigned int* visited;
    uint64_t words;
    int lo_bits;
    uint64_t* log;
    uint64_t cap;
    Ctl* ctl;
    DevStatus* st;
    unsigned int* visited_t;  // square components: the transpose, brought along
};

// A warp's collected tuples go to the log: one reservation, coalesced stores.
__device__ __forceinline__ void flush(const Out& o, uint64_t* stage, unsigned& staged) {
    if (!staged) return;
    unsigned long long at = 0;
    if (lane_id() == 0) at = atomicAdd(&o.ctl->tail, (unsigned long long)staged);
    at = __shfl_sync(FULL, at, 0);
    __syncwarp();
    for (unsigned i = lane_id(); i < staged; i += 32)
        if (at + i < o.cap) __stcg(&o.log[at + i], stage[i]);  // beyond the capacity: found again from the bitmap by the host
    __syncwarp();
    staged = 0;
}

__device__ __forceinline__ void mark_transposed(const Out& o, uint64_t t) {
    const uint32_t h = (uint32_t)(t >> 32);
    atomicOr(&o.visited_t[((uint32_t)t << (o.lo_bits - 5)) | (h >> 5)], 1u << (h & 31));
}

// What the warp's rows are, lane by lane (lane i: row i).
struct Lane {
    uint64_t row;
    uint32_t s1, s2, l2, before;  // first matches, second join's length, outputs of the rows before
};

// Outputs [from, to) of the warp's rows: marked, and the new ones collected.  `single`: all of them
// belong to lane 0's row.
__device__ __forceinline__ void emit(const Out& o, const Rule& ru, const Lane& me, uint64_t incl, uint64_t from, uint64_t to, bool single, uint64_t* stage, unsigned& staged) {
    const unsigned lane = lane_id();
    for (uint64_t base = from; base < to; base += DL_STEP) {
        uint64_t tup[DL_UNROLL];
        uint32_t x[DL_UNROLL];
        bool on[DL_UNROLL];
#pragma unroll
        for (int u = 0; u < DL_UNROLL; ++u) {
            const uint64_t t = base + u * 32 + lane;
            on[u] = t < to;
            int owner = 0;
            if (!single) {  // the row whose outputs hold t: rows before it end at or before t
#pragma unroll
                for (int d = 16; d; d >>= 1) {
                    const uint64_t end = __shfl_sync(FULL, incl, owner + d - 1);
                    if (end <= t) owner += d;
                }
            }
            const uint64_t row = __shfl_sync(FULL, me.row, owner);
            const uint32_t s1 = __shfl_sync(FULL, me.s1, owner);
            const uint32_t before = single ? 0u : __shfl_sync(FULL, me.before, owner);
            uint32_t m1 = 0, m2 = 0;
            if (ru.joins == 2) {
                const uint32_t s2 = __shfl_sync(FULL, me.s2, owner), l2 = __shfl_sync(FULL, me.l2, owner);
                if (on[u]) {
                    const uint64_t j = t - before;
                    const uint32_t a = j >> 32 ? (uint32_t)(j / l2) : (uint32_t)j / l2, b = (uint32_t)(j - (uint64_t)a * l2);
                    m1 = other_of(ru.ix[0], s1 + a);
                    m2 = other_of(ru.ix[1], s2 + b);
                }
            } else if (on[u]) m1 = other_of(ru.ix[0], s1 + (uint32_t)(t - before));
            const uint32_t h = pick(ru.hi_src, row, m1, m2), l = pick(ru.lo_src, row, m1, m2);
            tup[u] = ((uint64_t)h << 32) | l;
            const uint64_t at = ((uint64_t)h << o.lo_bits) | l;
            x[u] = (uint32_t)at;
            if (on[u] && ((uint64_t)l >> o.lo_bits || (at >> 5) >= o.words)) {
                set_status(o.st, XLB_ERR_CAPACITY, 13, tup[u]);  // outside the domain the host derived: report, never write
                on[u] = false;
            }
        }
        unsigned word[DL_UNROLL];
#pragma unroll
        for (int u = 0; u < DL_UNROLL; ++u) word[u] = on[u] ? o.visited[x[u] >> 5] : 0xFFFFFFFFu;  // (a stale line only costs an atomic)
#pragma unroll
        for (int u = 0; u < DL_UNROLL; ++u) {
            const unsigned bit = 1u << (x[u] & 31);
            on[u] = on[u] && !(word[u] & bit) && !(atomicOr(&o.visited[x[u] >> 5], bit) & bit);
        }
        if (o.visited_t)
#pragma unroll
            for (int u = 0; u < DL_UNROLL; ++u)
                if (on[u]) mark_transposed(o, tup[u]);
        if (staged + DL_STEP > DL_STAGE) flush(o, stage, staged);
#pragma unroll
        for (int u = 0; u < DL_UNROLL; ++u) {
            const unsigned b = __ballot_sync(FULL, on[u]);
            if (on[u]) stage[staged + __popc(b & lanemask_lt())] = tup[u];
            staged += __popc(b);
        }
        __syncwarp();
    }
}

// Rows log[at, at + rows) of the delta (rows <= 32) under every rule.
__device__ __forceinline__ void take_rows(const Out& o, const Rules& rules, uint64_t at, unsigned rows, Heavy* heavy, uint64_t* stage, unsigned& staged, unsigned long long& cand) {
    const unsigned lane = lane_id();
    Lane me;
    me.row = lane < rows ? __ldcg(&o.log[at + lane]) : 0;
    for (int q = 0; q < rules.n; ++q) {
        const Rule& ru = rules.r[q];
        uint32_t l1 = 0;
        me.s1 = me.s2 = me.l2 = 0;
        uint64_t cnt = 0;
        if (lane < rows) {
            find(ru.ix[0], ru.key_src[0] == 0 ? (uint32_t)(me.row >> 32) : (uint32_t)me.row, me.s1, l1);
            cnt = l1;
            if (ru.joins == 2 && l1) {
                find(ru.ix[1], ru.key_src[1] == 0 ? (uint32_t)(me.row >> 32) : (uint32_t)me.row, me.s2, me.l2);
                cnt *= me.l2;
            }
        }
        cand += cnt;
        // long rows: listed for whole blocks; one that finds the list full stays here
        unsigned alone = 0;
        if (cnt > DL_HEAVY) {
            const uint64_t pieces = (cnt + DL_PIECE - 1) / DL_PIECE;
            bool listed = false;
            if (pieces <= DL_HEAVY_MAX) {
                const unsigned h = atomicAdd(&o.ctl->heavy_n, (unsigned)pieces);
                if (h <= DL_HEAVY_MAX - pieces) {
                    for (unsigned k = 0; k < pieces; ++k) heavy[h + k] = {me.row, (unsigned)q, k};
                    listed = true;
                } else {
                    for (unsigned k = h; k < DL_HEAVY_MAX; ++k) heavy[k] = {0, ~0u, 0};  // the room that was left: nothing to do there
                }
            }
            if (!listed) alone = 1;
        }
        const uint64_t mine = cnt > DL_HEAVY ? 0 : cnt;
        uint64_t incl = mine;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint64_t v = __shfl_up_sync(FULL, incl, d);
            if (lane >= (unsigned)d) incl += v;
        }
        me.before = (uint32_t)(incl - mine);
        const uint64_t total = __shfl_sync(FULL, incl, 31);
        if (total) emit(o, ru, me, incl, 0, total, rows == 1, stage, staged);
        for (unsigned left = __ballot_sync(FULL, alone); left; left &= left - 1) {
            const int r = __ffs(left) - 1;
            Lane one;
            one.row = __shfl_sync(FULL, me.row, r);
            one.s1 = __shfl_sync(FULL, me.s1, r);
            one.s2 = __shfl_sync(FULL, me.s2, r);
            one.l2 = __shfl_sync(FULL, me.l2, r);
            one.before = 0;
            emit(o, ru, one, 0, 0, __shfl_sync(FULL, cnt, r), true, stage, staged);
        }
    }
}

// One delta row under every variant of the rules with two recursive atoms, by the whole warp.
__device__ __forceinline__ void square_row(const Out& o, const Square& sq, uint64_t row, uint64_t* stage, unsigned& staged, unsigned long long& cand) {
    const unsigned lane = lane_id(), row_words = 1u << (sq.bits - 5);
    for (int q = 0; q < sq.n; ++q) {
        const Variant& v = sq.v[q];
        uint32_t s = 0, len = 1;
        if (v.a_key >= 0) find(v.a, v.a_key == 0 ? (uint32_t)(row >> 32) : (uint32_t)row, s, len);
        for (uint32_t i = 0; i < len; i += SQ_UNROLL) {
            uint32_t fixed[SQ_UNROLL];
            bool on_row[SQ_UNROLL];
            const unsigned int *from[SQ_UNROLL], *known[SQ_UNROLL];
#pragma unroll
            for (int k = 0; k < SQ_UNROLL; ++k) {
                uint32_t e = 0;
                if (v.a_key >= 0 && i + k < len) e = other_of(v.a, s + i + k);
                const uint32_t key = pick(v.row_key, row, e, 0);
                fixed[k] = pick(v.fixed, row, e, 0);
                // (a stored value beyond the head's domain has no row in it)
                on_row[k] = i + k < len && !(key >> sq.bits);
                if (on_row[k] && fixed[k] >> sq.bits) {
                    set_status(o.st, XLB_ERR_CAPACITY, 16, fixed[k]);
                    on_row[k] = false;
                }
                from[k] = v.rows + ((uint64_t)key << (sq.bits - 5));
                known[k] = (v.bits_are_hi ? sq.known_t : o.visited) + ((uint64_t)fixed[k] << (sq.bits - 5));
                if (v.counts && lane == 0 && on_row[k]) cand += __ldcg(&v.counts[key]);
            }
            for (unsigned w0 = 0; w0 < row_words; w0 += 32) {
                const unsigned w = w0 + lane;
                unsigned m[SQ_UNROLL];
#pragma unroll
                for (int k = 0; k < SQ_UNROLL; ++k) {
                    m[k] = on_row[k] && w < row_words ? __ldcg(&from[k][w]) : 0u;  // (what the last iteration left: never from the L1)
                    if (!v.counts) cand += __popc(m[k]);
                }
#pragma unroll
                for (int k = 0; k < SQ_UNROLL; ++k)
                    if (m[k]) m[k] &= ~known[k][w];  // (a stale line only costs an atomic)
#pragma unroll
                for (int k = 0; k < SQ_UNROLL; ++k)
                    while (__any_sync(FULL, m[k] != 0)) {  // what is left is new, or was found a moment ago
                        bool on = m[k] != 0;
                        uint64_t t = 0;
                        if (on) {
                            const uint32_t x = (w << 5) | (__ffs(m[k]) - 1);
                            m[k] &= m[k] - 1;
                            t = v.bits_are_hi ? ((uint64_t)x << 32) | fixed[k] : ((uint64_t)fixed[k] << 32) | x;
                            const uint32_t at = ((uint32_t)(t >> 32) << sq.bits) | (uint32_t)t;
                            const unsigned bit = 1u << (at & 31);
                            on = !(atomicOr(&o.visited[at >> 5], bit) & bit);
                            if (on) mark_transposed(o, t);
                        }
                        const unsigned b = __ballot_sync(FULL, on);
                        if (staged + 32 > DL_STAGE) flush(o, stage, staged);
                        if (on) stage[staged + __popc(b & lanemask_lt())] = t;
                        staged += __popc(b);
                        __syncwarp();
                    }
            }
        }
    }
}
// A row of the delta joins the head as the iteration finds it, and the composites over it.
__device__ __forceinline__ void square_full(const Out& o, const Square& sq, uint64_t row) {
    const uint32_t h = (uint32_t)(row >> 32), l = (uint32_t)row;
    atomicOr(&sq.full[(h << (sq.bits - 5)) | (l >> 5)], 1u << (l & 31));
    atomicOr(&sq.full_t[(l << (sq.bits - 5)) | (h >> 5)], 1u << (h & 31));
    for (int q = 0; q < sq.n_aux; ++q) {
        const Composite& x = sq.aux[q];
        uint32_t s, len;
        find(x.ix, x.list_key == 0 ? h : l, s, len);
        if (!len) continue;
        const uint32_t key = x.row_key == 0 ? h : l;
        atomicAdd(&x.counts[key], (unsigned long long)len);
        for (uint32_t i = 0; i < len; ++i) {
            const uint32_t m = other_of(x.ix, s + i);
            if (m >> sq.bits) {
                set_status(o.st, XLB_ERR_CAPACITY, 17, m);
                continue;
            }
            unsigned int* word = &x.rows[(key << (sq.bits - 5)) | (m >> 5)];
            const unsigned bit = 1u << (m & 31);
            if (!(__ldcg(word) & bit)) atomicOr(word, bit);
        }
    }
}

// One piece of a long row, by all warps of the block.
__device__ __forceinline__ void take_piece(const Out& o, const Rules& rules, const Heavy& h, uint64_t* stage, unsigned& staged) {
    if (h.rule >= (unsigned)rules.n) return;
    const Rule& ru = rules.r[h.rule];
    Lane me;
    me.row = h.row;
    me.before = 0;
    uint32_t l1;
    find(ru.ix[0], ru.key_src[0] == 0 ? (uint32_t)(me.row >> 32) : (uint32_t)me.row, me.s1, l1);
    uint64_t cnt = l1;
    me.s2 = me.l2 = 0;
    if (ru.joins == 2) {
        find(ru.ix[1], ru.key_src[1] == 0 ? (uint32_t)(me.row >> 32) : (uint32_t)me.row, me.s2, me.l2);
        cnt *= me.l2;
    }
    const uint64_t lo = (uint64_t)h.piece * DL_PIECE, hi = lo + DL_PIECE < cnt ? lo + DL_PIECE : cnt;
    const uint64_t per = ((hi - lo + DL_WARPS - 1) / DL_WARPS + 31) & ~31ull;
    const uint64_t from = lo + (threadIdx.x >> 5) * per, to = from + per < hi ? from + per : hi;
    if (from < to) emit(o, ru, me, 0, from, to, true, stage, staged);
}

// The end of an iteration: its new tuples become the delta.  (One thread, everybody else waiting.)
// Returns what comes next.
__device__ unsigned next_iteration(const Out& o, uint64_t max_iterations, bool square) {
    Ctl* c = o.ctl;
    volatile Ctl* v = c;
    const uint64_t tail = v->tail, end = v->end, rows = end - v->start, cands = v->candidates - v->cand_before;
    v->iterations = v->iterations + 1;
    v->cand_before = v->candidates;
    v->start = end;
    v->end = tail;
    v->next_chunk = 0;
    v->heavy_n = 0;
    v->next_heavy = 0;
    const uint64_t next = tail - end;
    if (next == 0) v->fix = 1;
    else if (tail > o.cap) v->overflow = 1;
    if (next == 0 || tail > o.cap || v->iterations >= max_iterations) return PH_DONE;
    if (square) return PH_FULL;
    return next <= DL_SOLO_ROWS && cands * next <= DL_SOLO_OUTPUTS * rows ? PH_SOLO : PH_ROWS;
}

template <bool SQUARE>
__global__ void __launch_bounds__(DL_THREADS, 1) delta_loop_k(Out o, Rules rules, Heavy* heavy, uint64_t max_iterations, Square sq) {
    extern __shared__ uint64_t stage_s[];
    __shared__ uint64_t range_s[2];
    __shared__ unsigned phase_s, item_s, go_s;
    const unsigned lane = lane_id(), warp = threadIdx.x >> 5;
    uint64_t* stage = stage_s + warp * DL_STAGE;
    unsigned staged = 0, generation = 0;
    Ctl* ctl = o.ctl;
    volatile Ctl* v = ctl;
    // What thread 0 has seen of the sync word.  Between a barrier and the next, a solo phase may begin
    // and end without the other blocks: one that is late finds the word two generations on, never a
    // phase that does not belong to the generation beside it.
    auto read_phase = [&]() {
        if (threadIdx.x == 0) {
            const unsigned w = v->sync;
            __threadfence();
            generation = w >> 3;
            phase_s = w & 7;
            range_s[0] = v->start;
            range_s[1] = v->end;
        }
        __syncthreads();
    };
    auto publish = [&](unsigned phase) {
        __threadfence();
        v->sync = ((generation + 1) << 3) | phase;
    };
    // Thread 0 waits until the generation has passed; false: it never did.
    auto wait_next = [&]() {
        for (unsigned polls = 0; v->sync >> 3 == generation; ++polls) {
            if (polls > DL_SPIN_LIMIT || v->abort) {
                v->abort = 1;
                set_status(o.st, XLB_ERR_TIMEOUT, 14, generation);
                return false;
            }
            __nanosleep(polls < 64 ? 20 : 100);
        }
        return true;
    };
    // All blocks arrive; the last one asks `then` what comes next and lets the others go.
    auto barrier = [&](auto then) {
        __syncthreads();
        if (threadIdx.x == 0) {
            __threadfence();
            go_s = 1;
            if (atomicAdd(&ctl->arrived, 1u) == gridDim.x - 1) {
                __threadfence();
                v->arrived = 0;
                publish(then());
            } else go_s = wait_next();
        }
        __syncthreads();
        return go_s != 0;
    };
    auto end_warp = [&](unsigned long long cand) {
        flush(o, stage, staged);
#pragma unroll
        for (int d = 16; d; d >>= 1) cand += __shfl_xor_sync(FULL, cand, d);
        if (lane == 0 && cand) atomicAdd(&ctl->candidates, cand);
    };
    read_phase();
    for (;;) {
        const unsigned phase = phase_s;
        const uint64_t start = range_s[0], n = range_s[1] - range_s[0];
        if (phase == PH_DONE) return;
        unsigned long long cand = 0;
        if (phase == PH_ROWS) {
            // rows of the delta in chunks: few rows per warp while there are few of them
            const uint64_t warps = (uint64_t)gridDim.x * DL_WARPS;
            // (a row of a square component can stand for any amount of work: smaller chunks)
            const unsigned most = SQUARE ? 8 : 32, per = (unsigned)(n >= warps * most ? most : (n + warps - 1) / warps);
            for (uint64_t chunk = (uint64_t)warp * gridDim.x + blockIdx.x; chunk * per < n;) {
                const uint64_t at = chunk * per;
                const unsigned rows = (unsigned)(n - at < per ? n - at : per);
                take_rows(o, rules, start + at, rows, heavy, stage, staged, cand);
                if (SQUARE)
                    for (unsigned r = 0; r < rows; ++r) square_row(o, sq, __ldcg(&o.log[start + at + r]), stage, staged, cand);
                if (n <= warps * per) break;
                unsigned next = 0;
                if (lane == 0) next = atomicAdd(&ctl->next_chunk, 1u);
                chunk = warps + __shfl_sync(FULL, next, 0);
            }
            end_warp(cand);
            if (!barrier([&]() -> unsigned { return v->heavy_n ? (unsigned)PH_HEAVY : next_iteration(o, max_iterations, SQUARE); })) return;
        } else if (phase == PH_HEAVY) {
            const unsigned listed = v->heavy_n, pieces = listed < DL_HEAVY_MAX ? listed : (unsigned)DL_HEAVY_MAX;
            for (;;) {
                __syncthreads();
                if (threadIdx.x == 0) item_s = atomicAdd(&ctl->next_heavy, 1u);
                __syncthreads();
                const unsigned item = item_s;
                if (item >= pieces) break;
                Heavy h;
                h.row = __ldcg(&heavy[item].row);
                h.rule = __ldcg(&heavy[item].rule);
                h.piece = __ldcg(&heavy[item].piece);
                take_piece(o, rules, h, stage, staged);
            }
            end_warp(0);
            if (!barrier([&] { return next_iteration(o, max_iterations, SQUARE); })) return;
        } else if (SQUARE && phase == PH_FULL) {
            for (uint64_t i = (uint64_t)blockIdx.x * DL_THREADS + threadIdx.x; i < n; i += (uint64_t)gridDim.x * DL_THREADS) square_full(o, sq, __ldcg(&o.log[start + i]));
            if (!barrier([&]() -> unsigned { return PH_ROWS; })) return;
        } else if (!SQUARE) {  // PH_SOLO
            if (blockIdx.x == 0) {
                const unsigned per = (unsigned)((n + DL_WARPS - 1) / DL_WARPS);  // at most 32 (DL_SOLO_ROWS)
                if ((uint64_t)warp * per < n) {
                    const uint64_t at = (uint64_t)warp * per;
                    take_rows(o, rules, start + at, (unsigned)(n - at < per ? n - at : per), heavy, stage, staged, cand);
                }
                end_warp(cand);
                __syncthreads();
                if (threadIdx.x == 0) {
                    __threadfence();
                    const unsigned next = v->heavy_n ? (unsigned)PH_HEAVY : next_iteration(o, max_iterations, SQUARE);
                    if (next != PH_SOLO) publish(next);  // everybody again
                }
            } else {
                if (threadIdx.x == 0) go_s = wait_next();
                __syncthreads();
                if (!go_s) return;
            }
        }
        __syncthreads();
        read_phase();
    }
}

// Rows of a bag into the head: new ones (their bit was clear) are appended to the log.
__global__ void __launch_bounds__(BLOCK) delta_seed_k(const uint64_t* __restrict__ rows, uint64_t n, Out o) {
    __shared__ uint64_t stage_s[BLOCK / 32][64];
    uint64_t* stage = stage_s[threadIdx.x >> 5];
    const uint64_t step = (uint64_t)gridDim.x * BLOCK;
    unsigned staged = 0;
    for (uint64_t base = (uint64_t)blockIdx.x * BLOCK + (threadIdx.x & ~31u); base < n; base += step) {
        const uint64_t i = base + lane_id();
        const uint64_t k = i < n ? rows[i] : 0;
        const uint64_t at = ((k >> 32) << o.lo_bits) | (k & 0xFFFFFFFFull);
        bool on = i < n;
        if (on && ((k & 0xFFFFFFFFull) >> o.lo_bits || (at >> 5) >= o.words)) {
            set_status(o.st, XLB_ERR_CAPACITY, 15, k);
            on = false;
        }
        const unsigned bit = 1u << (at & 31);
        on = on && !(o.visited[at >> 5] & bit) && !(atomicOr(&o.visited[at >> 5], bit) & bit);
        if (on && o.visited_t) mark_transposed(o, k);
        const unsigned b = __ballot_sync(FULL, on);
        if (on) stage[staged + __popc(b & lanemask_lt())] = k;
        staged += __popc(b);
        __syncwarp();
        if (staged > 32) flush(o, stage, staged);
    }
    flush(o, stage, staged);
}

__global__ void delta_begin_k(Ctl* c, bool square) {
    const unsigned long long n = c->tail;
    c->start = 0;
    c->end = n;
    if (n == 0) {  // an iteration over nothing finds nothing
        c->iterations = 1;
        c->fix = 1;
    }
    c->sync = n == 0 ? PH_DONE : square ? PH_FULL : PH_ROWS;  // (never solo: a block that starts late would miss it)
}

// On with the delta at hand, once the log has the room for it.
__global__ void delta_resume_k(Ctl* c, uint64_t max_iterations, bool square) {
    c->overflow = 0;
    c->sync = c->iterations >= max_iterations ? PH_DONE : square ? PH_FULL : PH_ROWS;
}

}  // namespace

static Out out_of(xlb_ctx* c, const DeltaLoop& d) {
    return Out{d.visited->as<unsigned int>(), d.words, d.lo_bits, d.log->as<uint64_t>(), d.cap, d.ctl->as<Ctl>(), c->d_status, d.visited_t ? d.visited_t->as<unsigned int>() : nullptr};
}

DeltaLoop ops_delta_begin(xlb_ctx* c, int hi_bits, int lo_bits, bool square) {
    DeltaLoop d;
    d.hi_bits = hi_bits;
    d.lo_bits = lo_bits;
    d.words = ((1ull << (hi_bits + lo_bits)) + 31) / 32;
    const uint64_t bytes = std::max<uint64_t>(d.words * 4, 16);
    d.visited = make_buf(c, bytes);
    d.ctl = make_buf(c, sizeof(Ctl));
    CUDA_OK(set_async(c, d.visited->p, 0, bytes));
    CUDA_OK(set_async(c, d.ctl->p, 0, sizeof(Ctl)));
    if (square) {
        d.visited_t = make_buf(c, bytes);
        d.full = make_buf(c, 2 * bytes);
        CUDA_OK(set_async(c, d.visited_t->p, 0, bytes));
        CUDA_OK(set_async(c, d.full->p, 0, 2 * bytes));
    }
    return d;
}

void ops_delta_known(xlb_ctx* c, DeltaLoop& d, const Keys& rows) {
    if (!rows.n) return;
    prof_begin(c, "dense_mark", rows.n * 8ull);
    dense_mark_k<true><<<grid_for(c, rows.n), BLOCK, 0, c->stream>>>(rows.ptr(), rows.n, d.lo_bits, d.visited->as<unsigned int>(), d.words, c->d_status);
    check_launch(c, "dense_mark");
}

// Room in the log for `more` tuples beyond the `d.room` that may be in it.
static void log_room(xlb_ctx* c, DeltaLoop& d, uint64_t more) {
    const uint64_t need = d.room + more;
    d.room = need;
    if (d.log && d.cap >= need) return;
    const uint64_t domain = 1ull << (d.hi_bits + d.lo_bits);
    uint64_t cap = std::min<uint64_t>(domain, std::max<uint64_t>(4 * need, 1ull << 24));  // (beyond the domain nothing can be new)
    Buf log = make_buf(c, std::max<uint64_t>(cap, 1) * 8);
    if (d.log && need > more) CUDA_OK(copy_async(c, log->p, d.log->p, std::min(d.cap, need - more) * 8, cudaMemcpyDeviceToDevice));
    d.log = log;
    d.cap = cap;
}

void ops_delta_seed(xlb_ctx* c, DeltaLoop& d, const Keys& bag) {
    if (!bag.n) return;
    log_room(c, d, bag.n);
    prof_begin(c, "dense_mark", bag.n * 16ull);
    delta_seed_k<<<grid_for(c, bag.n), BLOCK, 0, c->stream>>>(bag.ptr(), bag.n, out_of(c, d));
    check_launch(c, "dense_mark");
}

void ops_delta_append(xlb_ctx* c, DeltaLoop& d, const Keys& rows) {
    if (!rows.n) return;
    log_room(c, d, rows.n);
    CUDA_OK(copy_async(c, d.log->as<uint64_t>() + (d.room - rows.n), rows.ptr(), rows.n * 8, cudaMemcpyDeviceToDevice));
    const unsigned long long tail = d.room;
    c->h_scalar[48] = tail;
    CUDA_OK(copy_async(c, &d.ctl->as<Ctl>()->tail, &c->h_scalar[48], 8, cudaMemcpyHostToDevice));
    stream_wait(c);  // (the staging word is used again)
}

static Ix view_of(const Index& ix) {
    return Ix{ix.cursor ? ix.cursor->as<unsigned long long>() : nullptr, ix.domain, ix.table ? ix.table->as<ulonglong2>() : nullptr, ix.mask,
              ix.S ? ix.S->as<uint64_t>() : nullptr, ix.pay ? ix.pay->as<uint32_t>() : nullptr};
}

bool ops_delta_run(xlb_ctx* c, DeltaLoop& d, const std::vector<DeltaRule>& rules, const std::vector<DeltaVariant>& variants, uint64_t max_iterations, const Keys& known,
                   DeltaResult* res) {
    if (rules.size() > DL_RULES || variants.size() > SQ_VARIANTS) xlb_fail(XLB_ERR_INVALID, "internal: %zu rules and %zu variants in a delta loop", rules.size(), variants.size());
    if (!c->delta_attr_set) {
        CUDA_OK(cudaFuncSetAttribute(delta_loop_k<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, DL_WARPS * DL_STAGE * 8));
        CUDA_OK(cudaFuncSetAttribute(delta_loop_k<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, DL_WARPS * DL_STAGE * 8));
    }
    c->delta_attr_set = true;
    const bool square = d.visited_t != nullptr;
    Square sq{};
    std::vector<Buf> composites;
    if (square) {
        const uint64_t bytes = d.visited->bytes;
        sq.bits = d.lo_bits;
        sq.known_t = d.visited_t->as<unsigned int>();
        sq.full = d.full->as<unsigned int>();
        sq.full_t = sq.full + bytes / 4;
        for (auto& in : variants) {
            Variant& v = sq.v[sq.n++];
            v.a_key = in.list ? in.list_key : -1;
            if (in.list) v.a = view_of(*in.list);
            v.row_key = in.row_key;
            v.fixed = in.fixed;
            v.bits_are_hi = in.bits_are_hi;
            if (in.rows == DeltaVariant::HEAD) v.rows = sq.full;
            else if (in.rows == DeltaVariant::HEAD_T) v.rows = sq.full_t;
            else {
                if (sq.n_aux == SQ_AUX) xlb_fail(XLB_ERR_INVALID, "internal: too many composites in a delta loop");
                Buf b = make_buf(c, bytes + (8ull << d.lo_bits));
                CUDA_OK(set_async(c, b->p, 0, b->bytes));
                composites.push_back(b);
                Composite& x = sq.aux[sq.n_aux++];
                x.ix = view_of(*in.composed);
                x.list_key = in.composed_list_key;
                x.row_key = in.composed_row_key;
                x.rows = b->as<unsigned int>();
                x.counts = (unsigned long long*)(x.rows + bytes / 4);
                v.rows = x.rows;
                v.counts = x.counts;
            }
        }
    }
    log_room(c, d, 0);
    Rules rs{};
    rs.n = (int)rules.size();
    for (int q = 0; q < rs.n; ++q) {
        Rule& r = rs.r[q];
        r.joins = rules[q].joins;
        r.hi_src = rules[q].hi_src;
        r.lo_src = rules[q].lo_src;
        for (int k = 0; k < r.joins; ++k) {
            r.key_src[k] = rules[q].key_src[k];
            r.ix[k] = view_of(*rules[q].ix[k]);
        }
    }
    Buf heavy = make_buf(c, (uint64_t)DL_HEAVY_MAX * sizeof(Heavy));
    delta_begin_k<<<1, 1, 0, c->stream>>>(d.ctl->as<Ctl>(), square);
    check_launch(c, "delta_begin");
    for (;;) {
        Out o = out_of(c, d);
        Heavy* hp = heavy->as<Heavy>();
        void* args[] = {&o, &rs, &hp, &max_iterations, &sq};
        prof_begin(c, "expand_mark", 0);
        CUDA_OK(cudaLaunchCooperativeKernel(square ? (const void*)delta_loop_k<true> : (const void*)delta_loop_k<false>, dim3((unsigned)c->sm_count), dim3(DL_THREADS), args, (size_t)DL_WARPS * DL_STAGE * 8, c->stream));
        check_launch(c, "expand_mark");
        unsigned long long w[7];  // tail, start, end, iterations, candidates, fix, overflow
        read_words(c, d.ctl->p, 7, w);
        if (c->status_code) return false;
        res->rows = w[0];
        res->iterations = w[3];
        res->candidates = w[4];
        res->fix = w[5] != 0;
        prof_add_bytes(c, "expand_mark", w[4] * 4ull + w[0] * 16ull);
        if (!w[6]) return true;
        // The log was too short for the last iteration: its delta is what the head's bitmap holds
        // beyond the known rows and the log before it.  A longer log takes up from there.
        const uint64_t tail = w[0], stored = d.cap;
        Keys done;
        done.buf = d.log;
        done.n = stored;
        Buf before = make_buf(c, d.visited->bytes);
        CUDA_OK(set_async(c, before->p, 0, before->bytes));
        for (const Keys* k : {&known, (const Keys*)&done}) {
            if (!k->n) continue;
            prof_begin(c, "dense_mark", k->n * 8ull);
            dense_mark_k<true><<<grid_for(c, k->n), BLOCK, 0, c->stream>>>(k->ptr(), k->n, d.lo_bits, before->as<unsigned int>(), d.words, c->d_status);
            check_launch(c, "dense_mark");
        }
        DenseSet lost;
        lost.hi_bits = d.hi_bits;
        lost.lo_bits = d.lo_bits;
        lost.words = d.words;
        lost.bitmap = d.visited;
        lost.visited = before->as<unsigned int>();
        lost.counts_buf = make_buf(c, 24);
        lost.counts = lost.counts_buf->as<uint64_t>();
        CUDA_OK(set_async(c, lost.counts_buf->p, 0, 24));
        Keys none;
        Keys rows = ops_dense_finish(c, lost, none);
        if (rows.n != tail - stored) xlb_fail(XLB_ERR_CUDA, "internal: %llu of %llu tuples found again", (unsigned long long)rows.n, (unsigned long long)(tail - stored));
        before.reset();
        lost = DenseSet();
        d.room = tail;
        log_room(c, d, tail);
        CUDA_OK(copy_async(c, d.log->as<uint64_t>() + stored, rows.ptr(), rows.n * 8, cudaMemcpyDeviceToDevice));
        d.room = tail;
        delta_resume_k<<<1, 1, 0, c->stream>>>(d.ctl->as<Ctl>(), max_iterations, square);
        check_launch(c, "delta_resume");
    }
}
