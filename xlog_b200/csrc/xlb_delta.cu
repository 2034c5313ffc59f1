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

// (Measured on the cases the comment above names, 32 warps with 2 outputs a lane in flight against 24
// warps, 16 warps, 4 outputs and 8 outputs: closure 299 us against 320 to 504, banded DAG 935 against
// 993 to 1503, same generation 779 against 846 to 1300.  The loop is bound by the latency of short rows'
// chains and by warps that wait for the others at the barriers, not by bandwidth or issue slots, of which 17 to
// 24 % are used: more in flight per warp is work for rows that are not there.)
constexpr int DL_THREADS = 1024, DL_WARPS = DL_THREADS / 32;
constexpr int DL_UNROLL = 2;                             // outputs a lane has in flight
constexpr int DL_STAGE = 128;                            // new tuples a warp collects before it reserves room in the log
constexpr unsigned DL_HEAVY = 512;                       // a row with more outputs than this is taken apart
constexpr unsigned DL_PIECE = 512;                       // ... into pieces that any warp can take
constexpr unsigned DL_HEAVY_MAX = 1u << 18;              // pieces an iteration can list (rows beyond stay with their warp)
constexpr uint64_t DL_SOLO_ROWS = 2048, DL_SOLO_OUTPUTS = 8192;  // iterations of at most this size run on one block
constexpr unsigned SOLO_NEXT = 2048;                     // tuples of a solo iteration that stay in shared memory
constexpr size_t DL_SMEM = std::max<size_t>((size_t)DL_WARPS * 2 * DL_STAGE * 8, 2 * SOLO_NEXT * 16);
static_assert(2 * SOLO_NEXT * 16 <= DL_SMEM, "the solo phase uses the warps' stages");

struct Ix {
    const unsigned long long* cursor;  // direct form: ends of the groups in `pay`, for keys below `domain`
    uint64_t domain;
    const ulonglong2* table;           // hash form
    uint64_t mask;
    const uint32_t* other;             // the rows' other column: a payload array, or the low halves of packed rows (step 1)
    int step;
};
struct Rule {
    Ix ix[2];
    int key_src[2];  // which half of the delta row is the key: 0 high, 1 low
    int joins;       // 1 or 2
    int hi_src, lo_src;  // output halves: 0 / 1 the delta row's, 2 / 3 the joined rows' other column, 4 zero
    unsigned long long rows;  // of the first relation
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
    uint32_t rows;     // bit rows joined with (head, transpose or a composite), as a word offset from the head's bitmap
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
    uint32_t rows;
    unsigned long long* counts;
};
// Bitmaps of `words` words each, back to back: the head, its transpose, the two as the iteration found
// them, the composites.
struct Square {
    Variant v[SQ_VARIANTS];
    Composite aux[SQ_AUX];
    int n, n_aux;
    uint32_t words;
    int bits;  // of a value
};
enum Phase { PH_ROWS = 0, PH_HEAVY = 1, PH_SOLO = 2, PH_DONE = 3, PH_FULL = 4 };
// What the blocks share about one iteration.  Three are used in turn: while one is filled the next is
// cleared (by block 0, in every phase that ends an iteration at a grid barrier: the rows and the pieces of
// long rows, which a solo phase goes over to directly), and the one before may still be read by a block
// that is late.  A solo phase that ends an iteration by itself touches none.
struct Slot {
    unsigned long long count, cand;  // tuples appended to the log; candidates
    unsigned long long heavy_n;      // pieces of long rows, listed or not (rows that found the list full go on raising it); of bit rows: rows that the delta's were led to
    unsigned next_heavy;             // pieces taken
    unsigned next_chunk;             // rows are taken in batches
};
struct Ctl {
    // in: where the loop stands; out: where it stopped (read by the host)
    unsigned long long tail;        // tuples in the log (may pass its capacity: see overflow)
    unsigned long long start, end;  // the delta at hand: log[start, end)
    unsigned long long iterations, candidates, fix, overflow;
    unsigned phase, check;          // check: most candidates of the last iteration were known already
    unsigned arrived;               // blocks that arrived at the grid barriers so far
    unsigned abort;
    // what block 0 found when it ran on alone
    unsigned solo_turns;            // solo phases that are over
    unsigned solo_phase, solo_check;
    // Work that touches none of the slots' counters for long counts up here, so that those who wait for it
    // can tell it from work that is not going on.
    unsigned beat;
    unsigned long long solo_start, solo_end, solo_iterations, solo_candidates;
    Slot slot[3];
    // rows evaluated one warp each: what they came to, and what was given up (read by the host)
    unsigned long long rows_tuples, rows_candidates, rows_levels, rows_left, rows_given_up, rows_seeds;
    unsigned rows_ticket, rows_idle;
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
__device__ __forceinline__ uint32_t other_of(const Ix& ix, uint32_t at) { return __ldg(&ix.other[(uint64_t)at << ix.step]); }
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
    unsigned spin_limit;      // polls without anything going on before a block gives up waiting
};
constexpr unsigned DL_BEAT_OUTPUTS = 1u << 22, DL_BEAT_ITEMS = 4096, DL_BEAT_GROUPS = 8, DL_BEAT_TURNS = 1024;  // work between two beats
__device__ __forceinline__ void beat(const Out& o) { atomicAdd(&o.ctl->beat, 1u); }

__device__ __forceinline__ void mark_transposed(const Out& o, uint64_t t) {
    const uint32_t h = (uint32_t)(t >> 32);
    atomicOr(&o.visited_t[((uint32_t)t << (o.lo_bits - 5)) | (h >> 5)], 1u << (h & 31));
}

// Where new tuples go.  A warp collects its own in shared memory and reserves room in the log for a
// batch of them with one atomic add (added one warp step at a time, the queue on that one counter
// held a same-generation closure at 24 G tuples/s); it does not wait for the reservation, but fills
// the other half of its stage meanwhile.
struct WarpSink {
    const Out& o;
    uint64_t* stage;              // two halves of DL_STAGE
    Slot* slot = nullptr;         // of the iteration under way ...
    uint64_t base = 0;            // ... whose tuples follow here in the log
    unsigned staged = 0, pending = 0, half = 0;
    unsigned long long at = 0;    // lane 0: where the pending half goes

    __device__ __forceinline__ void write(uint64_t to, const uint64_t* from, unsigned n) {
        for (unsigned i = lane_id(); i < n; i += 32)
            if (to + i < o.cap) o.log[to + i] = from[i];  // beyond the capacity: found again from the bitmap by the host
        __syncwarp();
    }
    __device__ __forceinline__ void finish() {
        if (!pending) return;
        write(__shfl_sync(FULL, at, 0), stage + (half ^ 1) * DL_STAGE, pending);
        pending = 0;
    }
    __device__ __forceinline__ void rotate() {
        finish();
        if (!staged) return;
        __syncwarp();
        if (lane_id() == 0) at = base + atomicAdd(&slot->count, (unsigned long long)staged);
        pending = staged;
        staged = 0;
        half ^= 1;
    }
    __device__ __forceinline__ void write_left(uint64_t to) {  // what is staged, to a place somebody else reserved
        write(to, stage + half * DL_STAGE, staged);
        staged = 0;
    }
    template <int N>
    __device__ __forceinline__ void look_ahead(const uint64_t (&)[N]) {}
    template <int N>
    __device__ __forceinline__ void push(const bool (&on)[N], const uint64_t (&tup)[N]) {
        unsigned b[N], total = 0;
#pragma unroll
        for (int u = 0; u < N; ++u) {
            b[u] = __ballot_sync(FULL, on[u]);
            total += __popc(b[u]);
        }
        if (staged + total > DL_STAGE) rotate();  // (what fits is staged: half-empty reservations queue on the counter)
        uint64_t* to = stage + half * DL_STAGE;
#pragma unroll
        for (int u = 0; u < N; ++u) {
            if (on[u]) to[staged + __popc(b[u] & lanemask_lt())] = tup[u];
            staged += __popc(b[u]);
        }
    }
};
// Block 0 alone: the next delta is built in shared memory; the log gets its copy on the side.  With one
// join a tuple's own matches are looked up while the atomic that decides about it is on its way, and
// kept beside it.
struct SoloShared {
    unsigned count[3], cand[3], listed[3];  // of three turns: a fast warp is in the next one while a slow one still reads
};
template <bool AHEAD>
struct SoloSink {
    const Out& o;
    const Rules& rules;
    uint64_t* next;
    uint32_t *next_s, *next_l;
    unsigned *count, *listed;
    uint64_t base;  // the log's tail
    uint32_t s[DL_UNROLL], l[DL_UNROLL];
    template <int N>
    __device__ __forceinline__ void look_ahead(const uint64_t (&tup)[N]) {
        if constexpr (AHEAD) {
#pragma unroll
            for (int u = 0; u < N; ++u) find(rules.r[0].ix[0], rules.r[0].key_src[0] == 0 ? (uint32_t)(tup[u] >> 32) : (uint32_t)tup[u], s[u], l[u]);
        }
    }
    template <int N>
    __device__ __forceinline__ void push(const bool (&on)[N], const uint64_t (&tup)[N]) {
        unsigned b[N], total = 0, at = 0;
#pragma unroll
        for (int u = 0; u < N; ++u) {
            b[u] = __ballot_sync(FULL, on[u]);
            total += __popc(b[u]);
        }
        if (!total) return;
        if (lane_id() == 0) at = atomicAdd(count, total);
        at = __shfl_sync(FULL, at, 0);
#pragma unroll
        for (int u = 0; u < N; ++u) {
            const unsigned p = at + __popc(b[u] & lanemask_lt());
            if (on[u]) {
                if (p < SOLO_NEXT) {
                    next[p] = tup[u];
                    if (AHEAD) {
                        next_s[p] = s[u];
                        next_l[p] = l[u];
                        if (l[u] > DL_HEAVY) *listed = 1;  // a long row: not for one block
                    }
                }
                if (base + p < o.cap) o.log[base + p] = tup[u];
            }
            at += __popc(b[u]);
        }
    }
};

// What the warp's rows are, lane by lane (lane i: row i).
struct Lane {
    uint64_t row;
    uint32_t s1, s2, l2, before;  // first matches, second join's length, outputs of the rows before
};

// Outputs of the warp's rows: marked, and the new ones handed to the sink.
//   BALANCED  `count` outputs in all, dealt out over the lanes; `incl`: outputs up to and with lane's row
//   SINGLE    `count` outputs of lane 0's row, from `first` on
//   SERIAL    every lane its own row's `incl` outputs, at most `count`: no searching for owners, where
//             the rows are about equally long
// `check`: most of what an iteration finds is known already; then a look at the bitmap saves the
// atomic, else it only delays it.
enum Deal { BALANCED, SINGLE, SERIAL };
template <Deal DEAL, int N, class Sink>
__device__ __forceinline__ void emit(const Out& o, const Rule& ru, const Lane& me, uint32_t incl, uint64_t first, uint32_t count, bool check, Sink& sink) {
    const unsigned lane = lane_id();
    for (uint32_t base = 0; base < count; base += DEAL == SERIAL ? N : 32 * N) {
        // (every load below is issued whether its lane has an output or not, from a place that exists:
        // a branch around it would make each wait for the one before)
        uint64_t tup[N];
        uint32_t at1[N], at2[N], x[N];
        bool on[N], bad = false;
#pragma unroll
        for (int u = 0; u < N; ++u) {
            const uint32_t t = DEAL == SERIAL ? base + u : base + u * 32 + lane;
            on[u] = t < (DEAL == SERIAL ? incl : count);
            int owner = DEAL == SERIAL ? (int)lane : 0;
            if (DEAL == BALANCED) {  // the row whose outputs hold t: rows before it end at or before t
#pragma unroll
                for (int d = 16; d; d >>= 1)
                    if (__shfl_sync(FULL, incl, owner + d - 1) <= t) owner += d;
            }
            tup[u] = DEAL == SERIAL ? me.row : __shfl_sync(FULL, me.row, owner);
            const uint32_t s1 = DEAL == SERIAL ? me.s1 : __shfl_sync(FULL, me.s1, owner);
            const uint64_t j = DEAL == SINGLE ? first + t : DEAL == SERIAL ? t : (uint64_t)(t - __shfl_sync(FULL, me.before, owner));
            at1[u] = s1 + (uint32_t)j;
            at2[u] = 0;
            if (ru.joins == 2) {
                const uint32_t s2 = DEAL == SERIAL ? me.s2 : __shfl_sync(FULL, me.s2, owner), l2 = max(DEAL == SERIAL ? me.l2 : __shfl_sync(FULL, me.l2, owner), 1u);
                const uint32_t a = DEAL == SINGLE && j >> 32 ? (uint32_t)(j / l2) : (uint32_t)j / l2, b = (uint32_t)(j - (uint64_t)a * l2);
                at1[u] = s1 + a;
                at2[u] = s2 + b;
            }
            if (!on[u]) at1[u] = at2[u] = 0;
        }
        uint32_t m1[N], m2[N];
#pragma unroll
        for (int u = 0; u < N; ++u) m1[u] = other_of(ru.ix[0], at1[u]);
#pragma unroll
        for (int u = 0; u < N; ++u) m2[u] = ru.joins == 2 ? other_of(ru.ix[1], at2[u]) : 0u;
#pragma unroll
        for (int u = 0; u < N; ++u) {
            const uint32_t h = pick(ru.hi_src, tup[u], m1[u], m2[u]), l = pick(ru.lo_src, tup[u], m1[u], m2[u]);
            tup[u] = ((uint64_t)h << 32) | l;
            const uint64_t at = ((uint64_t)h << o.lo_bits) | l;
            x[u] = (uint32_t)at;
            const bool outside = (uint64_t)l >> o.lo_bits || (at >> 5) >= o.words;
            bad |= on[u] && outside;
            on[u] = on[u] && !outside;
            if (!on[u]) x[u] = 0;
        }
        if (bad) set_status(o.st, XLB_ERR_CAPACITY, 13, tup[0]);  // outside the domain the host derived: reported, never written
        if (check) {
            unsigned word[N];
#pragma unroll
            for (int u = 0; u < N; ++u) word[u] = o.visited[x[u] >> 5];  // (a stale line only costs an atomic)
#pragma unroll
            for (int u = 0; u < N; ++u) on[u] = on[u] && !((word[u] >> (x[u] & 31)) & 1u);
        }
        unsigned old[N];
#pragma unroll
        for (int u = 0; u < N; ++u) {
            old[u] = 0;
            if (on[u]) old[u] = atomicOr(&o.visited[x[u] >> 5], 1u << (x[u] & 31));
        }
        sink.look_ahead(tup);
#pragma unroll
        for (int u = 0; u < N; ++u) on[u] = on[u] && !((old[u] >> (x[u] & 31)) & 1u);
        if (o.visited_t)
#pragma unroll
            for (int u = 0; u < N; ++u)
                if (on[u]) mark_transposed(o, tup[u]);
        sink.push(on, tup);
    }
}

// Outputs of rows whose matches are known (lane's own: `mine`, none of them long) under one rule.
template <class Sink>
__device__ __forceinline__ void deal(const Out& o, const Rule& ru, Lane& me, uint32_t mine, unsigned rows, bool check, Sink& sink) {
    const uint32_t longest = __reduce_max_sync(FULL, mine);
    if (longest <= 1) {
        if (longest) emit<SERIAL, 1>(o, ru, me, mine, 0, 1, check, sink);
        return;
    }
    const uint32_t total = __reduce_add_sync(FULL, mine);
    if (longest * 16 <= total) {  // at least half of the lanes' steps would bring an output
        emit<SERIAL, DL_UNROLL>(o, ru, me, mine, 0, longest, check, sink);
    } else if (rows == 1) {
        emit<SINGLE, DL_UNROLL>(o, ru, me, 0, 0, total, check, sink);
    } else {
        uint32_t incl = mine;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t v = __shfl_up_sync(FULL, incl, d);
            if (lane_id() >= (unsigned)d) incl += v;
        }
        me.before = incl - mine;
        emit<BALANCED, DL_UNROLL>(o, ru, me, incl, 0, total, check, sink);
    }
}

// The warp's rows (lane i < rows: me_row of the delta) under every rule with one recursive atom.
// `cand` += this lane's candidates (at most 512 a row and rule; those of longer rows are counted
// in global memory).  Returns whether a long row was listed in pieces.
template <class Sink>
__device__ __forceinline__ bool take_rows(const Out& o, const Rules& rules, uint64_t me_row, unsigned rows, Heavy* heavy, Slot* slot, bool check, Sink& sink, unsigned& cand) {
    const unsigned lane = lane_id();
    bool any_listed = false;
    Lane me;
    me.row = me_row;
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
        if (cnt <= DL_HEAVY) cand += (unsigned)cnt;
        else atomicAdd(&slot->cand, (unsigned long long)cnt);
        // long rows: listed in pieces; one that finds the list full stays here
        unsigned alone = 0;
        if (cnt > DL_HEAVY) {
            const uint64_t pieces = (cnt + DL_PIECE - 1) / DL_PIECE;
            bool listed = false;
            if (pieces <= DL_HEAVY_MAX) {
                const uint64_t h = atomicAdd(&slot->heavy_n, (unsigned long long)pieces);
                if (h <= DL_HEAVY_MAX - pieces) {
                    for (unsigned k = 0; k < pieces; ++k) heavy[h + k] = {me.row, (unsigned)q, k};
                    listed = true;
                } else {
                    for (uint64_t k = h; k < DL_HEAVY_MAX; ++k) heavy[k] = {0, ~0u, 0};  // the room that was left: nothing to do there
                }
            }
            any_listed = true;  // (the count was raised either way)
            if (!listed) alone = 1;
        }
        deal(o, ru, me, cnt > DL_HEAVY ? 0 : (uint32_t)cnt, rows, check, sink);
        for (unsigned left = __ballot_sync(FULL, alone); left; left &= left - 1) {
            const int r = __ffs(left) - 1;
            Lane one;
            one.row = __shfl_sync(FULL, me.row, r);
            one.s1 = __shfl_sync(FULL, me.s1, r);
            one.s2 = __shfl_sync(FULL, me.s2, r);
            one.l2 = __shfl_sync(FULL, me.l2, r);
            one.before = 0;
            const uint64_t all = __shfl_sync(FULL, cnt, r);
            for (uint64_t at = 0; at < all; at += DL_BEAT_OUTPUTS) {
                emit<SINGLE, DL_UNROLL>(o, ru, one, 0, at, (uint32_t)(all - at < DL_BEAT_OUTPUTS ? all - at : DL_BEAT_OUTPUTS), check, sink);
                if (lane == 0) beat(o);
            }
        }
    }
    return any_listed;
}

// One piece of a long row.
__device__ __forceinline__ void take_piece(const Out& o, const Rules& rules, const Heavy& h, bool check, WarpSink& sink) {
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
    const uint64_t from = (uint64_t)h.piece * DL_PIECE;
    if (from < cnt) emit<SINGLE, DL_UNROLL>(o, ru, me, 0, from, (uint32_t)(cnt - from < DL_PIECE ? cnt - from : DL_PIECE), check, sink);
}

// The warp's rows (lane i < rows: me_row) under every variant of the rules with two recursive atoms.  A variant
// of a row stands for one bit row per stored match (or for one).  The warp looks the matches up
// lane by lane for all rows and variants at once, then takes the bit rows SQ_UNROLL at a time, two
// words per lane: what a single row costs is the latency of its loads, so they are kept in flight.
__device__ __forceinline__ void take_square(const Out& o, const Square& sq, uint64_t me_row, unsigned rows, WarpSink& sink, unsigned long long& cand) {
    const unsigned lane = lane_id(), shift = sq.bits - 5, row_words = 1u << shift, work = rows * sq.n;
    const unsigned int* bits = o.visited;
    for (unsigned t0 = 0; t0 < work; t0 += 32) {
        const unsigned t = t0 + lane;
        const uint64_t row = __shfl_sync(FULL, me_row, t / sq.n);
        unsigned q = 0;
        uint32_t s = 0, len = 0;
        if (t < work) {
            q = t % sq.n;
            len = 1;
            if (sq.v[q].a_key >= 0) find(sq.v[q].a, sq.v[q].a_key == 0 ? (uint32_t)(row >> 32) : (uint32_t)row, s, len);
        }
        uint64_t incl = len;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint64_t v = __shfl_up_sync(FULL, incl, d);
            if (lane >= (unsigned)d) incl += v;
        }
        const uint64_t total = __shfl_sync(FULL, incl, 31), before = incl - len;
        for (uint64_t i0 = 0; i0 < total; i0 += 32) {
            if (i0 && i0 % DL_BEAT_ITEMS == 0 && lane == 0) beat(o);
            const uint64_t i = i0 + lane;
            int owner = 0;
#pragma unroll
            for (int d = 16; d; d >>= 1)
                if (__shfl_sync(FULL, incl, owner + d - 1) <= i) owner += d;
            const uint64_t r = __shfl_sync(FULL, row, owner);
            const unsigned vq = __shfl_sync(FULL, q, owner);
            const uint32_t from_s = __shfl_sync(FULL, s, owner);
            const uint64_t from_before = __shfl_sync(FULL, before, owner);
            bool ok = i < total;
            uint32_t from = 0, known = 0;
            if (ok) {
                const Variant& v = sq.v[vq];
                const uint32_t e = v.a_key >= 0 ? other_of(v.a, from_s + (uint32_t)(i - from_before)) : 0;
                const uint32_t key = pick(v.row_key, r, e, 0), fixed = pick(v.fixed, r, e, 0);
                ok = !(key >> sq.bits);  // (a stored value beyond the head's domain has no row in it)
                if (ok && fixed >> sq.bits) {
                    set_status(o.st, XLB_ERR_CAPACITY, 16, fixed);
                    ok = false;
                }
                from = v.rows + (key << shift);
                known = (v.bits_are_hi ? sq.words : 0u) + (fixed << shift);
                if (ok && v.counts) cand += __ldcg(&v.counts[key]);
            }
            for (unsigned left = __ballot_sync(FULL, ok); left;) {
                uint32_t f[SQ_UNROLL], kn[SQ_UNROLL];
                int items = 0;
#pragma unroll
                for (int k = 0; k < SQ_UNROLL; ++k) {
                    const int src = left ? __ffs(left) - 1 : 0;
                    items += left ? 1 : 0;
                    f[k] = __shfl_sync(FULL, from, src);
                    kn[k] = __shfl_sync(FULL, known, src);
                    left &= left - 1;
                }
                for (unsigned w0 = 0; w0 < row_words; w0 += 64) {
                    const unsigned w = w0 + 2 * lane;
                    uint64_t m[SQ_UNROLL], have[SQ_UNROLL];
#pragma unroll
                    for (int k = 0; k < SQ_UNROLL; ++k) {
                        const bool in = k < items && w < row_words;
                        m[k] = in ? *reinterpret_cast<const unsigned long long*>(bits + f[k] + w) : 0ull;        // (the barrier's fence has emptied the L1)
                        have[k] = in ? *reinterpret_cast<const unsigned long long*>(bits + kn[k] + w) : 0ull;     // (a stale line only costs an atomic)
                    }
                    uint64_t any = 0;
#pragma unroll
                    for (int k = 0; k < SQ_UNROLL; ++k) {
                        if (f[k] < 4 * sq.words) cand += __popcll(m[k]);
                        m[k] &= ~have[k];
                        any |= m[k];
                    }
                    if (!__any_sync(FULL, any != 0)) continue;
                    // What is left is new, or was found a moment ago: one atomic a pair of words tells.  A row of the
                    // head decides; where the bits are the tuples' high halves the pair is the transpose's,
                    // which lets one of those who find a tuple through, and the head's bit then decides.  (One atomic a
                    // bit, several turns of them one after the other: points-to over 1500 values 483 us, now 395.)
                    uint64_t was[SQ_UNROLL];
#pragma unroll
                    for (int k = 0; k < SQ_UNROLL; ++k) was[k] = m[k] ? atomicOr(reinterpret_cast<unsigned long long*>(o.visited + kn[k] + w), (unsigned long long)m[k]) : 0ull;
                    any = 0;
#pragma unroll
                    for (int k = 0; k < SQ_UNROLL; ++k) {
                        m[k] &= ~was[k];
                        any |= m[k];
                    }
                    while (__any_sync(FULL, any != 0)) {  // a few bits of one pair per lane and turn
                        bool on[SQ_UNROLL];
                        uint64_t tup[SQ_UNROLL];
                        uint64_t mine = 0;
                        uint32_t where = 0;
#pragma unroll
                        for (int k = SQ_UNROLL - 1; k >= 0; --k)
                            if (m[k]) {
                                mine = m[k];
                                where = kn[k];
                            }
                        const bool hi = where >= sq.words;
                        const uint32_t fixed = (hi ? where - sq.words : where) >> shift;
                        unsigned old[SQ_UNROLL];
                        uint64_t rest = mine;
#pragma unroll
                        for (int u = 0; u < SQ_UNROLL; ++u) {
                            on[u] = rest != 0;
                            const uint32_t x = (w << 5) + (on[u] ? __ffsll(rest) - 1 : 0);
                            rest &= rest - 1;
                            tup[u] = hi ? ((uint64_t)x << 32) | fixed : ((uint64_t)fixed << 32) | x;
                            old[u] = 0;
                            if (on[u] && hi) old[u] = atomicOr(&o.visited[(x << shift) + (fixed >> 5)], 1u << (fixed & 31));
                            if (on[u] && !hi) mark_transposed(o, tup[u]);
                        }
#pragma unroll
                        for (int u = 0; u < SQ_UNROLL; ++u) on[u] = on[u] && !((old[u] >> (fixed & 31)) & 1u);
                        bool taken = mine == 0;
                        any = 0;
#pragma unroll
                        for (int k = 0; k < SQ_UNROLL; ++k) {
                            if (!taken && m[k]) {
                                m[k] = rest;
                                taken = true;
                            }
                            any |= m[k];
                        }
                        sink.push(on, tup);
                    }
                }
            }
        }
    }
}
// A row of the delta joins the head as the iteration finds it, and the composites over it.
__device__ __forceinline__ void square_full(const Out& o, const Square& sq, uint64_t row) {
    const uint32_t h = (uint32_t)(row >> 32), l = (uint32_t)row, shift = sq.bits - 5;
    atomicOr(&o.visited[2 * sq.words + ((h << shift) | (l >> 5))], 1u << (l & 31));
    atomicOr(&o.visited[3 * sq.words + ((l << shift) | (h >> 5))], 1u << (h & 31));
    for (int q = 0; q < sq.n_aux; ++q) {
        const Composite& x = sq.aux[q];
        uint32_t s, len;
        find(x.ix, x.list_key == 0 ? h : l, s, len);
        if (!len) continue;
        const uint32_t key = x.row_key == 0 ? h : l;
        atomicAdd(&x.counts[key], (unsigned long long)len);
        for (uint32_t i = 0; i < len; ++i) {
            if ((i + 1) % DL_BEAT_ITEMS == 0) beat(o);
            const uint32_t m = other_of(x.ix, s + i);
            if (m >> sq.bits) {
                set_status(o.st, XLB_ERR_CAPACITY, 17, m);
                continue;
            }
            unsigned int* word = &o.visited[x.rows + ((key << shift) | (m >> 5))];
            const unsigned bit = 1u << (m & 31);
            if (!(__ldcg(word) & bit)) atomicOr(word, bit);
        }
    }
}

// Where the loop stands, as every block works it out for itself.
struct State {
    uint64_t start, end, iterations, candidates;
    unsigned phase, check, slot;
    bool fix, overflow;
};
// The end of an iteration that appended `count` tuples: they become the delta.
__device__ __forceinline__ void next_iteration(State& st, uint64_t count, uint64_t cands, uint64_t cap, uint64_t max_iterations, bool square) {
    const uint64_t rows = st.end - st.start;
    ++st.iterations;
    st.candidates += cands;
    st.start = st.end;
    st.end += count;
    st.check = count * 2 < cands;
    st.fix = count == 0;
    st.overflow = !st.fix && st.end > cap;
    if (st.fix || st.overflow || st.iterations >= max_iterations) st.phase = PH_DONE;
    else if (square) st.phase = PH_FULL;
    else st.phase = count <= DL_SOLO_ROWS && cands * count <= DL_SOLO_OUTPUTS * rows ? PH_SOLO : PH_ROWS;
}

// Small iterations, by block 0 alone while the others wait: the delta, the next one and the counts
// stay in shared memory, one block barrier per iteration.  Leaves `st` (of all threads) at what needs all
// blocks.
template <bool AHEAD>
__device__ __forceinline__ void solo(const Out& o, const Rules& rules, Heavy* heavy, Slot* slot, uint64_t max_iterations, uint64_t* buf, SoloShared& sh, State& st) {
    const unsigned lane = lane_id(), warp = threadIdx.x >> 5;
    uint32_t *buf_s = reinterpret_cast<uint32_t*>(buf + 2 * SOLO_NEXT), *buf_l = buf_s + 2 * SOLO_NEXT;
    unsigned n = (unsigned)(st.end - st.start), cur = 0;
    bool thin = true;  // about one output a row: as few warps as hold the rows, each pays the whole chain of instructions
    if (threadIdx.x < 3) {
        sh.count[threadIdx.x] = 0;
        sh.cand[threadIdx.x] = 0;
        sh.listed[threadIdx.x] = 0;
    }
    __syncthreads();
    for (unsigned i = threadIdx.x; i < n; i += DL_THREADS) {
        const uint64_t row = __ldcg(&o.log[st.start + i]);
        buf[i] = row;
        if (AHEAD) {
            find(rules.r[0].ix[0], rules.r[0].key_src[0] == 0 ? (uint32_t)(row >> 32) : (uint32_t)row, buf_s[i], buf_l[i]);
            if (buf_l[i] > DL_HEAVY) sh.listed[2] = 1;
        }
    }
    __syncthreads();
    if (AHEAD && sh.listed[2]) {  // a long row: all blocks
        st.phase = PH_ROWS;
        return;
    }
    for (unsigned turn = 0;; turn = turn == 2 ? 0 : turn + 1) {
        if (threadIdx.x == 0 && st.iterations % DL_BEAT_TURNS == 0) beat(o);
        const unsigned after = turn == 2 ? 0 : turn + 1;  // (its counters were read last two barriers ago)
        if (threadIdx.x == 0) {
            sh.count[after] = 0;
            sh.cand[after] = 0;
            sh.listed[after] = 0;
        }
        const unsigned per = thin || n >= DL_THREADS ? 32 : (n + DL_WARPS - 1) / DL_WARPS;
        unsigned cand = 0;
        const unsigned to = (cur ^ 1) * SOLO_NEXT, from = cur * SOLO_NEXT;
        for (unsigned at = warp * per; at < n; at += DL_WARPS * per) {
            const unsigned rows = n - at < per ? n - at : per;
            SoloSink<AHEAD> sink{o, rules, buf + to, buf_s + to, buf_l + to, &sh.count[turn], &sh.listed[turn], st.end};
            const uint64_t row = lane < rows ? buf[from + at + lane] : 0;
            if (AHEAD) {
                Lane me;
                me.row = row;
                me.s1 = lane < rows ? buf_s[from + at + lane] : 0;
                me.s2 = me.l2 = 0;
                const uint32_t mine = lane < rows ? buf_l[from + at + lane] : 0;
                cand += mine;
                deal(o, rules.r[0], me, mine, rows, false, sink);
            } else if (take_rows(o, rules, row, rows, heavy, slot, false, sink, cand)) sh.listed[turn] = 1;
        }
        cand = __reduce_add_sync(FULL, cand);
        if (lane == 0 && cand) atomicAdd(&sh.cand[turn], cand);
        __syncthreads();
        const unsigned next = sh.count[turn];
        const uint64_t cands = sh.cand[turn];
        if (!AHEAD && sh.listed[turn]) {  // the iteration is not over: its long rows are listed
            if (threadIdx.x == 0) {
                slot->count = next;
                atomicAdd(&slot->cand, (unsigned long long)cands);
            }
            st.phase = PH_HEAVY;
            return;
        }
        next_iteration(st, next, cands, o.cap, max_iterations, false);
        if (AHEAD && sh.listed[turn] && st.phase == PH_SOLO) st.phase = PH_ROWS;
        if (st.phase != PH_SOLO) return;
        thin = cands <= 2ull * n;
        n = next;
        cur ^= 1;
    }
}

// A bounded wait (one thread): until the word has come to `want`.  An iteration may take any time, so
// what is bounded is the time in which nothing that the others do can be seen.
__device__ __forceinline__ unsigned going_on(const Ctl* ctl) {
    unsigned v = *(const volatile unsigned*)&ctl->beat;
    for (int k = 0; k < 3; ++k) {
        const volatile Slot* s = &ctl->slot[k];
        v += (unsigned)s->count + s->next_heavy + s->next_chunk;
    }
    return v;
}
__device__ __forceinline__ bool wait_for(const Out& o, const unsigned* word, unsigned want, unsigned sleep, unsigned passed) {
    unsigned v, seen = going_on(o.ctl);
    for (unsigned polls = 0;; ++polls) {
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(word) : "memory");
        if ((int)(v - want) >= 0) return true;
        if (polls >= o.spin_limit) {
            const unsigned now = going_on(o.ctl);
            if (now != seen && o.spin_limit) {  // (a limit of 0: what is not over when it is first looked at has run out)
                seen = now;
                polls = 0;
                continue;
            }
            *(volatile unsigned*)&o.ctl->abort = 1;
            set_status(o.st, XLB_ERR_TIMEOUT, 14, passed);
            return false;
        }
        if (*(volatile unsigned*)&o.ctl->abort) return false;
        if (sleep) __nanosleep(sleep);
    }
}

template <bool SQUARE>
__global__ void __launch_bounds__(DL_THREADS, 1) delta_loop_k(const __grid_constant__ Out o, const __grid_constant__ Rules rules, Heavy* heavy, uint64_t max_iterations, const __grid_constant__ Square sq) {
    extern __shared__ uint64_t stage_s[];
    __shared__ State state_s;
    __shared__ unsigned go_s;
    __shared__ SoloShared solo_s;
    __shared__ unsigned left_s[32];
    __shared__ unsigned long long cand_s[32];
    const unsigned lane = lane_id(), warp = threadIdx.x >> 5;
    WarpSink sink{o, stage_s + warp * (2 * DL_STAGE)};
    unsigned passed = 0, solo_turns = 0;
    Ctl* ctl = o.ctl;
    // All blocks arrive; then thread 0 of each runs `then`, which all threads see the effects of.
    auto barrier = [&](auto then) {
        __syncthreads();
        if (threadIdx.x == 0) {
            passed += gridDim.x;
            asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(&ctl->arrived) : "memory");
            const unsigned want = passed;
            go_s = wait_for(o, &ctl->arrived, want, 0, passed);
            if (go_s) then(state_s);
        }
        __syncthreads();
        return go_s != 0;
    };
    auto end_iteration = [&](State& st) {
        const Slot* s = &ctl->slot[st.slot];
        const unsigned long long count = __ldcg(&s->count), cands = __ldcg(&s->cand);
        next_iteration(st, count, cands, o.cap, max_iterations, SQUARE);
        st.slot = st.slot == 2 ? 0 : st.slot + 1;
    };
    // (The next slot was last read by blocks that have since arrived at another barrier.)
    auto clear_next = [&]() {
        if (blockIdx.x == 0 && threadIdx.x == 0) ctl->slot[state_s.slot == 2 ? 0 : state_s.slot + 1] = Slot{};
    };
    // The block's last tuples and its count of candidates go out with one atomic each (a warp with a
    // tuple or two each would queue on them for longer than a small iteration takes).
    auto end_block = [&](unsigned long long cand) {
        sink.finish();
#pragma unroll
        for (int d = 16; d; d >>= 1) cand += __shfl_xor_sync(FULL, cand, d);
        if (lane == 0) {
            left_s[warp] = sink.staged;
            cand_s[warp] = cand;
        }
        __syncthreads();
        if (warp == 0) {
            const unsigned mine = left_s[lane];
            unsigned incl = mine;
            unsigned long long c = cand_s[lane], at = 0;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const unsigned x = __shfl_up_sync(FULL, incl, d);
                if (lane >= (unsigned)d) incl += x;
            }
#pragma unroll
            for (int d = 16; d; d >>= 1) c += __shfl_xor_sync(FULL, c, d);
            const unsigned total = __shfl_sync(FULL, incl, 31);
            if (lane == 0) {
                if (total) at = atomicAdd(&sink.slot->count, (unsigned long long)total);
                if (c) atomicAdd(&sink.slot->cand, c);
            }
            cand_s[lane] = sink.base + __shfl_sync(FULL, at, 0) + incl - mine;
        }
        __syncthreads();
        sink.write_left(cand_s[warp]);
    };
    static_assert(DL_WARPS == 32, "end_block adds up one value a lane");
    if (threadIdx.x == 0) {
        const Ctl* c = ctl;
        state_s = State{__ldcg(&c->start), __ldcg(&c->end), __ldcg(&c->iterations), __ldcg(&c->candidates), __ldcg(&c->phase), __ldcg(&c->check), 0, __ldcg(&c->fix) != 0, false};
    }
    __syncthreads();
    for (;;) {
        const unsigned phase = state_s.phase;
        const uint64_t start = state_s.start, n = state_s.end - state_s.start;
        const bool check = state_s.check != 0;
        Slot* slot = &ctl->slot[state_s.slot];
        sink.slot = slot;
        sink.base = state_s.end;
        if (phase == PH_DONE) break;
        if (phase == PH_ROWS) {
            clear_next();
            unsigned long long cand = 0;
            const uint64_t warps = (uint64_t)gridDim.x * DL_WARPS, me = (uint64_t)warp * gridDim.x + blockIdx.x;
            if (SQUARE) {
                // A row of a square component can stand for any amount of work, and rows of one hub lie
                // side by side: every warp takes rows far apart, eight at a time.
                unsigned groups = 0;
                for (uint64_t first = me; first < n; first += 8 * warps) {
                    if (++groups % DL_BEAT_GROUPS == 0 && lane == 0) beat(o);
                    const unsigned rows = (unsigned)min((n - first + warps - 1) / warps, (uint64_t)8);
                    const uint64_t row = lane < rows ? o.log[start + first + lane * warps] : 0;
                    unsigned linear = 0;
                    take_rows(o, rules, row, rows, heavy, slot, check, sink, linear);
                    cand += linear;
                    take_square(o, sq, row, rows, sink, cand);
                }
            } else {
                // Few rows per warp while there are few of them; many are taken in batches from a counter
                // (32 at a time, 14 M rows queued on it for longer than their work took).
                const unsigned per = (unsigned)(n >= warps * 32 ? 32 : (n + warps - 1) / warps);
                uint64_t batch = n / (warps * 8) & ~31ull;
                batch = per < 32 ? per : batch < 32 ? 32 : batch > 2048 ? 2048 : batch;
                for (uint64_t at = me * batch; at < n;) {
                    const uint64_t stop = at + batch < n ? at + batch : n;
                    uint64_t row = at + lane < stop ? o.log[start + at + lane] : 0;
                    for (; at < stop; at += per) {
                        const unsigned rows = (unsigned)(stop - at < per ? stop - at : per);
                        const uint64_t next_row = at + per + lane < stop ? o.log[start + at + per + lane] : 0;
                        unsigned linear = 0;
                        take_rows(o, rules, row, rows, heavy, slot, check, sink, linear);
                        cand += linear;
                        row = next_row;
                    }
                    if (n <= warps * batch) break;
                    unsigned next = 0;
                    if (lane == 0) next = atomicAdd(&slot->next_chunk, 1u);
                    at = (warps + __shfl_sync(FULL, next, 0)) * batch;
                }
            }
            end_block(cand);
            if (!barrier([&](State& st) {
                    if (__ldcg(&slot->heavy_n)) st.phase = PH_HEAVY;
                    else end_iteration(st);
                }))
                return;
        } else if (phase == PH_HEAVY) {
            clear_next();
            const uint64_t listed = __ldcg(&slot->heavy_n);
            const unsigned pieces = listed < DL_HEAVY_MAX ? (unsigned)listed : (unsigned)DL_HEAVY_MAX;
            for (;;) {
                unsigned item = 0;
                if (lane == 0) item = atomicAdd(&slot->next_heavy, 1u);
                item = __shfl_sync(FULL, item, 0);
                if (item >= pieces) break;
                Heavy h;
                h.row = __ldcg(&heavy[item].row);
                h.rule = __ldcg(&heavy[item].rule);
                h.piece = __ldcg(&heavy[item].piece);
                take_piece(o, rules, h, check, sink);
            }
            end_block(0);
            if (!barrier(end_iteration)) return;
        } else if (SQUARE && phase == PH_FULL) {
            for (uint64_t i = (uint64_t)blockIdx.x * DL_THREADS + threadIdx.x; i < n; i += (uint64_t)gridDim.x * DL_THREADS) square_full(o, sq, o.log[start + i]);
            if (!barrier([&](State& st) { st.phase = PH_ROWS; })) return;
        } else if (!SQUARE) {  // PH_SOLO
            if (blockIdx.x == 0) {
                State st = state_s;
                if (rules.n == 1 && rules.r[0].joins == 1) solo<true>(o, rules, heavy, slot, max_iterations, stage_s, solo_s, st);
                else solo<false>(o, rules, heavy, slot, max_iterations, stage_s, solo_s, st);
                __syncthreads();
                if (threadIdx.x == 0) {  // everybody again
                    state_s = st;
                    volatile Ctl* v = ctl;
                    v->solo_start = st.start;
                    v->solo_end = st.end;
                    v->solo_iterations = st.iterations;
                    v->solo_candidates = st.candidates;
                    v->solo_phase = st.phase;
                    v->solo_check = st.check;
                    asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(&ctl->solo_turns), "r"(++solo_turns) : "memory");
                }
                __syncthreads();
            } else {
                if (threadIdx.x == 0) {
                    const unsigned want = ++solo_turns;
                    go_s = wait_for(o, &ctl->solo_turns, want, 100, passed);
                    state_s.start = __ldcg(&ctl->solo_start);
                    state_s.end = __ldcg(&ctl->solo_end);
                    state_s.iterations = __ldcg(&ctl->solo_iterations);
                    state_s.candidates = __ldcg(&ctl->solo_candidates);
                    state_s.phase = __ldcg(&ctl->solo_phase);
                    state_s.check = __ldcg(&ctl->solo_check);
                }
                __syncthreads();
                if (!go_s) return;
            }
        }
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        volatile Ctl* v = ctl;
        v->tail = state_s.end;
        v->start = state_s.start;
        v->end = state_s.end;
        v->iterations = state_s.iterations;
        v->candidates = state_s.candidates;
        v->fix = state_s.fix;
        v->overflow = state_s.overflow;
        v->check = state_s.check;
    }
}

__device__ __forceinline__ void flush(const Out& o, const uint64_t* stage, unsigned& staged) {
    if (!staged) return;
    unsigned long long at = 0;
    if (lane_id() == 0) at = atomicAdd(&o.ctl->tail, (unsigned long long)staged);
    at = __shfl_sync(FULL, at, 0);
    __syncwarp();
    for (unsigned i = lane_id(); i < staged; i += 32)
        if (at + i < o.cap) o.log[at + i] = stage[i];
    __syncwarp();
    staged = 0;
}
__device__ __forceinline__ void ready(Ctl* ctl, bool square) {
    volatile Ctl* c = ctl;
    const unsigned long long n = c->tail;
    c->check = 1;
    c->start = 0;
    c->end = n;
    c->iterations = n == 0 ? 1 : 0;  // an iteration over nothing finds nothing
    c->fix = n == 0 ? 1 : 0;
    c->phase = n == 0 ? PH_DONE : square ? PH_FULL : PH_ROWS;  // (never solo: a block that starts late would miss it)
}
// Rows of a bag into the head: new ones (their bit was clear) are appended to the log, where there is one.
__global__ void __launch_bounds__(BLOCK) delta_seed_k(const uint64_t* __restrict__ rows, uint64_t n, const __grid_constant__ Out o, bool square) {
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
        if (!o.log) continue;
        const unsigned b = __ballot_sync(FULL, on);
        if (on) stage[staged + __popc(b & lanemask_lt())] = k;
        staged += __popc(b);
        __syncwarp();
        if (staged > 32) flush(o, stage, staged);
    }
    flush(o, stage, staged);
    // the block that finishes last leaves the loop ready to start on what has been seeded so far
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        if (atomicAdd(&o.ctl->arrived, 1u) == gridDim.x - 1) {
            __threadfence();
            o.ctl->arrived = 0;
            ready(o.ctl, square);
        }
    }
}

__global__ void delta_begin_k(Ctl* c, bool square) { ready(c, square); }

// On with the delta at hand, once the log has the room for it.
__global__ void delta_resume_k(Ctl* c, uint64_t max_iterations, bool square) {
    c->overflow = 0;
    c->arrived = 0;
    c->solo_turns = 0;
    for (int k = 0; k < 3; ++k) c->slot[k] = Slot{};
    c->phase = c->iterations >= max_iterations ? PH_DONE : square ? PH_FULL : PH_ROWS;
}

// ---- rules that keep a column: a block (one warp or a few) for each value of it
// Where every rule hands the head's first column on and joins on the second (a closure: reach(x, z) :-
// reach(x, y), edge(y, z)), what is derived for one x depends on nothing derived for another.  A
// block takes an x, holds its row of the head's bitmap and the frontier of its search in shared memory and
// goes level by level to the end: no barrier between blocks, no atomics and no log in global memory.
// Its levels are the iterations of the loop, and its candidates the loop's.  Instructions one after the
// other bound it (issue slots 68 % used on 2000 nodes of degree 5; 20 % on a chain, where one warp of four has
// something to do), not memory: hence several warps a row where rows are few, four outputs a
// lane in flight, and a path of its own for a frontier of one value.  (Loop -> this, B200: chain of 1500
// nodes 3279 -> 498 us (70 with `walk`), banded DAG of 2^14 nodes 961 -> 472, 2000 nodes of degree 5 276 -> 113, four
// blocks of 128 nodes 181 -> 66; one warp a row with one output a lane in flight: 1089, 1238, 185, 698.)
//   What a block is too slow for is left to the loop: a row is given up when its frontier outgrows its
// queue, or when it is long and most blocks have nothing left to do; its seeds are all that remains
// of it.  Once a quarter of the blocks have given one up, the rest of the rows are not tried.
constexpr int RW_UNROLL = 4;
constexpr int RW_BITS_MIN = 5, RW_BITS_MAX = 16;  // of the second column: a row is whole words, a value 16 bits
constexpr unsigned RW_QUEUE = 16384;              // values the frontier of a row may hold (and the row's seeds)
constexpr unsigned RW_LONG = 16384;               // candidates of a warp (some 50 us) from which a row may be given up
constexpr unsigned RW_UNITED = 4;                 // words of rows of bits that take as long as a candidate (counted by their candidates, rows were given up long before they took long: band of 2000 nodes of degree 66 876 us, now 280; by matches 732)
constexpr unsigned RW_LIST = 64;                  // a value with so many matches is a warp's work by itself
constexpr unsigned RW_FOLLOW = 32, RW_PATH = 96;  // levels of one value each after which a row is taken for a path, and entries of the table for each
constexpr int RW_LISTS_BITS = 11;                 // values whose matches are taken as rows of bits: at most 64 words
constexpr uint64_t RW_LISTS_MIN = 1u << 13;       // rows of the relation below which the copy costs what it saves (four blocks of 44 nodes, 7744 rows: 162 us by matches, 165 by rows; of 46 162 and 162; of 80 205 and 192)
constexpr unsigned RW_SQUARED = 16;               // entries a thread of the path's table
struct RowsShape {
    unsigned rows, words;  // rows of the bitmap, words of each
    unsigned queue;        // entries, a power of two
    unsigned chunk;        // rows taken at a time
    const unsigned* lists;  // the relation as rows of bits like the head's, or null
};
constexpr unsigned rows_queue(int bits) { return 1u << bits < RW_QUEUE ? 1u << bits : RW_QUEUE; }
constexpr unsigned rows_bytes(int bits) { return (1u << bits) / 8 + rows_queue(bits) * 2; }
struct RowsShared {
    unsigned head, tail;  // of the queue's ring; the tail counts the row's tuples
    unsigned failed, next;
    unsigned long long level, cand, tuples, cands, levels;
};
__device__ __forceinline__ unsigned warp_sum_before(unsigned mine, unsigned* total) {
    unsigned incl = mine;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const unsigned v = __shfl_up_sync(FULL, incl, d);
        if (lane_id() >= (unsigned)d) incl += v;
    }
    *total = __shfl_sync(FULL, incl, 31);
    return incl - mine;
}
template <int W>
struct RowsWarp {
    unsigned* seen;
    unsigned short* queue;
    uint2* match;  // of the warp's 32 values: start, length
    RowsShared* sh;
    unsigned mask, head;

    // New values among z join the row and the queue.
    template <int N>
    __device__ __forceinline__ void offer(const Out& o, const uint32_t (&z)[N], bool (&on)[N]) {
        unsigned word[N];
        bool any = false, bad = false;
#pragma unroll
        for (int u = 0; u < N; ++u) {
            bad |= on[u] && z[u] >> o.lo_bits;
            on[u] = on[u] && !(z[u] >> o.lo_bits);
            word[u] = on[u] ? seen[z[u] >> 5] : ~0u;  // (a look first: most are known, and many lanes share a word)
        }
#pragma unroll
        for (int u = 0; u < N; ++u) {
            on[u] = on[u] && !((word[u] >> (z[u] & 31)) & 1u);
            any |= on[u];
        }
        if (bad) set_status(o.st, XLB_ERR_CAPACITY, 22, z[0]);  // outside the domain the host derived
        if (!__any_sync(FULL, any)) return;
#pragma unroll
        for (int u = 0; u < N; ++u)
            if (on[u]) word[u] = atomicOr(&seen[z[u] >> 5], 1u << (z[u] & 31));
        unsigned b[N], count = 0;
#pragma unroll
        for (int u = 0; u < N; ++u) {
            on[u] = on[u] && !((word[u] >> (z[u] & 31)) & 1u);
            b[u] = __ballot_sync(FULL, on[u]);
            count += __popc(b[u]);
        }
        if (!count) return;
        unsigned to = 0;
        if (lane_id() == 0) to = atomicAdd(&sh->tail, count);
        to = __shfl_sync(FULL, to, 0);
        if (to + count - head > mask + 1) {  // (the level at hand is still in the ring)
            if (lane_id() == 0) sh->failed = 1;
            return;
        }
#pragma unroll
        for (int u = 0; u < N; ++u) {
            if (on[u]) queue[(to + __popc(b[u] & lanemask_lt())) & mask] = (unsigned short)z[u];
            to += __popc(b[u]);
        }
    }
    // The matches [at, at + len) of one value.
    __device__ __forceinline__ void list(const Out& o, const Ix& ix, uint32_t at, uint32_t len) {
        for (uint32_t base = 0; base < len; base += 32 * RW_UNROLL) {
            uint32_t z[RW_UNROLL];
            bool on[RW_UNROLL];
#pragma unroll
            for (int u = 0; u < RW_UNROLL; ++u) {
                const uint32_t t = base + u * 32 + lane_id();
                on[u] = t < len;
                z[u] = other_of(ix, at + (on[u] ? t : 0u));
            }
            offer(o, z, on);
        }
    }
    // `total` matches of the lanes' values, dealt out evenly; lanes below m have some, lane's first is output `before`.
    template <int N>
    __device__ __forceinline__ void dealt(const Out& o, const Ix& ix, uint32_t from, uint32_t total, unsigned m, uint32_t before, uint32_t shift) {
        const unsigned lane = lane_id();
        uint32_t z[N];
        bool on[N];
#pragma unroll
        for (int u = 0; u < N; ++u) {
            const uint32_t base = from + u * 32, t = base + lane, d = before - base;
            const unsigned starts = __reduce_or_sync(FULL, lane < m && before >= base && d < 32 ? 1u << d : 0u);
            // the last lane whose outputs start at or before t
            const unsigned owner = __popc(__ballot_sync(FULL, lane < m && before < base)) + __popc(starts & (lanemask_lt() | (1u << lane))) - 1;
            const uint32_t at = __shfl_sync(FULL, shift, owner) + t;
            on[u] = t < total;
            z[u] = other_of(ix, on[u] ? at : 0u);
        }
        offer(o, z, on);
    }
    // All matches of up to 32 values by one rule; their number.
    __device__ __forceinline__ uint32_t expand(const Out& o, const Ix& ix, bool on, unsigned y) {
        const unsigned lane = lane_id();
        uint32_t start = 0, len = 0;
        if (on) find(ix, y, start, len);
        uint32_t all = 0;
        for (unsigned far = __ballot_sync(FULL, len >= RW_LIST); far; far &= far - 1) {
            const uint32_t n = __shfl_sync(FULL, len, __ffs(far) - 1);
            list(o, ix, __shfl_sync(FULL, start, __ffs(far) - 1), n);
            all += n;
        }
        if (len >= RW_LIST) len = 0;
        const unsigned some = __ballot_sync(FULL, len != 0), m = __popc(some);
        if (!some) return all;
        if (some & (some + 1)) {  // values without matches between others: closed up, so that every lane below m has outputs
            if (len) match[__popc(some & lanemask_lt())] = make_uint2(start, len);
            __syncwarp();
            const uint2 p = lane < m ? match[lane] : make_uint2(0, 0);
            __syncwarp();
            start = p.x;
            len = p.y;
        }
        uint32_t incl = len;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t v = __shfl_up_sync(FULL, incl, d);
            if (lane >= (unsigned)d) incl += v;
        }
        const uint32_t total = __shfl_sync(FULL, incl, 31), before = incl - len, shift = start - before;
        uint32_t from = 0;
        for (; total - from > 64; from += 32 * RW_UNROLL) {
            dealt<RW_UNROLL>(o, ix, from, total, m, before, shift);
            if (total - from <= 32 * RW_UNROLL) return all + total;
        }
        for (; from < total; from += 32) dealt<1>(o, ix, from, total, m, before, shift);
        return all + total;
    }
    // All matches of up to 32 values [at, at + m) of the queue, as rows of bits: a row is `words` (at most 64) of them, and
    // narrow rows are taken several at a time.
    __device__ __forceinline__ void unite(const unsigned* __restrict__ rows, unsigned n_rows, unsigned words, unsigned at, unsigned m) {
        const unsigned lane = lane_id(), side = words < 32 ? 32 / words : 1, mine = words < 32 ? lane / words : 0;
        const unsigned w = lane & (min(words, 32u) - 1);
        constexpr unsigned N = 8;
        unsigned acc[2] = {0, 0};
        for (unsigned j0 = mine; j0 - mine < m; j0 += N * side) {
            unsigned v[N][2];
#pragma unroll
            for (unsigned u = 0; u < N; ++u) {
                const unsigned y = j0 + u * side < m ? queue[(at + j0 + u * side) & mask] : ~0u;
                const bool on = y < n_rows;
                v[u][0] = on ? __ldg(&rows[y * words + w]) : 0u;
                v[u][1] = on && words > 32 ? __ldg(&rows[y * words + 32 + w]) : 0u;
            }
#pragma unroll
            for (unsigned u = 0; u < N; ++u) {
                acc[0] |= v[u][0];
                acc[1] |= v[u][1];
            }
        }
        for (unsigned d = words; d < 32; d *= 2) acc[0] |= __shfl_xor_sync(FULL, acc[0], d);
        unsigned count = 0, all;
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            if (lane != w) acc[k] = 0;  // (the lanes beside hold the same; a second word there is only of rows of 64)
            if (acc[k] && acc[k] & ~seen[w + 32 * k]) acc[k] &= ~atomicOr(&seen[w + 32 * k], acc[k]);
            else acc[k] = 0;
            count += __popc(acc[k]);
        }
        const unsigned before = warp_sum_before(count, &all);
        if (!all) return;
        unsigned to = 0;
        if (lane == 0) to = atomicAdd(&sh->tail, all);
        to = __shfl_sync(FULL, to, 0);
        if (to + all - head > mask + 1) {  // (the level at hand is still in the ring)
            if (lane == 0) sh->failed = 1;
            return;
        }
        to += before;
#pragma unroll
        for (int k = 0; k < 2; ++k)
            for (unsigned x = acc[k]; x; x &= x - 1, ++to) queue[to & mask] = (unsigned short)((w + 32 * k) * 32 + __ffs(x) - 1);
    }
    // A frontier of one value, followed by one warp while it stays one, for at most `most` levels: a value's
    // matches are looked up while the test whether it is new is under way.  Leaves the ring's ends and the
    // level in `sh`.
    __device__ __forceinline__ void follow(const Out& o, const Ix& ix, uint64_t max_iterations, unsigned most) {
        const unsigned lane = lane_id();
        unsigned at = sh->head, y = queue[at & mask];
        uint64_t cand = 0;
        uint32_t start, len;
        find(ix, y, start, len);
        const unsigned levels = (unsigned)min((unsigned long long)(max_iterations - sh->level), (unsigned long long)most);
        unsigned more = 1, done = 0;  // values in the frontier; levels done
        while (done < levels && len <= 32) {
            ++done;
            cand += len;
            bool fresh = lane < len;
            const uint32_t z = other_of(ix, fresh ? start + lane : 0u);
            if (fresh && z >> o.lo_bits) {
                set_status(o.st, XLB_ERR_CAPACITY, 22, z);
                fresh = false;
            }
            uint32_t next = 0, next_len = 0;
            unsigned word = ~0u;
            if (fresh) {
                word = seen[z >> 5];
                find(ix, z, next, next_len);
            }
            const unsigned bit = 1u << (z & 31);
            fresh = fresh && !(word & bit);
            unsigned b = __ballot_sync(FULL, fresh);
            if (b & (b - 1)) {  // several (or one more than once)
                if (fresh) fresh = !(atomicOr(&seen[z >> 5], bit) & bit);
                b = __ballot_sync(FULL, fresh);
                more = __popc(b);
                if (more > 1) {
                    const unsigned to = at + 1 + __popc(b & lanemask_lt());
                    if (fresh) queue[to & mask] = (unsigned short)z;  // (32 at most, and the one they came from is done with)
                    break;
                }
            } else if (fresh) seen[z >> 5] = word | bit;
            if (!b) {
                more = 0;
                break;
            }
            const unsigned from = __ffs(b) - 1;
            y = __shfl_sync(FULL, z, from);
            start = __shfl_sync(FULL, next, from);
            len = __shfl_sync(FULL, next_len, from);
            ++at;
            __syncwarp();
        }
        __syncwarp();
        if (lane == 0) {
            const bool still = more == 1;  // one value, not looked at yet
            if (still) queue[at & mask] = (unsigned short)y;
            sh->head = still ? at : at + 1;
            sh->tail = still ? at + 1 : at + 1 + more;
            sh->level += done;
            sh->cand += cand;
        }
    }
    // A path that has been followed for a while, by the whole block: the ring, which holds one value then, becomes
    // a table of every value's only match.  Squared five times over it leads 32 matches on, and 32 lanes of one
    // warp, which start on matches that follow one another, go down the path side by side: 32 levels for a
    // look-up of the table and of the row's bits.  (A value a lane is squared in registers; where the
    // table has more, one lane goes alone.)  Ends where a value has no or several matches (its level is not done),
    // where a value is known, or at the limit.  What bounds `follow` is some 600 cycles of dependent instructions a
    // level, one warp an SM partition; here 32 levels share them (chain of 1500 nodes, the whole kernel: 484 us
    // with `follow` alone, 135 with one lane on the table, 70 with 32).  Making the table takes what 40 levels of `follow` do,
    // with more values more: a path with a twig after every 40 of 7000 nodes, each of which ended a walk of eight
    // levels, took 22.0 ms, 8.1 now that a row whose walk was cut short is followed further before its next (7.9 by
    // `follow` alone); paths of 80 nodes, 8000 in all, 297 us, 222 since more values want more levels (217 by `follow` alone).
    __device__ __forceinline__ void walk(const Out& o, const Ix& ix, uint64_t max_iterations) {
        constexpr unsigned short STOP = 0xFFFF;  // (no value: the ring has fewer entries)
        const unsigned lane = lane_id(), at = sh->head, values = 1u << o.lo_bits;
        unsigned y = queue[at & mask];
        __syncthreads();
        constexpr unsigned N = 8;  // values a thread looks up together
        for (unsigned v0 = threadIdx.x; v0 < values; v0 += N * W * 32) {
            uint32_t start[N], len[N];
#pragma unroll
            for (unsigned u = 0; u < N; ++u) {
                start[u] = len[u] = 0;
                if (v0 + u * W * 32 < values) find(ix, v0 + u * W * 32, start[u], len[u]);
            }
#pragma unroll
            for (unsigned u = 0; u < N; ++u) start[u] = len[u] == 1 ? other_of(ix, start[u]) : ~0u;
#pragma unroll
            for (unsigned u = 0; u < N; ++u)
                if (v0 + u * W * 32 < values) queue[v0 + u * W * 32] = start[u] >> o.lo_bits ? STOP : (unsigned short)start[u];  // (a match outside the domain is left to the other paths to report)
        }
        __syncthreads();
        const unsigned width = values <= RW_SQUARED * W * 32 ? 32 : 1;
        unsigned z = queue[y];  // lane l's: the match l + 1 steps on
        for (unsigned k = 1; k < width; k *= 2) {
            const unsigned from = __shfl_up_sync(FULL, z, k);
            if (lane >= k && lane < 2 * k) z = from == STOP ? STOP : queue[from];
            unsigned short twice[RW_SQUARED];
#pragma unroll
            for (int i = 0; i < (int)RW_SQUARED; ++i) {
                const unsigned v = threadIdx.x + i * W * 32, next = v < values ? queue[v] : STOP;
                twice[i] = next == STOP ? STOP : queue[next];
            }
            __syncthreads();
#pragma unroll
            for (int i = 0; i < (int)RW_SQUARED; ++i)
                if (threadIdx.x + i * W * 32 < values) queue[threadIdx.x + i * W * 32] = twice[i];
            __syncthreads();
        }
        if (threadIdx.x >= 32) return;
        const unsigned levels = (unsigned)min((unsigned long long)(max_iterations - sh->level), 0xFFFFFFFFull);
        unsigned done = 0;
        bool known = false;
        for (;;) {
            const bool here = z != STOP && lane < width && lane < levels - done;
            const unsigned word = here ? seen[z >> 5] : 0u, next = here ? queue[z] : STOP, bit = 1u << (z & 31);
            const unsigned before = __match_any_sync(FULL, z) & lanemask_lt();  // a loop shorter than the warp is wide
            const unsigned ends = __ballot_sync(FULL, !here), old = __ballot_sync(FULL, here && ((word & bit) || before));
            const unsigned count = min(ends ? __ffs(ends) - 1 : 32, old ? __ffs(old) - 1 : 32);
            if (lane < count) atomicOr(&seen[z >> 5], bit);
            if (count) y = __shfl_sync(FULL, z, count - 1);
            done += count;
            if (count < width) {
                known = (old >> count) & 1;
                break;
            }
            z = next;
            __syncwarp();
        }
        if (lane) return;
        // (as many tuples as levels, but for the level that ended on a known value; y is in the frontier unless there was one)
        const unsigned to = at + done;
        done += known ? 1 : 0;
        if (!known) queue[to & mask] = (unsigned short)y;
        sh->head = known ? to + 1 : to;
        sh->tail = to + 1;
        sh->level += done;
        sh->cand += done;
    }
};
// The seeds of a row that is given up, for the loop.
__device__ __noinline__ void rows_give_up(const Out& o, const RowsShape& sh, unsigned row) {
    for (unsigned at = threadIdx.x; at < sh.words; at += blockDim.x) {
        unsigned word = o.visited[(uint64_t)row * sh.words + at];
        if (!word) continue;
        unsigned long long to = atomicAdd(&o.ctl->rows_seeds, (unsigned long long)__popc(word));
        for (; word; word &= word - 1, ++to)
            if (to < o.cap) o.log[to] = ((uint64_t)row << 32) | (at * 32 + __ffs(word) - 1);
    }
    if (threadIdx.x == 0) atomicAdd(&o.ctl->rows_given_up, 1ull);
}
template <int W>
__global__ void __launch_bounds__(W * 32) delta_rows_k(const __grid_constant__ Out o, const __grid_constant__ Rules rules, const __grid_constant__ RowsShape sh, uint64_t max_iterations) {
    extern __shared__ __align__(16) unsigned char rw_smem[];
    __shared__ RowsShared s;
    __shared__ uint2 match_s[W][32];
    const unsigned lane = lane_id(), warp = threadIdx.x >> 5;
    RowsWarp<W> w;
    w.seen = reinterpret_cast<unsigned*>(rw_smem);
    w.queue = reinterpret_cast<unsigned short*>(w.seen + sh.words);
    w.match = match_s[warp];
    w.sh = &s;
    w.mask = sh.queue - 1;
    volatile RowsShared* v = &s;
    Ctl* ctl = o.ctl;
    if (threadIdx.x == 0) s.tuples = s.cands = s.levels = 0;
    bool left = false;
    for (uint64_t chunk = blockIdx.x;;) {
        const uint64_t first = chunk * sh.chunk;
        if (first >= sh.rows) break;
        if (threadIdx.x == 0) s.next = *(volatile unsigned long long*)&ctl->rows_given_up * 4 <= gridDim.x;
        __syncthreads();
        const bool tried = v->next;
        for (unsigned row = (unsigned)first; row < sh.rows && row < first + sh.chunk; ++row) {
            // the row's bits and the queue they start
            unsigned mine = 0;
            for (unsigned at = threadIdx.x; at < sh.words; at += W * 32) {
                const unsigned word = o.visited[(uint64_t)row * sh.words + at];
                w.seen[at] = word;
                mine += __popc(word);
            }
            if (threadIdx.x == 0) {
                s.head = s.tail = s.failed = 0;
                s.level = s.cand = 0;
            }
            const int any = __syncthreads_or(mine != 0);
            if (!any) continue;
            if (mine) {
                unsigned to = atomicAdd(&s.tail, mine);
                for (unsigned at = threadIdx.x; at < sh.words; at += W * 32)
                    for (unsigned word = w.seen[at]; word; word &= word - 1, ++to)
                        if (to < sh.queue) w.queue[to] = (unsigned short)(at * 32 + __ffs(word) - 1);
            }
            __syncthreads();
            unsigned head = 0, end = v->tail;
            __syncthreads();  // (read by all before a warp adds to it)
            bool ok = tried && end <= sh.queue;
            uint64_t level = 0, cand = 0;
            int patience = RW_LONG;  // candidates (or what takes as long) until it is asked whether the others are done
            const unsigned least = max(RW_FOLLOW, sh.queue / RW_PATH);
            unsigned path = least;  // levels of one value each after which the row is taken for a path
            while (ok && head != end && level < max_iterations) {
                if (end - head == 1 && rules.n == 1) {
                    const bool table = sh.queue >> o.lo_bits;  // the ring has an entry for every value
                    const unsigned from = head;
                    if (warp == 0) w.follow(o, rules.r[0].ix[0], max_iterations, table ? path : ~0u);
                    __syncthreads();
                    head = v->head;
                    end = v->tail;
                    if (table && head - from == path && end - head == 1) {
                        w.walk(o, rules.r[0].ix[0], max_iterations);
                        __syncthreads();
                        head = v->head;
                        end = v->tail;
                        path = head - from < least * 9 / 4 ? 2 * path : least;  // (a short one, as the next may be: later)
                    }
                    level = v->level;
                    __syncthreads();
                    if (head == end || level >= max_iterations) break;
                }
                ++level;
                w.head = head;
                const unsigned per = min(32u, (end - head + W - 1) / W);
                for (unsigned at = head + warp * per; at - head < end - head; at += W * per) {
                    const bool on = lane < per && end - at > lane;
                    const unsigned y = on ? w.queue[(at + lane) & w.mask] : 0u;
                    if (sh.lists) {
                        uint32_t start = 0, len = 0;
                        if (on) find(rules.r[0].ix[0], y, start, len);
                        const unsigned all = __reduce_add_sync(FULL, len), m = min(per, end - at);
                        cand += all;
                        if (all) {
                            patience -= (int)(m * sh.words / RW_UNITED);
                            w.unite(sh.lists, sh.rows, sh.words, at, m);
                        }
                    } else
                        for (int q = 0; q < rules.n; ++q) {
                            const uint32_t all = w.expand(o, rules.r[q].ix[0], on, y);
                            cand += all;
                            patience -= (int)min(all, 1u << 20);
                        }
                    if (patience < 0) {
                        patience = 4096;
                        if (lane == 0 && *(volatile unsigned*)&ctl->rows_idle * 4ull > gridDim.x * 3ull) s.failed = 1;
                    }
                    if (__any_sync(FULL, v->failed)) break;
                }
                __syncthreads();
                head = end;
                end = v->tail;
                ok = !v->failed;
                if (threadIdx.x == 0) {
                    s.head = head;
                    s.level = level;
                }
                __syncthreads();
            }
            if (!ok) {
                rows_give_up(o, sh, row);
                __syncthreads();
                continue;
            }
            if (lane == 0) atomicAdd(&s.cand, (unsigned long long)cand);
            for (unsigned at = threadIdx.x; at < sh.words; at += W * 32) o.visited[(uint64_t)row * sh.words + at] = w.seen[at];
            left |= head != end;
            __syncthreads();
            if (threadIdx.x == 0) {
                s.tuples += end;
                s.cands += s.cand;
                s.levels = level > s.levels ? level : s.levels;
            }
            __syncthreads();
        }
        __syncthreads();
        if (threadIdx.x == 0) s.next = atomicAdd(&ctl->rows_ticket, 1u);
        __syncthreads();
        chunk = (uint64_t)gridDim.x + v->next;
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        atomicAdd(&ctl->rows_idle, 1u);
        if (s.levels) {
            atomicAdd(&ctl->rows_tuples, s.tuples);
            atomicAdd(&ctl->rows_candidates, s.cands);
            if (*(volatile unsigned long long*)&ctl->rows_levels < s.levels) atomicMax(&ctl->rows_levels, s.levels);
        }
        if (left) ctl->rows_left = 1;
    }
}
// ---- rules that take the head's columns apart: bit rows
// Where each rule leads a delta row's first column through one stored relation (or none) to the new first column,
// and its second through another to the new second (same generation: sg(X, Y) :- edge(A, X), sg(A, B),
// edge(B, Y)), an iteration is two products with sparse matrices: new = A^T delta B.  A block owns every
// 148th row.  It takes its rows of the delta as bits, leads the bits through B into rows in shared memory, and ORs
// those into the rows that A leads to; what they gain over the head is found by their own block in the next
// iteration.  A tuple so costs no atomic in global memory, no entry in a log and no look at a word of its
// own: same generation over 7001 nodes (26.8 M tuples) took 718 us in the loop, bound by its atomics on single
// bits, 282 with a warp for each row (five rows in seven have nothing to lead to), and takes 180 here: a phase is
// some 20 K cycles of dependent steps between two barriers, then atomics on words of shared memory (what neighbours
// lead to shares words; setting a lane's bits of one word together cost more than it saved).
//   Rows that nobody reached are passed over by a stamp.  Lists of A are shared out among a block's warps only: where one
// is longer than BT_ROWS, the loop does it all.  A fixpoint whose iterations come out cheaper there is handed to the
// loop, whose small ones meet at no barrier.
constexpr int BT_BITS_MIN = 5, BT_BITS_MAX = 13;
constexpr int BT_BITS_BOTH = 20;                    // of both columns: below, the loop is as fast (same generation over 300 and 511 nodes 139 and 149 us of device time by the loop, 155 and 161 here; 1023 nodes 195 and 166)
constexpr unsigned BT_WORDS = 1u << (BT_BITS_MAX - 5);
constexpr unsigned BT_OWN = 56;                     // rows of a block
constexpr unsigned BT_LIST = 16;                    // a value with more matches is a whole warp's work
constexpr unsigned BT_ROWS = 1024;                  // rows that a row may lead to; where the head has more than four times as many, a quarter of those (7000 nodes of degree 2 and 2000 more into one: 2.39 ms by the loop, 2.02; 4000 into one 2.48 and 3.67; 2000 nodes and 1900 into one 0.72 and 0.85)
// What an iteration takes beside what it would take the loop, counted in candidates of the loop (80 a ns).  One of next
// to nothing took 1.4 us more with heads of 11 bits a column, 1.7 with 12 and 4 to 11 with 13: the rows every block looks
// through.  Then a word a lane of every place.  Going on in the loop costs some 40 us.
constexpr float BT_FIXED = 80e3f, BT_MAP = 0.16f, BT_WORD = 1 / 16.f, BT_CHANGE = 3200e3f;
// Seeds, times the matches of a value, a row of the head has to have for bit rows to be begun.  Same generation over
// trees has 1.8 to 3.6 (gains of 1.2 to 2.6 x), 2000 nodes of degree 2 3.8 (338 us by the loop, 252), of degree 1.1
// 1.15 (262 and 302; 8000 nodes 690 and 865), a path 1 or less (8000 nodes 38 and 72 ms), 5 values led on by a relation of
// 10^6 rows 0.07 (207 and 622), 3000 of them 45 (16.0 and 1.1 ms).
constexpr double BT_SEEDS = 1.5;
constexpr unsigned BT_SCANNED = 1u << 14;           // rows of A that every block looks through, for the rows that only one leads to (more: none is taken for such a row)
constexpr unsigned BT_LISTED = 16384;               // rows of the stored relation whose lists a block keeps in shared memory
constexpr unsigned BT_SMEM = ((DL_RULES + 2) * BT_WORDS + 2 * BT_OWN * BT_WORDS + DL_WARPS * 256 + (1u << BT_BITS_MAX)) * 4 + BT_LISTED * 2;
static_assert(BT_SMEM <= (222u << 10), "a block an SM");
struct BitsRule {
    Ix a, b;
    bool a_list, b_list;
    unsigned listed;  // rows of B's index, if it is the one kept in shared memory
    unsigned a_rows;  // of A's
};
struct BitsRules {
    BitsRule r[DL_RULES];
    int n;
};
struct Bits {
    unsigned *next[2], *stamp[2];  // what rows are reached by in this iteration and the next; rows that are
    unsigned rows, words;          // of the head's bitmap, words of each
};
struct Active {  // a row of the delta that A leads on: the block's k-th, its list, the entries of those before it
    unsigned k;
    uint32_t at, len, before;
};
struct BitsState {
    unsigned long long tuples, cands, pending, iterations;
    float regret, before;  // time lost to the loop so far, in its candidates; tuples of the iteration before
    unsigned slot, leaving, over, fix, go;
    // Whether the loop should go on, after an iteration of so many tuples, candidates and words written (of `all` there
    // can be; the head's bitmap has `map`).  Looks two iterations ahead by the growth of this one: a few seeds may be about to fill the head.
    __device__ __forceinline__ bool leave(float found, float cand, float words, float all, float map) {
        const float fixed = BT_FIXED + map * BT_MAP, growth = iterations ? found / fmaxf(before, 1.f) : cand / fmaxf(found, 1.f);
        regret = fmaxf(0.f, regret + fixed + words * BT_WORD - cand);
        before = found;
        return regret >= BT_CHANGE && fixed + fminf(words * growth, all) * BT_WORD > cand * growth * fmaxf(growth, 1.f);
    }
};
// B as a block keeps it: per value its matches' start and number, and the matches.
struct Lists {
    const unsigned* at;
    const unsigned short* other;
};
// Up to 16 words of a row led through B: where `word` (lane's own, of values from `first` on) has bits, their matches
// are set in `led`.  Their number, lane by lane.
template <bool KEPT>
__device__ __forceinline__ unsigned lead(const Out& o, const Ix& ix, const Lists& kept, unsigned word, unsigned first, unsigned short* queue, unsigned* led) {
    const unsigned lane = lane_id();
    unsigned n, c = 0;
    unsigned to = warp_sum_before(__popc(word), &n);
    if (!n) return 0;
    for (; word; word &= word - 1) queue[to++] = (unsigned short)(first + __ffs(word) - 1);
    __syncwarp();
    auto other = [&](uint32_t at) { return KEPT ? (uint32_t)kept.other[at] : other_of(ix, at); };
    auto mark = [&](uint32_t v) {
        if (v >> o.lo_bits) set_status(o.st, XLB_ERR_CAPACITY, 18, v);
        else atomicOr(&led[v >> 5], 1u << (v & 31));
    };
    for (unsigned base = 0; base < n; base += 64) {  // two values a lane, so that their look-ups are under way together
        uint32_t s[2], len[2];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const unsigned i = base + u * 32 + lane;
            s[u] = len[u] = 0;
            if (i >= n) continue;
            if (KEPT) {
                const unsigned p = kept.at[queue[i]];
                s[u] = p & 0xFFFF;
                len[u] = p >> 16;
            } else find(ix, queue[i], s[u], len[u]);
        }
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            c += len[u];
            for (unsigned far = __ballot_sync(FULL, len[u] > BT_LIST); far; far &= far - 1) {
                const uint32_t all = __shfl_sync(FULL, len[u], __ffs(far) - 1), from = __shfl_sync(FULL, s[u], __ffs(far) - 1);
                for (uint32_t j = lane; j < all; j += 32) mark(other(from + j));
            }
            if (len[u] > BT_LIST) len[u] = 0;
        }
        const unsigned most = __reduce_max_sync(FULL, max(len[0], len[1]));
        for (unsigned j = 0; j < most; j += 4) {
            uint32_t v[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) v[u] = j + (u & 3) < len[u >> 2] ? other(s[u >> 2] + j + (u & 3)) : 0u;
#pragma unroll
            for (int u = 0; u < 8; ++u)
                if (j + (u & 3) < len[u >> 2]) mark(v[u]);
        }
    }
    __syncwarp();
    return c;
}
__global__ void __launch_bounds__(DL_THREADS, 1) delta_bits_k(const __grid_constant__ Out o, const __grid_constant__ BitsRules rules, const __grid_constant__ Bits b, uint64_t max_iterations) {
    extern __shared__ unsigned bt_smem[];
    __shared__ BitsState st;
    __shared__ unsigned long long sum_s[3];
    __shared__ unsigned total_s[BT_OWN];                    // tuples of the block's rows of the delta
    __shared__ Active act_s[BT_OWN];
    __shared__ unsigned active_s;
    const unsigned lane = lane_id(), warp = threadIdx.x >> 5, W = b.words;
    constexpr int N = BT_WORDS / 32;
    unsigned* has = bt_smem;                                // per rule, the values that B leads anywhere
    unsigned* rows_s = has + DL_RULES * BT_WORDS;           // the block's rows of the delta ...
    unsigned* led_s = rows_s + BT_OWN * BT_WORDS;           // ... and what B leads them to
    unsigned* once_s = led_s + BT_OWN * BT_WORDS;           // rows that something leads to,
    unsigned* more_s = once_s + BT_WORDS;                   // that several things lead to
    unsigned short* queue = reinterpret_cast<unsigned short*>(more_s + BT_WORDS + warp * 256);
    unsigned* lists_at = more_s + BT_WORDS + DL_WARPS * 256;
    unsigned short* lists_other = reinterpret_cast<unsigned short*>(lists_at + (1u << BT_BITS_MAX));
    const Lists kept{lists_at, lists_other};
    const unsigned own = b.rows > blockIdx.x ? (b.rows - blockIdx.x + gridDim.x - 1) / gridDim.x : 0;
    const unsigned parts = W > 16 ? 31 - __clz(W / 16) : 0;  // a row is led in 2^parts pieces of work
    Ctl* ctl = o.ctl;
    bool bad = false;
    float all_places = 0;
    for (int q = 0; q < rules.n; ++q) all_places += rules.r[q].a_list ? rules.r[q].a_rows : b.rows;
    for (unsigned i = threadIdx.x; i < 2 * BT_WORDS; i += DL_THREADS) once_s[i] = 0;
    __syncthreads();
    for (int q = 0; q < rules.n; ++q) {
        const BitsRule& ru = rules.r[q];
        constexpr int T = (1 << BT_BITS_MAX) / DL_THREADS;  // (their look-ups are under way together)
        uint32_t s[T], len[T];
#pragma unroll
        for (int i = 0; i < T; ++i) {
            const unsigned v = threadIdx.x + i * DL_THREADS;
            s[i] = 0;
            len[i] = v < W * 32 ? 1 : 0;
            if (ru.b_list && v < W * 32) find(ru.b, v, s[i], len[i]);
        }
#pragma unroll
        for (int i = 0; i < T; ++i) {
            const unsigned v = threadIdx.x + i * DL_THREADS, word = __ballot_sync(FULL, len[i] != 0);
            if (v >= W * 32) continue;
            if (ru.listed) lists_at[v] = len[i] ? s[i] | (len[i] << 16) : 0u;
            if (lane == 0) has[q * BT_WORDS + (v >> 5)] = word;
        }
#pragma unroll 4
        for (unsigned i = threadIdx.x; i < ru.listed; i += DL_THREADS) lists_other[i] = (unsigned short)min(other_of(ru.b, i), 0xFFFFu);
        auto leads_to = [&](uint32_t to) {
            if (to < b.rows && (atomicOr(&once_s[to >> 5], 1u << (to & 31)) >> (to & 31) & 1u)) atomicOr(&more_s[to >> 5], 1u << (to & 31));
        };
        if (!ru.a_list) {
            for (unsigned v = threadIdx.x; v < b.rows; v += DL_THREADS) leads_to(v);
            continue;
        }
#pragma unroll
        for (int i = 0; i < T; ++i) {
            const unsigned v = threadIdx.x + i * DL_THREADS;
            len[i] = 0;
            if (v < b.rows) find(ru.a, v, s[i], len[i]);
        }
#pragma unroll
        for (int i = 0; i < T; ++i) bad |= len[i] > max(BT_ROWS, b.rows / 4);
        if (ru.a_rows > BT_SCANNED) {
            for (unsigned i = threadIdx.x; i < BT_WORDS; i += DL_THREADS) more_s[i] = ~0u;
            continue;
        }
#pragma unroll 4
        for (unsigned i = threadIdx.x; i < ru.a_rows; i += DL_THREADS) leads_to(other_of(ru.a, i));
    }
    if (threadIdx.x == 0) st = BitsState{};
    if (__syncthreads_or(bad)) {  // (all blocks find the same)
        if (blockIdx.x == 0 && threadIdx.x == 0) ctl->rows_given_up = 1;
        return;
    }
    unsigned passed = 0;
    for (unsigned phase = 0;; ++phase) {
        const unsigned cur = phase & 1;
        const bool leaving = st.leaving != 0;
        unsigned *next = b.next[cur ^ 1], *reached = b.next[cur];
        Slot* slot = &ctl->slot[st.slot];
        if (threadIdx.x < 3) sum_s[threadIdx.x] = 0;
        if (blockIdx.x == 0 && threadIdx.x == 0) ctl->slot[st.slot == 2 ? 0 : st.slot + 1] = Slot{};
        __syncthreads();
        // the rows of the delta: what they were reached by beyond the head (at first: the seeds)
        bool some = false;
        static_assert(BT_OWN <= 2 * DL_WARPS, "a warp has two rows at most");
        unsigned stamp[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) stamp[i] = warp + i * DL_WARPS < own && phase ? __ldcg(&b.stamp[cur][blockIdx.x + (warp + i * DL_WARPS) * gridDim.x]) : 1u;
        for (unsigned k = warp; k < own; k += DL_WARPS) {
            const unsigned row = blockIdx.x + k * gridDim.x;
            unsigned mine = 0;
            if (stamp[k >= DL_WARPS]) {
                unsigned have[N], r[N];
#pragma unroll
                for (int i = 0; i < N; ++i) {
                    const unsigned w = lane + 32 * i;
                    have[i] = w < W ? __ldcg(&o.visited[(uint64_t)row * W + w]) : 0u;
                    r[i] = w < W && phase ? __ldcg(&reached[(uint64_t)row * W + w]) : 0u;
                }
#pragma unroll
                for (int i = 0; i < N; ++i) {
                    const unsigned w = lane + 32 * i, d = phase ? r[i] & ~have[i] : have[i];
                    if (r[i]) reached[(uint64_t)row * W + w] = 0;
                    if (r[i] & ~have[i]) o.visited[(uint64_t)row * W + w] = have[i] | d;
                    if (w < W) rows_s[k * W + w] = d;
                    mine += __popc(d);
                }
                if (lane == 0) b.stamp[cur][row] = 0;
            }
            const unsigned all = __reduce_add_sync(FULL, mine);
            if (lane == 0) {
                total_s[k] = all;
                if (all) atomicAdd(&sum_s[0], (unsigned long long)all);
            }
            some |= all != 0;
            if (leaving && all) {
                unsigned before;
                before = warp_sum_before(mine, &before);
                unsigned long long to = 0;
                if (lane == 0) to = atomicAdd(&ctl->rows_seeds, (unsigned long long)all);
                to = __shfl_sync(FULL, to, 0) + before;
                __syncwarp();
                for (unsigned w = lane; w < W; w += 32)
                    for (unsigned word = rows_s[k * W + w]; word; word &= word - 1, ++to)
                        if (to < o.cap) o.log[to] = ((uint64_t)row << 32) | (w * 32 + __ffs(word) - 1);
            }
        }
        some = __syncthreads_or(some) && !leaving;
        if (some && threadIdx.x == 0) beat(o);
        unsigned long long cand = 0;
        for (int q = 0; some && q < rules.n; ++q) {
            const BitsRule& ru = rules.r[q];
            if (warp == 0) {  // the rows that A leads anywhere, and how many places those before each are led to
                unsigned rows = 0, places = 0;
                for (unsigned k0 = 0; k0 < own; k0 += 32) {
                    const unsigned k = k0 + lane, all = k < own ? total_s[k] : 0;
                    uint32_t at = 0, len = all ? 1 : 0;
                    if (ru.a_list && all) find(ru.a, blockIdx.x + k * gridDim.x, at, len);
                    if (!ru.b_list) cand += (unsigned long long)all * len;
                    unsigned more;
                    const unsigned before = warp_sum_before(len, &more), some = __ballot_sync(FULL, len != 0);
                    if (len) act_s[rows + __popc(some & lanemask_lt())] = Active{k, at, len, places + before};
                    rows += __popc(some);
                    places += more;
                }
                if (lane == 0) {
                    active_s = rows;
                    sum_s[2] += places;  // (nobody else's until the iteration is over)
                }
            }
            if (ru.b_list)
                for (unsigned i = threadIdx.x; i < own * W; i += DL_THREADS) led_s[i] = 0;
            __syncthreads();
            const unsigned active = active_s;
            if (ru.b_list) {
                for (unsigned i = warp; i < active << parts; i += DL_WARPS) {
                    // (the same part of all rows first: values that lead on may lie in a few parts only)
                    const Active& on = act_s[i % active];
                    const unsigned k = on.k, w = i / active * 16 + lane;
                    const unsigned word = lane < 16 && w < W ? rows_s[k * W + w] & has[q * BT_WORDS + w] : 0u;
                    cand += (unsigned long long)(ru.listed ? lead<true>(o, ru.b, kept, word, w * 32, queue, led_s + k * W) : lead<false>(o, ru.b, kept, word, w * 32, queue, led_s + k * W)) * on.len;
                }
                __syncthreads();
            }
            const unsigned* led = ru.b_list ? led_s : rows_s;
            for (unsigned i = 0; i < active; ++i) {
                const unsigned k = act_s[i].k;
                for (unsigned j = (warp - act_s[i].before) % DL_WARPS; j < act_s[i].len; j += DL_WARPS) {  // (a place a warp, one after the other)
                    const uint32_t to = ru.a_list ? other_of(ru.a, act_s[i].at + j) : blockIdx.x + k * gridDim.x;
                    if (to >= b.rows) {
                        if (lane == 0) set_status(o.st, XLB_ERR_CAPACITY, 19, to);
                        continue;
                    }
                    // A row that nothing else leads to is written as it is; it is its own block that looks what is new
                    // in it.
                    const bool shared = (more_s[to >> 5] >> (to & 31)) & 1u;
                    unsigned *out = next + (uint64_t)to * W, any = 0;
                    if (shared) {
                        constexpr unsigned H = 4;  // words a lane has under way
                        for (unsigned w0 = lane; w0 < W; w0 += 32 * H) {
                            unsigned v[H];
#pragma unroll
                            for (unsigned u = 0; u < H; ++u) v[u] = w0 + 32 * u < W ? led[k * W + w0 + 32 * u] : 0u;
                            // (a word of the head that is being brought up to date only costs an atomic)
#pragma unroll
                            for (unsigned u = 0; u < H; ++u)
                                if (v[u]) v[u] &= ~__ldcg(&o.visited[(uint64_t)to * W + w0 + 32 * u]);
#pragma unroll
                            for (unsigned u = 0; u < H; ++u)
                                if (v[u]) {
                                    atomicOr(&out[w0 + 32 * u], v[u]);
                                    any = 1;
                                }
                        }
                    } else {
                        for (unsigned w = lane; w < W; w += 32) {
                            const unsigned v = led[k * W + w];
                            if (v) out[w] = v;
                            any |= v;
                        }
                    }
                    if (__any_sync(FULL, any) && lane == 0) b.stamp[cur ^ 1][to] = 1;
                }
            }
            __syncthreads();
        }
#pragma unroll
        for (int d = 16; d; d >>= 1) cand += __shfl_xor_sync(FULL, cand, d);
        if (lane == 0 && cand) atomicAdd(&sum_s[1], cand);
        __syncthreads();
        if (threadIdx.x == 0) {
            if (sum_s[0]) atomicAdd(&slot->count, sum_s[0]);
            if (sum_s[1]) atomicAdd(&slot->cand, sum_s[1]);
            if (sum_s[2]) atomicAdd(&slot->heavy_n, sum_s[2]);
            passed += gridDim.x;
            asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(&ctl->arrived) : "memory");
            st.go = wait_for(o, &ctl->arrived, passed, 0, passed);
            const unsigned long long found = __ldcg(&slot->count);
            st.tuples += found;
            st.cands += st.pending;  // of the joins that found them
            st.pending = __ldcg(&slot->cand);
            st.iterations = phase;
            st.fix = found == 0;
            st.over = st.fix || leaving || phase >= max_iterations;
            // (the log takes whatever the next iteration finds)
            st.leaving = st.leave((float)found, (float)st.pending, (float)__ldcg(&slot->heavy_n) * W, all_places * W, (float)b.rows * W) && st.pending <= o.cap;
            st.slot = st.slot == 2 ? 0 : st.slot + 1;
        }
        __syncthreads();
        if (!st.go) return;
        if (st.over) break;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        ctl->rows_tuples = st.tuples;
        ctl->rows_candidates = st.cands;
        ctl->rows_levels = st.iterations ? st.iterations : 1;  // an iteration over nothing finds nothing
        ctl->rows_left = st.fix ? 0 : 1;
    }
}
// ---- two recursive atoms, by rows of the head
// The rules of DeltaRows give whole rows of bits to rows of the head, so an iteration is unions of rows: for a value P
// that a rule has a list for, the rows Q that its row names (of the head where (P, Q) is in the delta, of the
// delta where it is in the head) are ORed in registers, warp by warp, then in shared memory, and the union goes
// to the rows it belongs to as far as these gain by it.  (Tuple by tuple, each against bit rows of the head, its
// transpose and its composites, as delta_loop_k does, a tuple cost an atomic a candidate word, one on the transpose and its
// place in the log, and few warps had most of them: points-to over 1500 values 395 us, here 184.)  An iteration has two
// phases: the rows' own warps add what was derived to the head, which makes the delta; then groups of eight warps
// take the values of all rules in turn, up to four groups a value where there are few of them.  What bounds it is the chain of
// loads a value costs, some 6 K cycles, and two barriers an iteration.
//   Against the loop: points-to programs of 300, 600, 1500, 3000 and 6000 values 328, 530, 623, 1236 and 3937 us by the loop, 198,
// 237, 287, 502 and 1506 by rows, as their relations are skewed.  An item costs whole rows, which are long where the head has
// many bits, whatever is in them; so from 12 bits on there has to be enough (ops_delta_by_rows_pays): seeds a
// value of the head, times the sum of the squares of the lists' lengths a value and rule, since a tuple is led on by
// a list of average length weighted by itself.  Over uniform relations, by the loop and by rows: COPY and STEPS over 8192
// values 1.0 seeds and 0.3 rows a value (0.4 by this measure) 416 and 509 us, 0.3 and 1.0 (0.6) 2.95 and 2.63 ms, 1.0 and
// 1.0 (2) 13.9 and 6.7; COPY, STEPS and ACROSS 0.4 14.2 and 20.5, 0.6 9.8 and 10.7, 2 31.8 and 22.4; STEPS 0.6 1.02 and
// 1.20; ACROSS alone, whose values have a row or none, 0.6 0.84 and 1.86, 2 8.7 and 9.7, 6 18.8 and 12.7.  Over 4096 values
// 0.12 183 and 204 us, 0.39 289 and 309, 3.02 and 2.54 ms, 0.6 995 and 866 us; ACROSS 1.8 604 and 796 us, 2 1.84 and
// 1.92 ms, 6 3.43 and 2.45.  Points-to over uniform relations of 6000 values 0.1 2.08 and 2.52, 0.3 3.90 and 4.86, 0.9 5.28 and 3.40; over skewed ones
// the measure is 1.2 to 10.  Up to 11 bits the two differ by a tenth at most where rows lose (ACROSS by a
// quarter); long copy chains in such programs, 2000 iterations of next to nothing, 17.4 and 20.0 ms.
//   (A warp a value for rows of few tuples, before the groups, did
// better on sparse relations and took points-to 242.)  h(P, Y) :- h(P, Q), h(Q, Y) stays with the loop: every row is a value
// then, and on a sparse graph of 8000 nodes rows took 1320 us and the loop 284 (dense, 2000 nodes: 713 and 966).
constexpr int WD_BITS_MIN = 6, WD_BITS_MAX = 13;
constexpr int WD_ALWAYS = 11;     // bits up to which rows are taken whatever is stored (but for ACROSS alone)
constexpr unsigned WD_WARPS = 8, WD_THREADS = WD_WARPS * 32, WD_GROUPS = DL_THREADS / WD_THREADS;
constexpr unsigned WD_SPLIT = 4;  // groups that share a value, at most
constexpr unsigned WD_FEW = 64;   // tuples of a row up to which it is not
struct WideRule {
    Ix ix;
    int kind;
};
struct WideRules {
    WideRule r[DELTA_ROWS_MAX];
    int n;
};
struct Wide {
    unsigned *delta, *reached, *stamp;  // bitmaps like the head's; rows that were reached
    unsigned *n_delta, *n_head;         // tuples of each row
    unsigned* active[2];                // rows of the delta that hold any, as bits: this iteration's, the next one's
    unsigned* keys;                     // per rule, the values it has something to do for ...
    unsigned* n_keys;                   // ... and how many
    unsigned rows, words;
};
// four rows, a list of twice a row's values, counters, items
__host__ __device__ constexpr size_t wide_group_bytes(unsigned words) { return words * 16 + words * 128 + 16 + WD_THREADS * 4; }
struct WideGroup {
    unsigned *led[2], *row_d, *row_h, *count, *items;
    unsigned short* list;
    unsigned id, warp, thread;
    __device__ __forceinline__ void sync() const { asm volatile("bar.sync %0, %1;" ::"r"(id + 1), "n"(WD_THREADS) : "memory"); }
};
// What `led` brings row `to` beyond the head, for up to four rows a warp at a time (entries first, first + step, ... of n).
template <class Row, class From>
__device__ __forceinline__ void give(const Out& o, const Wide& b, unsigned first, unsigned step, unsigned n, Row row, From from) {
    const unsigned W = b.words, lane = lane_id();
    constexpr int N = 4;
    for (unsigned e0 = first; e0 < n; e0 += N * step) {
        unsigned to[N];
        const unsigned* led[N];
#pragma unroll
        for (int u = 0; u < N; ++u) {
            const bool on = e0 + u * step < n;
            to[u] = on ? row(e0 + u * step) : ~0u;
            led[u] = on ? from(e0 + u * step) : nullptr;
            if (on && to[u] >= b.rows) {
                if (lane == 0) set_status(o.st, XLB_ERR_CAPACITY, 24, to[u]);
                to[u] = ~0u;
            }
        }
        for (unsigned w = 2 * lane; w < W; w += 64) {
            unsigned long long gain[N];
#pragma unroll
            for (int u = 0; u < N; ++u) {
                gain[u] = to[u] != ~0u ? *reinterpret_cast<const unsigned long long*>(led[u] + w) : 0ull;
                if (gain[u]) gain[u] &= ~__ldcg(reinterpret_cast<const unsigned long long*>(o.visited + (uint64_t)to[u] * W + w));
            }
#pragma unroll
            for (int u = 0; u < N; ++u)
                if (gain[u]) gain[u] &= ~__ldcg(reinterpret_cast<const unsigned long long*>(b.reached + (uint64_t)to[u] * W + w));  // (found a moment ago)
#pragma unroll
            for (int u = 0; u < N; ++u)
                if (gain[u]) {
                    atomicOr(reinterpret_cast<unsigned long long*>(b.reached + (uint64_t)to[u] * W + w), gain[u]);
                    b.stamp[to[u]] = 1;
                }
        }
    }
}
// The union of rows: entries of the group's list, a row number and the matrix (bit 15: the delta) each, into led[0].
__device__ __forceinline__ void unite(const Out& o, const Wide& b, const WideGroup& g, unsigned n) {
    const unsigned W = b.words, lane = lane_id();
    constexpr int N = 8;
    for (unsigned w = 2 * lane; w - 2 * lane < W; w += 64) {
        unsigned long long acc = 0;
        for (unsigned e0 = g.warp; e0 < n; e0 += N * WD_WARPS) {
            unsigned long long v[N];
#pragma unroll
            for (int u = 0; u < N; ++u) {
                const unsigned e = e0 + u * WD_WARPS < n ? g.list[e0 + u * WD_WARPS] : ~0u;
                const unsigned* m = e & 0x8000u ? b.delta : o.visited;
                v[u] = e != ~0u && w < W ? __ldcg(reinterpret_cast<const unsigned long long*>(m + (uint64_t)(e & 0x7FFF) * W + w)) : 0ull;
            }
#pragma unroll
            for (int u = 0; u < N; ++u) acc |= v[u];
        }
        if (acc) atomicOr(reinterpret_cast<unsigned long long*>(g.led[0] + w), acc);
    }
}
__global__ void __launch_bounds__(DL_THREADS, 1) delta_wide_k(const __grid_constant__ Out o, const __grid_constant__ WideRules rules, const __grid_constant__ Wide b, uint64_t max_iterations) {
    extern __shared__ __align__(16) unsigned char wd_smem[];
    __shared__ BitsState st;
    __shared__ unsigned long long sum_s[2];
    __shared__ unsigned n_keys_s[DELTA_ROWS_MAX];
    const unsigned lane = lane_id(), warp = threadIdx.x >> 5, W = b.words;
    WideGroup g;
    g.id = warp / WD_WARPS;
    g.warp = warp % WD_WARPS;
    g.thread = threadIdx.x % WD_THREADS;
    unsigned* base = reinterpret_cast<unsigned*>(wd_smem + g.id * wide_group_bytes(W));
    g.led[0] = base;
    g.led[1] = base + W;
    g.row_d = base + 2 * W;
    g.row_h = base + 3 * W;
    g.list = reinterpret_cast<unsigned short*>(base + 4 * W);
    g.count = base + 4 * W + 32 * W;
    g.items = g.count + 4;
    Ctl* ctl = o.ctl;
    if (threadIdx.x == 0) st = BitsState{};
    // the values each rule has something to do for
    for (int q = blockIdx.x; q < rules.n; q += gridDim.x)
        for (unsigned v = threadIdx.x; v < b.rows; v += DL_THREADS) {
            uint32_t s, len;
            find(rules.r[q].ix, v, s, len);
            if (len) b.keys[q * b.rows + atomicAdd(&b.n_keys[q], 1u)] = v;
        }
    unsigned passed = 0;
    const auto meet = [&]() {  // (thread 0)
        passed += gridDim.x;
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(&ctl->arrived) : "memory");
        st.go = wait_for(o, &ctl->arrived, passed, 0, passed);
    };
    for (unsigned phase = 0;; ++phase) {
        __syncthreads();
        if (threadIdx.x < 2) sum_s[threadIdx.x] = 0;
        if (blockIdx.x == 0 && threadIdx.x == 0) ctl->slot[st.slot == 2 ? 0 : st.slot + 1] = Slot{};
        __syncthreads();
        Slot* slot = &ctl->slot[st.slot];
        // what was derived joins the head (at first: the seeds are in it)
        for (unsigned row = warp * gridDim.x + blockIdx.x; row < b.rows; row += gridDim.x * DL_WARPS) {
            const unsigned held = __ldcg(&b.n_delta[row]), reached = phase ? __ldcg(&b.stamp[row]) : 1u;
            if (!held && !reached) continue;
            unsigned mine = 0;
            for (unsigned w = 2 * lane; w < W; w += 64) {
                const uint64_t at = (uint64_t)row * W + w;
                unsigned long long d = 0;
                if (reached) {
                    const unsigned long long have = __ldcg(reinterpret_cast<const unsigned long long*>(o.visited + at));
                    d = have;
                    if (phase) {
                        const unsigned long long r = __ldcg(reinterpret_cast<const unsigned long long*>(b.reached + at));
                        d = r & ~have;
                        if (r) *reinterpret_cast<unsigned long long*>(b.reached + at) = 0;
                        if (d) *reinterpret_cast<unsigned long long*>(o.visited + at) = have | d;
                    }
                }
                *reinterpret_cast<unsigned long long*>(b.delta + at) = d;
                mine += __popcll(d);
            }
            const unsigned all = __reduce_add_sync(FULL, mine);
            if (lane == 0) {
                if (reached) b.stamp[row] = 0;
                b.n_delta[row] = all;
                if (all) {
                    b.n_head[row] += all;
                    atomicOr(&b.active[phase & 1][row >> 5], 1u << (row & 31));
                    atomicAdd(&sum_s[0], (unsigned long long)all);
                }
            }
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            if (sum_s[0]) atomicAdd(&slot->count, sum_s[0]);
            meet();
            const unsigned long long found = __ldcg(&slot->count);
            st.tuples += found;
            st.cands += st.pending;  // of the joins that found them
            st.iterations = phase;
            st.fix = found == 0;
            st.over = st.fix || phase >= max_iterations;
        }
        __syncthreads();
        if (!st.go) return;
        if (st.over) break;
        if (phase == 0 && threadIdx.x < (unsigned)rules.n) n_keys_s[threadIdx.x] = __ldcg(&b.n_keys[threadIdx.x]);
        for (unsigned w = blockIdx.x * DL_THREADS + threadIdx.x; w < (b.rows + 31) / 32; w += gridDim.x * DL_THREADS) b.active[(phase & 1) ^ 1][w] = 0;  // (read by nobody now)
        __syncthreads();
        const unsigned* active = b.active[phase & 1];
        unsigned long long cand = 0;
        const unsigned groups = gridDim.x * WD_GROUPS;
        unsigned turns = 0;
        unsigned first = g.id * gridDim.x + blockIdx.x;  // (items are numbered through all rules)
        for (int q = 0; q < rules.n; ++q) {
            const WideRule& ru = rules.r[q];
            unsigned split = ru.kind == DeltaRows::COPY ? 1 : WD_SPLIT;  // (fewer where there are enough values to go round)
            while (split > 1 && 2 * n_keys_s[q] * split > 3 * groups) split /= 2;
            const unsigned items = n_keys_s[q] * split;
            const unsigned all = items > first ? (items - first + groups - 1) / groups : 0;
            const bool direct = all <= 2;  // (else they are first looked at side by side: what has nothing to do costs no turn)
            unsigned done = 0, left = direct ? all : 0;
            while (left || (!direct && done < all)) {
                if (!left) {
                    g.sync();
                    if (g.thread == 0) g.count[2] = 0;
                    g.sync();
                    if (done + g.thread < all) {
                        const unsigned i = first + (done + g.thread) * groups, key = __ldcg(&b.keys[q * b.rows + i / split]), nd = __ldcg(&b.n_delta[key]), nh = __ldcg(&b.n_head[key]);
                        if ((nd || (nh && ru.kind != DeltaRows::COPY)) && (nh > WD_FEW || i % split == 0)) g.items[atomicAdd(&g.count[2], 1u)] = i;
                    }
                    g.sync();
                    left = g.count[2];
                    done += WD_THREADS;
                    continue;
                }
                --left;
                const unsigned item = direct ? first + left * groups : g.items[left];
                if (++turns % 64 == 0 && g.thread == 0) beat(o);
                const unsigned key = __ldcg(&b.keys[q * b.rows + item / split]), part = item % split;
                const unsigned nd = __ldcg(&b.n_delta[key]), nh = __ldcg(&b.n_head[key]);
                if (!nh || (ru.kind == DeltaRows::COPY && !nd) || (part && nh <= WD_FEW)) continue;
                uint32_t s, len;
                find(ru.ix, key, s, len);
                const unsigned mask = split == 1 || nh <= WD_FEW ? ~0u : (split == 4 ? 0x11111111u : 0x55555555u) << part;  // the values of the row that are this group's
                g.sync();  // (the one before is done with the rows and the list)
                if (g.thread == 0) g.count[0] = g.count[1] = 0;
                for (unsigned w = g.thread; w < W; w += WD_THREADS) {
                    g.led[0][w] = g.led[1][w] = 0;
                    g.row_d[w] = nd ? __ldcg(&b.delta[(uint64_t)key * W + w]) : 0u;
                    g.row_h[w] = ru.kind != DeltaRows::COPY ? __ldcg(&o.visited[(uint64_t)key * W + w]) : 0u;
                }
                g.sync();
                if (ru.kind == DeltaRows::COPY) {
                    if (g.thread == 0) cand += (unsigned long long)nd * len;
                    give(o, b, g.warp, WD_WARPS, len, [&](unsigned e) { return other_of(ru.ix, s + e); }, [&](unsigned) { return (const unsigned*)g.row_d; });
                    continue;
                }
                if (ru.kind == DeltaRows::ACROSS) {
                    // rows listed for the value: of the head into one union, of the delta into the other
                    unsigned long long all = 0, fresh = 0;
                    for (unsigned w0 = 0; w0 < W; w0 += 64) {
                        const unsigned w = w0 + 2 * lane;
                        unsigned long long x = 0, y = 0;
                        for (uint32_t j = g.warp; j < len; j += WD_WARPS) {
                            const uint32_t m = other_of(ru.ix, s + j);
                            if (m >= b.rows) continue;  // (no row: never derived)
                            const unsigned mh = __ldcg(&b.n_head[m]), md = __ldcg(&b.n_delta[m]);
                            if (w0 == 0) {
                                all += mh;
                                fresh += md;
                            }
                            if (w < W && nd && mh) x |= __ldcg(reinterpret_cast<const unsigned long long*>(o.visited + (uint64_t)m * W + w));
                            if (w < W && md) y |= __ldcg(reinterpret_cast<const unsigned long long*>(b.delta + (uint64_t)m * W + w));
                        }
                        if (x) atomicOr(reinterpret_cast<unsigned long long*>(g.led[0] + w), x);
                        if (y) atomicOr(reinterpret_cast<unsigned long long*>(g.led[1] + w), y);
                    }
                    if (lane == 0 && part == 0) cand += nd * all + nh * fresh;
                    if (lane == 0 && fresh) g.count[1] = 1;
                    g.sync();
                    const bool any_fresh = g.count[1] != 0;
                    for (unsigned w = g.thread; w < W; w += WD_THREADS) {  // the row's values: those of the delta get the one, the others the other
                        const unsigned d = g.row_d[w] & mask, h = any_fresh ? g.row_h[w] & ~g.row_d[w] & mask : 0u;
                        unsigned at = d | h ? atomicAdd(&g.count[0], (unsigned)(__popc(d) + __popc(h))) : 0u;
                        for (unsigned x = d; x; x &= x - 1) g.list[at++] = (unsigned short)(w * 32 + __ffs(x) - 1);
                        for (unsigned x = h; x; x &= x - 1) g.list[at++] = (unsigned short)((w * 32 + __ffs(x) - 1) | 0x8000u);
                    }
                    g.sync();
                    give(o, b, g.warp, WD_WARPS, g.count[0], [&](unsigned e) { return (unsigned)(g.list[e] & 0x7FFF); }, [&](unsigned e) { return (const unsigned*)(g.list[e] >> 15 ? g.led[1] : g.led[0]); });
                    continue;
                }
                // STEPS: rows of the head for values of the delta, rows of the delta for values of the head
                unsigned long long c = 0;
                for (unsigned w = g.thread; w < W; w += WD_THREADS) {
                    const unsigned d = g.row_d[w] & mask, h = g.row_h[w] & __ldcg(&active[w]) & mask;
                    unsigned at = d | h ? atomicAdd(&g.count[0], (unsigned)(__popc(d) + __popc(h))) : 0u;
                    for (unsigned x = d; x; x &= x - 1) {
                        const unsigned v = w * 32 + __ffs(x) - 1;
                        c += __ldcg(&b.n_head[v]);
                        g.list[at++] = (unsigned short)v;
                    }
                    for (unsigned x = h; x; x &= x - 1) {
                        const unsigned v = w * 32 + __ffs(x) - 1;
                        c += __ldcg(&b.n_delta[v]);
                        g.list[at++] = (unsigned short)(v | 0x8000u);
                    }
                }
                cand += c * len;
                g.sync();
                const unsigned n = g.count[0];
                if (!n) continue;
                unite(o, b, g, n);
                g.sync();
                give(o, b, g.warp, WD_WARPS, len, [&](unsigned e) { return other_of(ru.ix, s + e); }, [&](unsigned) { return (const unsigned*)g.led[0]; });
            }
            first = (first + groups - items % groups) % groups;
        }
#pragma unroll
        for (int d = 16; d; d >>= 1) cand += __shfl_xor_sync(FULL, cand, d);
        if (lane == 0 && cand) atomicAdd(&sum_s[1], cand);
        __syncthreads();
        if (threadIdx.x == 0) {
            if (sum_s[1]) atomicAdd(&slot->cand, sum_s[1]);
            beat(o);
            meet();
            st.pending = __ldcg(&slot->cand);
            st.slot = st.slot == 2 ? 0 : st.slot + 1;
        }
        __syncthreads();
        if (!st.go) return;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        ctl->rows_tuples = st.tuples;
        ctl->rows_candidates = st.cands;
        ctl->rows_levels = st.iterations ? st.iterations : 1;  // an iteration over nothing finds nothing
        ctl->rows_left = st.fix ? 0 : 1;
    }
}
// Squares of the lists' lengths, of all rules: what a tuple is led on to, summed over the stored rows.
__global__ void __launch_bounds__(DL_THREADS) list_squares_k(const __grid_constant__ WideRules rules, unsigned rows, unsigned long long* sum, const Publish pub) {
    __shared__ unsigned long long sum_s;
    if (threadIdx.x == 0) sum_s = 0;
    __syncthreads();
    unsigned long long mine = 0;
    for (int q = 0; q < rules.n; ++q)
#pragma unroll 4
        for (unsigned v = threadIdx.x; v < rows; v += DL_THREADS) {
            uint32_t s, len;
            find(rules.r[q].ix, v, s, len);
            mine += (unsigned long long)len * len;
        }
#pragma unroll
    for (int d = 16; d; d >>= 1) mine += __shfl_xor_sync(FULL, mine, d);
    if (lane_id() == 0 && mine) atomicAdd(&sum_s, mine);
    __syncthreads();
    if (threadIdx.x == 0) *sum = sum_s;
    publish_now(pub);
}
// The loop starts on what was given up, or left.
__global__ void delta_rows_left_k(Ctl* c) {
    c->tail = c->rows_seeds;
    c->arrived = 0;
    for (int k = 0; k < 3; ++k) c->slot[k] = Slot{};
    ready(c, false);
}

}  // namespace

static Out out_of(xlb_ctx* c, const DeltaLoop& d) {
    return Out{d.visited->as<unsigned int>(), d.words, d.lo_bits, d.log ? d.log->as<uint64_t>() : nullptr, d.cap, (Ctl*)d.ctl, c->d_status, d.square ? d.visited->as<unsigned int>() + d.words : nullptr, c->delta_spin_limit};
}

DeltaLoop ops_delta_begin(xlb_ctx* c, int hi_bits, int lo_bits, bool square, int composites) {
    DeltaLoop d;
    d.hi_bits = hi_bits;
    d.lo_bits = lo_bits;
    d.square = square;
    d.words = ((1ull << (hi_bits + lo_bits)) + 31) / 32;
    // the bitmaps, then the control block: one fill for both
    const uint64_t bitmaps = std::max<uint64_t>(d.words * 4, 16) * (square ? 4 + composites : 1);
    d.visited = make_buf(c, bitmaps + sizeof(Ctl));
    d.ctl = (char*)d.visited->p + bitmaps;
    CUDA_OK(set_async(c, d.visited->p, 0, d.visited->bytes));
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
    // Four times what is in it, and from the start as much as a large fixpoint derives where that is a
    // small part of the free budget (running out costs a pass over the bitmap and a second launch);
    // never more than the domain, beyond which nothing can be new.
    const uint64_t domain = 1ull << (d.hi_bits + d.lo_bits);
    const uint64_t spare = c->budget > c->allocated ? (c->budget - c->allocated) / 32 / 8 : 0;
    const uint64_t cap = std::min<uint64_t>(domain, std::max<uint64_t>({4 * need, 1ull << 20, std::min<uint64_t>(spare, 1ull << 26)}));
    Buf log = make_buf(c, std::max<uint64_t>(cap, 1) * 8);
    if (d.log && need > more) CUDA_OK(copy_async(c, log->p, d.log->p, std::min(d.cap, need - more) * 8, cudaMemcpyDeviceToDevice));
    d.log = log;
    d.cap = cap;
}

void ops_delta_seed(xlb_ctx* c, DeltaLoop& d, const Keys& bag) {
    if (!bag.n) return;
    if (d.logged) log_room(c, d, bag.n);
    prof_begin(c, "dense_mark", bag.n * 16ull);
    delta_seed_k<<<grid_for(c, bag.n), BLOCK, 0, c->stream>>>(bag.ptr(), bag.n, out_of(c, d), d.square);
    d.seeded = true;
    check_launch(c, "dense_mark");
}

void ops_delta_append(xlb_ctx* c, DeltaLoop& d, const Keys& rows) {
    if (!rows.n) return;
    log_room(c, d, rows.n);
    CUDA_OK(copy_async(c, d.log->as<uint64_t>() + (d.room - rows.n), rows.ptr(), rows.n * 8, cudaMemcpyDeviceToDevice));
    const unsigned long long tail = d.room;
    c->h_scalar[48] = tail;
    CUDA_OK(copy_async(c, &((Ctl*)d.ctl)->tail, &c->h_scalar[48], 8, cudaMemcpyHostToDevice));
    stream_wait(c);  // (the staging word is used again)
}

static Ix view_of(const Index& ix) {
    return Ix{ix.cursor ? ix.cursor->as<unsigned long long>() : nullptr, ix.domain, ix.table ? ix.table->as<ulonglong2>() : nullptr, ix.mask,
              ix.pay ? ix.pay->as<uint32_t>() : ix.S->as<uint32_t>(), ix.pay ? 0 : 1};
}

// Rules that keep the head's first column and join its second with one stored relation, from seeds alone.
static bool rows_apart(const DeltaLoop& d, const std::vector<DeltaRule>& rules, const std::vector<DeltaVariant>& variants, const Keys& known) {
    if (d.square || !d.seeded || known.n || rules.empty() || !variants.empty() || d.lo_bits < RW_BITS_MIN || d.lo_bits > RW_BITS_MAX || d.hi_bits > 31) return false;
    for (auto& r : rules)
        if (r.joins != 1 || r.hi_src != 0 || r.lo_src != 2 || r.key_src[0] != SRC_LO) return false;
    return true;
}
static_assert(rows_bytes(RW_BITS_MAX) <= (46u << 10), "a row's shared memory needs no opt-in");
static unsigned rows_per_sm(int lo_bits) { return std::min(32u, (220u << 10) / (rows_bytes(lo_bits) + 2048u)); }
template <int W>
static void launch_rows(xlb_ctx* c, const DeltaLoop& d, const Rules& rs, RowsShape sh, uint64_t max_iterations) {
    const unsigned smem = rows_bytes(d.lo_bits);
    const unsigned per_sm = std::min(2048u / (W * 32), rows_per_sm(d.lo_bits));
    const unsigned blocks = std::min(per_sm * (unsigned)c->sm_count, sh.rows);
    sh.chunk = std::max(1u, sh.rows / (blocks * 8));  // (a domain much larger than what is in use: few tickets)
    delta_rows_k<W><<<blocks, W * 32, smem, c->stream>>>(out_of(c, d), rs, sh, max_iterations);
}
// False: rows are left for the loop, which is ready to start on them.
static bool run_rows(xlb_ctx* c, DeltaLoop& d, const Rules& rs, uint64_t max_iterations, DeltaResult* res) {
    RowsShape sh{};
    sh.rows = 1u << d.hi_bits;
    sh.words = 1u << (d.lo_bits - 5);
    sh.queue = rows_queue(d.lo_bits);
    // Where the seeds are the relation itself and a value has as many matches as a row has words, a level takes the
    // values' rows and not their matches one by one (four blocks of 128 nodes, 33 M candidates: 62 us, now 19
    // and 4 for the copy; 2000 nodes of degree 5, rows of 64 words, stay with their matches.)
    Buf lists;
    if (d.seeds_listed && d.lo_bits <= RW_LISTS_BITS && rs.r[0].rows >= std::max<uint64_t>(d.words, RW_LISTS_MIN)) {
        lists = make_buf(c, std::max<uint64_t>(d.words * 4, 16));
        CUDA_OK(copy_async(c, lists->p, d.visited->p, d.words * 4, cudaMemcpyDeviceToDevice));
        sh.lists = lists->as<unsigned>();
    }
    Ctl* ctl = (Ctl*)d.ctl;
    prof_begin(c, "expand_mark", 0);
    // Four warps a row keep rows of a few thousand candidates short (one: twice the time); eight where an SM
    // has few rows, or room for few.
    if (std::min((sh.rows + (unsigned)c->sm_count - 1) / (unsigned)c->sm_count, rows_per_sm(d.lo_bits)) <= 6) launch_rows<8>(c, d, rs, sh, max_iterations);
    else launch_rows<4>(c, d, rs, sh, max_iterations);
    check_launch(c, "expand_mark");
    unsigned long long w[6];  // tuples, candidates, levels, left, given up, seeds
    read_words(c, &ctl->rows_tuples, 6, w);
    res->rows = w[0];
    res->candidates = w[1];
    res->iterations = w[2];
    res->fix = w[3] == 0;
    prof_add_bytes(c, "expand_mark", w[1] * 4ull + d.words * 8ull);
    if (w[4] == 0) {
        res->iterations = std::max<uint64_t>(res->iterations, 1);  // an iteration over nothing finds nothing
        return true;
    }
    delta_rows_left_k<<<1, 1, 0, c->stream>>>(ctl);
    check_launch(c, "delta_begin");
    d.room = w[5];
    return false;
}

// Rules whose new first column comes from the old first, and the second from the second, by lists of their own or as
// they are; from seeds alone.
static bool bits_apart(const DeltaLoop& d, const std::vector<DeltaRule>& rules, const std::vector<DeltaVariant>& variants, const Keys& known, BitsRules* out) {
    if (d.square || !d.seeded || known.n || rules.empty() || !variants.empty() || d.lo_bits < BT_BITS_MIN || d.lo_bits > BT_BITS_MAX || d.hi_bits > BT_BITS_MAX || d.hi_bits + d.lo_bits < BT_BITS_BOTH) return false;
    out->n = (int)rules.size();
    bool listed = false;  // one rule's B is kept in shared memory
    double first = 0;     // candidates of the first iteration, at least (a value of a stored relation has a match)
    for (size_t q = 0; q < rules.size(); ++q) {
        const DeltaRule& r = rules[q];
        BitsRule& x = out->r[q];
        x.a_list = r.hi_src == 2 || r.hi_src == 3;
        x.b_list = r.lo_src == 2 || r.lo_src == 3;
        if ((!x.a_list && r.hi_src != 0) || (!x.b_list && r.lo_src != 1) || r.joins != (x.a_list ? 1 : 0) + (x.b_list ? 1 : 0)) return false;
        if (x.a_list && x.b_list && r.hi_src == r.lo_src) return false;
        if (x.a_list && r.key_src[r.hi_src - 2] != SRC_HI) return false;
        if (x.b_list && r.key_src[r.lo_src - 2] != SRC_LO) return false;
        if (x.a_list) x.a = view_of(*r.ix[r.hi_src - 2]);
        x.a_rows = x.a_list ? (unsigned)r.ix[r.hi_src - 2]->n : 0;
        if (x.b_list) x.b = view_of(*r.ix[r.lo_src - 2]);
        x.listed = 0;
        const double rows = (double)(1u << d.hi_bits), cols = (double)(1u << d.lo_bits);
        first += (double)d.room * (x.a_list ? std::max(1.0, r.ix[r.hi_src - 2]->n / rows) : 1) * (x.b_list ? std::max(1.0, r.ix[r.lo_src - 2]->n / cols) : 1);
        if (x.b_list && !listed && r.ix[r.lo_src - 2]->n <= BT_LISTED) {
            x.listed = (unsigned)r.ix[r.lo_src - 2]->n;
            listed = true;
        }
    }
    return first >= BT_SEEDS * (1u << d.hi_bits);
}
enum class BitsEnd { DONE, DECLINED, LEFT };
static BitsEnd run_bits(xlb_ctx* c, DeltaLoop& d, BitsRules rules, uint64_t max_iterations, DeltaResult* res, uint64_t* left) {
    Bits b{};
    b.rows = 1u << d.hi_bits;
    b.words = 1u << (d.lo_bits - 5);
    const uint64_t map = (uint64_t)b.rows * b.words;
    if (b.rows > BT_OWN * (unsigned)c->sm_count) return BitsEnd::DECLINED;
    if (c->budget && c->allocated + (map + b.rows) * 8 > c->budget) return BitsEnd::DECLINED;
    Buf reached = make_buf(c, (map + b.rows) * 8);
    CUDA_OK(set_async(c, reached->p, 0, reached->bytes));
    for (int k = 0; k < 2; ++k) {
        b.next[k] = reached->as<unsigned>() + k * map;
        b.stamp[k] = reached->as<unsigned>() + 2 * map + k * b.rows;
    }
    Out o = out_of(c, d);
    Ctl* ctl = (Ctl*)d.ctl;
    void* args[] = {&o, &rules, &b, &max_iterations};
    prof_begin(c, "expand_mark", 0);
    CUDA_OK(cudaLaunchCooperativeKernel((const void*)delta_bits_k, dim3((unsigned)c->sm_count), dim3(DL_THREADS), args, BT_SMEM, c->stream));
    check_launch(c, "expand_mark");
    unsigned long long w[6];  // tuples, candidates, iterations, left, declined, listed
    read_words(c, &ctl->rows_tuples, 6, w);
    if (w[4]) return BitsEnd::DECLINED;
    res->rows = w[0];
    res->candidates = w[1];
    res->iterations = w[2];
    res->fix = w[3] == 0;
    *left = w[5];
    prof_add_bytes(c, "expand_mark", w[0] / 8 + map * 8);
    return w[5] ? BitsEnd::LEFT : BitsEnd::DONE;
}

void ops_delta_run(xlb_ctx* c, DeltaLoop& d, const std::vector<DeltaRule>& rules, const std::vector<DeltaVariant>& variants, uint64_t max_iterations, const Keys& known,
                   DeltaResult* res) {
    if (rules.size() > DL_RULES || variants.size() > SQ_VARIANTS) xlb_fail(XLB_ERR_INVALID, "internal: %zu rules and %zu variants in a delta loop", rules.size(), variants.size());
    if (!c->delta_attr_set) {
        CUDA_OK(cudaFuncSetAttribute(delta_loop_k<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)DL_SMEM));
        CUDA_OK(cudaFuncSetAttribute(delta_loop_k<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)DL_SMEM));
        CUDA_OK(cudaFuncSetAttribute(delta_bits_k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)BT_SMEM));
    }
    c->delta_attr_set = true;
    const bool square = d.square;
    Square sq{};
    std::vector<Buf> counts;
    if (square) {
        sq.bits = d.lo_bits;
        sq.words = (uint32_t)d.words;
        for (auto& in : variants) {
            Variant& v = sq.v[sq.n++];
            v.a_key = in.list ? in.list_key : -1;
            if (in.list) v.a = view_of(*in.list);
            v.row_key = in.row_key;
            v.fixed = in.fixed;
            v.bits_are_hi = in.bits_are_hi;
            if (in.rows != DeltaVariant::COMPOSED) {
                v.rows = (in.rows == DeltaVariant::HEAD ? 2 : 3) * sq.words;
                continue;
            }
            if (sq.n_aux == SQ_AUX || d.visited->bytes < (uint64_t)(5 + sq.n_aux) * sq.words * 4 + sizeof(Ctl)) xlb_fail(XLB_ERR_INVALID, "internal: too many composites in a delta loop");
            Buf b = make_buf(c, 8ull << sq.bits);
            CUDA_OK(set_async(c, b->p, 0, b->bytes));
            counts.push_back(b);
            Composite& x = sq.aux[sq.n_aux];
            x.ix = view_of(*in.composed);
            x.list_key = in.composed_list_key;
            x.row_key = in.composed_row_key;
            x.rows = v.rows = (4 + sq.n_aux++) * sq.words;
            v.counts = x.counts = b->as<unsigned long long>();
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
        r.rows = rules[q].ix[0]->n;
    }
    Buf by_rows;  // the head after rows were evaluated, and some are left
    BitsRules bits{};
    uint64_t earlier = 0;  // iterations before the loop's
    bool left = false;
    if (rows_apart(d, rules, variants, known)) {
        if (run_rows(c, d, rs, max_iterations, res)) return;
        left = true;
    } else if (bits_apart(d, rules, variants, known, &bits)) {
        uint64_t listed = 0;
        const BitsEnd end = run_bits(c, d, bits, max_iterations, res, &listed);
        if (end == BitsEnd::DONE || (end == BitsEnd::LEFT && res->iterations >= max_iterations)) return;
        if (end == BitsEnd::LEFT) {  // its last tuples are the loop's first delta
            res->rows -= listed;
            earlier = res->iterations;
            max_iterations -= earlier;
            delta_rows_left_k<<<1, 1, 0, c->stream>>>((Ctl*)d.ctl);
            check_launch(c, "delta_begin");
            d.room = listed;
            left = true;
        }
    }
    if (left) {
        by_rows = make_buf(c, std::max<uint64_t>(d.words * 4, 16));
        CUDA_OK(copy_async(c, by_rows->p, d.visited->p, d.words * 4, cudaMemcpyDeviceToDevice));
    }
    DeltaResult rows_done = *res;
    if (!by_rows || earlier) rows_done.fix = true;
    Buf heavy = make_buf(c, (uint64_t)DL_HEAVY_MAX * sizeof(Heavy));
    if (!d.seeded) {
        delta_begin_k<<<1, 1, 0, c->stream>>>((Ctl*)d.ctl, square);
        check_launch(c, "delta_begin");
    }
    for (;;) {
        Out o = out_of(c, d);
        Heavy* hp = heavy->as<Heavy>();
        void* args[] = {&o, &rs, &hp, &max_iterations, &sq};
        prof_begin(c, "expand_mark", 0);
        CUDA_OK(cudaLaunchCooperativeKernel(square ? (const void*)delta_loop_k<true> : (const void*)delta_loop_k<false>, dim3((unsigned)c->sm_count), dim3(DL_THREADS), args, DL_SMEM, c->stream));
        check_launch(c, "expand_mark");
        unsigned long long w[7];  // tail, start, end, iterations, candidates, fix, overflow
        read_words(c, d.ctl, 7, w);
        res->rows = rows_done.rows + w[0];
        res->iterations = earlier ? earlier + w[3] : std::max<uint64_t>(rows_done.iterations, w[3]);
        res->candidates = rows_done.candidates + w[4];
        res->fix = rows_done.fix && w[5] != 0;
        prof_add_bytes(c, "expand_mark", w[4] * 4ull + w[0] * 16ull);
        if (!w[6]) return;
        // The log was too short for the last iteration: its delta is what the head's bitmap holds
        // beyond the known rows and the log before it.  A longer log takes up from there.
        const uint64_t tail = w[0], stored = d.cap;
        Keys done;
        done.buf = d.log;
        done.n = stored;
        Buf before = make_buf(c, std::max<uint64_t>(d.words * 4, 16));
        if (by_rows) CUDA_OK(copy_async(c, before->p, by_rows->p, d.words * 4, cudaMemcpyDeviceToDevice));
        else CUDA_OK(set_async(c, before->p, 0, before->bytes));
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
        delta_resume_k<<<1, 1, 0, c->stream>>>((Ctl*)d.ctl, max_iterations, square);
        check_launch(c, "delta_resume");
    }
}

static uint64_t wide_bytes(int bits) {
    const uint64_t rows = 1ull << bits, map = rows * rows / 32;
    return (2 * map + 3 * rows + 2 * std::max<uint64_t>(rows / 32, 2) + DELTA_ROWS_MAX * rows + DELTA_ROWS_MAX) * 4;
}
static WideRules wide_rules(const std::vector<DeltaRows>& rules) {
    WideRules rs{};
    for (auto& r : rules) {
        if (rules.size() > DELTA_ROWS_MAX || !r.list) xlb_fail(XLB_ERR_INVALID, "internal: %zu rules by rows", rules.size());
        WideRule& x = rs.r[rs.n++];
        x.kind = r.kind;
        x.ix = view_of(*r.list);
    }
    return rs;
}
bool ops_delta_by_rows_pays(xlb_ctx* c, int bits, double seeds, const std::vector<DeltaRows>& rules) {
    bool across = true;
    for (auto& r : rules) across = across && r.kind == DeltaRows::ACROSS;
    const double least = across ? (bits <= WD_ALWAYS - 1 ? 0 : bits <= WD_ALWAYS ? 2 : 4) : bits <= WD_ALWAYS ? 0 : bits <= WD_ALWAYS + 1 ? 0.25 : 0.7;
    if (least == 0 || rules.empty()) return true;
    // (what the squares are between: rows as even as they can be, and all of one value)
    const double values = (double)(1u << bits), scale = seeds / values / (values * rules.size());
    double low = 0, high = 0;
    for (auto& r : rules) {
        const double n = (double)r.list->n;
        low += n * std::max(1.0, n / values);
        high += n * n;
    }
    if (low * scale >= least || high * scale < least) return low * scale >= least;
    const WideRules rs = wide_rules(rules);
    Buf sum = make_buf(c, 8);
    prof_begin(c, "list_squares", 0);
    const Publish pub = publish_by(c, 1, sum->p, 1);
    list_squares_k<<<1, DL_THREADS, 0, c->stream>>>(rs, 1u << bits, sum->as<unsigned long long>(), pub);
    check_launch(c, "list_squares");
    unsigned long long squares;
    read_published(c, pub, sum->p, 1, &squares);
    return squares * scale >= least;
}
bool ops_delta_by_rows_fits(xlb_ctx* c, int bits) {
    return bits >= WD_BITS_MIN && bits <= WD_BITS_MAX && (!c->budget || c->allocated + (1ull << (2 * bits)) / 8 * 2 + wide_bytes(bits) <= c->budget);
}
void ops_delta_by_rows(xlb_ctx* c, DeltaLoop& d, const std::vector<DeltaRows>& rules, uint64_t max_iterations, DeltaResult* res) {
    Wide b{};
    b.rows = 1u << d.hi_bits;
    b.words = b.rows / 32;
    WideRules rs = wide_rules(rules);
    const size_t smem = wide_group_bytes(b.words) * WD_GROUPS;
    if (!c->delta_wide_attr_set) CUDA_OK(cudaFuncSetAttribute(delta_wide_k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(wide_group_bytes(1u << (WD_BITS_MAX - 5)) * WD_GROUPS)));
    c->delta_wide_attr_set = true;
    const uint64_t map = (uint64_t)b.rows * b.words, marks = std::max(b.rows / 32, 2u);
    Buf all = make_buf(c, wide_bytes(d.hi_bits));
    CUDA_OK(set_async(c, all->p, 0, all->bytes));
    unsigned* at = all->as<unsigned>();
    b.delta = at, at += map;
    b.reached = at, at += map;
    b.stamp = at, at += b.rows;
    b.n_delta = at, at += b.rows;
    b.n_head = at, at += b.rows;
    b.active[0] = at, at += marks;
    b.active[1] = at, at += marks;
    b.keys = at, at += (uint64_t)DELTA_ROWS_MAX * b.rows;
    b.n_keys = at;
    Out o = out_of(c, d);
    Ctl* ctl = (Ctl*)d.ctl;
    void* args[] = {&o, &rs, &b, &max_iterations};
    prof_begin(c, "expand_mark", 0);
    CUDA_OK(cudaLaunchCooperativeKernel((const void*)delta_wide_k, dim3((unsigned)c->sm_count), dim3(DL_THREADS), args, smem, c->stream));
    check_launch(c, "expand_mark");
    unsigned long long w[4];  // tuples, candidates, iterations, left
    read_words(c, &ctl->rows_tuples, 4, w);
    res->rows = w[0];
    res->candidates = w[1];
    res->iterations = w[2];
    res->fix = w[3] == 0;
    prof_add_bytes(c, "expand_mark", w[0] / 8 + map * 12);
}
