// Joins and aggregation over column-major relations without sorting where no order is asked for:
// semi and anti joins, inner joins (equal keys grouped by counting), group-by over small domains.
#include <algorithm>

#include "xlb_kernels.cuh"
#include "xlb_ops.h"
#include "xlb_place.h"

using namespace xk;

namespace {

// The key word of a row: a column's value, or (a << 32) | b for two 32-bit columns.
struct KeyCols {
    const void* c0;
    const uint32_t* c1;
    int w0;
    __device__ __forceinline__ uint64_t operator()(uint64_t i) const {
        if (c1) {
            const uint32_t a = __ldg((const uint32_t*)c0 + i), b = __ldg(c1 + i);
            return ((uint64_t)a << 32) | b;
        }
        if (w0 == 4) return __ldg((const uint32_t*)c0 + i);
        return w0 == 8 ? (uint64_t)__ldg((const unsigned long long*)c0 + i) : (uint64_t)__ldg((const uint8_t*)c0 + i);
    }
};
struct Cols {  // columns in and out, with the side a joined column comes from
    const void* in[XLB_MAX_ARITY];
    void* out[XLB_MAX_ARITY];
    int width[XLB_MAX_ARITY];
    int n, left;  // the first `left` columns come from the left side
};
// A row out: all columns are read before any is written, so that a row costs one trip and not one a column
// (joined rows of five columns, 2.6 M of them: 80 us one by one, against 71; a selection of three columns 41, against 34).
__device__ __forceinline__ void copy_row(const Cols& c, uint64_t left, uint64_t right, uint64_t to) {
    unsigned long long v[XLB_MAX_ARITY];
#pragma unroll
    for (int k = 0; k < (int)XLB_MAX_ARITY; ++k) {
        if (k >= c.n) break;
        const uint64_t from = k < c.left ? left : right;
        if (c.width[k] == 4) v[k] = __ldg((const uint32_t*)c.in[k] + from);
        else if (c.width[k] == 8) v[k] = __ldg((const unsigned long long*)c.in[k] + from);
        else v[k] = __ldg((const uint8_t*)c.in[k] + from);
    }
#pragma unroll
    for (int k = 0; k < (int)XLB_MAX_ARITY; ++k) {
        if (k >= c.n) break;
        if (c.width[k] == 4) ((uint32_t*)c.out[k])[to] = (uint32_t)v[k];
        else if (c.width[k] == 8) ((unsigned long long*)c.out[k])[to] = v[k];
        else ((uint8_t*)c.out[k])[to] = (uint8_t)v[k];
    }
}

// ---- keys of the build side: open addressing over the keys themselves, zero where a slot is free.  The key 0 has
// the slot behind the last one.  (Slots that named a row, whose key was then looked up: 4 M probes of 400 000 keys
// 73 us, now 45; their insertion 18, now 14: what is left is a random sector of the L2 a probe, 90 G/s.)
__device__ __forceinline__ uint64_t slot_of(uint64_t key, uint64_t mask) { return key ? mix64(key) & mask : mask + 1; }
__device__ __forceinline__ void claim(unsigned long long* slots, uint64_t mask, uint64_t key, DevStatus* st) {
    uint64_t h = slot_of(key, mask);
    if (!key) {
        slots[h] = 1;
        return;
    }
    for (uint64_t probe = 0; probe <= mask; ++probe) {  // bounded by the table size
        unsigned long long cur = slots[h];
        if (cur == 0) cur = atomicCAS(&slots[h], 0ull, (unsigned long long)key);
        if (cur == 0 || cur == key) return;
        h = (h + 1) & mask;
    }
    set_status(st, XLB_ERR_CAPACITY, 20, key);
}
__global__ void __launch_bounds__(BLOCK) exists_build_k(KeyCols keys, uint64_t n, unsigned long long* __restrict__ slots, uint64_t mask, DevStatus* st) {
    for (uint64_t i = (uint64_t)blockIdx.x * BLOCK + threadIdx.x; i < n; i += (uint64_t)gridDim.x * BLOCK) claim(slots, mask, keys(i), st);
}
// One bit per probe row (has a match == want), and for each tile of SCAN_TILE rows how many were selected before it.
constexpr int QT_ROUNDS = SCAN_TILE / BLOCK;
__global__ void __launch_bounds__(BLOCK) exists_probe_k(KeyCols probe, uint64_t n, const unsigned long long* __restrict__ slots, uint64_t mask, bool want,
                                                       unsigned int* __restrict__ bits, SelectTiles tiles, uint64_t* __restrict__ tile_offs, uint64_t* __restrict__ total,
                                                       const Publish pub) {
    __shared__ uint32_t sm[33];
    __shared__ unsigned tile_s;
    const unsigned tile = tiles.take(tile_s);
    const uint64_t base = (uint64_t)tile * SCAN_TILE + (threadIdx.x & ~31u) * QT_ROUNDS;  // a warp's rows side by side
    uint32_t cnt = 0;
    uint64_t key[QT_ROUNDS];
    unsigned long long cur[QT_ROUNDS];
#pragma unroll
    for (int r = 0; r < QT_ROUNDS; ++r) {
        const uint64_t i = base + r * 32 + lane_id();
        key[r] = i < n ? probe(i) : 0;
    }
#pragma unroll
    for (int r = 0; r < QT_ROUNDS; ++r) cur[r] = base + r * 32 + lane_id() < n ? __ldg(&slots[slot_of(key[r], mask)]) : 0ull;
#pragma unroll
    for (int r = 0; r < QT_ROUNDS; ++r) {
        const uint64_t i = base + r * 32 + lane_id();
        if (key[r]) {
            uint64_t h = mix64(key[r]) & mask;
            for (uint64_t p = 0; p < mask && cur[r] && cur[r] != key[r]; ++p) {  // bounded by the table size
                h = (h + 1) & mask;
                cur[r] = __ldg(&slots[h]);
            }
        }
        const bool found = cur[r] && (!key[r] || cur[r] == key[r]);
        const unsigned b = __ballot_sync(FULL, i < n && found == want);
        if (lane_id() == 0 && base + r * 32 < n) bits[(base + r * 32) >> 5] = b;
        cnt += __popc(b);
    }
    uint32_t tot;
    block_exclusive_scan<uint32_t>(lane_id() == 0 ? cnt : 0u, &tot, sm);
    if (threadIdx.x < 32) leave_tile(tiles, tile, tot, tile_offs, total);
    publish_last(pub);
}
// The selected rows, all columns, in order.  (A third of 4 M rows of 16 bytes: 29 us with a lane for every row, selected or
// not; 20 closed up first.)
__global__ void __launch_bounds__(BLOCK) select_rows_k(Cols cols, const unsigned int* __restrict__ bits, uint64_t n, const uint64_t* __restrict__ tile_offs, const Publish pub) {
    __shared__ uint32_t sm[33];
    __shared__ unsigned char row_s[BLOCK / 32][32 * QT_ROUNDS];
    static_assert(32 * QT_ROUNDS <= 256, "a row of the warp's is a byte");
    const uint64_t base = (uint64_t)blockIdx.x * SCAN_TILE + (threadIdx.x & ~31u) * QT_ROUNDS;
    unsigned w[QT_ROUNDS];
    uint32_t cnt = 0;
#pragma unroll
    for (int r = 0; r < QT_ROUNDS; ++r) {
        w[r] = base + r * 32 < n ? bits[(base + r * 32) >> 5] : 0u;
        cnt += __popc(w[r]);
    }
    uint32_t tot;
    uint32_t ex = block_exclusive_scan<uint32_t>(lane_id() == 0 ? cnt : 0u, &tot, sm);
    // The warp's selected rows are closed up first, so that every lane has one to copy.
    const uint64_t pos = tile_offs[blockIdx.x] + __shfl_sync(FULL, ex, 0);
    unsigned char* mine = row_s[threadIdx.x >> 5];
    unsigned at = 0;
#pragma unroll
    for (int r = 0; r < QT_ROUNDS; ++r) {
        if ((w[r] >> lane_id()) & 1u) mine[at + __popc(w[r] & lanemask_lt())] = (unsigned char)(r * 32 + lane_id());
        at += __popc(w[r]);
    }
    __syncwarp();
    for (unsigned t = lane_id(); t < at; t += 32) copy_row(cols, base + mine[t], base + mine[t], pos + t);
    publish_last(pub);
}

// ---- inner join: the build rows grouped by key
// A slot holds a key, the number of its rows and the last of them; every row names the one before it.  Where the
// rows go out a few times and groups are short, the chains are followed when they do (join_chains_k), and a
// handful of rows is put in order by a few compares.  Else lists are made of them first: starts, places,
// then each group put in row order (three kernels, 92 us for 2 M rows, which used to come before every join).  The
// line, 1 M build rows, chains / lists: groups of 2, 8 outputs a build row 257 / 322 us, 16 outputs 422 / 503; groups
// of 8, 8 outputs 249 / 284, 16 outputs 427 / 422; groups of 32, one output 277 / 254 (16 384 rows: 159 / 80).
//   A group above JOIN_GROUP_MAX rows is reported when it is met, the launches behind end at once, and the caller
// sorts instead.
//   The rows of a hub queue for its slot and on its count, some 13 ns each, so a build side of JOIN_SAMPLED
// rows and more is looked at first: while the other blocks clear the slots, one picks rows evenly and
// reports a key that it meets JOIN_OFTEN times, which one of JOIN_GROUP_MAX rows cannot be.  (2 M build rows,
// 4 M probe rows, B200: one key of 1000 rows 947 us without the sample, 787 with it, one of 1 M that no probe row asks
// for 1592 and 691; the sort alone 768 and 673; keys of at most 64 rows 330.  The sample costs some 3 us of 200,
// so smaller build sides go without: 32 768 rows all of one key 122 us sampled, 157 counted.)
constexpr unsigned JOIN_GROUP_MAX = 64;
static_assert(JOIN_GROUP_MAX <= 1u << PLACE_NUMBER_BITS, "a row's number in its group");
constexpr uint64_t JOIN_CHAIN_OUTPUTS = 8;  // outputs a build row, and rows of the longest group, up to which they
constexpr unsigned JOIN_CHAIN_ROWS = 16;    // go out from the chains
constexpr uint64_t JOIN_CHAIN_NEAR = 1ull << 18, JOIN_CHAIN_FAR = 52;  // above so many build rows, outputs a build row times rows of the longest group (1 M rows by chains / lists: groups of 16 two outputs 162 / 214, four 253 / 244, eight 373 / 298; groups of 12 four 161 / 234, eight 290 / 290; 131 072 rows, groups of 16, eight 85 / 116)
constexpr unsigned JOIN_SAMPLE = 1024, JOIN_OFTEN = 16;  // (a row a thread: a chain of latencies as long as the clearing)
constexpr uint64_t JOIN_SAMPLED = 1ull << 16;
__global__ void __launch_bounds__(JOIN_SAMPLE) group_clear_k(KeyCols keys, uint64_t n, uint4* __restrict__ slots, uint64_t slot_vecs, uint64_t* __restrict__ words, uint64_t nwords,
                                                            unsigned int* too_long) {
    if (blockIdx.x > 0) {  // (the first block, which starts at once, has the words and the sample)
        const uint64_t step = (uint64_t)(gridDim.x - 1) * JOIN_SAMPLE;
        for (uint64_t i = (uint64_t)(blockIdx.x - 1) * JOIN_SAMPLE + threadIdx.x; i < slot_vecs; i += step) slots[i] = make_uint4(0, 0, 0, 0);
        return;
    }
    __shared__ uint64_t key_s[JOIN_SAMPLE];
    __shared__ unsigned count_s[JOIN_SAMPLE], rep_s[2 * JOIN_SAMPLE];
    const unsigned me = threadIdx.x;
    const uint64_t key = keys(me * n / JOIN_SAMPLE);
    for (uint64_t i = me; i < nwords; i += JOIN_SAMPLE) words[i] = 0;
    count_s[me] = rep_s[me] = rep_s[me + JOIN_SAMPLE] = 0;
    key_s[me] = key;
    __syncthreads();
    for (unsigned h = (unsigned)mix64(key);; ++h) {  // (half of the slots stay free)
        const unsigned at = h & (2 * JOIN_SAMPLE - 1), cur = atomicCAS(&rep_s[at], 0u, me + 1);
        if (cur && key_s[cur - 1] != key) continue;
        if (atomicAdd(&count_s[cur ? cur - 1 : me], 1u) + 1 >= JOIN_OFTEN) *too_long = 1;
        break;
    }
}
// (16 bytes at once, of 16-byte aligned memory; what was there)
__device__ __forceinline__ ulonglong2 cas16(ulonglong2* at, ulonglong2 want, ulonglong2 to) {
    ulonglong2 was;
    asm volatile(
        "{ .reg .b128 w, t, o; mov.b128 w, {%2, %3}; mov.b128 t, {%4, %5}; atom.global.cas.b128 o, [%6], w, t; mov.b128 {%0, %1}, o; }"
        : "=l"(was.x), "=l"(was.y)
        : "l"(want.x), "l"(want.y), "l"(to.x), "l"(to.y), "l"(at)
        : "memory");
    return was;
}
// The first row of a key brings key, count and link by one exchange, the others count and link by one each (an
// exchange in a loop for them, too, took 1 ms on 32 768 rows of one key, against 157 us).  place: what the lists need.
// A slot is met by accesses of three sizes: the exchange of 16 bytes, the look at its key, and the additions and
// exchanges on the halves of its entry.  The PTX memory model promises nothing for overlapping accesses of different
// sizes, so this rests on the hardware: atomics, and volatile loads, of one sector are served one by one at the L2, and
// a row adds to an entry only after its look, or its exchange, has brought the key back.  (Within the model: a
// key claimed by 8 bytes and an atomic each for count and link, 71 us for the 60 below.)
// Bound by atomics whose answer is waited for, some 50 G/s on a table of 64 MB: 2 M rows 60 us (an atomic each for key,
// count and link 71; four rows a thread under way together 60 as well).
__global__ void __launch_bounds__(BLOCK) group_chain_k(KeyCols keys, uint64_t n, ulonglong2* __restrict__ slots, uint64_t mask, uint32_t* __restrict__ before, uint64_t* __restrict__ place,
                                                      volatile unsigned int* too_long, DevStatus* st) {
    for (uint64_t i = (uint64_t)blockIdx.x * BLOCK + threadIdx.x; i < n; i += (uint64_t)gridDim.x * BLOCK) {
        const unsigned stop = *too_long;
        const uint64_t key = keys(i);
        if (stop) return;
        uint64_t h = slot_of(key, mask);
        unsigned number = 0, link = 0;
        for (uint64_t probe = 0;; ++probe) {
            if (probe > mask) {  // bounded by the table size
                set_status(st, XLB_ERR_CAPACITY, 20, i);
                break;
            }
            unsigned long long there = *(volatile unsigned long long*)&slots[h].x;
            if (key && !there) {
                there = cas16(&slots[h], make_ulonglong2(0, 0), make_ulonglong2(key, ((unsigned long long)(i + 1) << 32) | 1)).x;
                if (!there) break;
            }
            if (there == key) {
                unsigned* entry = reinterpret_cast<unsigned*>(&slots[h].y);  // [0] rows, [1] the last one (plus one)
                number = atomicAdd(&entry[0], 1u);
                if (number >= JOIN_GROUP_MAX) {
                    *too_long = 1;
                    return;
                }
                if (number < JOIN_CHAIN_ROWS) link = atomicExch(&entry[1], (unsigned)i + 1);  // (longer chains are not followed)
                break;
            }
            h = (h + 1) & mask;
        }
        before[i] = link;
        place[i] = place_of(h, number);
    }
}
// Lists, for joins whose rows go out often or whose groups are long: a slot's entry becomes start << 32 | rows, and
// starts[last row of a chain] is the start as well.  Groups may lie in any order: a block takes the room for its slots'
// rows with one atomic.
__global__ void __launch_bounds__(BLOCK) group_start_k(ulonglong2* __restrict__ slots, uint64_t count, uint32_t* __restrict__ starts, unsigned int* __restrict__ used) {
    __shared__ uint32_t sm[33], room_s;
    const uint64_t base = (uint64_t)blockIdx.x * SCAN_TILE + threadIdx.x;
    unsigned len[SCAN_IPT], last[SCAN_IPT], mine = 0;
#pragma unroll
    for (int k = 0; k < SCAN_IPT; ++k) {
        const uint64_t h = base + (uint64_t)k * BLOCK;
        const unsigned long long e = h < count ? slots[h].y : 0ull;
        len[k] = (unsigned)e;
        last[k] = (unsigned)(e >> 32);
        mine += len[k];
    }
    uint32_t tot;
    uint32_t at = block_exclusive_scan<uint32_t>(mine, &tot, sm);
    if (threadIdx.x == 0) room_s = tot ? atomicAdd(used, tot) : 0u;
    __syncthreads();
    at += room_s;
#pragma unroll
    for (int k = 0; k < SCAN_IPT; ++k) {
        if (!len[k]) continue;
        reinterpret_cast<unsigned*>(&slots[base + (uint64_t)k * BLOCK].y)[1] = at;
        starts[last[k] - 1] = at;
        at += len[k];
    }
}
__global__ void __launch_bounds__(BLOCK) group_fill_k(const uint64_t* __restrict__ place, uint64_t n, const ulonglong2* __restrict__ slots, uint32_t* __restrict__ rows) {
    for (uint64_t i = (uint64_t)blockIdx.x * BLOCK + threadIdx.x; i < n; i += (uint64_t)gridDim.x * BLOCK) {
        const uint64_t p = place[i];
        rows[(uint32_t)(slots[place_slot(p)].y >> 32) + place_number(p)] = (uint32_t)i;
    }
}
// Four slots a thread at a time: a slot is a chain of loads (60 us one at a time for 4 M slots, against 50).
__global__ void __launch_bounds__(BLOCK) group_order_k(const ulonglong2* __restrict__ slots, uint64_t count, uint32_t* __restrict__ rows) {
    constexpr int S = 4, SHORT = 4;
    const uint64_t step = (uint64_t)gridDim.x * BLOCK;
    for (uint64_t h0 = (uint64_t)blockIdx.x * BLOCK + threadIdx.x; h0 < count; h0 += S * step) {
        unsigned len[S], at[S];
        uint32_t v[S][SHORT];
#pragma unroll
        for (int s = 0; s < S; ++s) {
            const unsigned long long e = h0 + s * step < count ? slots[h0 + s * step].y : 0ull;
            len[s] = (unsigned)e;
            at[s] = (unsigned)(e >> 32);
        }
#pragma unroll
        for (int s = 0; s < S; ++s)
#pragma unroll
            for (int k = 0; k < SHORT; ++k) v[s][k] = len[s] > 1 && len[s] <= SHORT && k < (int)len[s] ? rows[at[s] + k] : 0xFFFFFFFFu;
#pragma unroll
        for (int s = 0; s < S; ++s) {
            if (len[s] < 2) continue;
            if (len[s] <= SHORT) {  // most groups: placed by rank (row numbers differ)
#pragma unroll
                for (int k = 0; k < SHORT; ++k) {
                    unsigned rank = 0;
#pragma unroll
                    for (int q = 0; q < SHORT; ++q) rank += v[s][q] < v[s][k];  // (what is past the end is above all)
                    if (k < (int)len[s]) rows[at[s] + rank] = v[s][k];
                }
                continue;
            }
            uint32_t* g = rows + at[s];
            for (unsigned a = 1; a < len[s]; ++a) {  // insertion sort in place
                const uint32_t x = g[a];
                unsigned b = a;
                while (b && g[b - 1] > x) {
                    g[b] = g[b - 1];
                    --b;
                }
                g[b] = x;
            }
        }
    }
}
// What each probe row meets (its slot's entry) and how many outputs come before it: in its tile, and before the tile.
__global__ void __launch_bounds__(BLOCK) join_probe_k(KeyCols probe, uint64_t n, const ulonglong2* __restrict__ table, uint64_t mask, uint64_t* __restrict__ match,
                                                     uint32_t* __restrict__ in_tile, SelectTiles tiles, uint64_t* __restrict__ tile_offs, uint64_t* __restrict__ total,
                                                     unsigned int* __restrict__ longest, const unsigned int* __restrict__ too_long, const Publish pub) {
    __shared__ uint64_t sm[33];
    __shared__ unsigned tile_s;
    const unsigned stop = *too_long;
    const unsigned tile = tiles.take(tile_s), lane = lane_id();
    if (stop) n = 0;  // (the tiles still leave their sums, all zero, and the words)
    const uint64_t base = (uint64_t)tile * SCAN_TILE + (threadIdx.x & ~31u) * QT_ROUNDS + lane;  // a warp's rows side by side
    uint64_t key[QT_ROUNDS];
    ulonglong2 m[QT_ROUNDS];
#pragma unroll
    for (int r = 0; r < QT_ROUNDS; ++r) key[r] = base + r * 32 < n ? probe(base + r * 32) : 0;
#pragma unroll
    for (int r = 0; r < QT_ROUNDS; ++r) m[r] = base + r * 32 < n ? __ldg(&table[slot_of(key[r], mask)]) : make_ulonglong2(0, 0);
    uint64_t mine = 0;
    uint32_t most = 0;
#pragma unroll
    for (int r = 0; r < QT_ROUNDS; ++r) {
        uint64_t h = mix64(key[r]) & mask;
        for (uint64_t p = 0; p < mask && m[r].y && m[r].x != key[r]; ++p) {  // bounded by the table size
            h = (h + 1) & mask;
            m[r] = __ldg(&table[h]);
        }
        if (m[r].x != key[r]) m[r].y = 0;
        mine += (uint32_t)m[r].y;
        most = max(most, (uint32_t)m[r].y);
    }
    most = __reduce_max_sync(FULL, most);
    if (lane == 0 && most > *longest) atomicMax(longest, most);  // (a look first: it settles soon)
    for (int d = 16; d; d >>= 1) mine += __shfl_xor_sync(FULL, mine, d);
    uint64_t tot;
    uint64_t at = block_exclusive_scan<uint64_t>(lane == 0 ? mine : 0ull, &tot, sm);
    if (threadIdx.x < 32) leave_tile(tiles, tile, tot, tile_offs, total);
    at = __shfl_sync(FULL, at, 0);
#pragma unroll
    for (int r = 0; r < QT_ROUNDS; ++r) {
        uint32_t run = (uint32_t)m[r].y;  // (32 groups of at most JOIN_GROUP_MAX rows; longer ones are not used)
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t v = __shfl_up_sync(FULL, run, d);
            if (lane >= (unsigned)d) run += v;
        }
        if (base + r * 32 < n) {
            match[base + r * 32] = m[r].y;
            in_tile[base + r * 32] = (uint32_t)at + run - (uint32_t)m[r].y;
        }
        at += __shfl_sync(FULL, run, 31);
    }
    publish_last(pub);
}
struct OutputsBefore {
    const uint64_t* tile;
    const uint32_t* in_tile;
    __device__ __forceinline__ uint64_t operator[](uint64_t row) const { return tile[row / SCAN_TILE] + in_tile[row]; }
};
// Load-balanced output of an inner join (the scheme of expand_k), all columns of both sides written
// at once: the pairs of row numbers never touch memory.  IPT outputs a thread, each step for all of them
// before the next; one where that still leaves SMs without a block (1848 outputs: 22 us -> 14; 2.6 M: 71 -> 61).
template <int IPT>
__global__ void __launch_bounds__(BLOCK) join_emit_k(const uint64_t* __restrict__ match, const OutputsBefore off, uint64_t nrows, uint64_t total, const uint32_t* __restrict__ rows,
                                                    const uint32_t* __restrict__ starts, Cols cols, const Publish pub) {
    constexpr int TILE = BLOCK * IPT;
    __shared__ unsigned rel[TILE + 2];
    __shared__ uint64_t row_s[2];
    const uint64_t o0 = (uint64_t)blockIdx.x * TILE, o1 = o0 + TILE < total ? o0 + TILE : total;
    if (threadIdx.x < 64) {
        const uint64_t o = threadIdx.x < 32 ? o0 : o0 + TILE;
        const uint64_t ub = o < total ? warp_partition_point(nrows, [&](uint64_t i) { return off[i] <= o; }) : nrows + 1;
        if (lane_id() == 0) row_s[threadIdx.x >> 5] = ub - 1;
    }
    __syncthreads();
    const uint64_t r0 = row_s[0], r1 = row_s[1] < nrows ? row_s[1] : nrows - 1, span = r1 - r0 + 1;
    const bool in_smem = span <= (uint64_t)(TILE + 2);
    if (in_smem)
        for (unsigned i = threadIdx.x; i < (unsigned)span; i += BLOCK) {
            const uint64_t at = off[r0 + i];
            rel[i] = at <= o0 ? 0u : (at - o0 < (uint64_t)TILE ? (unsigned)(at - o0) : (unsigned)TILE);
        }
    const uint64_t skip0 = o0 - off[r0];
    __syncthreads();
    uint64_t l[IPT], r[IPT];
#pragma unroll
    for (int u = 0; u < IPT; ++u) {
        const unsigned t = u * BLOCK + threadIdx.x;
        l[u] = r0;
        r[u] = 0;
        if (t >= (unsigned)(o1 - o0)) continue;
        uint64_t lo = 0, hi = span;
        if (in_smem) {
            while (lo < hi) {
                const uint64_t mid = (lo + hi) >> 1;
                if (rel[mid] <= t) lo = mid + 1;
                else hi = mid;
            }
            r[u] = lo == 1 ? skip0 + t : (uint64_t)(t - rel[lo - 1]);
        } else {
            while (lo < hi) {
                const uint64_t mid = (lo + hi) >> 1;
                if (off[r0 + mid] <= o0 + t) lo = mid + 1;
                else hi = mid;
            }
            r[u] = o0 + t - off[r0 + lo - 1];
        }
        l[u] = r0 + lo - 1;
    }
#pragma unroll
    for (int u = 0; u < IPT; ++u) {
        const unsigned t = u * BLOCK + threadIdx.x;
        if (t < (unsigned)(o1 - o0)) r[u] += starts[(match[l[u]] >> 32) - 1];
    }
#pragma unroll
    for (int u = 0; u < IPT; ++u) {
        const unsigned t = u * BLOCK + threadIdx.x;
        if (t < (unsigned)(o1 - o0)) r[u] = rows[r[u]];
    }
#pragma unroll
    for (int u = 0; u < IPT; ++u) {
        const unsigned t = u * BLOCK + threadIdx.x;
        if (t < (unsigned)(o1 - o0)) copy_row(cols, l[u], r[u], o0 + t);
    }
    publish_last(pub);
}

// The same from the chains: a warp takes 32 probe rows, follows their chains together, puts the rows in order in
// shared memory and writes their outputs side by side.  (2.6 M outputs of five columns 64 us, bound by the random
// sectors of the build side's columns; from lists 57, whose making took 92.)
constexpr int GL_SHORT = 4;
constexpr unsigned JC_ROOM = 512;  // outputs at a time; a row's are fewer
static_assert(JOIN_GROUP_MAX <= JC_ROOM, "a probe row fits");
__global__ void __launch_bounds__(BLOCK) join_chains_k(const uint64_t* __restrict__ match, const OutputsBefore off, uint64_t nrows, const uint32_t* __restrict__ before, Cols cols,
                                                      const Publish pub) {
    __shared__ uint32_t right_s[BLOCK / 32][JC_ROOM];
    __shared__ unsigned char left_s[BLOCK / 32][JC_ROOM];
    const unsigned lane = lane_id();
    uint32_t* right = right_s[threadIdx.x >> 5];
    unsigned char* left = left_s[threadIdx.x >> 5];
    const uint64_t base = (uint64_t)blockIdx.x * BLOCK + (threadIdx.x & ~31u);
    const uint64_t m = base + lane < nrows ? match[base + lane] : 0ull;
    const unsigned len = (unsigned)m;
    unsigned incl = len;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const unsigned v = __shfl_up_sync(FULL, incl, d);
        if (lane >= (unsigned)d) incl += v;
    }
    const unsigned all = __shfl_sync(FULL, incl, 31);
    const uint64_t to = all ? off[base] : 0;
    uint32_t v[GL_SHORT];
    v[0] = (uint32_t)(m >> 32);
#pragma unroll
    for (int k = 1; k < GL_SHORT; ++k) v[k] = k < (int)len ? __ldg(&before[v[k - 1] - 1]) : 0xFFFFFFFFu;
    for (unsigned done = 0; done < all;) {  // as many rows at a time as there is room for
        const bool mine = incl > done && incl - done <= JC_ROOM;
        const unsigned at = incl - len - done, stop = __shfl_sync(FULL, incl, 31 - __clz(__ballot_sync(FULL, mine)));
        if (mine && len <= GL_SHORT) {  // placed by rank (row numbers differ)
#pragma unroll
            for (int k = 0; k < GL_SHORT; ++k) {
                unsigned rank = 0;
#pragma unroll
                for (int q = 0; q < GL_SHORT; ++q) rank += v[q] < v[k];  // (what is past the end is above all)
                if (k < (int)len) {
                    right[at + rank] = v[k] - 1;
                    left[at + k] = (unsigned char)lane;
                }
            }
        } else if (mine) {
            uint32_t x = v[0];
            for (unsigned a = 0; a < len; ++a, x = x ? __ldg(&before[x - 1]) : 0) {  // insertion sort in place
                unsigned b = a;
                while (b && right[at + b - 1] > x - 1) {
                    right[at + b] = right[at + b - 1];
                    --b;
                }
                right[at + b] = x - 1;
                left[at + a] = (unsigned char)lane;
            }
        }
        __syncwarp();
        for (unsigned t = lane; t < stop - done; t += 32) copy_row(cols, base + left[t], right[t], to + done + t);
        __syncwarp();
        done = stop;
    }
    publish_last(pub);
}

// ---- a few thousand rows: an operation by one block
// What a small join or group-by cost was its launches (some 5 us each with the gap before it) and its read-backs (10 us)
// and nothing of its sizes: 3001 facts through semi join, inner join and group-by took 17 launches and 6
// read-backs, 164 us; one launch and one read-back each, 87.  Tables lie in shared memory; results go straight into
// columns with room for the most there can be.  The block takes eight rows a thread: 8192 facts 109 us (by grids 190;
// 12 000, with the smaller operations still by one block, 150 against 190, 20 000 177 against 203).
constexpr unsigned SMALL_THREADS = 1024, SMALL_IPT = 8, SMALL_PROBE = SMALL_THREADS * SMALL_IPT, SMALL_BUILD = 4096;
constexpr unsigned SMALL_SLOTS = 2 * SMALL_BUILD;  // (half of them stay free)
constexpr unsigned SMALL_CHAIN = 12;   // rows of a key up to which a thread puts them in order by itself (groups of 20: 98 us, ranked row by row 45; by grids 75)
constexpr unsigned SMALL_GROUP = 256;  // rows of a key, at most: each is ranked among the others
constexpr uint64_t SMALL_OUTPUTS = 3 * SMALL_PROBE / 2;  // of a join; more go out by a grid
constexpr unsigned SMALL_GROUPS_BYTES = 160u << 10;
constexpr unsigned GROUP_PEERS = 4;  // lanes of one key from which a warp puts their values together first ...
constexpr unsigned GROUP_HUB = 256;  // ... where some group has more rows than this (looking for them costs 7 us for 8192 rows; 30 groups of 273: 38 us either way)
__device__ __forceinline__ unsigned small_slots(uint64_t build) {
    unsigned cap = 64;
    while (cap < 2 * build) cap <<= 1;
    return cap;
}
// Exclusive sums over the rows of a block that has SMALL_IPT rounds of them (row = round * SMALL_THREADS + thread);
// warp_s: SMALL_IPT * 32 + 1 words.  `mine` becomes what comes before.
__device__ __forceinline__ unsigned rounds_before(unsigned (&mine)[SMALL_IPT], unsigned* warp_s) {
    const unsigned lane = lane_id(), warp = threadIdx.x >> 5;
    unsigned len[SMALL_IPT];
#pragma unroll
    for (unsigned r = 0; r < SMALL_IPT; ++r) {
        len[r] = mine[r];
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const unsigned v = __shfl_up_sync(FULL, mine[r], d);
            if (lane >= (unsigned)d) mine[r] += v;
        }
        if (lane == 31) warp_s[r * 32 + warp] = mine[r];
    }
    __syncthreads();
    if (warp == 0) {
        unsigned before = 0;
        for (unsigned r = 0; r < SMALL_IPT; ++r) {
            const unsigned v = warp_s[r * 32 + lane];
            unsigned incl = v;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const unsigned x = __shfl_up_sync(FULL, incl, d);
                if (lane >= (unsigned)d) incl += x;
            }
            warp_s[r * 32 + lane] = before + incl - v;
            before += __shfl_sync(FULL, incl, 31);
        }
        if (lane == 0) warp_s[SMALL_IPT * 32] = before;
    }
    __syncthreads();
#pragma unroll
    for (unsigned r = 0; r < SMALL_IPT; ++r) mine[r] = mine[r] - len[r] + warp_s[r * 32 + warp];
    return warp_s[SMALL_IPT * 32];
}
__device__ __forceinline__ unsigned small_claim(unsigned long long* slots, unsigned mask, uint64_t key) {  // (a slot is free: twice as many as keys)
    for (unsigned h = (unsigned)mix64(key) & mask;; h = (h + 1) & mask) {
        const unsigned long long cur = atomicCAS(&slots[h], 0ull, (unsigned long long)key);
        if (cur == 0 || cur == key) return h;
    }
}
__global__ void __launch_bounds__(SMALL_THREADS, 1) exists_small_k(KeyCols keys, unsigned build, KeyCols probe, unsigned n, bool want, Cols cols, unsigned long long* total, const Publish pub) {
    extern __shared__ unsigned long long small_s[];
    __shared__ unsigned warp_s[SMALL_IPT * 32 + 1], zero_s;
    const unsigned cap = small_slots(build), mask = cap - 1;
    unsigned short* list = reinterpret_cast<unsigned short*>(small_s + cap);
    uint64_t key[SMALL_IPT];
#pragma unroll
    for (unsigned r = 0; r < SMALL_IPT; ++r) key[r] = r * SMALL_THREADS + threadIdx.x < n ? probe(r * SMALL_THREADS + threadIdx.x) : 0;
    for (unsigned h = threadIdx.x; h < cap; h += SMALL_THREADS) small_s[h] = 0;
    if (threadIdx.x == 0) zero_s = 0;
    __syncthreads();
    for (unsigned i = threadIdx.x; i < build; i += SMALL_THREADS) {
        const uint64_t k = keys(i);
        if (k) small_claim(small_s, mask, k);
        else zero_s = 1;
    }
    __syncthreads();
    unsigned at[SMALL_IPT];
    bool on[SMALL_IPT];
#pragma unroll
    for (unsigned r = 0; r < SMALL_IPT; ++r) {
        bool found = zero_s != 0;
        if (key[r]) {
            unsigned h = (unsigned)mix64(key[r]) & mask;
            while (small_s[h] && small_s[h] != key[r]) h = (h + 1) & mask;
            found = small_s[h] != 0;
        }
        on[r] = r * SMALL_THREADS + threadIdx.x < n && found == want;
        at[r] = on[r];
    }
    const unsigned m = rounds_before(at, warp_s);
#pragma unroll
    for (unsigned r = 0; r < SMALL_IPT; ++r)
        if (on[r]) list[at[r]] = (unsigned short)(r * SMALL_THREADS + threadIdx.x);
    __syncthreads();
    for (unsigned t = threadIdx.x; t < m; t += SMALL_THREADS) copy_row(cols, list[t], list[t], t);
    if (threadIdx.x == 0) *total = m;
    publish_now(pub);
}
// What is left for join_emit_k where there are more outputs than room or a key has many rows, so that the grids need
// not find it out again (8000 probe rows, 80 000 outputs: 98 us when they did, 66 without the attempt, 45 now; 32 000
// written by the one block 82 to 96, now 44; 100 rows of one key on either side 107, by a sort of all, now 36).  Per probe row, the outputs before it, its group and the group's start ...
struct SmallLists {
    uint64_t* match;
    uint32_t *before, *start;
    uint64_t* tile;  // (nothing: `before` counts from the first row)
    uint32_t* rows;  // ... in the build rows by group
};
struct Rounds {
    unsigned v[SMALL_IPT];
};
// (a function of its own: as part of the kernel it took registers from the way without it, 32.6 us for 2392 probe rows, now 30.8; 963 21.8, 20.7)
__device__ __noinline__ void leave_lists(KeyCols keys, unsigned build, unsigned n, unsigned long long* small_s, const unsigned* count, const unsigned* chain, const unsigned short* after, unsigned cap,
                                         unsigned* warp_s, Rounds at, Rounds slot, SmallLists lists) {
    constexpr unsigned NONE = ~0u;
    const unsigned mask = cap - 1;
    unsigned start[SMALL_IPT];  // of each slot's rows
    static_assert(SMALL_SLOTS <= SMALL_PROBE, "rounds of slots");
    __syncthreads();  // (warp_s)
#pragma unroll
    for (unsigned r = 0; r < SMALL_IPT; ++r) start[r] = r * SMALL_THREADS + threadIdx.x < cap ? count[r * SMALL_THREADS + threadIdx.x] : 0u;
    const unsigned others = rounds_before(start, warp_s);
    unsigned rank[SMALL_BUILD / SMALL_THREADS], in[SMALL_BUILD / SMALL_THREADS];
#pragma unroll
    for (unsigned r = 0; r < SMALL_BUILD / SMALL_THREADS; ++r) {  // of each build row in its chain
        const unsigned i = r * SMALL_THREADS + threadIdx.x;
        in[r] = NONE;
        rank[r] = 0;
        if (i >= build) continue;
        const uint64_t k = keys(i);
        unsigned h = cap;
        if (k)
            for (h = (unsigned)mix64(k) & mask; small_s[h] != k;) h = (h + 1) & mask;
        in[r] = h;
        for (unsigned x = chain[h]; x; x = after[x - 1]) rank[r] += x - 1 < i;
    }
    __syncthreads();
    unsigned* starts = reinterpret_cast<unsigned*>(small_s);  // (the keys have been looked up)
#pragma unroll
    for (unsigned r = 0; r < SMALL_IPT; ++r)
        if (r * SMALL_THREADS + threadIdx.x < cap) starts[r * SMALL_THREADS + threadIdx.x] = start[r];
    if (threadIdx.x == 0) starts[cap] = others;
    __syncthreads();
#pragma unroll
    for (unsigned r = 0; r < SMALL_BUILD / SMALL_THREADS; ++r)
        if (in[r] != NONE) lists.rows[starts[in[r]] + rank[r]] = r * SMALL_THREADS + threadIdx.x;
#pragma unroll
    for (unsigned r = 0; r < SMALL_IPT; ++r) {
        const unsigned i = r * SMALL_THREADS + threadIdx.x;
        if (i >= n) break;
        lists.match[i] = ((uint64_t)(i + 1) << 32) | (slot.v[r] != NONE ? count[slot.v[r]] : 0u);
        lists.before[i] = at.v[r];
        lists.start[i] = slot.v[r] != NONE ? starts[slot.v[r]] : 0u;
        if (i % SCAN_TILE == 0) lists.tile[i / SCAN_TILE] = 0;
    }
}
// words: outputs; what became of them: 0 written, 1 listed, 2 nothing, as a group is too long.
__global__ void __launch_bounds__(SMALL_THREADS, 1) join_small_k(KeyCols keys, unsigned build, KeyCols probe, unsigned n, Cols cols, uint64_t room, SmallLists lists, unsigned long long* words,
                                                               const Publish pub) {
    extern __shared__ unsigned long long small_s[];
    __shared__ unsigned warp_s[SMALL_IPT * 32 + 1], long_s, too_long_s;
    const unsigned cap = small_slots(build), mask = cap - 1;
    unsigned* count = reinterpret_cast<unsigned*>(small_s + cap);  // rows of a slot's key (of the key 0: behind the others) ...
    unsigned* chain = count + cap + 1;                             // ... the first of them, plus one
    unsigned short* after = reinterpret_cast<unsigned short*>(chain + cap + 1);
    uint64_t key[SMALL_IPT];
#pragma unroll
    for (unsigned r = 0; r < SMALL_IPT; ++r) key[r] = r * SMALL_THREADS + threadIdx.x < n ? probe(r * SMALL_THREADS + threadIdx.x) : 0;
    for (unsigned h = threadIdx.x; h <= cap; h += SMALL_THREADS) {
        if (h < cap) small_s[h] = 0;
        count[h] = chain[h] = 0;
    }
    if (threadIdx.x == 0) long_s = too_long_s = 0;
    __syncthreads();
    for (unsigned i = threadIdx.x; i < build; i += SMALL_THREADS) {
        const uint64_t k = keys(i);
        const unsigned h = k ? small_claim(small_s, mask, k) : cap;
        // (both by one native atomic each: a compare-and-swap of both together cost 40 us where all rows have one key)
        const unsigned number = atomicAdd(&count[h], 1u);
        if (number >= SMALL_CHAIN) long_s = 1;
        if (number >= SMALL_GROUP) too_long_s = 1;
        if (number < SMALL_GROUP) after[i] = (unsigned short)atomicExch(&chain[h], i + 1);
    }
    __syncthreads();
    if (too_long_s) {
        if (threadIdx.x == 0) words[1] = 2;
        publish_now(pub);
        return;
    }
    constexpr unsigned NONE = ~0u;
    Rounds at, slot;
#pragma unroll
    for (unsigned r = 0; r < SMALL_IPT; ++r) {
        slot.v[r] = NONE;
        if (key[r]) {
            unsigned h = (unsigned)mix64(key[r]) & mask;
            while (small_s[h] && small_s[h] != key[r]) h = (h + 1) & mask;
            if (small_s[h]) slot.v[r] = h;
        } else if (r * SMALL_THREADS + threadIdx.x < n) slot.v[r] = cap;
        at.v[r] = slot.v[r] != NONE ? count[slot.v[r]] : 0u;
    }
    const unsigned m = rounds_before(at.v, warp_s);
    const bool listed = m > room || long_s;
    if (!listed) {
        for (unsigned h = threadIdx.x; h <= cap; h += SMALL_THREADS) {  // chains put in row order
            if (count[h] < 2) continue;
            unsigned sorted = 0;
            for (unsigned x = chain[h]; x;) {
                const unsigned next = after[x - 1];
                if (!sorted || sorted > x) {
                    after[x - 1] = (unsigned short)sorted;
                    sorted = x;
                } else {
                    unsigned p = sorted;
                    while (after[p - 1] && after[p - 1] < x) p = after[p - 1];
                    after[x - 1] = after[p - 1];
                    after[p - 1] = (unsigned short)x;
                }
                x = next;
            }
            chain[h] = sorted;
        }
        __syncthreads();
#pragma unroll
        for (unsigned r = 0; r < SMALL_IPT; ++r)
            for (unsigned x = slot.v[r] != NONE ? chain[slot.v[r]] : 0u, to = at.v[r]; x; x = after[x - 1], ++to) copy_row(cols, r * SMALL_THREADS + threadIdx.x, x - 1, to);
    } else {
        leave_lists(keys, build, n, small_s, count, chain, after, cap, warp_s, at, slot, lists);
    }
    if (threadIdx.x == 0) {
        words[0] = m;
        words[1] = listed;
    }
    publish_now(pub);
}

// ---- group-by over a small domain of keys: tables indexed by the key itself
// Rows per key (the tile's rows are combined in shared memory first: one hub key would serialise
// the atomics), whose maximum tells whether the values may be added up by atomics as well.
struct GroupKey {
    KeyCols cols;
    int lo_bits;  // two columns: index = (a << lo_bits) | b
    __device__ __forceinline__ uint32_t operator()(uint64_t i) const {
        const uint64_t k = cols(i);
        return cols.c1 ? (uint32_t)(((k >> 32) << lo_bits) | (k & 0xFFFFFFFFull)) : (uint32_t)k;
    }
};
__global__ void __launch_bounds__(BLOCK) group_bound_k(KeyCols keys, uint64_t n, unsigned long long* __restrict__ bound, const Publish pub) {
    uint64_t o = 0;
    for (uint64_t i = (uint64_t)blockIdx.x * BLOCK + threadIdx.x; i < n; i += (uint64_t)gridDim.x * BLOCK) o |= keys(i);
    block_or(o, bound);
    publish_last(pub);
}
__global__ void __launch_bounds__(BLOCK) group_rows_k(GroupKey key, uint64_t n, unsigned int* __restrict__ count) {
    __shared__ uint32_t skey[DX_SLOTS], scnt[DX_SLOTS];
    const uint64_t ntiles = (n + DX_TILE - 1) / DX_TILE;
    for (uint64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        for (int s = threadIdx.x; s < DX_SLOTS; s += BLOCK) {
            skey[s] = DX_EMPTY;
            scnt[s] = 0;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < DX_IPT; ++k) {
            const uint64_t i = tile * DX_TILE + (uint64_t)k * BLOCK + threadIdx.x;
            if (i >= n) break;
            const uint32_t x = key(i), h = dx_slot(skey, x);
            if (h != DX_NONE) atomicAdd(&scnt[h], 1u);
            else atomicAdd(&count[x], 1u);
        }
        __syncthreads();
        for (int s = threadIdx.x; s < DX_SLOTS; s += BLOCK)
            if (scnt[s]) atomicAdd(&count[skey[s]], scnt[s]);
        __syncthreads();
    }
}
__global__ void __launch_bounds__(BLOCK) group_tiles_k(const unsigned int* __restrict__ count, uint64_t domain, SelectTiles tiles, uint64_t* __restrict__ tile_offs, uint64_t* __restrict__ total,
                                                      unsigned long long* __restrict__ longest, const Publish pub) {
    __shared__ uint32_t sm[33];
    __shared__ unsigned tile_s;
    const unsigned tile = tiles.take(tile_s);
    const uint64_t base = (uint64_t)tile * SCAN_TILE;
    uint32_t groups = 0, most = 0;
#pragma unroll
    for (int k = 0; k < SCAN_IPT; ++k) {
        const uint64_t x = base + (uint64_t)k * BLOCK + threadIdx.x;
        const uint32_t c = x < domain ? count[x] : 0u;
        groups += c != 0;
        most = c > most ? c : most;
    }
    most = __reduce_max_sync(FULL, most);
    if (lane_id() == 0 && most) atomicMax(longest, (unsigned long long)most);
    uint32_t tot;
    block_exclusive_scan<uint32_t>(groups, &tot, sm);
    if (threadIdx.x < 32) leave_tile(tiles, tile, tot, tile_offs, total);
    publish_last(pub);
}
struct Aggs {
    const void* val[XLB_MAX_ARITY];
    unsigned long long* table[XLB_MAX_ARITY];  // null: a count, which the row counts hold
    void* out[XLB_MAX_ARITY];
    uint8_t op[XLB_MAX_ARITY], width[XLB_MAX_ARITY], out_width[XLB_MAX_ARITY];
    int n;
};
__global__ void __launch_bounds__(BLOCK) group_add_k(GroupKey key, uint64_t n, Aggs a) {
    for (uint64_t i = (uint64_t)blockIdx.x * BLOCK + threadIdx.x; i < n; i += (uint64_t)gridDim.x * BLOCK) {
        const uint32_t x = key(i);
        for (int q = 0; q < a.n; ++q) {
            unsigned long long* t = a.table[q];
            if (!t) continue;
            const unsigned long long v = a.width[q] == 4 ? __ldg((const uint32_t*)a.val[q] + i) : __ldg((const unsigned long long*)a.val[q] + i);
            // (a look first: once a group has settled most values change nothing; a stale look only costs an atomic)
            if (a.op[q] == XLB_AGG_SUM) atomicAdd(&t[x], v);
            else if (a.op[q] == XLB_AGG_MIN) {
                if (v < t[x]) atomicMin(&t[x], v);
            } else if (v > t[x]) atomicMax(&t[x], v);
        }
    }
}
__global__ void __launch_bounds__(BLOCK) group_emit_k(const unsigned int* __restrict__ count, uint64_t domain, const uint64_t* __restrict__ tile_offs, Aggs a, int lo_bits, int w0, void* key0,
                                                     uint32_t* key1, const Publish pub) {
    __shared__ uint32_t sm[33];
    const uint64_t base = (uint64_t)blockIdx.x * SCAN_TILE + (uint64_t)threadIdx.x * SCAN_IPT;
    uint32_t c[SCAN_IPT], groups = 0;
#pragma unroll
    for (int k = 0; k < SCAN_IPT; ++k) {
        c[k] = base + k < domain ? count[base + k] : 0u;
        groups += c[k] != 0;
    }
    uint32_t tot;
    uint64_t pos = tile_offs[blockIdx.x] + block_exclusive_scan<uint32_t>(groups, &tot, sm);
    for (int k = 0; k < SCAN_IPT; ++k) {
        if (!c[k]) continue;
        const uint64_t x = base + k;
        if (key1) {
            ((uint32_t*)key0)[pos] = (uint32_t)(x >> lo_bits);
            key1[pos] = (uint32_t)(x & ((1ull << lo_bits) - 1));
        } else if (w0 == 4) ((uint32_t*)key0)[pos] = (uint32_t)x;
        else ((unsigned long long*)key0)[pos] = x;
        for (int q = 0; q < a.n; ++q) {
            const unsigned long long v = a.table[q] ? a.table[q][x] : c[k];
            if (a.out_width[q] == 4) ((uint32_t*)a.out[q])[pos] = (uint32_t)v;
            else ((unsigned long long*)a.out[q])[pos] = v;
        }
        ++pos;
    }
    publish_last(pub);
}

// Lanes of one key: each knows those after it, 1, 2, 4 ... further on, so that their values come to the first of them.
// An atomic of 64 bits on shared memory is a loop that lanes and warps on one address go through one after the other,
// some 17 ns each: 8192 rows of one key, a count, a sum and a minimum, 311 us, now 39 (by the grids 62).
struct Peers {
    unsigned char after[5];  // lane, or 32: none
    unsigned rounds;         // of the warp
    bool first;
    __device__ __forceinline__ void find(unsigned x, bool on) {
        rounds = 0;
        first = on;
        const unsigned lane = lane_id(), all = __match_any_sync(FULL, on ? x : ~0u), rest = all & ~lanemask_lt() & ~(1u << lane);
        const unsigned most = __reduce_max_sync(FULL, on ? __popc(all) : 0);
        if (most < GROUP_PEERS) return;
        rounds = 32 - __clz(most - 1);
        first = on && !(all & lanemask_lt());
        unsigned next = on && rest ? __ffs(rest) - 1 : 32;
#pragma unroll
        for (unsigned k = 0; k < 5; ++k) {
            if (k >= rounds) break;
            after[k] = (unsigned char)next;
            const unsigned then = __shfl_sync(FULL, next, next & 31);
            if (next != 32) next = then;
        }
    }
    template <class Op>
    __device__ __forceinline__ unsigned long long gather(unsigned long long v, Op op) const {
#pragma unroll
        for (unsigned k = 0; k < 5; ++k) {
            if (k >= rounds) break;
            const unsigned long long theirs = __shfl_sync(FULL, v, after[k] & 31);
            if (after[k] != 32) v = op(v, theirs);
        }
        return v;
    }
};
// words: bound of the keys, groups.  All ones for the groups: the tables do not fit, nothing was done.
__global__ void __launch_bounds__(SMALL_THREADS, 1) group_small_k(GroupKey key, unsigned n, Aggs a, int tables, int w0, void* key0, uint32_t* key1, unsigned long long* words, const Publish pub) {
    extern __shared__ unsigned long long small_s[];
    __shared__ unsigned long long bound_s;
    __shared__ unsigned warp_s[33];
    const unsigned lane = lane_id(), warp = threadIdx.x >> 5;
    uint64_t k[SMALL_IPT], all = 0;
#pragma unroll
    for (unsigned r = 0; r < SMALL_IPT; ++r) {
        k[r] = r * SMALL_THREADS + threadIdx.x < n ? key.cols(r * SMALL_THREADS + threadIdx.x) : 0;
        all |= k[r];
    }
    if (threadIdx.x == 0) bound_s = 0;
    __syncthreads();
#pragma unroll
    for (int d = 16; d; d >>= 1) all |= __shfl_xor_sync(FULL, all, d);
    if (lane == 0 && all) atomicOr(&bound_s, (unsigned long long)all);
    __syncthreads();
    const unsigned long long bound = bound_s;
    int bits = 64 - __clzll(bound);
    if (key.cols.c1) {
        key.lo_bits = max(64 - __clzll(bound & 0xFFFFFFFFull), 1);
        bits = 64 - __clzll(bound >> 32) + key.lo_bits;
    }
    if (bits > 20 || ((8u * tables + 4u) << bits) > SMALL_GROUPS_BYTES) {
        if (threadIdx.x == 0) {
            words[0] = bound;
            words[1] = ~0ull;
        }
        publish_now(pub);
        return;
    }
    const unsigned domain = 1u << bits;
    unsigned* count = reinterpret_cast<unsigned*>(small_s + (size_t)tables * domain);
    int t = 0;
    for (int q = 0; q < a.n; ++q) {
        if (a.op[q] == XLB_AGG_COUNT) continue;
        for (unsigned x = threadIdx.x; x < domain; x += SMALL_THREADS) small_s[t * domain + x] = a.op[q] == XLB_AGG_MIN ? ~0ull : 0ull;
        ++t;
    }
    for (unsigned x = threadIdx.x; x < domain; x += SMALL_THREADS) count[x] = 0;
    __syncthreads();
    const auto key_of = [&](unsigned r) { return key.cols.c1 ? (unsigned)(((k[r] >> 32) << key.lo_bits) | (k[r] & 0xFFFFFFFFull)) : (unsigned)k[r]; };
    bool hub = false;
#pragma unroll
    for (unsigned r = 0; r < SMALL_IPT; ++r)
        if (r * SMALL_THREADS + threadIdx.x < n) hub |= atomicAdd(&count[key_of(r)], 1u) >= GROUP_HUB;
    const auto add_up = [&](auto together) {
        constexpr bool TOGETHER = decltype(together)::value;
#pragma unroll
        for (unsigned r = 0; r < SMALL_IPT; ++r) {
            const unsigned i = r * SMALL_THREADS + threadIdx.x, x = key_of(r);
            if ((TOGETHER ? i - lane : i) >= n) break;  // (a warp's rows together)
            const bool on = i < n;
            Peers peers;
            if (TOGETHER) peers.find(x, on);
            int t = 0;
            for (int q = 0; q < a.n; ++q) {
                if (a.op[q] == XLB_AGG_COUNT) continue;
                unsigned long long* to = &small_s[t++ * domain + x];
                unsigned long long v = !on ? 0ull : a.width[q] == 4 ? __ldg((const uint32_t*)a.val[q] + i) : __ldg((const unsigned long long*)a.val[q] + i);
                if (TOGETHER) {
                    v = a.op[q] == XLB_AGG_SUM   ? peers.gather(v, [](unsigned long long y, unsigned long long z) { return y + z; })
                        : a.op[q] == XLB_AGG_MIN ? peers.gather(v, [](unsigned long long y, unsigned long long z) { return min(y, z); })
                                                 : peers.gather(v, [](unsigned long long y, unsigned long long z) { return max(y, z); });
                    if (!peers.first) continue;
                }
                if (a.op[q] == XLB_AGG_SUM) atomicAdd(to, v);
                else if (a.op[q] == XLB_AGG_MIN) atomicMin(to, v);
                else atomicMax(to, v);
            }
        }
    };
    if (__syncthreads_or(hub)) add_up(std::true_type());
    else add_up(std::false_type());
    __syncthreads();
    unsigned groups = 0;
    for (unsigned x0 = 0; x0 < domain; x0 += SMALL_THREADS) {  // in the order of the keys
        const unsigned x = x0 + threadIdx.x, c = x < domain ? count[x] : 0u, some = __ballot_sync(FULL, c != 0);
        if (lane == 0) warp_s[warp] = __popc(some);
        __syncthreads();
        unsigned before = 0, total = 0;
        for (unsigned w = 0; w < SMALL_THREADS / 32; ++w) {
            if (w < warp) before += warp_s[w];
            total += warp_s[w];
        }
        if (c) {
            const unsigned pos = groups + before + __popc(some & lanemask_lt());
            if (key1) {
                ((uint32_t*)key0)[pos] = x >> key.lo_bits;
                key1[pos] = x & ((1u << key.lo_bits) - 1);
            } else if (w0 == 4) ((uint32_t*)key0)[pos] = x;
            else ((unsigned long long*)key0)[pos] = x;
            t = 0;
            for (int q = 0; q < a.n; ++q) {
                const unsigned long long v = a.op[q] == XLB_AGG_COUNT ? c : small_s[t++ * domain + x];
                if (a.out_width[q] == 4) ((uint32_t*)a.out[q])[pos] = (uint32_t)v;
                else ((unsigned long long*)a.out[q])[pos] = v;
            }
        }
        groups += total;
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        words[0] = bound;
        words[1] = groups;
    }
    publish_now(pub);
}

KeyCols key_cols(const xlb_rel* r, const uint32_t* keys, uint32_t nk) {
    KeyCols k{r->cols[keys[0]]->p, nullptr, (int)type_width(r->schema.types[keys[0]])};
    if (nk == 2) k.c1 = r->cols[keys[1]]->as<uint32_t>();
    return k;
}
int bit_length(uint64_t v) { return v ? 64 - __builtin_clzll(v) : 0; }
uint64_t row_bytes(const xlb_schema& s) {
    uint64_t bytes = 0;
    for (uint32_t i = 0; i < s.arity; ++i) bytes += type_width(s.types[i]);
    return bytes;
}
// out: a fresh relation of `rows` rows with the columns of `from` in place `at` and after
void add_columns(xlb_ctx* c, xlb_rel* out, Cols& cols, const xlb_rel* from, uint64_t rows) {
    for (uint32_t i = 0; i < from->schema.arity; ++i) {
        const int k = cols.n++;
        cols.width[k] = (int)type_width(from->schema.types[i]);
        out->cols[k] = make_buf(c, rows * cols.width[k]);
        cols.in[k] = from->cols[i]->p;
        cols.out[k] = out->cols[k]->p;
    }
}
// A relation whose columns had room for more rows than there are.  Giving a rest back costs 0.2 us, and as much when the
// relation goes (semi join, inner join and group-by of 3001 facts 87 us, 90 with every rest): only those worth it.
constexpr uint64_t REST_KEPT = 16u << 10;  // bytes a column
xlb_rel* with_rows(std::unique_ptr<xlb_rel>& o, uint64_t rows) {
    o->rows = rows;
    for (uint32_t i = 0; i < o->schema.arity; ++i) {
        const uint64_t bytes = rows * type_width(o->schema.types[i]);
        if (o->cols[i]->bytes - bytes > REST_KEPT) o->cols[i]->keep(bytes);
    }
    return o.release();
}

// The sums before each tile of a kernel that calls leave_tile: the kernel's own doing, or by a scan after it.
struct Sweep {
    SelectTiles tiles;
    uint64_t* leave_at;
    Sweep(xlb_ctx* c_, uint64_t n_, uint64_t* zeroed, uint64_t* offs_, uint64_t* total_) : leave_at(offs_), c(c_), n(n_), offs(offs_), total(total_) {
        if (n <= 4ull * c->sm_count) tiles = sweep_tiles(c, zeroed, n);  // (four blocks of 256 threads and more fit an SM)
        else {
            tiles.n = (unsigned)n;
            counts = make_buf(c, n * 8);
            leave_at = counts->as<uint64_t>();
        }
    }
    // For the kernel to leave `words` words from `from` (the total among them) when it places its tiles itself.
    Publish publish(const void* from, int words) const { return counts ? Publish() : publish_by(c, n, from, words); }
    void finish() {
        if (counts) exclusive_scan<LoadU64, uint64_t>(c, LoadU64{counts->as<uint64_t>()}, n, offs, total);
    }

   private:
    xlb_ctx* c;
    uint64_t n, *offs, *total;
    Buf counts;
};

}  // namespace

// Whether one block takes it; the shared memory its kernels may ask for.  Its columns have room for the most rows there
// can be (`room` bytes); where the budget has not, the grids make them as long as the result.
static bool one_block(xlb_ctx* c, uint64_t build, uint64_t probe, uint64_t room) {
    if (!build || build > SMALL_BUILD || !probe || probe > SMALL_PROBE || !within_budget(c, room + 64)) return false;
    if (!c->query_attr_set) {
        CUDA_OK(cudaFuncSetAttribute(exists_small_k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(SMALL_SLOTS * 8 + SMALL_PROBE * 2)));
        CUDA_OK(cudaFuncSetAttribute(join_small_k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(SMALL_SLOTS * 16 + 16 + SMALL_BUILD * 2)));
        CUDA_OK(cudaFuncSetAttribute(group_small_k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMALL_GROUPS_BYTES));
        c->query_attr_set = true;
    }
    return true;
}
static unsigned slots_of(uint64_t build) {
    unsigned cap = 64;
    while (cap < 2 * build) cap <<= 1;
    return cap;
}

xlb_rel* query_exists(xlb_ctx* c, const xlb_rel* l, const xlb_rel* r, const uint32_t* lk, const uint32_t* rk, uint32_t nk, bool want) {
    if (r->rows >= 0xFFFFFFFFull) xlb_fail(XLB_ERR_CAPACITY, "join build side of %llu rows exceeds the 2^32 - 1 row limit", (unsigned long long)r->rows);
    if (one_block(c, r->rows, l->rows, l->rows * row_bytes(l->schema))) {
        std::unique_ptr<xlb_rel> o(new xlb_rel);
        o->ctx = c;
        o->schema = l->schema;
        Cols cols{};
        add_columns(c, o.get(), cols, l, l->rows);
        Buf total = make_buf(c, 8);
        prof_begin(c, "exists_small", 0);
        const Publish pub = publish_by(c, 1, total->p, 1);
        exists_small_k<<<1, SMALL_THREADS, slots_of(r->rows) * 8 + SMALL_PROBE * 2, c->stream>>>(key_cols(r, rk, nk), (unsigned)r->rows, key_cols(l, lk, nk), (unsigned)l->rows, want, cols,
                                                                                              total->as<unsigned long long>(), pub);
        check_launch(c, "exists_small");
        unsigned long long m;
        read_published(c, pub, total->p, 1, &m);
        return with_rows(o, m);
    }
    uint64_t cap = 1024;
    while (cap < 2 * r->rows) cap <<= 1;
    const uint64_t n = l->rows, tiles = (n + SCAN_TILE - 1) / SCAN_TILE;
    const uint64_t words = cap + 1 + sweep_words(tiles);
    Buf slots = make_buf(c, words * 8);
    CUDA_OK(set_async(c, slots->p, 0, words * 8));
    const KeyCols build = key_cols(r, rk, nk), probe = key_cols(l, lk, nk);
    if (r->rows) {
        prof_begin(c, "hash_insert", 0);
        exists_build_k<<<grid_for(c, r->rows), BLOCK, 0, c->stream>>>(build, r->rows, slots->as<unsigned long long>(), cap - 1, c->d_status);
        check_launch(c, "hash_insert");
    }
    Buf bits = make_buf(c, (n + 31) / 32 * 4), offs = make_buf(c, tiles * 8 + 8);
    uint64_t* total = offs->as<uint64_t>() + tiles;
    Sweep sweep(c, tiles, slots->as<uint64_t>() + cap + 1, offs->as<uint64_t>(), total);
    prof_begin(c, "hash_probe", n * 12ull);
    const Publish pub = sweep.publish(total, 1);
    exists_probe_k<<<(unsigned)tiles, BLOCK, 0, c->stream>>>(probe, n, slots->as<unsigned long long>(), cap - 1, want, bits->as<unsigned int>(), sweep.tiles, sweep.leave_at, total, pub);
    check_launch(c, "hash_probe");
    sweep.finish();
    unsigned long long m;
    read_published(c, pub, total, 1, &m);
    std::unique_ptr<xlb_rel> o(new xlb_rel);
    o->ctx = c;
    o->schema = l->schema;
    o->rows = m;
    Cols cols{};
    add_columns(c, o.get(), cols, l, m);
    if (m) {
        prof_begin(c, "select_rows", 0);
        const Publish last = publish_by(c, tiles);
        select_rows_k<<<(unsigned)tiles, BLOCK, 0, c->stream>>>(cols, bits->as<unsigned int>(), n, offs->as<uint64_t>(), last);
        check_launch(c, "select_rows");
        status_published(c, last);
    }
    return o.release();
}

// The outputs of a join from its rows by group.
static void emit_joined(xlb_ctx* c, const uint64_t* match, const OutputsBefore& outputs, uint64_t probes, uint64_t total, const uint32_t* rows, const uint32_t* starts, const Cols& cols) {
    const bool few = total <= (uint64_t)c->sm_count * BLOCK * 4;
    const uint64_t tile = few ? BLOCK : BLOCK * 4, blocks = (total + tile - 1) / tile;
    prof_begin(c, "join_emit", 0);
    const Publish last = publish_by(c, blocks);
    if (few) join_emit_k<1><<<(unsigned)blocks, BLOCK, 0, c->stream>>>(match, outputs, probes, total, rows, starts, cols, last);
    else join_emit_k<4><<<(unsigned)blocks, BLOCK, 0, c->stream>>>(match, outputs, probes, total, rows, starts, cols, last);
    check_launch(c, "join_emit");
    status_published(c, last);
}

xlb_rel* query_join(xlb_ctx* c, const xlb_rel* l, const xlb_rel* r, const uint32_t* lk, const uint32_t* rk, uint32_t nk, const xlb_schema& os) {
    const uint64_t n = r->rows;
    if (n >= 0xFFFFFFFFull) xlb_fail(XLB_ERR_CAPACITY, "join build side of %llu rows exceeds the 2^32 - 1 row limit", (unsigned long long)n);
    const uint64_t room = std::min<uint64_t>(SMALL_OUTPUTS, 4 * l->rows + 1024);
    if (one_block(c, n, l->rows, room * row_bytes(os) + l->rows * 24 + n * 4)) {
        std::unique_ptr<xlb_rel> o(new xlb_rel);
        o->ctx = c;
        o->schema = os;
        Cols cols{};
        cols.left = (int)l->schema.arity;
        add_columns(c, o.get(), cols, l, room);
        add_columns(c, o.get(), cols, r, room);
        const uint64_t tiles = (l->rows + SCAN_TILE - 1) / SCAN_TILE;
        Buf words = make_buf(c, 16 + (tiles + l->rows * 2) * 8 + n * 4);
        SmallLists lists{};
        lists.tile = words->as<uint64_t>() + 2;
        lists.match = lists.tile + tiles;
        lists.before = (uint32_t*)(lists.match + l->rows);
        lists.start = lists.before + l->rows;
        lists.rows = lists.start + l->rows;
        prof_begin(c, "join_small", 0);
        const Publish pub = publish_by(c, 1, words->p, 2);
        const unsigned cap = slots_of(n);
        join_small_k<<<1, SMALL_THREADS, cap * 16 + 16 + (unsigned)n * 2, c->stream>>>(key_cols(r, rk, nk), (unsigned)n, key_cols(l, lk, nk), (unsigned)l->rows, cols, room, lists,
                                                                                     words->as<unsigned long long>(), pub);
        check_launch(c, "join_small");
        unsigned long long w[2];
        read_published(c, pub, words->p, 2, w);
        if (w[1] == 2) return nullptr;
        if (w[1] == 0 || w[0] == 0) return with_rows(o, w[0]);
        if (w[0] > room) {
            for (uint32_t i = 0; i < os.arity; ++i) o->cols[i].reset();
            cols.n = 0;
            add_columns(c, o.get(), cols, l, w[0]);
            add_columns(c, o.get(), cols, r, w[0]);
        }
        emit_joined(c, lists.match, OutputsBefore{lists.tile, lists.before}, l->rows, w[0], lists.rows, lists.start, cols);
        return with_rows(o, w[0]);
    }
    uint64_t cap = 1024;
    while (cap < 2 * n) cap <<= 1;
    const KeyCols build = key_cols(r, rk, nk), probe = key_cols(l, lk, nk);
    const uint64_t tiles = (l->rows + SCAN_TILE - 1) / SCAN_TILE, nwords = 4 + sweep_words(tiles);
    Buf table = make_buf(c, (cap + 1) * 16 + nwords * 8), before = make_buf(c, n * 4), place = make_buf(c, n * 8);
    ulonglong2* slots = table->as<ulonglong2>();
    uint64_t* words = (uint64_t*)(slots + cap + 1);  // [0] outputs, [1] a group is too long, [2] rows of the longest group met, [3] room taken for groups, then the sweep's
    unsigned int* too_long = (unsigned int*)(words + 1);
    if (n < JOIN_SAMPLED) {
        CUDA_OK(set_async(c, table->p, 0, (cap + 1) * 16 + nwords * 8));
    } else {
        prof_begin(c, "group_clear", cap * 16ull);
        group_clear_k<<<(unsigned)std::min<uint64_t>((cap + JOIN_SAMPLE - 1) / JOIN_SAMPLE, 2ull * c->sm_count) + 1, JOIN_SAMPLE, 0, c->stream>>>(build, n, table->as<uint4>(), cap + 1, words, nwords, too_long);
        check_launch(c, "group_clear");
    }
    prof_begin(c, "hash_insert", n * 8ull);
    group_chain_k<<<grid_for(c, n), BLOCK, 0, c->stream>>>(build, n, slots, cap - 1, before->as<uint32_t>(), place->as<uint64_t>(), too_long, c->d_status);
    check_launch(c, "hash_insert");
    Buf match = make_buf(c, l->rows * 8), in_tile = make_buf(c, l->rows * 4), offs = make_buf(c, tiles * 8);
    Sweep sweep(c, tiles, words + 4, offs->as<uint64_t>(), words);
    prof_begin(c, "hash_probe", l->rows * 32ull);
    const Publish pub = sweep.publish(words, 3);
    join_probe_k<<<(unsigned)tiles, BLOCK, 0, c->stream>>>(probe, l->rows, slots, cap - 1, match->as<uint64_t>(), in_tile->as<uint32_t>(), sweep.tiles, sweep.leave_at, words, (unsigned int*)(words + 2), too_long, pub);
    check_launch(c, "hash_probe");
    sweep.finish();
    unsigned long long w[3];
    read_published(c, pub, words, 3, w);
    if (w[1]) return nullptr;
    std::unique_ptr<xlb_rel> o(new xlb_rel);
    o->ctx = c;
    o->schema = os;
    o->rows = w[0];
    Cols cols{};
    cols.left = (int)l->schema.arity;
    add_columns(c, o.get(), cols, l, w[0]);
    add_columns(c, o.get(), cols, r, w[0]);
    if (w[0]) {
        const OutputsBefore outputs{offs->as<uint64_t>(), in_tile->as<uint32_t>()};
        const bool far = n > JOIN_CHAIN_NEAR && w[2] > JOIN_CHAIN_ROWS / 2;
        if (w[0] > JOIN_CHAIN_OUTPUTS * n || w[2] > JOIN_CHAIN_ROWS || (far && w[0] * w[2] > JOIN_CHAIN_FAR * n)) {
            Buf rows = make_buf(c, n * 8);
            prof_begin(c, "group_start", cap * 16ull);
            group_start_k<<<(unsigned)((cap + SCAN_TILE) / SCAN_TILE), BLOCK, 0, c->stream>>>(slots, cap + 1, rows->as<uint32_t>() + n, (unsigned int*)(words + 3));
            check_launch(c, "group_start");
            prof_begin(c, "group_fill", n * 16ull);
            group_fill_k<<<grid_for(c, n), BLOCK, 0, c->stream>>>(place->as<uint64_t>(), n, slots, rows->as<uint32_t>());
            check_launch(c, "group_fill");
            prof_begin(c, "group_order", cap * 16ull);
            group_order_k<<<grid_for(c, cap + 1), BLOCK, 0, c->stream>>>(slots, cap + 1, rows->as<uint32_t>());
            check_launch(c, "group_order");
            emit_joined(c, match->as<uint64_t>(), outputs, l->rows, w[0], rows->as<uint32_t>(), rows->as<uint32_t>() + n, cols);
        } else {
            prof_begin(c, "join_emit", 0);
            const uint64_t blocks = (l->rows + BLOCK - 1) / BLOCK;
            const Publish last = publish_by(c, blocks);
            join_chains_k<<<(unsigned)blocks, BLOCK, 0, c->stream>>>(match->as<uint64_t>(), outputs, l->rows, before->as<uint32_t>(), cols, last);
            check_launch(c, "join_emit");
            status_published(c, last);
        }
    }
    return o.release();
}

// The tables cost a clear and a pass over the domain, four entries a row at most; a long group's atomics
// queue, some 2 us for every 1000 of its rows and three tables.  4 M rows, 250 000 groups: 162 us, with one of
// 60 000 rows 279; sorted, with one of 100 000 rows, 527 of which the attempt is some 70 (540 before there was
// one).  200 000 rows: 105 with a group of 60 000, sorted 210.
constexpr int GROUP_BITS_MAX = 26;
constexpr uint64_t GROUP_DOMAIN_FREE = 1ull << 16, GROUP_ROWS_MAX = 1ull << 16;

xlb_rel* query_groupby(xlb_ctx* c, const xlb_rel* in, const uint32_t* key_cols_in, uint32_t nk, const uint32_t* agg_cols, const uint32_t* agg_ops, uint32_t na, const xlb_schema& os) {
    if (nk > 2 || (nk == 2 && (type_width(in->schema.types[key_cols_in[0]]) != 4 || type_width(in->schema.types[key_cols_in[1]]) != 4))) return nullptr;
    const uint64_t n = in->rows;
    GroupKey key{key_cols(in, key_cols_in, nk), 0};
    uint32_t tables = 0;
    for (uint32_t a = 0; a < na; ++a) tables += agg_ops[a] != XLB_AGG_COUNT;
    std::unique_ptr<xlb_rel> o(new xlb_rel);
    o->ctx = c;
    o->schema = os;
    Aggs ag{};
    ag.n = (int)na;
    const auto results = [&](uint64_t rows) {
        for (uint32_t i = 0; i < os.arity; ++i) o->cols[i] = make_buf(c, rows * type_width(os.types[i]));
        for (uint32_t a = 0; a < na; ++a) {
            ag.val[a] = in->cols[agg_cols[a]]->p;
            ag.op[a] = (uint8_t)agg_ops[a];
            ag.width[a] = (uint8_t)type_width(in->schema.types[agg_cols[a]]);
            ag.out[a] = o->cols[nk + a]->p;
            ag.out_width[a] = (uint8_t)type_width(os.types[nk + a]);
        }
    };
    Buf words = make_buf(c, 24);  // [0] key bound, [1] groups, [2] rows of the largest
    unsigned long long w[2];
    const bool small = one_block(c, 1, n, n * row_bytes(os));
    if (small) {
        results(n);
        prof_begin(c, "group_small", 0);
        const Publish pub = publish_by(c, 1, words->p, 2);
        group_small_k<<<1, SMALL_THREADS, SMALL_GROUPS_BYTES, c->stream>>>(key, (unsigned)n, ag, (int)tables, (int)type_width(os.types[0]), o->cols[0]->p, nk == 2 ? o->cols[1]->as<uint32_t>() : nullptr,
                                                                         words->as<unsigned long long>(), pub);
        check_launch(c, "group_small");
        read_published(c, pub, words->p, 2, w);
        if (w[1] != ~0ull) return with_rows(o, w[1]);
        for (uint32_t i = 0; i < os.arity; ++i) o->cols[i].reset();
    }
    CUDA_OK(set_async(c, words->p, 0, 24));
    if (!small) {
        prof_begin(c, "group_bound", 0);
        const unsigned bound_grid = std::min(grid_for(c, n, BLOCK * 4), PUBLISH_BLOCKS_MAX);
        const Publish bound_pub = publish_by(c, bound_grid, words->p, 1);
        group_bound_k<<<bound_grid, BLOCK, 0, c->stream>>>(key.cols, n, words->as<unsigned long long>(), bound_pub);
        check_launch(c, "group_bound");
        read_published(c, bound_pub, words->p, 1, w);
    }
    int bits = bit_length(w[0]);
    if (nk == 2) {
        key.lo_bits = std::max(bit_length(w[0] & 0xFFFFFFFFull), 1);
        bits = bit_length(w[0] >> 32) + key.lo_bits;
    }
    if (bits > GROUP_BITS_MAX || (1ull << bits) > std::max<uint64_t>(4 * n, GROUP_DOMAIN_FREE)) return nullptr;
    const uint64_t domain = 1ull << bits, tiles = (domain + SCAN_TILE - 1) / SCAN_TILE;
    const uint64_t clear = (domain * 4 + 7) / 8 * 8 + sweep_words(tiles) * 8;
    Buf count = make_buf(c, clear), offs = make_buf(c, tiles * 8);
    CUDA_OK(set_async(c, count->p, 0, clear));
    prof_begin(c, "group_rows", 0);
    group_rows_k<<<grid_for(c, n, DX_TILE), BLOCK, 0, c->stream>>>(key, n, count->as<unsigned int>());
    check_launch(c, "group_rows");
    Sweep sweep(c, tiles, count->as<uint64_t>() + (domain * 4 + 7) / 8, offs->as<uint64_t>(), words->as<uint64_t>() + 1);
    prof_begin(c, "group_tiles", domain * 4ull);
    const Publish pub = sweep.publish(words->as<uint64_t>() + 1, 2);
    group_tiles_k<<<(unsigned)tiles, BLOCK, 0, c->stream>>>(count->as<unsigned int>(), domain, sweep.tiles, sweep.leave_at, words->as<uint64_t>() + 1, words->as<unsigned long long>() + 2, pub);
    check_launch(c, "group_tiles");
    sweep.finish();
    read_published(c, pub, words->as<uint64_t>() + 1, 2, w);
    const uint64_t m = w[0];
    if (tables && w[1] > GROUP_ROWS_MAX) return nullptr;
    o->rows = m;
    results(m);
    // sums and maxima start from zero, minima from all ones: two fills
    Buf acc = make_buf(c, std::max<uint64_t>(tables * domain * 8, 8));
    uint64_t at = 0, minima = 0;
    for (int pass = 0; pass < 2; ++pass) {
        for (uint32_t a = 0; a < na; ++a) {
            if (agg_ops[a] == XLB_AGG_COUNT || (agg_ops[a] == XLB_AGG_MIN) != (pass == 1)) continue;
            ag.table[a] = acc->as<unsigned long long>() + at;
            at += domain;
        }
        if (pass == 0) minima = at;
    }
    if (minima) CUDA_OK(set_async(c, acc->p, 0, minima * 8));
    if (at > minima) CUDA_OK(set_async(c, acc->as<uint64_t>() + minima, 0xFF, (at - minima) * 8));
    if (tables) {
        prof_begin(c, "groupby_reduce", 0);
        group_add_k<<<grid_for(c, n), BLOCK, 0, c->stream>>>(key, n, ag);
        check_launch(c, "groupby_reduce");
    }
    prof_begin(c, "group_emit", 0);
    const Publish last = publish_by(c, tiles);
    group_emit_k<<<(unsigned)tiles, BLOCK, 0, c->stream>>>(count->as<unsigned int>(), domain, offs->as<uint64_t>(), ag, key.lo_bits, (int)type_width(os.types[0]), o->cols[0]->p,
                                                          nk == 2 ? o->cols[1]->as<uint32_t>() : nullptr, last);
    check_launch(c, "group_emit");
    status_published(c, last);
    return o.release();
}
