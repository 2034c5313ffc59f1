// Rows put in order by key columns of any type: the key columns become one or a few 64-bit words that
// hold nothing but the bits that differ, the words are sorted, and the result's columns are written in
// one launch.
#include <algorithm>

#include "xlb_kernels.cuh"
#include "xlb_ops.h"

using namespace xk;

namespace {

enum : unsigned char { KIND_UNSIGNED = 0, KIND_SIGNED = 1, KIND_FLOAT = 2 };
unsigned char kind_of(uint8_t t) { return (t == XLB_I32 || t == XLB_I64) ? KIND_SIGNED : (t == XLB_F32 || t == XLB_F64) ? KIND_FLOAT : KIND_UNSIGNED; }

// Unsigned image of a value that orders as the values do (signed: sign flipped; float: IEEE
// totalOrder), and back.
__device__ __forceinline__ uint64_t image_of(const void* col, int width, int kind, uint64_t row) {
    if (width == 8) {
        const uint64_t x = ((const uint64_t*)col)[row], sign = 1ull << 63;
        if (kind == KIND_UNSIGNED) return x;
        return kind == KIND_FLOAT && (x & sign) ? ~x : x ^ sign;
    }
    if (width == 1) return ((const uint8_t*)col)[row];
    const uint32_t x = ((const uint32_t*)col)[row], sign = 1u << 31;
    if (kind == KIND_UNSIGNED) return x;
    return kind == KIND_FLOAT && (x & sign) ? ~x : x ^ sign;
}
__device__ __forceinline__ uint64_t value_of(uint64_t image, int width, int kind) {
    if (kind == KIND_UNSIGNED) return image;
    const uint64_t sign = 1ull << (8 * width - 1);
    return kind == KIND_FLOAT && !(image & sign) ? ~image : image ^ sign;  // (of a narrower value the low bytes count)
}

struct KeyPart {  // a key column's bits in a word: (image - base) << shift
    const void* col;
    uint64_t base, mask;
    unsigned char width, kind, shift, column;
};
struct KeyWord {
    KeyPart p[XLB_MAX_ARITY];
    int n = 0, bits = 0;
    bool with_row = false;  // the row number lies below the keys' bits
    __device__ __forceinline__ uint64_t operator()(uint64_t row) const {
        uint64_t w = with_row ? row : 0;
        for (int k = 0; k < n; ++k) w |= (image_of(p[k].col, p[k].width, p[k].kind, row) - p[k].base) << p[k].shift;
        return w;
    }
};
struct OutCol {
    const void* from;  // null: decoded from the key word, or (width 0) the row number itself
    void* to;
    uint64_t base, mask;
    unsigned char width, kind, shift;
};
// What is written of row `row`, whose last key word is `word`, at place `i`.
struct OutCols {
    OutCol c[XLB_MAX_ARITY];
    int n = 0;
    __device__ __forceinline__ void operator()(uint64_t i, uint64_t word, uint32_t row) const {
        for (int k = 0; k < n; ++k) {
            const OutCol& o = c[k];
            if (o.width == 0) {
                ((uint32_t*)o.to)[i] = row;
            } else if (!o.from) {
                const uint64_t x = value_of(((word >> o.shift) & o.mask) + o.base, o.width, o.kind);
                if (o.width == 4) ((uint32_t*)o.to)[i] = (uint32_t)x;
                else if (o.width == 8) ((uint64_t*)o.to)[i] = x;
                else ((uint8_t*)o.to)[i] = (uint8_t)x;
            } else if (o.width == 4) ((uint32_t*)o.to)[i] = __ldg((const uint32_t*)o.from + row);
            else if (o.width == 8) ((unsigned long long*)o.to)[i] = __ldg((const unsigned long long*)o.from + row);
            else ((uint8_t*)o.to)[i] = __ldg((const uint8_t*)o.from + row);
        }
    }
};

// Least image and the complement of the greatest one, per key column (from words of all ones).  A few
// blocks per SM with several loads in flight each: one atomic per block and word is all that meets.
template <int WIDTH>
__device__ __forceinline__ void range_of(const KeyPart& p, uint64_t n, uint64_t& a, uint64_t& b) {
    const uint64_t step = (uint64_t)gridDim.x * BLOCK;
#pragma unroll 8
    for (uint64_t i = (uint64_t)blockIdx.x * BLOCK + threadIdx.x; i < n; i += step) {
        const uint64_t v = image_of(p.col, WIDTH, p.kind, i);
        a = min(a, v);
        b = min(b, ~v);
    }
}
__global__ void __launch_bounds__(BLOCK) key_range_k(const KeyWord w, uint64_t n, unsigned long long* __restrict__ least, const Publish pub) {
    __shared__ unsigned long long s[2];
    for (int k = 0; k < w.n; ++k) {
        uint64_t a = ~0ull, b = ~0ull;
        if (threadIdx.x < 2) s[threadIdx.x] = ~0ull;
        if (w.p[k].width == 4) range_of<4>(w.p[k], n, a, b);
        else if (w.p[k].width == 8) range_of<8>(w.p[k], n, a, b);
        else range_of<1>(w.p[k], n, a, b);
        for (int d = 16; d; d >>= 1) {
            a = min(a, (uint64_t)__shfl_xor_sync(FULL, a, d));
            b = min(b, (uint64_t)__shfl_xor_sync(FULL, b, d));
        }
        __syncthreads();
        if (lane_id() == 0) {
            atomicMin(&s[0], (unsigned long long)a);
            atomicMin(&s[1], (unsigned long long)b);
        }
        __syncthreads();
        if (threadIdx.x < 2) atomicMin(&least[2 * k + threadIdx.x], s[threadIdx.x]);
    }
    publish_last(pub);
}
// A row number that came out of a sort.  One that gave up (its status says so) leaves places unwritten, and
// this kernel runs before the host has read the status: no row is looked for outside the relation.
__device__ __forceinline__ uint32_t row_of(uint32_t row, uint64_t n) { return row < n ? row : 0u; }
__global__ void __launch_bounds__(BLOCK) key_word_k(const KeyWord w, const uint32_t* __restrict__ rows, uint64_t* __restrict__ out, uint64_t n) {
    for (uint64_t i = (uint64_t)blockIdx.x * BLOCK + threadIdx.x; i < n; i += (uint64_t)gridDim.x * BLOCK) out[i] = w(rows ? row_of(rows[i], n) : i);
}
// Words that were sorted by their bits from `mend` on only: each row finds the others of its prefix next to
// it and counts those that come before it.  *unmended: a prefix has more rows than that is done for.
constexpr unsigned MEND_MAX = 32;
template <bool MEND>
__global__ void __launch_bounds__(BLOCK) rows_out_k(const OutCols out, const uint64_t* __restrict__ words, const uint32_t* __restrict__ rows, uint64_t row_mask, uint64_t n, int mend,
                                                    unsigned long long* __restrict__ unmended, const Publish pub) {
    for (uint64_t i = (uint64_t)blockIdx.x * BLOCK + threadIdx.x; i < n; i += (uint64_t)gridDim.x * BLOCK) {
        const uint64_t w = words ? words[i] : 0;
        uint64_t to = i;
        if (MEND) {
            const uint64_t prefix = w >> mend;
            unsigned left = 0, right = 0;
            for (; left < MEND_MAX && left < i; ++left) {
                const uint64_t v = words[i - left - 1];
                if (v >> mend != prefix) break;
                if (v > w) --to;
            }
            for (; right < MEND_MAX && i + right + 1 < n; ++right) {
                const uint64_t v = words[i + right + 1];
                if (v >> mend != prefix) break;
                if (v < w) ++to;
            }
            if (left == MEND_MAX || right == MEND_MAX) *unmended = 1;
        }
        out(to, w, row_of(rows ? rows[i] : row_mask ? (uint32_t)(w & row_mask) : (uint32_t)i, n));
    }
    publish_last(pub);
}
// How often rows picked evenly meet one with the same bits from `mend` on.
constexpr unsigned SAMPLE = 2048, SAMPLE_SLOTS = 4096, SAMPLE_MEET = SAMPLE / 16;
__global__ void __launch_bounds__(1024) prefix_sample_k(const KeyWord w, uint64_t n, int mend, unsigned long long* __restrict__ met, const Publish pub) {
    __shared__ unsigned long long table[SAMPLE_SLOTS];
    __shared__ unsigned met_s;
    for (unsigned i = threadIdx.x; i < SAMPLE_SLOTS; i += 1024) table[i] = ~0ull;  // (no prefix: mend > 0)
    if (threadIdx.x == 0) met_s = 0;
    __syncthreads();
    for (unsigned i = threadIdx.x; i < SAMPLE; i += 1024) {
        const unsigned long long prefix = w(i * n / SAMPLE) >> mend;
        unsigned h = (unsigned)mix64(prefix) & (SAMPLE_SLOTS - 1);
        for (unsigned probe = 0; probe < SAMPLE_SLOTS; ++probe) {
            const unsigned long long cur = atomicCAS(&table[h], ~0ull, prefix);
            if (cur == prefix) atomicAdd(&met_s, 1u);
            if (cur == ~0ull || cur == prefix) break;
            h = (h + 1) & (SAMPLE_SLOTS - 1);
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) *met = met_s;
    publish_now(pub);
}

// a few thousand rows: words made, sorted and (the last one) turned into columns in one launch each
struct LoadRow {
    KeyWord word;
    const uint32_t* rows;  // in and out may be one buffer: the block reads all before it writes
    __device__ __forceinline__ uint64_t operator()(unsigned i, uint32_t& val) const {
        val = rows ? rows[i] : i;
        return word(val);
    }
};
struct StoreRow {
    uint32_t* rows;
    __device__ __forceinline__ void operator()(unsigned i, uint64_t, uint32_t val) const { rows[i] = val; }
};
struct StoreOut {
    OutCols out;
    __device__ __forceinline__ void operator()(unsigned i, uint64_t key, uint32_t val) const { out(i, key, val); }
};

int bits_of(uint64_t v) { return v ? 64 - __builtin_clzll(v) : 1; }

// The key columns cut into words, least significant word first; a column that came before is no key again.
// `range`: least and complement of the greatest image of each part, or null: all bits of the type.
std::vector<KeyWord> words_of(const KeyWord& all, const unsigned long long* range) {
    std::vector<KeyWord> words;
    for (int k = all.n - 1; k >= 0; --k) {
        KeyPart p = all.p[k];
        int bits = 8 * p.width;
        p.base = 0;
        if (range) {
            const uint64_t least = range[2 * k], most = ~range[2 * k + 1];
            bits = most > least ? 64 - __builtin_clzll(most - least) : 0;
            p.base = least;
        }
        if (bits == 0) continue;
        if (words.empty() || words.back().bits + bits > 64) words.emplace_back();
        KeyWord& w = words.back();
        p.shift = (unsigned char)w.bits;
        p.mask = bits == 64 ? ~0ull : (1ull << bits) - 1;
        w.bits += bits;
        w.p[w.n++] = p;
    }
    return words;
}

// Puts the rows of `r` in (stable) order by `keys` and writes `out`: columns of the result, with `from` the
// column of `r`.  What a pass of the sort moves is what this costs: columns shrink to the bits in which
// their values differ (ids below 2^19 and times within 2^40 us are one word of 59 bits), row numbers lie
// in the word's free bits where they fit (16 bytes moved per row and pass, not 24), and columns that the
// last word holds come out of it in order, so that only the others are gathered.  4 M rows (u32 id, i64
// time, f32) by (id, time): 11 passes, three gathers and four passes of sign mapping before, now
// 8 passes and one gather; see sort_rows for the times.
void order_rows(xlb_ctx* c, const xlb_rel* r, const uint32_t* keys, uint32_t nk, OutCols out) {
    const uint64_t n = r->rows;
    if (n == 0) return;
    if (n >= (1ull << 32)) xlb_fail(XLB_ERR_CAPACITY, "sort of %llu rows exceeds the 2^32 row limit", (unsigned long long)n);
    KeyWord all;
    unsigned seen = 0;
    for (uint32_t k = 0; k < nk; ++k) {
        if ((seen >> keys[k]) & 1u) continue;
        seen |= 1u << keys[k];
        const uint8_t t = r->schema.types[keys[k]];
        all.p[all.n++] = KeyPart{r->cols[keys[k]]->p, 0, 0, (unsigned char)type_width(t), kind_of(t), 0, (unsigned char)keys[k]};
    }
    const bool small = n <= (uint64_t)SS_MAX && !c->lb_first_tile;
    std::vector<KeyWord> words;
    if (small) {
        words = words_of(all, nullptr);
    } else if (all.n) {
        Buf least = make_buf(c, 16 * XLB_MAX_ARITY);
        CUDA_OK(set_async(c, least->p, 0xFF, 16 * XLB_MAX_ARITY));
        prof_begin(c, "key_range", n * 8ull * all.n);
        const unsigned grid = std::min(grid_for(c, n, BLOCK * 8), 6u * c->sm_count);
        const Publish pub = publish_by(c, grid, least->p, 2 * all.n);
        key_range_k<<<grid, BLOCK, 0, c->stream>>>(all, n, least->as<unsigned long long>(), pub);
        check_launch(c, "key_range");
        unsigned long long range[2 * XLB_MAX_ARITY];
        read_published(c, pub, least->p, 2 * all.n, range);
        words = words_of(all, range);
    }
    bool rows_wanted = words.size() > 1;
    if (!words.empty())
        for (int k = 0; k < out.n; ++k) {  // columns that the last word holds
            OutCol& o = out.c[k];
            const KeyPart* p = nullptr;
            if (o.from)
                for (int q = 0; q < words.back().n; ++q)
                    if (words.back().p[q].col == o.from && words.back().p[q].width == o.width) p = &words.back().p[q];
            if (!p) {
                rows_wanted = true;
                continue;
            }
            o.from = nullptr;
            o.base = p->base;
            o.mask = p->mask;
            o.shift = p->shift;
            o.kind = p->kind;
        }
    Buf rows;
    if (small) {
        for (size_t q = 0; q < words.size(); ++q) {
            const LoadRow load{words[q], rows ? rows->as<uint32_t>() : nullptr};
            if (q + 1 == words.size()) {
                radix_small(c, load, StoreOut{out}, n, 0xFFu);
            } else {
                if (!rows) rows = make_buf(c, n * 4);
                radix_small(c, load, StoreRow{rows->as<uint32_t>()}, n, 0xFFu);
            }
        }
        if (!words.empty()) return;
    }
    Buf last;
    uint64_t row_mask = 0;
    int row_bits = 0;
    if (words.size() == 1) {
        KeyWord& w = words[0];
        row_bits = rows_wanted ? bits_of(n - 1) : 0;
        if (w.bits + row_bits > 64) row_bits = 0;
        w.with_row = row_bits > 0;
        row_mask = (1ull << row_bits) - 1;
        for (int k = 0; k < w.n; ++k) w.p[k].shift = (unsigned char)(w.p[k].shift + row_bits);
        for (int k = 0; k < out.n; ++k) out.c[k].shift = (unsigned char)(out.c[k].shift + row_bits);
    }
    const auto sort_word = [&](const KeyWord& w, int from, int bits) {
        last = make_buf(c, n * 8);
        prof_begin(c, "key_word", n * 8ull);
        key_word_k<<<grid_for(c, n), BLOCK, 0, c->stream>>>(w, rows ? rows->as<uint32_t>() : nullptr, last->as<uint64_t>(), n);
        check_launch(c, "key_word");
        const Digits digits = run_of_digits(from, bits);
        radix_sort(c, last, rows_wanted && !row_bits ? &rows : nullptr, n, 0xFFu, ~0ull, false, &digits);
    };
    const unsigned grid = grid_for(c, n);
    // Many bits and values spread over them: the highest log2(n) bits tell nearly all rows apart, so only
    // they are sorted by, and rows_out puts the few of one prefix in order.  A sample says whether they do
    // (ids that are few or lie close together do not); a prefix of many rows that it missed costs the
    // passes made so far.  (4 M rows of 59 bits: three passes of 50 us and not eight.)
    if (words.size() == 1) {
        const KeyWord& w = words[0];
        const int high = (bits_of(n - 1) + 7) / 8 * 8, mend = row_bits + w.bits - high;
        if ((w.bits + 7) / 8 > high / 8 + 1) {
            Buf flags = make_buf(c, 16);
            CUDA_OK(set_async(c, flags->p, 0, 16));
            unsigned long long *met = flags->as<unsigned long long>(), *unmended = met + 1, h;
            const Publish asked = publish_by(c, 1, met, 1);
            prof_begin(c, "prefix_sample", 0);
            prefix_sample_k<<<1, 1024, 0, c->stream>>>(w, n, mend, met, asked);
            check_launch(c, "prefix_sample");
            read_published(c, asked, met, 1, &h);
            if (h <= SAMPLE_MEET) {
                sort_word(w, mend, high);
                const Publish pub = publish_by(c, grid, unmended, 1);
                prof_begin(c, "rows_out", 0);
                rows_out_k<true><<<grid, BLOCK, 0, c->stream>>>(out, last->as<uint64_t>(), rows ? rows->as<uint32_t>() : nullptr, row_mask, n, mend, unmended, pub);
                check_launch(c, "rows_out");
                read_published(c, pub, unmended, 1, &h);
                if (!h) return;
                rows.reset();
            }
        }
    }
    for (const KeyWord& w : words) sort_word(w, row_bits, w.bits);
    const Publish pub = publish_by(c, grid);
    prof_begin(c, "rows_out", 0);
    rows_out_k<false><<<grid, BLOCK, 0, c->stream>>>(out, last ? last->as<uint64_t>() : nullptr, rows ? rows->as<uint32_t>() : nullptr, row_mask, n, 0, nullptr, pub);
    check_launch(c, "rows_out");
    status_published(c, pub);
}

}  // namespace

Buf sort_permutation(xlb_ctx* c, const xlb_rel* r, const uint32_t* keys, uint32_t nk) {
    Buf idx = make_buf(c, r->rows * 4);
    OutCols out;
    out.n = 1;
    out.c[0] = OutCol{nullptr, idx->p, 0, 0, 0, 0, 0};
    order_rows(c, r, keys, nk, out);
    return idx;
}

xlb_rel* sort_rows(xlb_ctx* c, const xlb_rel* in, const uint32_t* keys, uint32_t nk) {
    ops_rel_columns(c, in);
    std::unique_ptr<xlb_rel> o(new xlb_rel);
    o->ctx = c;
    o->schema = in->schema;
    o->rows = in->rows;
    OutCols out;
    for (uint32_t i = 0; i < in->schema.arity; ++i) {
        const uint32_t w = type_width(in->schema.types[i]);
        o->cols[i] = make_buf(c, in->rows * w);
        if (in->rows) out.c[out.n++] = OutCol{in->cols[i]->p, o->cols[i]->p, 0, 0, (unsigned char)w, 0, 0};
    }
    order_rows(c, in, keys, nk, out);
    return o.release();
}
