// A column of runs, written out by host threads: no device in it.
#pragma once
#if defined(__SSE2__)
#include <emmintrin.h>
#endif

#include <algorithm>
#include <atomic>
#include <chrono>
#include <condition_variable>
#include <cstdint>
#include <exception>
#include <mutex>
#include <thread>
#include <vector>

template <class T>
struct Run {
    T row, value;
};

// Rows [lo, hi) of the column, a cache line at a time.  A line that runs meet in is put together first: written
// in parts, some of them around the cache, it cost 0.3 us.
template <class T>
inline void fill_rows(T* to, const Run<T>* runs, uint64_t n_runs, uint64_t n, uint64_t lo, uint64_t hi) {
    constexpr uint64_t line = 64 / sizeof(T);
    uint64_t r = std::upper_bound(runs, runs + n_runs, lo, [](uint64_t row, const Run<T>& x) { return row < x.row; }) - runs - 1;
    const auto end_of = [&](uint64_t run) { return run + 1 < n_runs ? (uint64_t)runs[run + 1].row : n; };
    uint64_t end = end_of(r);
    for (uint64_t at = lo; at < hi;) {
        alignas(64) T buf[line];
        const bool whole = (uintptr_t)(to + at) % 64 == 0 && hi - at >= line;
        const uint64_t m = whole ? line : 1;
        for (uint64_t k = 0; k < m; ++k) {
            while (at + k >= end) end = end_of(++r);
            buf[k] = runs[r].value;
        }
        if (!whole) {
            to[at++] = buf[0];
            continue;
        }
        // this line, and those behind it that lie in the run it ends with
        const uint64_t lines = end >= at + 2 * line ? (std::min(end, hi) - at) / line : 1;
#if defined(__SSE2__)
        __m128i v[4];
        for (int k = 0; k < 4; ++k) v[k] = _mm_load_si128(reinterpret_cast<const __m128i*>(buf) + k);
        __m128i* out = reinterpret_cast<__m128i*>(to + at);
        for (int k = 0; k < 4; ++k) _mm_stream_si128(out + k, v[k]);
        v[0] = v[1] = v[2] = v[3] = sizeof(T) == 4 ? _mm_set1_epi32((int)buf[line - 1]) : _mm_set1_epi64x((long long)buf[line - 1]);
        for (out += 4; out < reinterpret_cast<__m128i*>(to + at) + 4 * lines; out += 4)
            for (int k = 0; k < 4; ++k) _mm_stream_si128(out + k, v[k]);
#else
        std::copy(buf, buf + line, to + at);
        std::fill(to + at + line, to + at + lines * line, buf[line - 1]);
#endif
        at += lines * line;
    }
#if defined(__SSE2__)
    _mm_sfence();
#endif
}
// Threads that write a column out.  They are started (11 us each) while the runs are on their way, and wait for them
// awake, for a while (the runs take some 60 us; a sleeping thread is 50 us late): what was on the stream before may
// take any time, and nobody else's cores.  Without any thread to be had the caller does all of it.
template <class T>
class Filler {
    enum { WAIT, FILL, LEAVE };
    static constexpr uint64_t CHUNK = 256ull << 10;  // bytes a thread takes at a time
    static constexpr std::chrono::microseconds AWAKE{1000};
    std::atomic<int> go{WAIT};
    std::atomic<uint64_t> next{0};
    std::mutex mu;
    std::condition_variable told;
    T* to = nullptr;
    const Run<T>* runs = nullptr;
    uint64_t n_runs = 0, n = 0;
    std::vector<std::thread> helpers;

    void work() {
        constexpr uint64_t rows = CHUNK / sizeof(T);
        for (uint64_t at; (at = next.fetch_add(rows, std::memory_order_relaxed)) < n;) fill_rows(to, runs, n_runs, n, at, std::min(n, at + rows));
    }
    void wait() {
        const auto until = std::chrono::steady_clock::now() + AWAKE;
        while (go.load(std::memory_order_acquire) == WAIT) {
            if (std::chrono::steady_clock::now() > until) {
                std::unique_lock<std::mutex> lock(mu);
                told.wait(lock, [this] { return go.load(std::memory_order_acquire) != WAIT; });
                return;
            }
            std::this_thread::yield();
        }
    }
    void tell(int what) {
        {
            std::lock_guard<std::mutex> lock(mu);
            go.store(what, std::memory_order_release);
        }
        told.notify_all();
    }

   public:
    explicit Filler(unsigned threads) {
        try {
            helpers.reserve(threads);
            for (unsigned t = 1; t < threads; ++t)
                helpers.emplace_back([this] {
                    wait();
                    if (go.load(std::memory_order_acquire) == FILL) work();
                });
        } catch (const std::exception&) {  // no thread (or memory for one) to be had
        }
    }
    void fill(T* column, const Run<T>* r, uint64_t count, uint64_t rows) {
        to = column;
        runs = r;
        n_runs = count;
        n = rows;
        tell(FILL);
        work();
    }
    ~Filler() {
        if (go.load(std::memory_order_relaxed) == WAIT) tell(LEAVE);
        for (auto& t : helpers) t.join();
    }
};
