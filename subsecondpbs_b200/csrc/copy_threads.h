// Helper threads for copies between a caller's memory and page-locked memory.
#pragma once

#include <unistd.h>
#if defined(__SSE2__)
#include <emmintrin.h>
#endif

#include <algorithm>
#include <condition_variable>
#include <cstddef>
#include <cstdint>
#include <cstring>
#include <exception>
#include <memory>
#include <mutex>
#include <thread>

namespace pbs {

// memcpy past the caches, for memory that the device reads next: lines that other cores
// hold dirty come out of their caches at a fraction of the link's rate. 5.2 MB filled by
// four threads and copied up in one piece: 177 us, with memcpy 699; by the driver from
// pageable memory 288.
inline void stream_copy(void* to, const void* from, size_t bytes) {
#if defined(__SSE2__)
    char* d = static_cast<char*>(to);
    const char* s = static_cast<const char*>(from);
    const size_t head = std::min<size_t>(bytes, (16 - (reinterpret_cast<uintptr_t>(d) & 15)) & 15);
    std::memcpy(d, s, head);
    size_t i = head;
    for (; i + 64 <= bytes; i += 64) {
        const __m128i* v = reinterpret_cast<const __m128i*>(s + i);
        __m128i* o = reinterpret_cast<__m128i*>(d + i);
        const __m128i a = _mm_loadu_si128(v), b = _mm_loadu_si128(v + 1), c = _mm_loadu_si128(v + 2),
                      e = _mm_loadu_si128(v + 3);
        _mm_stream_si128(o, a);
        _mm_stream_si128(o + 1, b);
        _mm_stream_si128(o + 2, c);
        _mm_stream_si128(o + 3, e);
    }
    std::memcpy(d + i, s + i, bytes - i);
    _mm_sfence();
#else
    std::memcpy(to, from, bytes);
#endif
}

// Up to three helpers beside the calling thread, started by the first call that needs
// them and kept until the object goes: waking them takes 8 us where creating and joining
// three threads takes 35. One call at a time.
class CopyThreads {
public:
    CopyThreads() = default;
    CopyThreads(const CopyThreads&) = delete;
    CopyThreads& operator=(const CopyThreads&) = delete;
    ~CopyThreads() {
        if (!s_) return;
        // In a forked child the helpers do not exist and what they wait on cannot be
        // destroyed.
        if (pid_ != getpid()) {
            (void)s_.release();
            return;
        }
        {
            std::lock_guard<std::mutex> lk(s_->m);
            s_->quit = true;
        }
        s_->wake.notify_all();
        for (std::thread& t : s_->helpers)
            if (t.joinable()) t.join();
    }

    // Calls f(first, last) for parts that cover the rows [0, n) of a copy of `bytes`
    // bytes; returns once all are done. f must not throw. Where no helper can be had the
    // calling thread does their parts.
    template <typename F>
    void split(size_t n, size_t bytes, F f) {
        const size_t cores = std::max(1u, std::thread::hardware_concurrency());
        const size_t want = std::min({kHelpers + 1, cores, n, bytes / kBytesPerPart});
        if (want < 2 || !start()) {
            f(size_t(0), n);
            return;
        }
        // A type-erased view of f for the helpers; it lives until they are done.
        struct Call {
            static void run(void* fn, size_t first, size_t last) { (*static_cast<F*>(fn))(first, last); }
        };
        State& s = *s_;
        const size_t parts = std::min(want, s.count + 1);
        {
            std::lock_guard<std::mutex> lk(s.m);
            s.run = &Call::run;
            s.fn = &f;
            s.n = n;
            s.parts = parts;
            s.left = parts - 1;
            ++s.call;
        }
        s.wake.notify_all();
        f(size_t(0), n / parts);
        std::unique_lock<std::mutex> lk(s.m);
        s.done.wait(lk, [&] { return s.left == 0; });
    }

private:
    static constexpr size_t kHelpers = 3, kBytesPerPart = size_t(64) << 10;

    struct State {
        std::mutex m;
        std::condition_variable wake, done;
        std::thread helpers[kHelpers];
        size_t count = 0;  // helpers that run
        bool quit = false;
        unsigned call = 0;
        void (*run)(void*, size_t, size_t) = nullptr;
        void* fn = nullptr;
        size_t n = 0, parts = 0, left = 0;
    };

    static void serve(State* s, size_t me) {
        std::unique_lock<std::mutex> lk(s->m);
        for (unsigned seen = 0;;) {
            s->wake.wait(lk, [&] { return s->quit || s->call != seen; });
            if (s->quit) return;
            seen = s->call;
            if (me >= s->parts) continue;
            const size_t first = s->n * me / s->parts, last = s->n * (me + 1) / s->parts;
            void (*run)(void*, size_t, size_t) = s->run;
            void* fn = s->fn;
            lk.unlock();
            run(fn, first, last);
            lk.lock();
            if (--s->left == 0) s->done.notify_one();
        }
    }

    // Whether there is a helper.
    bool start() {
        if (s_) return pid_ == getpid() && s_->count > 0;
        try {
            std::unique_ptr<State> s(new State);
            s_ = std::move(s);
            pid_ = getpid();
            for (; s_->count < kHelpers; ++s_->count)
                s_->helpers[s_->count] = std::thread(&CopyThreads::serve, s_.get(), s_->count + 1);
        } catch (const std::exception&) {  // no memory or no thread to be had: those that there are
        }
        return s_ && s_->count > 0;
    }

    std::unique_ptr<State> s_;
    pid_t pid_ = 0;
};

}  // namespace pbs
