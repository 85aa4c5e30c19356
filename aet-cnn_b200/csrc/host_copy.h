// Host-side copies between a caller's pageable memory and the library's page-locked staging memory.
//
// cudaMemcpyAsync on pageable memory goes through the driver's own staging buffer on the calling thread (measured on the
// target hosts: 12.7 GB/s up for an 80 MB batch, 21 GB/s down).  A memcpy on one core is bound by that core (19 GB/s from
// memory) while the link takes 53 GB/s, so large copies are cut into chunks that a few helper threads share with the
// calling thread, and finished pieces are sent to the device while the rest is still being copied.
#pragma once
#include <atomic>
#include <chrono>
#include <condition_variable>
#include <mutex>
#include <string.h>
#include <thread>
#include <vector>

// One per context: its helpers are started by the first large copy and end with the context.  One job at a time (one host
// thread drives one context).  The calling thread never waits for a helper to wake up: it takes chunks like the helpers
// do, closes the job when none is left, and waits only for helpers that are inside a chunk.
class HostCopier {
public:
    // Waking a sleeping thread costs the waker about 10 us and the woken one 30 to 50 us (virtual machines), so all helpers
    // are woken only for a copy that takes several times that on one core.
    static constexpr size_t kWakeFrom = 4 * 1024 * 1024;
    // Two helpers stay awake for a millisecond after a job, which is longer than a serving or training loop takes to come
    // back; while they are, smaller copies are shared too (1.5 MB: 76 us alone).  With nobody awake a copy from here on
    // wakes one helper, 10 us that the copy itself gets little for: it is for the copies that follow.
    static constexpr size_t kParallelFrom = 512 * 1024;
    static constexpr int kHelpers = 5, kLingering = 2;   // six copying threads saturate the host's memory on this path
    static constexpr size_t kChunk = 128 * 1024;

    ~HostCopier() {
        {
            std::lock_guard<std::mutex> g(m_);
            stop_ = true;
            quit_.store(true);
        }
        wake_.notify_all();
        for (std::thread &t : threads_) t.join();
    }

    // Copies `bytes` from src to dst.  `whole`: the size of the copy that this one is a piece of.
    void copy(void *dst, const void *src, size_t bytes, size_t whole = 0) {
        if (bytes < kParallelFrom || !reserve((bytes + kChunk - 1) / kChunk)) {
            memcpy(dst, src, bytes);
            return;
        }
        open_job(dst, src, bytes, (bytes + kChunk - 1) / kChunk, whole > bytes ? whole : bytes);
        for (size_t i, done = 0; done < chunks_;) {
            if ((i = next_.fetch_add(1, std::memory_order_relaxed)) < chunks_) copy_chunk(i);
            while (done < chunks_ && finished_[done].load(std::memory_order_acquire)) ++done;
        }
        close_job();
    }

    // Copies `bytes` from src through the ring of `ring_bytes` (a multiple of kChunk) at `ring`: send(ring offset, source
    // offset, length) is called on the calling thread for consecutive pieces as they are complete (a piece never wraps),
    // and freed() says how many bytes from the start have been consumed, i.e. may be overwritten in the ring.
    // send returns 0, freed what it says, or a (negative) error code, which ends the copy; `no_memory` is the code for that.
    template <typename Send, typename Freed>
    int stream(void *ring, size_t ring_bytes, const void *src, size_t bytes, Send send, Freed freed, int no_memory) {
        const size_t ring_chunks = ring_bytes / kChunk, chunks = (bytes + kChunk - 1) / kChunk;
        if (!reserve(chunks)) return no_memory;
        size_t piece = chunks / 4;   // what is left to send when the copy is done costs time: small pieces, of small copies too
        if (piece > ring_chunks / 4) piece = ring_chunks / 4;
        if (piece < 1) piece = 1;
        open_job(ring, src, bytes, ring_chunks, bytes);
        size_t done = 0, sent = 0, released = 0;
        int rc = 0;
        while (sent < chunks && rc == 0) {
            if (chunks > ring_chunks && released < sent) {
                const long long f = freed();
                if (f < 0) {   // nothing will be consumed any more
                    rc = (int)f;
                    break;
                }
                released = (size_t)f >= bytes ? chunks : (size_t)f / kChunk;
                released_.store(released, std::memory_order_release);
            }
            size_t i = next_.load(std::memory_order_relaxed);
            if (i < chunks && i < released + ring_chunks && next_.compare_exchange_strong(i, i + 1, std::memory_order_relaxed)) copy_chunk(i);
            while (done < chunks && finished_[done].load(std::memory_order_acquire)) ++done;
            while (rc == 0 && done > sent && (done - sent >= piece || done == chunks)) {
                size_t n = ring_chunks - sent % ring_chunks;   // up to the ring's end
                if (n > done - sent) n = done - sent;
                const size_t lo = sent * kChunk, hi = sent + n == chunks ? bytes : (sent + n) * kChunk;
                rc = send(sent % ring_chunks * kChunk, lo, hi - lo);
                sent += n;
            }
        }
        released_.store(chunks, std::memory_order_release);   // after an error: nobody waits for the ring any more
        close_job();
        return rc;
    }

private:
    // Marks for that many chunks; the callers are C entry points, which nothing may leave as an exception.
    bool reserve(size_t chunks) {
        try {
            if (finished_.size() < chunks) finished_ = std::vector<std::atomic<unsigned char>>(chunks);
        } catch (...) {
            return false;
        }
        return true;
    }
    void open_job(void *dst, const void *src, size_t bytes, size_t ring_chunks, size_t whole) {
        const size_t chunks = (bytes + kChunk - 1) / kChunk;
        for (size_t i = 0; i < chunks; ++i) finished_[i].store(0, std::memory_order_relaxed);
        dst_ = static_cast<unsigned char *>(dst); src_ = static_cast<const unsigned char *>(src);
        bytes_ = bytes; ring_chunks_ = ring_chunks; chunks_ = chunks;
        all_ = whole >= kWakeFrom;
        released_.store(0, std::memory_order_relaxed);
        next_.store(0, std::memory_order_relaxed);
        open_.store(true, std::memory_order_seq_cst);
        start_helpers();
        if (lingering_.load(std::memory_order_relaxed) < (all_ ? (int)threads_.size() : 1)) {
            { std::lock_guard<std::mutex> g(m_); }   // a helper about to sleep has either seen the job or will be woken
            wake_.notify_one();                       // and wakes the next one itself
        }
    }
    void close_job() {   // a helper that joins from now on finds the job closed and leaves
        open_.store(false, std::memory_order_seq_cst);
        while (busy_.load(std::memory_order_seq_cst) != 0) pause();
    }
    void copy_chunk(size_t i) {
        while (i >= released_.load(std::memory_order_acquire) + ring_chunks_) pause();
        const size_t lo = i * kChunk, n = bytes_ - lo < kChunk ? bytes_ - lo : kChunk;
        memcpy(dst_ + i % ring_chunks_ * kChunk, src_ + lo, n);
        finished_[i].store(1, std::memory_order_release);
    }
    void start_helpers() {
        if (!threads_.empty()) return;
        int n = (int)std::thread::hardware_concurrency() - 1;
        if (n > kHelpers) n = kHelpers;
        try {
            for (int k = 0; k < n; ++k) threads_.emplace_back([this] { helper(); });
        } catch (...) {
        }   // fewer helpers (or none): the calling thread copies what nobody else takes
    }
    void helper() {
        std::unique_lock<std::mutex> g(m_);
        while (true) {
            wake_.wait(g, [&] { return stop_ || work_left(); });
            if (stop_) return;
            g.unlock();
            const bool lingers = lingering_.fetch_add(1, std::memory_order_relaxed) < kLingering;
            auto until = std::chrono::steady_clock::now();
            do {
                busy_.fetch_add(1, std::memory_order_seq_cst);
                if (open_.load(std::memory_order_seq_cst)) {   // counted as busy before the check: the job cannot be replaced now
                    if (all_) wake_.notify_one();
                    for (size_t i; (i = next_.fetch_add(1, std::memory_order_relaxed)) < chunks_;) copy_chunk(i);
                }
                busy_.fetch_sub(1, std::memory_order_seq_cst);
                // a caller's next copy often follows at once: all stay awake for it
                until = std::chrono::steady_clock::now() + std::chrono::microseconds(lingers ? 1000 : 50);
                while (!work_left() && !quit_.load(std::memory_order_relaxed) && std::chrono::steady_clock::now() < until) pause();
            } while (work_left());
            lingering_.fetch_sub(1, std::memory_order_relaxed);
            g.lock();
        }
    }
    static void pause() {
#if defined(__x86_64__)
        for (int i = 0; i < 8; ++i) __builtin_ia32_pause();
#else
        std::this_thread::yield();
#endif
    }
    bool work_left() const { return open_.load(std::memory_order_seq_cst) && next_.load(std::memory_order_relaxed) < chunks_.load(std::memory_order_relaxed); }
    std::mutex m_;
    std::condition_variable wake_;
    std::vector<std::thread> threads_;
    std::vector<std::atomic<unsigned char>> finished_;
    std::atomic<size_t> next_{0}, chunks_{0};
    std::atomic<bool> open_{false};
    std::atomic<int> busy_{0}, lingering_{0};
    std::atomic<bool> quit_{false};
    unsigned char *dst_ = nullptr;
    const unsigned char *src_ = nullptr;
    size_t bytes_ = 0, ring_chunks_ = 1;
    std::atomic<size_t> released_{0};
    bool all_ = false, stop_ = false;
};
