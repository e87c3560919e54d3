// Copies between ordinary (pageable) host memory and the device.
//
// cudaMemcpyAsync from pageable memory copies through the driver's own bounce buffers on the calling thread: about 15 GB/s,
// a quarter of what the link takes, and it is what a call on host arrays consists of (9.4 MB of float images: 0.6 of 0.7 ms).
// A context therefore keeps a ring of page-locked slots and a few copy threads.  A transfer is cut into slot-sized pieces;
// the threads (and the caller) fill slots in parallel while the caller issues the DMA of every piece as soon as it is
// filled, in order.  The caller's memory is not touched after the call returns, so no wait for the stream is needed.
// Small transfers (weights, tables) share slots: they are copied by the caller and leave as one DMA each.
//
// Ring and threads belong to the context: created on first use, bounded, released with it.  Like the rest of a context they
// are used by one thread at a time.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <condition_variable>
#include <cstddef>
#include <cstdint>
#include <cstring>
#include <memory>
#include <mutex>
#include <system_error>
#include <thread>
#include <vector>
#if defined(__x86_64__)
#include <immintrin.h>
#endif

namespace zb {

class HostStage {
  public:
    // A piece costs the caller about 5 us (enqueue, event), so pieces are large; the first ones are small so that the link
    // starts early.  9.4 MB: 1250 us with memcpy and one thread in pieces of 128 KB, 480 us with streaming stores and pieces of
    // 512 KB, 280 us with two more threads (the link alone: 185 us); further threads change nothing.
    static constexpr size_t kSlot = 1024 << 10;
    static constexpr int kSlots = 16;                // 16 MB of page-locked memory
    static constexpr int kThreads = 3;
    static size_t piece_begin(int i) {               // 128, 128, 256, 512 KB, then whole slots
        static constexpr size_t first[4] = {0, 128 << 10, 256 << 10, 512 << 10};
        return i < 4 ? first[i] : (size_t)(i - 3) * kSlot;
    }

    static HostStage* create() {
        HostStage* s = new HostStage();
        if (cudaHostAlloc((void**)&s->mem_, kSlot * kSlots, cudaHostAllocDefault) != cudaSuccess) { cudaGetLastError(); delete s; return nullptr; }
        for (int i = 0; i < kSlots; ++i)
            if (cudaEventCreateWithFlags(&s->ev_[i], cudaEventDisableTiming) != cudaSuccess) { cudaGetLastError(); delete s; return nullptr; }
        return s;
    }
    ~HostStage() {
        { std::lock_guard<std::mutex> l(mu_); quit_ = true; }
        cv_.notify_all();
        for (auto& t : threads_) t.join();
        for (int i = 0; i < kSlots; ++i) if (ev_[i]) cudaEventDestroy(ev_[i]);
        if (mem_) cudaFreeHost(mem_);
    }
    HostStage(const HostStage&) = delete;
    HostStage& operator=(const HostStage&) = delete;

    // dst (device) <- src (pageable host), ordered on the stream; src is free again when this returns.
    cudaError_t to_device(void* dst, const void* src, size_t bytes, cudaStream_t stream) {
        if (bytes <= kSlot / 4) {
            const Part one{src, bytes, 0};
            return to_device(dst, &one, 1, bytes, stream);
        }
        cudaError_t e = next_slot();                               // pieces own whole slots, from cur_ on
        if (e != cudaSuccess) return e;
        int pieces = bytes > kSlot ? (int)((bytes + kSlot - 1) / kSlot) + 3 : 1;
        while (piece_begin(pieces) < bytes) ++pieces;
        const int first = cur_;
        start_threads();
        // slot of piece i: first + i.  Slots whose last DMA is through may be filled; the threads stop at `limit_`.
        {
            std::lock_guard<std::mutex> l(mu_);
            src_ = (const char*)src; bytes_ = bytes; first_ = first; pieces_ = pieces;
            if ((size_t)pieces > done_cap_) { done_cap_ = (size_t)pieces; done_.reset(new std::atomic<uint8_t>[done_cap_]); }
            for (int i = 0; i < pieces; ++i) done_[i].store(0, std::memory_order_relaxed);
            next_.store(0); limit_.store(1);
            job_.fetch_add(1);
        }
        cv_.notify_all();
        int open = 1;                                              // pieces whose slot is free
        for (int i = 0; i < pieces && e == cudaSuccess; ++i) {
            while (open < pieces && open < i + kSlots) {
                const cudaError_t q = idle_ && open < kSlots ? cudaSuccess : cudaEventQuery(ev_[(first + open) % kSlots]);
                if (q == cudaErrorNotReady) {
                    if (open > i) break;                           // piece i is open: go on with it
                    continue;
                }
                if (q != cudaSuccess) { e = q; break; }
                limit_.store(++open, std::memory_order_release);
            }
            if (e != cudaSuccess) break;
            // help until piece i is filled
            while (!done(i)) { if (!copy_one()) pause(); }
            const size_t off = piece_begin(i), n = std::min(piece_begin(i + 1), bytes) - off;
            const int s = (first + i) % kSlots;
            e = cudaMemcpyAsync((char*)dst + off, slot(s), n, cudaMemcpyHostToDevice, stream);
            if (e == cudaSuccess) e = cudaEventRecord(ev_[s], stream);
        }
        // whatever was claimed is finished before src goes back to the caller, and nothing is claimed any more: a thread counts itself
        // busy before it looks at the limit, the limit falls before the count is read, and all four accesses are in one order
        limit_.store(0, std::memory_order_seq_cst);
        while (busy_.load(std::memory_order_seq_cst) != 0) pause();
        cur_ = (first + pieces) % kSlots;
        used_ = 0; dirty_ = false;
        const bool skip = idle_ && pieces < kSlots;
        idle_ = false;
        if (e == cudaSuccess && !skip) e = cudaEventSynchronize(ev_[cur_]);
        return e;
    }

    // Several small buffers whose places on the device lie within `span` bytes (at most a quarter of a slot): one copy, which also carries the gaps.
    struct Part { const void* src; size_t bytes, off; };
    cudaError_t to_device(void* dst, const Part* parts, size_t n, size_t span, cudaStream_t stream) {
        if (used_ + span > kSlot || (used_ > 0 && stream != stream_)) { cudaError_t e = next_slot(); if (e != cudaSuccess) return e; }
        char* p = slot(cur_) + used_;
        stream_ = stream;
        for (size_t i = 0; i < n; ++i) stream_copy(p + parts[i].off, (const char*)parts[i].src, parts[i].bytes);
        used_ += (span + 255) / 256 * 256;
        dirty_ = true; idle_ = false;
        return cudaMemcpyAsync(dst, p, span, cudaMemcpyHostToDevice, stream);
    }

    // The stream has been drained: every slot is free, and no stream is remembered.
    void drained() { idle_ = true; used_ = 0; dirty_ = false; stream_ = nullptr; }

    // Page-locked room for a result of at most a slot; valid until the next transfer of this context.
    void* result_slot(size_t bytes, cudaStream_t stream) {
        if (bytes > kSlot) return nullptr;
        if ((used_ + bytes > kSlot || (used_ > 0 && stream != stream_)) && next_slot() != cudaSuccess) { cudaGetLastError(); return nullptr; }
        return slot(cur_) + used_;
    }

  private:
    HostStage() = default;
    // The destination is read by the DMA engine only: streaming stores do not fetch its lines first and leave the caches alone.
#if defined(__x86_64__)
    __attribute__((target("avx2"))) static void copy_avx2(char* d, const char* s, size_t n) {
        size_t i = 0;
        for (; i + 128 <= n; i += 128) {
            const __m256i a = _mm256_loadu_si256((const __m256i*)(s + i)), b = _mm256_loadu_si256((const __m256i*)(s + i + 32));
            const __m256i c = _mm256_loadu_si256((const __m256i*)(s + i + 64)), e = _mm256_loadu_si256((const __m256i*)(s + i + 96));
            _mm256_stream_si256((__m256i*)(d + i), a); _mm256_stream_si256((__m256i*)(d + i + 32), b);
            _mm256_stream_si256((__m256i*)(d + i + 64), c); _mm256_stream_si256((__m256i*)(d + i + 96), e);
        }
        std::memcpy(d + i, s + i, n - i);
        _mm_sfence();
    }
#endif
    static void stream_copy(char* d, const char* s, size_t n) {      // d: 32-byte aligned
#if defined(__x86_64__)
        static const bool avx2 = __builtin_cpu_supports("avx2");
        if (avx2) { copy_avx2(d, s, n); return; }
#endif
        std::memcpy(d, s, n);
    }
    char* slot(int i) { return mem_ + (size_t)i * kSlot; }
    static void pause() {
#if defined(__x86_64__)
        _mm_pause();
#else
        std::this_thread::yield();
#endif
    }
    // closes the current slot (its event marks its last DMA, on the stream that its small copies share) and waits until the next one is free
    cudaError_t next_slot() {
        if (!dirty_ && used_ == 0) return cudaSuccess;
        cudaError_t e = cudaEventRecord(ev_[cur_], stream_);
        if (e != cudaSuccess) return e;
        cur_ = (cur_ + 1) % kSlots;
        used_ = 0; dirty_ = false;
        return cudaEventSynchronize(ev_[cur_]);
    }
    bool done(int i) { return done_[i].load(std::memory_order_acquire) != 0; }
    // claims and fills one open piece; false when there is none
    bool copy_one() {
        busy_.fetch_add(1, std::memory_order_seq_cst);
        int i = next_.load(std::memory_order_acquire);
        bool got = false;
        while (i < limit_.load(std::memory_order_seq_cst)) {
            if (next_.compare_exchange_weak(i, i + 1)) { got = true; break; }
        }
        if (got) {
            const size_t off = piece_begin(i), n = std::min(piece_begin(i + 1), bytes_) - off;
            stream_copy(slot((first_ + i) % kSlots), src_ + off, n);
            done_[i].store(1, std::memory_order_release);
        }
        busy_.fetch_sub(1, std::memory_order_acq_rel);
        return got;
    }
    void start_threads() {
        if (started_) return;
        started_ = true;
        const int n = std::min<int>(kThreads, (int)std::thread::hardware_concurrency() - 1);
        try {
            for (int i = 0; i < n; ++i) threads_.emplace_back([this] { work(); });
        } catch (const std::system_error&) {}                       // the caller copies alone
    }
    void work() {
        unsigned seen = 0;
        while (true) {
            {
                std::unique_lock<std::mutex> l(mu_);
                cv_.wait(l, [&] { return quit_ || job_.load() != seen; });
                if (quit_) return;
                seen = job_.load();
            }
            // until the job's last piece is claimed or the caller has closed it
            while (job_.load(std::memory_order_acquire) == seen) {
                if (copy_one()) continue;
                const int lim = limit_.load(std::memory_order_acquire);
                if (lim == 0 || next_.load(std::memory_order_acquire) >= pieces_.load(std::memory_order_acquire)) break;
                pause();
            }
        }
    }

    char* mem_ = nullptr;
    cudaEvent_t ev_[kSlots] = {};
    int cur_ = 0;
    size_t used_ = 0;
    cudaStream_t stream_ = nullptr;     // of the current slot's small copies
    bool dirty_ = false;
    bool idle_ = true;         // no DMA of this ring is in flight
    bool started_ = false;
    std::vector<std::thread> threads_;
    std::mutex mu_;
    std::condition_variable cv_;
    bool quit_ = false;
    // the current transfer
    std::atomic<unsigned> job_{0};
    std::atomic<int> next_{0}, limit_{0}, busy_{0}, pieces_{0};
    const char* src_ = nullptr;
    size_t bytes_ = 0;
    int first_ = 0;
    std::unique_ptr<std::atomic<uint8_t>[]> done_;
    size_t done_cap_ = 0;
};

// A context leaves its stream, which goes away with `destroy` or with whoever owns it: nothing of the ring may refer to it any more.
inline cudaError_t leave_stream(HostStage* stage, cudaStream_t stream, bool destroy) {
    const cudaError_t e = cudaStreamSynchronize(stream);
    if (e != cudaSuccess) return e;
    if (stage) stage->drained();
    return destroy ? cudaStreamDestroy(stream) : cudaSuccess;
}

}  // namespace zb
