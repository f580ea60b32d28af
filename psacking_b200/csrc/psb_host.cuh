// psb_host.cuh — host threads and large host-device copies.
//
// The public calls take and return host arrays of the tray's size (4-12 MB).
// A pageable cudaMemcpy moves those through the driver's staging buffer with
// one thread, and a fresh result array takes its page faults there as well:
// 0.4-0.6 ms per copy at 240x123x100, several copies per call.  Here they go
// through pinned blocks in chunks, the host cores copying one chunk while the
// next is on the bus.  The threads that do so are made once per process (one
// std::thread per core and call cost 0.2-0.4 ms per use).
#pragma once
#include <cuda_runtime.h>
#include <unistd.h>
#if defined(__SSE2__)
#include <emmintrin.h>
#endif

#include <algorithm>
#include <atomic>
#include <condition_variable>
#include <cstring>
#include <deque>
#include <functional>
#include <map>
#include <memory>
#include <mutex>
#include <system_error>
#include <thread>
#include <vector>

// Runs the chunks of one or several callers' jobs on all host cores.  Any
// thread may call run(); it takes part in its own job.  Never destroyed: its
// threads wait in the kernel until the process ends.  A forked child has no
// threads of it and runs its jobs alone.
class HostPool {
  public:
    static HostPool& get() {
        static HostPool* p = new HostPool();
        return *p;
    }

    struct Job {
        std::function<void(size_t)> fn;
        size_t n;
        std::atomic<size_t> next{0}, done{0};
        bool one() {
            const size_t i = next.fetch_add(1);
            if (i >= n) return false;
            fn(i);
            done.fetch_add(1, std::memory_order_release);
            return true;
        }
    };

    // queue fn(0) .. fn(n - 1); finish() waits for them
    std::shared_ptr<Job> start(size_t n, std::function<void(size_t)> fn) {
        auto j = std::make_shared<Job>();
        j->fn = std::move(fn);
        j->n = n;
        if (n > 1 && workers_ > 0 && getpid() == pid_) {
            {
                std::lock_guard<std::mutex> lk(mu_);
                jobs_.push_back(j);
            }
            if (n - 1 >= (size_t)workers_) cv_.notify_all();
            else for (size_t i = 1; i < n; ++i) cv_.notify_one();
        }
        return j;
    }
    void finish(const std::shared_ptr<Job>& j) {
        while (j->one()) {}
        while (j->done.load(std::memory_order_acquire) < j->n) std::this_thread::yield();
    }
    void run(size_t n, std::function<void(size_t)> fn) {
        if (n == 1) fn(0);
        else if (n > 1) finish(start(n, std::move(fn)));
    }

  private:
    HostPool() : pid_(getpid()) {
        const int want = (int)std::min(11u, std::max(1u, std::thread::hardware_concurrency()) - 1u);
        try {
            for (; workers_ < want; ++workers_) std::thread([this] { loop(); }).detach();
        } catch (const std::system_error&) {
            // no more threads to be had: the callers do the rest themselves
        }
    }
    void loop() {
        std::unique_lock<std::mutex> lk(mu_);
        for (;;) {
            cv_.wait(lk, [this] { return !jobs_.empty(); });
            std::shared_ptr<Job> j = jobs_.front();
            if (j->next.load() >= j->n) {   // every chunk is taken
                jobs_.pop_front();
                continue;
            }
            lk.unlock();
            while (j->one()) {}
            lk.lock();
        }
    }
    std::mutex mu_;
    std::condition_variable cv_;
    std::deque<std::shared_ptr<Job>> jobs_;
    int workers_ = 0;
    pid_t pid_;
};

// fn(begin, end) over [0, n) in chunks on the host cores
template <typename F>
void parallel_chunks(size_t n, size_t chunk, F fn) {
    const size_t nchunks = (n + chunk - 1) / chunk;
    HostPool::get().run(nchunks, [&](size_t c) { fn(c * chunk, std::min(n, (c + 1) * chunk)); });
}

// memcpy into pinned memory past the cache: lines left dirty in several
// cores' caches make the bus read them back one snoop at a time (11.8 MB
// written by 12 cores with plain stores took 1.3-1.9 ms on the bus, 0.23 ms
// once it lies in memory).  dst 16-byte aligned.
inline void stream_copy(void* dst, const void* src, size_t bytes) {
#if defined(__SSE2__)
    size_t i = 0;
    for (; i + 64 <= bytes; i += 64) {
        const __m128i* s = (const __m128i*)((const char*)src + i);
        __m128i* d = (__m128i*)((char*)dst + i);
        const __m128i a = _mm_loadu_si128(s), b = _mm_loadu_si128(s + 1), c = _mm_loadu_si128(s + 2),
                      e = _mm_loadu_si128(s + 3);
        _mm_stream_si128(d, a);
        _mm_stream_si128(d + 1, b);
        _mm_stream_si128(d + 2, c);
        _mm_stream_si128(d + 3, e);
    }
    if (i < bytes) memcpy((char*)dst + i, (const char*)src + i, bytes - i);
    _mm_sfence();
#else
    memcpy(dst, src, bytes);
#endif
}

inline void parallel_copy(void* dst, const void* src, size_t bytes) {
    if (bytes < ((size_t)2 << 20)) {
        memcpy(dst, src, bytes);
        return;
    }
    parallel_chunks(bytes, (size_t)1 << 19, [&](size_t b, size_t e) {
        memcpy((char*)dst + b, (const char*)src + b, e - b);
    });
}

// Pinned memory of the trays (staging, descriptors), kept when a tray is
// destroyed and handed to the next one: cudaMallocHost and cudaFreeHost take
// 0.5-5 ms each and stop the whole device, and a many-tray run makes a tray's
// worth of them per tray.  At most kKeep bytes are kept.
class PinCache {
  public:
    static constexpr size_t kKeep = (size_t)256 << 20;
    static PinCache& get() {
        static PinCache* p = new PinCache();
        return *p;
    }
    // *got: the bytes it really has
    cudaError_t take(void** out, size_t bytes, size_t* got) {
        bytes = std::max(bytes, (size_t)4096);
        {
            std::lock_guard<std::mutex> lk(mu_);
            auto it = free_.lower_bound(bytes);
            if (it != free_.end() && it->first <= std::max(4 * bytes, (size_t)1 << 20)) {
                *out = it->second;
                *got = it->first;
                kept_ -= it->first;
                free_.erase(it);
                return cudaSuccess;
            }
        }
        // room to grow: the next user may need a little more
        *got = (bytes + bytes / 4 + 4095) / 4096 * 4096;
        return cudaHostAlloc(out, *got, cudaHostAllocPortable);
    }
    // nothing queued may use it any more
    void give(void* p, size_t n) {
        if (!p) return;
        {
            std::lock_guard<std::mutex> lk(mu_);
            if (kept_ + n <= kKeep) {
                free_.emplace(n, p);
                kept_ += n;
                return;
            }
        }
        cudaFreeHost(p);
    }

  private:
    std::mutex mu_;
    std::multimap<size_t, void*> free_;
    size_t kept_ = 0;
};

// Pinned blocks, shared by all threads: at most kBlocks per process of at most
// kBlockMax bytes; a block is free again once the copies queued from it have
// run.  Larger copies, and copies while no block is free, are pageable.
struct PinBlock {
    char* p = nullptr;
    size_t n = 0;
    int dev = -1;
    bool held = false;
    static constexpr int kEvents = 5;
    cudaEvent_t ev[kEvents] = {};   // the last one marks the block's last use
};

class PinBlocks {
  public:
    static constexpr size_t kBlockMax = (size_t)64 << 20;
    static constexpr int kBlocks = 6;
    static PinBlocks& get() {
        static PinBlocks* p = new PinBlocks();
        return *p;
    }
    PinBlock* take(size_t bytes) {
        int dev = 0;
        if (bytes > kBlockMax || cudaGetDevice(&dev) != cudaSuccess) return nullptr;
        std::lock_guard<std::mutex> lk(mu_);
        PinBlock* best = nullptr;
        for (PinBlock& b : blocks_)
            if (b.p && !b.held && b.dev == dev && b.n >= bytes && (!best || b.n < best->n) &&
                cudaEventQuery(b.ev[PinBlock::kEvents - 1]) == cudaSuccess)
                best = &b;
        if (!best) {
            for (PinBlock& b : blocks_)
                if (!b.p && !b.held) { best = &b; break; }
            if (!best)   // every place is in use: replace an idle one that is too small or another device's
                for (PinBlock& b : blocks_)
                    if (!b.held && (b.dev != dev || b.n < bytes) &&
                        cudaEventQuery(b.ev[PinBlock::kEvents - 1]) == cudaSuccess) { best = &b; break; }
            if (!best || !make(best, bytes, dev)) return nullptr;
        }
        best->held = true;
        return best;
    }
    // the copies queued on st so far are the block's last use
    void give(PinBlock* b, cudaStream_t st) {
        const bool ok = cudaEventRecord(b->ev[PinBlock::kEvents - 1], st) == cudaSuccess;
        if (!ok) cudaStreamSynchronize(st);
        std::lock_guard<std::mutex> lk(mu_);
        b->held = false;
    }

  private:
    bool make(PinBlock* b, size_t bytes, int dev) {
        if (b->p) {
            cudaFreeHost(b->p);
            for (cudaEvent_t& e : b->ev) { cudaEventDestroy(e); e = nullptr; }
            b->p = nullptr;
            b->n = 0;
        }
        const size_t n = (bytes + ((size_t)2 << 20) - 1) >> 21 << 21;
        if (cudaMallocHost((void**)&b->p, n) != cudaSuccess) {
            cudaGetLastError();
            b->p = nullptr;
            return false;
        }
        for (cudaEvent_t& e : b->ev)
            if (cudaEventCreateWithFlags(&e, cudaEventDisableTiming) != cudaSuccess) {
                cudaGetLastError();
                for (cudaEvent_t& f : b->ev) { if (f) cudaEventDestroy(f); f = nullptr; }
                cudaFreeHost(b->p);
                b->p = nullptr;
                return false;
            }
        b->n = n;
        b->dev = dev;
        return true;
    }
    std::mutex mu_;
    PinBlock blocks_[kBlocks];
};

// Copies below this stay with the driver (one call, no thread woken): waking
// the cores costs about 0.05 ms, a pageable megabyte about 0.06 ms.  On the
// way back they also wait for the bus: 2 MB took 0.3 ms longer staged, 8 MB
// 0.2 ms shorter.
constexpr size_t kUploadMin = (size_t)3 << 19, kDownloadMin = (size_t)4 << 20;

// Whether the driver takes a copy's bytes before the call returns: of pageable
// memory only.  Page-locked memory (a pinned tensor's) is read when the copy
// runs, and memory that CUDA manages may be.
inline bool host_pageable(const void* p) {
    cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return a.type == cudaMemoryTypeUnregistered;
}

// Host array -> device on st.  The source may be reused on return; the copy
// itself is queued (waited for where it would still be reading the source).
inline cudaError_t upload_async(void* dst, const void* src, size_t bytes, cudaStream_t st) {
    PinBlock* b = bytes >= kUploadMin ? PinBlocks::get().take(bytes) : nullptr;
    if (!b) {
        const cudaError_t e = cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, st);
        return e != cudaSuccess || host_pageable(src) ? e : cudaStreamSynchronize(st);
    }
    // the cores copy 512 KiB at a time, the bus takes quarters: every bus copy
    // costs some 20 us besides its bytes
    const size_t chunk = (size_t)512 << 10, n = (bytes + chunk - 1) / chunk, group = (n + 3) / 4;
    std::unique_ptr<std::atomic<char>[]> ready(new std::atomic<char>[n]);
    for (size_t i = 0; i < n; ++i) ready[i] = 0;
    auto job = HostPool::get().start(n, [&](size_t i) {
        const size_t o = i * chunk, m = std::min(chunk, bytes - o);
        stream_copy(b->p + o, (const char*)src + o, m);
        ready[i].store(1, std::memory_order_release);
    });
    cudaError_t e = cudaSuccess;
    for (size_t i = 0; i < n; ++i) {
        while (!ready[i].load(std::memory_order_acquire))
            if (!job->one()) std::this_thread::yield();
        if ((i + 1) % group != 0 && i + 1 != n) continue;
        const size_t o = i / group * group * chunk, m = std::min(bytes, (i + 1) * chunk) - o;
        if (e == cudaSuccess) e = cudaMemcpyAsync((char*)dst + o, b->p + o, m, cudaMemcpyHostToDevice, st);
    }
    HostPool::get().finish(job);
    PinBlocks::get().give(b, st);
    return e;
}

// Device -> host array; the data is there on return, and st is synchronised.
inline cudaError_t download(void* dst, const void* src, size_t bytes, cudaStream_t st) {
    PinBlock* b = bytes >= kDownloadMin ? PinBlocks::get().take(bytes) : nullptr;
    if (!b) {
        cudaError_t e = cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, st);
        return e == cudaSuccess ? cudaStreamSynchronize(st) : e;
    }
    const size_t chunk = (size_t)512 << 10, n = (bytes + chunk - 1) / chunk, group = (n + 3) / 4;
    cudaError_t e = cudaSuccess;
    for (size_t i = 0; i < n && e == cudaSuccess; i += group) {
        const size_t o = i * chunk, m = std::min(bytes, (i + group) * chunk) - o;
        e = cudaMemcpyAsync(b->p + o, (const char*)src + o, m, cudaMemcpyDeviceToHost, st);
        if (e == cudaSuccess) e = cudaEventRecord(b->ev[i / group], st);
    }
    if (e == cudaSuccess) {
        std::atomic<int> bad{0};
        HostPool::get().run(n, [&](size_t i) {
            // the cores' threads start out on device 0, where a call for
            // another device's event would make a context
            cudaError_t w = cudaSetDevice(b->dev);
            if (w == cudaSuccess) w = cudaEventSynchronize(b->ev[i / group]);
            if (w != cudaSuccess) { bad = (int)w; return; }
            const size_t o = i * chunk, m = std::min(chunk, bytes - o);
            memcpy((char*)dst + o, b->p + o, m);
        });
        if (bad) e = (cudaError_t)bad.load();
    }
    const cudaError_t s = cudaStreamSynchronize(st);
    PinBlocks::get().give(b, st);
    return e != cudaSuccess ? e : s;
}
