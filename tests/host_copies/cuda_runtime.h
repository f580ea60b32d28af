// A stand-in for the CUDA runtime calls that psb_host.cuh makes, for the CPU:
// two devices, streams that run nothing until somebody waits for them, and
// page-locked memory, whose copies are therefore only queued when the call
// returns (a pageable copy has run by then).  It counts the event calls made
// by a thread whose current device is not the event's.
#pragma once
#include <algorithm>
#include <atomic>
#include <chrono>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <map>
#include <mutex>
#include <thread>
#include <vector>

enum cudaError_t { cudaSuccess = 0, cudaErrorInvalidValue = 1, cudaErrorNotReady = 600 };
enum cudaMemcpyKind { cudaMemcpyHostToDevice = 1, cudaMemcpyDeviceToHost = 2 };
enum cudaMemoryType { cudaMemoryTypeUnregistered = 0, cudaMemoryTypeHost = 1 };
constexpr unsigned cudaHostAllocPortable = 1, cudaEventDisableTiming = 2;
struct cudaPointerAttributes { cudaMemoryType type; };

struct FakeStream {
    std::vector<std::function<void()>> todo;
    size_t ran = 0;
};
using cudaStream_t = FakeStream*;
struct FakeEvent {
    int dev = 0;
    cudaStream_t st = nullptr;
    size_t at = 0;
};
using cudaEvent_t = FakeEvent*;

namespace fake {
inline std::recursive_mutex mu;
inline std::map<const char*, size_t> pinned;
inline std::atomic<int> wrong_device{0};
inline int& device() {
    thread_local int d = 0;
    return d;
}
inline bool is_pinned(const void* p) {
    std::lock_guard<std::recursive_mutex> lk(mu);
    for (auto& r : pinned)
        if ((const char*)p >= r.first && (const char*)p < r.first + r.second) return true;
    return false;
}
inline void run(cudaStream_t st, size_t to) {
    std::lock_guard<std::recursive_mutex> lk(mu);
    for (; st->ran < to; ++st->ran) st->todo[st->ran]();
}
}  // namespace fake

inline cudaError_t cudaGetDevice(int* d) { *d = fake::device(); return cudaSuccess; }
inline cudaError_t cudaSetDevice(int d) { fake::device() = d; return cudaSuccess; }
inline cudaError_t cudaGetLastError() { return cudaSuccess; }
inline cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) {
    std::lock_guard<std::recursive_mutex> lk(fake::mu);
    *p = aligned_alloc(4096, (n + 4095) / 4096 * 4096);
    fake::pinned[(const char*)*p] = n;
    return cudaSuccess;
}
inline cudaError_t cudaMallocHost(void** p, size_t n) { return cudaHostAlloc(p, n, 0); }
inline cudaError_t cudaFreeHost(void* p) {
    std::lock_guard<std::recursive_mutex> lk(fake::mu);
    fake::pinned.erase((const char*)p);
    free(p);
    return cudaSuccess;
}
inline cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p) {
    a->type = fake::is_pinned(p) ? cudaMemoryTypeHost : cudaMemoryTypeUnregistered;
    return cudaSuccess;
}
inline cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind k, cudaStream_t st) {
    std::lock_guard<std::recursive_mutex> lk(fake::mu);
    st->todo.push_back([=] { memcpy(d, s, n); });
    if (!fake::is_pinned(k == cudaMemcpyHostToDevice ? s : d)) fake::run(st, st->todo.size());
    return cudaSuccess;
}
inline cudaError_t cudaStreamSynchronize(cudaStream_t st) {
    fake::run(st, st->todo.size());
    return cudaSuccess;
}
inline cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) {
    *e = new FakeEvent;
    (*e)->dev = fake::device();
    return cudaSuccess;
}
inline cudaError_t cudaEventDestroy(cudaEvent_t e) { delete e; return cudaSuccess; }
inline cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t st) {
    std::lock_guard<std::recursive_mutex> lk(fake::mu);
    if (e->dev != fake::device()) return cudaErrorInvalidValue;   // as the runtime's: the stream's device has to match
    e->st = st;
    e->at = st->todo.size();
    return cudaSuccess;
}
inline cudaError_t cudaEventQuery(cudaEvent_t e) {
    std::lock_guard<std::recursive_mutex> lk(fake::mu);
    return !e->st || e->st->ran >= e->at ? cudaSuccess : cudaErrorNotReady;
}
inline cudaError_t cudaEventSynchronize(cudaEvent_t e) {
    if (e->dev != fake::device()) ++fake::wrong_device;
    std::this_thread::sleep_for(std::chrono::milliseconds(2));   // so that the other threads take a share
    if (e->st) fake::run(e->st, e->at);
    return cudaSuccess;
}
