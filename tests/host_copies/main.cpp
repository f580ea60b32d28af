// Runs one case of tests/test_host_copies.py against the stand-in runtime;
// prints "ok" or what went wrong.
#include "psb_host.cuh"

#include <cstdio>
#include <string>

#ifdef THREADS
// a process that may have no more than THREADS threads of its own
#include <cerrno>
#include <dlfcn.h>
#include <pthread.h>
extern "C" int pthread_create(pthread_t* t, const pthread_attr_t* a, void* (*f)(void*), void* x) noexcept {
    static int made = 0;
    if (made++ >= THREADS) return EAGAIN;
    return ((decltype(&pthread_create))dlsym(RTLD_NEXT, "pthread_create"))(t, a, f, x);
}
#endif

static FakeStream g_stream[2];

// upload_async, the source overwritten as soon as the call has returned
static bool upload(size_t bytes, bool pinned) {
    std::vector<char> pageable(pinned ? 0 : bytes), dev(bytes, 0);
    char* src = pageable.data();
    if (pinned && cudaHostAlloc((void**)&src, bytes, 0) != cudaSuccess) return false;
    for (size_t i = 0; i < bytes; ++i) src[i] = (char)(i * 7 + 1);
    if (upload_async(dev.data(), src, bytes, &g_stream[0]) != cudaSuccess) return false;
    memset(src, 0x55, bytes);
    cudaStreamSynchronize(&g_stream[0]);
    bool same = true;
    for (size_t i = 0; i < bytes; ++i) same = same && dev[i] == (char)(i * 7 + 1);
    if (pinned) cudaFreeHost(src);
    return same;
}

int main(int argc, char** argv) {
    const std::string what = argc > 1 ? argv[1] : "";
    bool ok = false;
    if (what == "upload") {
        ok = upload((size_t)atoll(argv[2]), argv[3][0] == 'p');
    } else if (what == "upload_no_block") {
        // every staging block in use elsewhere
        for (int i = 0; i < PinBlocks::kBlocks; ++i)
            if (!PinBlocks::get().take((size_t)2 << 20)) return 1;
        ok = upload((size_t)2 << 20, argv[2][0] == 'p');
    } else if (what == "download") {
        // every byte there on return, no event waited for from another device
        const size_t bytes = (size_t)atoll(argv[2]);
        cudaSetDevice(atoi(argv[3]));
        std::vector<char> dev(bytes), out(bytes, 0);
        for (size_t i = 0; i < bytes; ++i) dev[i] = (char)(i * 5 + 2);
        ok = download(out.data(), dev.data(), bytes, &g_stream[0]) == cudaSuccess && out == dev && !fake::wrong_device;
    } else if (what == "two_devices") {
        // the first device's idle blocks give way to the second's, and back
        ok = true;
        for (int dev : {0, 1, 0}) {
            cudaSetDevice(dev);
            PinBlock* b[PinBlocks::kBlocks];
            for (PinBlock*& x : b) ok = (x = PinBlocks::get().take((size_t)2 << 20)) != nullptr && x->dev == dev && ok;
            ok = PinBlocks::get().take((size_t)2 << 20) == nullptr && ok;   // none is left while they are held
            for (PinBlock* x : b) if (x) PinBlocks::get().give(x, &g_stream[dev]);
        }
    } else if (what == "chunks") {
        const size_t n = (size_t)atoll(argv[2]);
        std::vector<std::atomic<int>> seen(n);
        parallel_chunks(n, 10, [&](size_t b, size_t e) {
            for (size_t i = b; i < e; ++i) ++seen[i];
        });
        ok = true;
        for (auto& c : seen) ok = ok && c == 1;
    }
    puts(ok ? "ok" : "wrong");
    fflush(stdout);
    _Exit(0);   // the host threads wait for ever
}
