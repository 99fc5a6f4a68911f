// sp_stage.cu -- large copies of pageable host memory through pinned buffers.
//
// The driver moves pageable memory with one thread (11 GB/s in, 17 out, measured
// at 288 MB), a fifth of the link. Here up to eight threads copy pieces between the
// caller's memory and 16 MB of pinned buffers while the pieces before are on the
// link: 51 GB/s with four of 4 MB, 49 with eight of 2 MB, 32 with half as many of
// either; 55 for memory that is pinned already. Copies below 32 MB take the smaller
// pieces: their first and last are not overlapped.
//
// The buffers are made by the first copy that is large enough and
// given back when the library is unloaded. One copy uses them at a time; one that
// finds them taken, a small one, and one whose memory the driver knows (pinned,
// managed or device memory) goes to cudaMemcpyAsync as it is.
#include <omp.h>
#include <algorithm>
#include <cstdint>
#include <cstring>
#include <mutex>
#include "sp_stage.h"

namespace {

constexpr size_t kPool = 16u << 20;
constexpr int kMaxSlots = 8;
constexpr int kThreads = 8;
// below, the threads' start costs what they save (4 MB in: 0.36 ms as it is)
constexpr size_t kLeast = 4u << 20;

size_t piece_of(size_t bytes) { return bytes < (32u << 20) ? 2u << 20 : 4u << 20; }

struct Buffers {
    std::mutex m;
    char *p = nullptr;
    bool refused = false;
    ~Buffers()
    {
        if (p)
            cudaFreeHost(p);  // fails harmlessly when the context is gone
    }
};
Buffers g_buf;

void copy_threads(char *dst, const char *src, size_t n, int threads)
{
#pragma omp parallel for num_threads(threads) schedule(static)
    for (int t = 0; t < threads; ++t) {
        const size_t a = n * t / threads / 64 * 64;
        const size_t b = t + 1 < threads ? n * (t + 1) / threads / 64 * 64 : n;
        memcpy(dst + a, src + a, b - a);
    }
}

// Threads for a copy that takes the staged way, 0 for one that does not; the
// buffers are then held by `lock`.
int take(const void *host, size_t bytes, std::unique_lock<std::mutex> &lock)
{
    if (bytes < kLeast || omp_in_parallel())
        return 0;
    const int threads = std::min(kThreads, omp_get_max_threads());
    if (threads < 2)
        return 0;
    cudaPointerAttributes at;
    if (cudaPointerGetAttributes(&at, host) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    if (at.type != cudaMemoryTypeUnregistered || !lock.try_lock() || g_buf.refused)
        return 0;
    if (!g_buf.p &&
        cudaHostAlloc((void **)&g_buf.p, kPool, cudaHostAllocPortable) != cudaSuccess) {
        cudaGetLastError();
        g_buf.p = nullptr;
        g_buf.refused = true;
        return 0;
    }
    return threads;
}

struct Events {
    cudaEvent_t e[kMaxSlots] = {};
    bool make()
    {
        for (auto &x : e)
            if (cudaEventCreateWithFlags(&x, cudaEventDisableTiming) != cudaSuccess)
                return false;
        return true;
    }
    ~Events()
    {
        for (auto x : e)
            if (x)
                cudaEventDestroy(x);
    }
};

}  // namespace

cudaError_t sp_copy_in(void *dev, const void *host, size_t bytes, cudaStream_t s,
                       const std::function<cudaError_t(size_t)> &enqueued)
{
    std::unique_lock<std::mutex> lock(g_buf.m, std::defer_lock);
    const int threads = take(host, bytes, lock);
    Events ev;
    if (threads == 0 || !ev.make()) {
        const cudaError_t r = cudaMemcpyAsync(dev, host, bytes, cudaMemcpyHostToDevice, s);
        return r == cudaSuccess && enqueued ? enqueued(bytes) : r;
    }
    cudaError_t e = cudaSuccess;
    const size_t piece = piece_of(bytes), slots = kPool / piece;
    const size_t pieces = (bytes + piece - 1) / piece;
    for (size_t k = 0; k < pieces && e == cudaSuccess; ++k) {
        const size_t at = k * piece, n = std::min(piece, bytes - at);
        char *slot = g_buf.p + k % slots * piece;
        if (k >= slots)
            e = cudaEventSynchronize(ev.e[k % slots]);
        if (e != cudaSuccess)
            break;
        copy_threads(slot, (const char *)host + at, n, threads);
        e = cudaMemcpyAsync((char *)dev + at, slot, n, cudaMemcpyHostToDevice, s);
        if (e == cudaSuccess)
            e = cudaEventRecord(ev.e[k % slots], s);
        if (e == cudaSuccess && enqueued)
            e = enqueued(at + n);
    }
    // the buffers go to the next copy: nothing may still read them
    const cudaError_t done = cudaStreamSynchronize(s);
    return e != cudaSuccess ? e : done;
}

cudaError_t sp_copy_out(void *host, const void *dev, size_t bytes, cudaStream_t s)
{
    std::unique_lock<std::mutex> lock(g_buf.m, std::defer_lock);
    const int threads = take(host, bytes, lock);
    Events ev;
    if (threads == 0 || !ev.make())
        return cudaMemcpyAsync(host, dev, bytes, cudaMemcpyDeviceToHost, s);
    cudaError_t e = cudaSuccess;
    const size_t piece = piece_of(bytes), slots = kPool / piece;
    const size_t pieces = (bytes + piece - 1) / piece;
    auto start = [&](size_t k) {
        const size_t at = k * piece, n = std::min(piece, bytes - at);
        cudaError_t r = cudaMemcpyAsync(g_buf.p + k % slots * piece, (const char *)dev + at, n,
                                        cudaMemcpyDeviceToHost, s);
        return r == cudaSuccess ? cudaEventRecord(ev.e[k % slots], s) : r;
    };
    for (size_t k = 0; k < pieces && k < slots && e == cudaSuccess; ++k)
        e = start(k);
    for (size_t k = 0; k < pieces && e == cudaSuccess; ++k) {
        const size_t at = k * piece, n = std::min(piece, bytes - at);
        e = cudaEventSynchronize(ev.e[k % slots]);
        if (e != cudaSuccess)
            break;
        copy_threads((char *)host + at, g_buf.p + k % slots * piece, n, threads);
        if (k + slots < pieces)
            e = start(k + slots);
    }
    if (e != cudaSuccess)
        cudaStreamSynchronize(s);
    return e;
}

// 256 slots of 256 bytes, made by the first that is taken (a cudaHostAlloc of its
// own per reservoir would cost each one 2.5 ms) and given back when the library is
// unloaded.
namespace {

constexpr int kMailSlots = 256;
constexpr size_t kMailBytes = 256;

struct Mail {
    std::mutex m;
    char *p = nullptr;
    bool refused = false;
    bool used[kMailSlots] = {};
    ~Mail()
    {
        if (p)
            cudaFreeHost(p);
    }
};
Mail g_mail;

}  // namespace

void *sp_mail_take(size_t bytes)
{
    if (bytes > kMailBytes)
        return nullptr;
    std::lock_guard<std::mutex> lock(g_mail.m);
    if (!g_mail.p && !g_mail.refused &&
        cudaHostAlloc((void **)&g_mail.p, kMailSlots * kMailBytes,
                      cudaHostAllocPortable | cudaHostAllocMapped) != cudaSuccess) {
        cudaGetLastError();
        g_mail.p = nullptr;
        g_mail.refused = true;
    }
    for (int k = 0; g_mail.p && k < kMailSlots; ++k)
        if (!g_mail.used[k]) {
            g_mail.used[k] = true;
            return g_mail.p + k * kMailBytes;
        }
    return nullptr;
}

void sp_mail_give(void *slot)
{
    if (!slot)
        return;
    std::lock_guard<std::mutex> lock(g_mail.m);
    g_mail.used[((char *)slot - g_mail.p) / kMailBytes] = false;
}
