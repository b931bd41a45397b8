// Large copies between pageable host memory and a device state.
//
// cudaMemcpy from pageable memory stages through one driver buffer on one
// thread: 11 GB/s host->device and 21 GB/s device->host for a 16 GiB state
// on the B200 systems this engine targets.  Here a few host threads each
// own two page-locked chunks and a stream; a thread copies its share of the
// buffer chunk by chunk between host memory and a chunk (memcpy) and between
// the chunk and the device (cudaMemcpyAsync), with the two chunks taking
// turns, so the host copies, the page faults of first-touch host memory and
// the DMA all run in parallel (27-45 GB/s host->device and 42 GB/s
// device->host with four threads, the fastest count measured; more threads
// contend).  Registering the caller's
// buffer instead (cudaHostRegister) copies at 55 GB/s but registering and
// unregistering 16 GiB takes 2.8 s, more than the copy itself.
//
// Copies of kSmallMin to kLargeMin go the same way through a small set of
// chunks (8 MiB of page-locked memory), the calling thread taking a share
// itself.  In us, up / down, plain and staged: 0.5 MiB 70 / 74 and 69 / 58 (188
// once), 1 MiB 128 / 102 and 90 / 77, 16 MiB 1550 / 920 and 700 / 695, 128 MiB
// 12100 / 7350 and 4200 / 4400.  The line lies at 1 MiB, where a call that copies
// up, runs and copies down gains (1 MiB 346 -> 262 us, 2 MiB 524 -> 365, 8 MiB 1490
// -> 830); of copies one after another in one direction those of 1 to 2 MiB lose
// (up 78 -> 98 us, 135 -> 158).
//
// Each set of chunks (the large one is 256 MiB) is allocated on its first copy
// and kept until exit; copies below kSmallMin use a plain cudaMemcpyAsync.
// One staged copy of a set runs at a time (take_chunks).
#include <cuda_runtime.h>

#include <atomic>
#include <cstring>
#include <exception>
#include <functional>
#include <mutex>
#include <thread>
#include <vector>

#include "hgm_internal.h"

namespace hgm {

namespace {

constexpr int kThreads = 4;
constexpr size_t kLargeChunk = size_t(32) << 20, kSmallChunk = size_t(1) << 20, kMinChunk = size_t(256) << 10;
constexpr size_t kLargeMin = size_t(256) << 20, kSmallMin = size_t(1) << 20;

struct Stager {
    size_t capacity;  // bytes of a chunk
    std::mutex mu;
    int device = -1;
    char *buf[kThreads][2] = {};
    cudaStream_t stream[kThreads] = {};
    cudaEvent_t done[kThreads][2] = {};
    bool ready = false, failed = false;
    explicit Stager(size_t c) : capacity(c) {}
};

Stager g_large(kLargeChunk), g_small(kSmallChunk);

Stager &chunks_for(size_t bytes) { return bytes < kLargeMin ? g_small : g_large; }

void stager_free(Stager &s) {
    for (int t = 0; t < kThreads; t++) {
        for (int k = 0; k < 2; k++) {
            if (s.buf[t][k]) cudaFreeHost(s.buf[t][k]);
            if (s.done[t][k]) cudaEventDestroy(s.done[t][k]);
            s.buf[t][k] = nullptr;
            s.done[t][k] = nullptr;
        }
        if (s.stream[t]) cudaStreamDestroy(s.stream[t]);
        s.stream[t] = nullptr;
    }
}

int stager_alloc(Stager &s) {
    for (int t = 0; t < kThreads; t++) {
        cudaError_t e;
        if ((e = cudaStreamCreateWithFlags(&s.stream[t], cudaStreamNonBlocking)) != cudaSuccess)
            return fail(HGM_ERR_CUDA, "staging stream: %s", cudaGetErrorString(e));
        for (int k = 0; k < 2; k++) {
            if ((e = cudaMallocHost(&s.buf[t][k], s.capacity)) != cudaSuccess)
                return fail(HGM_ERR_NOMEM, "staging chunk: %s", cudaGetErrorString(e));
            if ((e = cudaEventCreateWithFlags(&s.done[t][k], cudaEventDisableTiming)) != cudaSuccess)
                return fail(HGM_ERR_CUDA, "staging event: %s", cudaGetErrorString(e));
        }
    }
    return HGM_OK;
}

int stager_init(Stager &s, int device) {
    if (s.ready) return HGM_OK;
    if (s.failed) return HGM_ERR_NOMEM;  // tried once; copy directly from now on
    int rc = stager_alloc(s);
    if (rc == HGM_OK) {
        s.device = device;
        s.ready = true;
    } else {
        stager_free(s);
        cudaGetLastError();
        s.failed = true;
    }
    return rc;
}

// Thread t's share: chunks t, t + kThreads, t + 2 kThreads, ...
void stage_h2d(Stager &s, size_t chunk, int t, char *dev, const char *host, size_t bytes, std::atomic<int> *err) {
    cudaSetDevice(s.device);
    int k = 0;
    for (size_t off = (size_t)t * chunk; off < bytes; off += (size_t)kThreads * chunk, k ^= 1) {
        const size_t n = off + chunk <= bytes ? chunk : bytes - off;
        if (cudaEventSynchronize(s.done[t][k]) != cudaSuccess) err->store(1);  // chunk free again
        memcpy(s.buf[t][k], host + off, n);
        if (cudaMemcpyAsync(dev + off, s.buf[t][k], n, cudaMemcpyHostToDevice, s.stream[t]) != cudaSuccess ||
            cudaEventRecord(s.done[t][k], s.stream[t]) != cudaSuccess)
            err->store(1);
    }
    if (cudaStreamSynchronize(s.stream[t]) != cudaSuccess) err->store(1);
}

void stage_d2h(Stager &s, size_t chunk, int t, char *host, const char *dev, size_t bytes, std::atomic<int> *err) {
    cudaSetDevice(s.device);
    size_t pending_off = 0, pending_n = 0;
    int pending_k = -1, k = 0;
    for (size_t off = (size_t)t * chunk; off < bytes; off += (size_t)kThreads * chunk, k ^= 1) {
        const size_t n = off + chunk <= bytes ? chunk : bytes - off;
        if (cudaMemcpyAsync(s.buf[t][k], dev + off, n, cudaMemcpyDeviceToHost, s.stream[t]) != cudaSuccess ||
            cudaEventRecord(s.done[t][k], s.stream[t]) != cudaSuccess)
            err->store(1);
        if (pending_k >= 0) {  // the previous chunk lands while this one is in flight
            if (cudaEventSynchronize(s.done[t][pending_k]) != cudaSuccess) err->store(1);
            memcpy(host + pending_off, s.buf[t][pending_k], pending_n);
        }
        pending_off = off;
        pending_n = n;
        pending_k = k;
    }
    if (pending_k >= 0) {
        if (cudaEventSynchronize(s.done[t][pending_k]) != cudaSuccess) err->store(1);
        memcpy(host + pending_off, s.buf[t][pending_k], pending_n);
    }
}

}  // namespace

// share(0) .. share(n - 1), each on a thread of its own and the first on this
// one; where no thread can be started (std::system_error, which must not leave
// a C entry), this one takes that share too.
void run_shares(int n, const std::function<void(int)> &share) {
    std::vector<std::thread> th;
    int t = 1;
    try {
        th.reserve(n);
        for (; t < n; t++) th.emplace_back(share, t);
    } catch (const std::exception &) {
    }
    share(0);
    for (; t < n; t++) share(t);
    for (std::thread &x : th) x.join();
}

int plain_copy(void *dst, const void *src, size_t bytes, bool to_device, cudaStream_t st) {
    cudaError_t e = cudaMemcpyAsync(dst, src, bytes, to_device ? cudaMemcpyHostToDevice : cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    return e == cudaSuccess ? HGM_OK : fail(HGM_ERR_CUDA, "state copy: %s", cudaGetErrorString(e));
}

// Whether a host buffer is copied through the chunks: pageable memory from
// kSmallMin on.  Page-locked memory (hgm_pinned_alloc, a registered or managed
// buffer) is what the copy engine reads by itself at the bus's rate: 16 MiB
// 320 us, 64 MiB 1.2 ms, 256 MiB 4.7 ms either way, against 610 us, 2.1-2.6 and
// 7.9-9.4 ms through the chunks.  Both ends are looked at: a buffer registered in part goes
// through the chunks.
bool staged(const void *host, size_t bytes) {
    if (bytes < kSmallMin) return false;
    for (const char *p : {(const char *)host, (const char *)host + bytes - 1}) {
        cudaPointerAttributes a;
        if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
            cudaGetLastError();
            return true;
        }
        if (a.type == cudaMemoryTypeUnregistered) return true;
    }
    return false;
}

// The right to the chunks that a copy of `bytes` goes through.  A copy that
// finds the small set taken gets none and goes directly beside the other: two
// threads copying at once, us a round up / down, taking turns and this way:
// 1 MiB 212 / 230 and 122 / 135, 4 MiB 490 / 680 and 315 / 520, 16 MiB 1150 / 1740 and
// 1045 / 1590 (both directly: 102 / 205, 422 / 560, 1750 / 1800).  Copies through
// the large set take turns.
std::unique_lock<std::mutex> take_chunks(size_t bytes) {
    Stager &s = chunks_for(bytes);
    return &s == &g_large ? std::unique_lock<std::mutex>(s.mu) : std::unique_lock<std::mutex>(s.mu, std::try_to_lock);
}

int copy_state(void *dst, const void *src, size_t bytes, bool to_device, void *stream) {
    cudaStream_t st = (cudaStream_t)stream;
    if (!staged(to_device ? src : dst, bytes)) return plain_copy(dst, src, bytes, to_device, st);
    // earlier work on the state's stream must be done before the staging
    // streams read or overwrite the state
    cudaError_t e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return fail(HGM_ERR_CUDA, "state copy: %s", cudaGetErrorString(e));
    int device = 0;
    cudaGetDevice(&device);
    Stager &s = chunks_for(bytes);
    std::unique_lock<std::mutex> lk = take_chunks(bytes);
    if (!lk.owns_lock()) return plain_copy(dst, src, bytes, to_device, st);
    // the chunks belong to the first device that made such a copy; other
    // devices, and hosts where page-locked memory ran out, copy directly
    if (stager_init(s, device) != HGM_OK || s.device != device) {
        lk.unlock();
        return plain_copy(dst, src, bytes, to_device, st);
    }
    // at least two chunks a thread, so that its host copies and transfers overlap
    const size_t share = bytes / (2 * kThreads), chunk = share >= s.capacity ? s.capacity : share < kMinChunk ? kMinChunk : share;
    std::atomic<int> err{0};
    auto run = [&](int t) {
        if (to_device) stage_h2d(s, chunk, t, (char *)dst, (const char *)src, bytes, &err);
        else stage_d2h(s, chunk, t, (char *)dst, (const char *)src, bytes, &err);
    };
    run_shares(kThreads, run);
    return err.load() ? fail(HGM_ERR_CUDA, "staged state copy failed") : HGM_OK;
}

}  // namespace hgm
