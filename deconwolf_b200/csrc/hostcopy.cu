// hostcopy.cu -- copies between pageable host memory and the device.
//
// The driver stages a pageable copy through a buffer of its own with one
// thread, about 10 GB/s, and the caller waits for it.  Here a few threads
// stage chunks through page-locked buffers, each keeping two chunks in
// flight, so the copy runs at the link's rate; a result's pages are also
// touched (and zeroed by the kernel) by several threads while the device
// iterates.  1024 x 1024 x 60, SHB 10, from and to NumPy arrays: 75 -> 47 ms.
//
// The page-locked buffers (kBuffers x kChunk bytes) are made at the first
// large copy, serve one copy at a time for as long as its bytes move (a second
// caller meanwhile takes the driver's path rather than wait) and are given
// back by dwcu_release_cache.
// Page-locked, registered and managed memory, and copies below kMinBytes,
// take the driver's path, which is at its best there.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstdint>
#include <cstring>
#include <mutex>
#include <new>
#include <system_error>
#include <thread>
#include <vector>

#include "hostcopy.h"

namespace dwcu {
namespace {

constexpr size_t kChunk = (size_t) 2 << 20;
constexpr int kThreads = 8;
constexpr int kBuffers = 2 * kThreads;
constexpr size_t kMinBytes = (size_t) 4 << 20;

std::mutex g_ring_mu;  // held for the length of a staged copy
char *g_ring = nullptr;

// the ring's buffers, made on first use (g_ring_mu held); null: not to be had
char *ring_locked()
{
    if (!g_ring && cudaHostAlloc((void **) &g_ring, kChunk * kBuffers, cudaHostAllocPortable) != cudaSuccess) {
        cudaGetLastError();
        g_ring = nullptr;
    }
    return g_ring;
}

bool pageable(const void *p)
{
    cudaPointerAttributes a;
    const cudaError_t e = cudaPointerGetAttributes(&a, p);
    cudaGetLastError();
    return e == cudaSuccess && a.type == cudaMemoryTypeUnregistered;
}

int worker_count(size_t chunks)
{
    const unsigned hw = std::thread::hardware_concurrency();
    return (int) std::max<size_t>(1, std::min<size_t>({(size_t) kThreads, chunks, hw > 2 ? hw / 2 : 1}));
}

// work(t, nt) on nt threads, this one among them; threads that cannot be
// started leave their share to none: returns how many t < nt ran
template <class F>
int on_threads(int nt, F work)
{
    std::vector<std::thread> th;
    int started = 1;
    try {
        th.reserve((size_t) nt);
        for (int t = 1; t < nt; ++t) {
            th.emplace_back(work, t);
            ++started;
        }
    } catch (const std::system_error &) {
    } catch (const std::bad_alloc &) {
    }
    work(0);
    for (auto &t : th) t.join();
    return started;
}

// One thread's share of a staged copy: chunks taken from a common counter.
// to_device: memcpy into a buffer, then its copy; otherwise the copy, then
// the memcpy out while the next chunk's copy runs.
cudaError_t stage(bool to_device, char *ring, int t, std::atomic<size_t> &next, size_t rows, size_t rows_per,
                  size_t row_bytes, char *host, char *dev, size_t dpitch, cudaStream_t st, int device)
{
    cudaError_t e = cudaSetDevice(device);
    cudaEvent_t ev[2] = {nullptr, nullptr};
    for (auto &v : ev)
        if (e == cudaSuccess) e = cudaEventCreateWithFlags(&v, cudaEventDisableTiming);
    struct Flight {
        size_t r0 = 0, n = 0;
    } fl[2];
    auto land = [&](int b) {
        if (!fl[b].n) return;
        const cudaError_t w = cudaEventSynchronize(ev[b]);
        if (e == cudaSuccess) e = w;
        if (!to_device && e == cudaSuccess)
            memcpy(host + fl[b].r0 * row_bytes, ring + (size_t) (2 * t + b) * kChunk, fl[b].n * row_bytes);
        fl[b].n = 0;
    };
    int b = 0;
    while (e == cudaSuccess) {
        const size_t r0 = next.fetch_add(rows_per);
        if (r0 >= rows) break;
        const size_t n = std::min(rows_per, rows - r0);
        char *buf = ring + (size_t) (2 * t + b) * kChunk;
        land(b);
        if (e != cudaSuccess) break;
        if (to_device) {
            memcpy(buf, host + r0 * row_bytes, n * row_bytes);
            e = dpitch == row_bytes
                    ? cudaMemcpyAsync(dev + r0 * dpitch, buf, n * row_bytes, cudaMemcpyHostToDevice, st)
                    : cudaMemcpy2DAsync(dev + r0 * dpitch, dpitch, buf, row_bytes, row_bytes, n, cudaMemcpyHostToDevice, st);
        } else {
            e = cudaMemcpyAsync(buf, dev + r0 * dpitch, n * row_bytes, cudaMemcpyDeviceToHost, st);
        }
        if (e == cudaSuccess) e = cudaEventRecord(ev[b], st);
        fl[b] = {r0, n};
        b ^= 1;
    }
    land(b);
    land(b ^ 1);
    for (auto v : ev)
        if (v) cudaEventDestroy(v);
    return e;
}

cudaError_t staged(bool to_device, char *host, char *dev, size_t dpitch, size_t row_bytes, size_t rows,
                   cudaStream_t st, int device, bool *done)
{
    *done = false;
    if (row_bytes * rows < kMinBytes || row_bytes > kChunk || !pageable(host)) return cudaSuccess;
    // what is queued on the stream (a result's whole run of iterations) is
    // waited for here, by one thread: not with the buffers held, nor by every
    // worker
    if (const cudaError_t e = cudaStreamSynchronize(st)) return e;
    std::unique_lock<std::mutex> lk(g_ring_mu, std::try_to_lock);
    if (!lk.owns_lock()) return cudaSuccess;
    char *ring = ring_locked();
    if (!ring) return cudaSuccess;
    const size_t rows_per = std::max<size_t>(1, kChunk / row_bytes);
    std::atomic<size_t> next{0};
    std::atomic<int> err{(int) cudaSuccess};
    on_threads(worker_count((rows + rows_per - 1) / rows_per), [&](int t) {
        const cudaError_t e =
            stage(to_device, ring, t, next, rows, rows_per, row_bytes, host, dev, dpitch, st, device);
        if (e != cudaSuccess) err.store((int) e);
    });
    *done = true;
    return (cudaError_t) err.load();
}

}  // namespace

cudaError_t copy_to_device(void *dev, size_t dpitch, const void *host, size_t row_bytes, size_t rows,
                           cudaStream_t st, int device)
{
    bool done = false;
    if (dpitch != row_bytes) {
        const cudaError_t e = staged(true, (char *) host, (char *) dev, dpitch, row_bytes, rows, st, device, &done);
        if (done || e != cudaSuccess) return e;
        return cudaMemcpy2DAsync(dev, dpitch, host, row_bytes, row_bytes, rows, cudaMemcpyHostToDevice, st);
    }
    // an unpitched copy is cut into pieces of its own
    const size_t bytes = row_bytes * rows, piece = 4096, whole = bytes / piece * piece;
    const cudaError_t e = staged(true, (char *) host, (char *) dev, piece, piece, whole / piece, st, device, &done);
    if (e != cudaSuccess) return e;
    const size_t from = done ? whole : 0;
    if (from == bytes) return cudaSuccess;
    return cudaMemcpyAsync((char *) dev + from, (const char *) host + from, bytes - from, cudaMemcpyHostToDevice, st);
}

cudaError_t copy_to_host(void *host, const void *dev, size_t bytes, cudaStream_t st, int device)
{
    bool done = false;
    const size_t piece = 4096, whole = bytes / piece * piece;
    cudaError_t e = staged(false, (char *) host, (char *) const_cast<void *>(dev), piece, piece, whole / piece, st,
                           device, &done);
    if (e != cudaSuccess) return e;
    const size_t from = done ? whole : 0;
    if (from == bytes) return cudaSuccess;
    return cudaMemcpyAsync((char *) host + from, (const char *) dev + from, bytes - from, cudaMemcpyDeviceToHost, st);
}

void copy_release()
{
    std::lock_guard<std::mutex> lk(g_ring_mu);
    if (g_ring) cudaFreeHost(g_ring);
    cudaGetLastError();
    g_ring = nullptr;
}

void Prefault::start(void *p, size_t bytes)
{
    if (!bytes || !pageable(p)) return;
    const size_t chunk = (size_t) 4 << 20, chunks = (bytes + chunk - 1) / chunk;
    const int nt = std::min(4, worker_count(chunks));
    try {
        next_.store(0);
        for (int t = 0; t < nt; ++t)
            th_.emplace_back([this, p, bytes, chunk]() {
                for (;;) {
                    const size_t o = next_.fetch_add(chunk);
                    if (o >= bytes) break;
                    memset((char *) p + o, 0, std::min(chunk, bytes - o));
                }
            });
    } catch (const std::system_error &) {  // fewer threads, or none: the copy faults the pages in
    } catch (const std::bad_alloc &) {
    }
}

void Prefault::join()
{
    for (auto &t : th_) t.join();
    th_.clear();
}

}  // namespace dwcu
