// A CUDA runtime of host threads for hostcopy.cu: streams run their work in
// order on a thread each, and copies say whether they came through page-locked
// memory or took the driver's path.
#include <cuda_runtime.h>

#include <atomic>
#include <condition_variable>
#include <cstdlib>
#include <cstring>
#include <deque>
#include <functional>
#include <map>
#include <mutex>
#include <thread>

#include "hostcopy.h"

namespace {

std::mutex g_mu;
std::map<const char *, size_t> g_locked;  // page-locked ranges
std::atomic<long long> g_staged{0}, g_driver{0};

bool locked(const void *p)
{
    std::lock_guard<std::mutex> lk(g_mu);
    auto it = g_locked.upper_bound((const char *) p);
    if (it == g_locked.begin()) return false;
    --it;
    return (const char *) p < it->first + it->second;
}

struct Stream {
    std::mutex mu;
    std::condition_variable cv;
    std::deque<std::function<void()>> work;
    bool busy = false, stop = false;
    std::thread th{[this] {
        std::unique_lock<std::mutex> lk(mu);
        for (;;) {
            cv.wait(lk, [&] { return stop || !work.empty(); });
            if (work.empty()) return;
            auto f = std::move(work.front());
            work.pop_front();
            busy = true;
            lk.unlock();
            f();
            lk.lock();
            busy = false;
            cv.notify_all();
        }
    }};
    void push(std::function<void()> f)
    {
        std::lock_guard<std::mutex> lk(mu);
        work.push_back(std::move(f));
        cv.notify_all();
    }
    ~Stream()
    {
        {
            std::lock_guard<std::mutex> lk(mu);
            stop = true;
            cv.notify_all();
        }
        th.join();
    }
};

struct Event {
    std::mutex mu;
    std::condition_variable cv;
    long long recorded = 0, reached = 0;
};

// waits for the work queued on the stream so far
void drain(Stream *s)
{
    Event e;
    s->push([&e] {
        std::lock_guard<std::mutex> lk(e.mu);
        e.reached = 1;
        e.cv.notify_all();
    });
    std::unique_lock<std::mutex> lk(e.mu);
    e.cv.wait(lk, [&] { return e.reached == 1; });
}

cudaError_t copy2d(void *dst, size_t dp, const void *src, size_t sp, size_t width, size_t rows, cudaMemcpyKind kind,
                   cudaStream_t st)
{
    auto *s = (Stream *) st;
    auto f = [=] {
        for (size_t r = 0; r < rows; ++r) memcpy((char *) dst + r * dp, (const char *) src + r * sp, width);
    };
    const bool through = locked(kind == cudaMemcpyHostToDevice ? src : dst);
    ++(through ? g_staged : g_driver);
    if (through) {
        s->push(f);
    } else {  // pageable memory: the caller waits
        drain(s);
        f();
    }
    return cudaSuccess;
}

}  // namespace

extern "C" {

cudaError_t cudaHostAlloc(void **p, size_t n, unsigned)
{
    *p = malloc(n);
    std::lock_guard<std::mutex> lk(g_mu);
    g_locked[(const char *) *p] = n;
    return cudaSuccess;
}
cudaError_t cudaFreeHost(void *p)
{
    {
        std::lock_guard<std::mutex> lk(g_mu);
        g_locked.erase((const char *) p);
    }
    free(p);
    return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *a, const void *p)
{
    memset(a, 0, sizeof *a);
    a->type = locked(p) ? cudaMemoryTypeHost : cudaMemoryTypeUnregistered;
    return cudaSuccess;
}
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned)
{
    *e = (cudaEvent_t) new Event();
    return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t e)
{
    delete (Event *) e;
    return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t ev, cudaStream_t st)
{
    auto *e = (Event *) ev;
    std::lock_guard<std::mutex> lk(e->mu);
    const long long k = ++e->recorded;
    ((Stream *) st)->push([e, k] {
        std::lock_guard<std::mutex> l2(e->mu);
        e->reached = k;
        e->cv.notify_all();
    });
    return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t ev)
{
    auto *e = (Event *) ev;
    std::unique_lock<std::mutex> lk(e->mu);
    const long long k = e->recorded;
    e->cv.wait(lk, [&] { return e->reached >= k; });
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t st)
{
    drain((Stream *) st);
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind kind, cudaStream_t st)
{
    return copy2d(d, n, s, n, n, 1, kind, st);
}
cudaError_t cudaMemcpy2DAsync(void *d, size_t dp, const void *s, size_t sp, size_t w, size_t h, cudaMemcpyKind kind,
                              cudaStream_t st)
{
    return copy2d(d, dp, s, sp, w, h, kind, st);
}

// ---- for the tests

void *fake_stream() { return new Stream(); }
void fake_stream_end(void *s) { delete (Stream *) s; }
// the stream stays busy until the returned gate is opened
void *fake_gate(void *s)
{
    auto *e = new Event();
    ((Stream *) s)->push([e] {
        std::unique_lock<std::mutex> lk(e->mu);
        e->cv.wait(lk, [&] { return e->reached == 1; });
    });
    return e;
}
void fake_open(void *gate)
{
    auto *e = (Event *) gate;
    std::lock_guard<std::mutex> lk(e->mu);
    e->reached = 1;
    e->cv.notify_all();
}
void fake_sync(void *s) { drain((Stream *) s); }
long long fake_staged() { return g_staged; }
long long fake_driver() { return g_driver; }
int to_device(void *dev, size_t dpitch, const void *host, size_t row_bytes, size_t rows, void *st)
{
    return (int) dwcu::copy_to_device(dev, dpitch, host, row_bytes, rows, (cudaStream_t) st, 0);
}
int to_host(void *host, const void *dev, size_t bytes, void *st)
{
    return (int) dwcu::copy_to_host(host, dev, bytes, (cudaStream_t) st, 0);
}
void release() { dwcu::copy_release(); }

}  // extern "C"
