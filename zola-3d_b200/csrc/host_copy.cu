// Large copies between pageable host memory and the device.
//
// The driver moves pageable memory through its own pinned buffers with one thread, 12 GB/s
// up and 4 GB/s down into fresh pages.  Here a few threads of the context each move every
// T-th segment through two pinned buffers of their own, so that their memcpys (and page
// faults) run side by side and overlap the copies: the 33 MB of 2,600 ROIs of 40 px and
// their variances take 0.9 ms instead of 2.9 (3,001 such fits 11.4 -> 10.0 ms).
#include <cuda_runtime.h>

#include <algorithm>
#include <condition_variable>
#include <cstring>
#include <memory>
#include <mutex>
#include <new>
#include <thread>

#include "zola_internal.h"

namespace zola {

// 512 KB a segment: a copy of 10 us, a memcpy of 50; four threads fill most of the link.
// Below 4 MB the driver's copy is as fast or faster: a gradient on 2.5 MB of bead stacks
// takes 0.56 ms with it and 0.70 with the threads, 2,000 fits of 16 px 2.70 and 2.87.
constexpr size_t HC_SEG = 512 << 10, HC_MIN = 4 << 20;
constexpr int HC_MAX_THREADS = 4;

struct HostCopy {
    // What the helpers share with the context.  They are detached, so that a context can be
    // given up in a process that has lost them (a forked child) without waiting for them.
    struct Shared {
        std::mutex mu;
        std::condition_variable wake, idle;
        unsigned job = 0;
        int pending = 0;
        bool stop = false;
        int device = 0, threads = 1;
        // the job
        bool in = false;
        char* dst = nullptr;
        const char* src = nullptr;
        size_t bytes = 0;
        cudaStream_t st = nullptr;
        char* buf[2 * HC_MAX_THREADS] = {};
        cudaEvent_t ev[2 * HC_MAX_THREADS] = {};
        cudaError_t err[HC_MAX_THREADS] = {};
    };
    std::shared_ptr<Shared> s;
};

// Segments t, t + T, ... of the job.
static cudaError_t hc_part(HostCopy::Shared& s, int t) {
    const size_t nseg = (s.bytes + HC_SEG - 1) / HC_SEG, step = s.threads;
    auto len = [&](size_t k) { return s.bytes - k * HC_SEG < HC_SEG ? s.bytes - k * HC_SEG : HC_SEG; };
    cudaError_t e = cudaSuccess;
    if (s.in) {
        int b = 2 * t;
        for (size_t k = t; k < nseg && e == cudaSuccess; k += step, b ^= 1) {
            e = cudaEventSynchronize(s.ev[b]);  // its last copy has left the buffer
            if (e != cudaSuccess) break;
            memcpy(s.buf[b], s.src + k * HC_SEG, len(k));
            e = cudaMemcpyAsync(s.dst + k * HC_SEG, s.buf[b], len(k), cudaMemcpyHostToDevice, s.st);
            if (e == cudaSuccess) e = cudaEventRecord(s.ev[b], s.st);
        }
        return e;
    }
    auto fetch = [&](size_t k, int b) {
        if (k >= nseg || e != cudaSuccess) return;
        e = cudaEventSynchronize(s.ev[b]);
        if (e == cudaSuccess)
            e = cudaMemcpyAsync(s.buf[b], s.src + k * HC_SEG, len(k), cudaMemcpyDeviceToHost, s.st);
        if (e == cudaSuccess) e = cudaEventRecord(s.ev[b], s.st);
    };
    fetch(t, 2 * t);
    fetch(t + step, 2 * t + 1);
    int b = 2 * t;
    for (size_t k = t; k < nseg && e == cudaSuccess; k += step, b ^= 1) {
        e = cudaEventSynchronize(s.ev[b]);
        if (e != cudaSuccess) break;
        memcpy(s.dst + k * HC_SEG, s.buf[b], len(k));
        fetch(k + 2 * step, b);
    }
    return e;
}

static void hc_thread(std::shared_ptr<HostCopy::Shared> s, int t) {
    const cudaError_t dev = cudaSetDevice(s->device);
    unsigned seen = 0;
    for (;;) {
        {
            std::unique_lock<std::mutex> lock(s->mu);
            s->wake.wait(lock, [&] { return s->stop || s->job != seen; });
            if (s->stop) return;
            seen = s->job;
        }
        s->err[t] = dev == cudaSuccess ? hc_part(*s, t) : dev;
        std::lock_guard<std::mutex> lock(s->mu);
        if (--s->pending == 0) s->idle.notify_one();
    }
}

// The context's helpers, or null where there are none to be had.
static HostCopy* hc_get(zola_ctx* ctx) {
    if (ctx->host_copy) return ctx->host_copy->s ? ctx->host_copy : nullptr;
    try {
        ctx->host_copy = new HostCopy();
        const int T = std::min<int>(HC_MAX_THREADS, (int)std::thread::hardware_concurrency());
        if (T < 2) return nullptr;
        auto s = std::make_shared<HostCopy::Shared>();
        s->device = ctx->device;
        s->threads = T;
        bool ok = cudaMallocHost((void**)&s->buf[0], 2 * T * HC_SEG) == cudaSuccess;
        for (int b = 0; b < 2 * T && ok; ++b) {
            s->buf[b] = s->buf[0] + b * HC_SEG;
            ok = cudaEventCreateWithFlags(&s->ev[b], cudaEventDisableTiming) == cudaSuccess;
        }
        ctx->host_copy->s = s;
        if (ok)
            for (int t = 1; t < T; ++t) std::thread(hc_thread, s, t).detach();
        if (!ok) {
            cudaGetLastError();
            host_copy_free(ctx);
            ctx->host_copy = new HostCopy();
            return nullptr;
        }
        return ctx->host_copy;
    } catch (...) {  // no memory or no threads: the driver's copies
        host_copy_free(ctx);
        ctx->host_copy = new (std::nothrow) HostCopy();
        return nullptr;
    }
}

void host_copy_free(zola_ctx* ctx) {
    HostCopy* h = ctx->host_copy;
    ctx->host_copy = nullptr;
    if (!h) return;
    if (h->s) {
        {
            std::lock_guard<std::mutex> lock(h->s->mu);
            h->s->stop = true;
        }
        h->s->wake.notify_all();
        for (cudaEvent_t e : h->s->ev)
            if (e) {
                cudaEventSynchronize(e);
                cudaEventDestroy(e);
            }
        if (h->s->buf[0]) cudaFreeHost(h->s->buf[0]);
    }
    delete h;
}

bool device_memory(const void* p) {
    cudaPointerAttributes a{};
    if (!p) return false;
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return a.type == cudaMemoryTypeDevice;
}

// Whether the driver would stage this host memory itself.
static bool pageable(const void* p) {
    cudaPointerAttributes a{};
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return a.type == cudaMemoryTypeUnregistered;
}

static cudaError_t hc_run(HostCopy* h, bool in, void* dst, const void* src, size_t bytes, cudaStream_t st) {
    HostCopy::Shared& s = *h->s;
    {
        std::lock_guard<std::mutex> lock(s.mu);
        s.in = in;
        s.dst = (char*)dst;
        s.src = (const char*)src;
        s.bytes = bytes;
        s.st = st;
        s.pending = s.threads - 1;
        ++s.job;
    }
    s.wake.notify_all();
    s.err[0] = hc_part(s, 0);
    std::unique_lock<std::mutex> lock(s.mu);
    s.idle.wait(lock, [&] { return s.pending == 0; });
    for (int t = 0; t < s.threads; ++t)
        if (s.err[t] != cudaSuccess) return s.err[t];
    return cudaSuccess;
}

cudaError_t copy_in(zola_ctx* ctx, void* dst, const void* src, size_t bytes, cudaStream_t st) {
    HostCopy* h = bytes >= HC_MIN && pageable(src) ? hc_get(ctx) : nullptr;
    if (!h) return cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, st);
    return hc_run(h, true, dst, src, bytes, st);
}

cudaError_t copy_out(zola_ctx* ctx, void* dst, const void* src, size_t bytes, cudaStream_t st) {
    HostCopy* h = bytes >= HC_MIN && pageable(dst) ? hc_get(ctx) : nullptr;
    if (!h) return cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, st);
    const cudaError_t e = cudaStreamSynchronize(st);
    return e == cudaSuccess ? hc_run(h, false, dst, src, bytes, st) : e;
}

}  // namespace zola
