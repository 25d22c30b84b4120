/*
 * Field transfers through page-locked staging.
 *
 * A copy between pageable memory and the device is staged by the driver on
 * one thread: 2-3 GB/s here for a pitched field, page faults of a fresh
 * destination included (a 2401 x 2001 forecast spent 30 ms of 108 reading five
 * fields).  These calls move a field in pieces through two page-locked
 * buffers: the copy engine fills or drains one at the link's rate while host
 * threads copy the other, each thread also taking the page faults of its part.
 *
 * The two buffers (8 MB each) are made at the first transfer of at least
 * 256 KB and kept for the process; a mutex gives them to one call at a time.
 * It is held while a field moves, never while a stream's earlier work runs: a
 * download, and an upload that fills a buffer twice, first wait for their
 * stream, and an upload whose stream is busy leaves its copies queued, marks
 * its buffers and returns.  A call that finds too few buffers free because
 * another stream's uploads are still queued takes the plain copy, so no caller
 * waits for another one's steps; so do smaller transfers, those whose caller's
 * side is not ordinary memory (page-locked memory needs no staging, device
 * memory no host thread can touch, and both may be what earlier work on the
 * stream writes or reads), and all where the buffers cannot be had.
 */
#include <string.h>

#include <algorithm>
#include <mutex>
#include <thread>
#include <vector>

#include "hostio.h"

namespace {

constexpr size_t kSlot = (size_t)8 << 20;
constexpr size_t kSmall = (size_t)256 << 10;

struct Staging {
    std::mutex mu;
    bool tried = false;
    char *slot[2] = {nullptr, nullptr};
    cudaEvent_t busy[2] = {nullptr, nullptr}; /* a transfer still using the slot */
    cudaStream_t by[2] = {nullptr, nullptr};  /* and its stream */

    bool ready() {
        if (!tried) {
            tried = true;
            for (auto &p : slot)
                if (cudaHostAlloc((void **)&p, kSlot, cudaHostAllocPortable) != cudaSuccess) {
                    p = nullptr;
                    cudaGetLastError(); /* refused: the plain copy */
                }
        }
        return slot[0] && slot[1];
    }
    /* Locks the slots for a transfer on `s` that needs `need` of them at once
     * and gives the first to use; -1, unlocked, where the plain copy is to be
     * taken.  Slots that earlier uploads on `s` still hold are waited for
     * outside the lock. */
    int take(std::unique_lock<std::mutex> &lock, int need, cudaStream_t s) {
        for (int attempt = 0; attempt < 2; attempt++) {
            lock.lock();
            if (!ready()) break;
            int nfree = 0, first = 0;
            bool own = false;
            for (int k = 1; k >= 0; k--) {
                if (busy[k] && cudaEventQuery(busy[k]) == cudaErrorNotReady) {
                    if (cudaPeekAtLastError() == cudaErrorNotReady) cudaGetLastError(); /* an answer, not an error */
                    own = own || by[k] == s;
                    continue;
                }
                nfree++;
                first = k;
            }
            if (nfree >= need) return first;
            if (!own) break;
            lock.unlock();
            if (cudaStreamSynchronize(s) != cudaSuccess) return -1; /* the plain copy meets the same error */
        }
        if (lock.owns_lock()) lock.unlock();
        return -1;
    }
    int wait(int k) {
        if (!busy[k]) return GC_OK;
        const cudaError_t e = cudaEventSynchronize(busy[k]);
        cudaEventDestroy(busy[k]);
        busy[k] = nullptr;
        GC_CUDA_OR_RET(e);
        return GC_OK;
    }
    /* the event belongs to the stream's device, whichever is current */
    static cudaError_t make_event(cudaEvent_t *ev, cudaStream_t s) {
        int dev = 0, cur = 0;
        cudaError_t e = cudaGetDevice(&cur);
        if (e == cudaSuccess) e = cudaStreamGetDevice(s, &dev);
        if (e == cudaSuccess && dev != cur) e = cudaSetDevice(dev);
        if (e != cudaSuccess) return e;
        e = cudaEventCreateWithFlags(ev, cudaEventDisableTiming);
        if (dev != cur) cudaSetDevice(cur);
        return e;
    }
    int mark(int k, cudaStream_t s) {
        cudaError_t e = make_event(&busy[k], s);
        if (e != cudaSuccess) busy[k] = nullptr;
        else e = cudaEventRecord(busy[k], s);
        by[k] = s;
        if (e != cudaSuccess) cudaStreamSynchronize(s); /* nobody else may find the slot in use */
        GC_CUDA_OR_RET(e);
        return GC_OK;
    }
};
Staging g_staging;

bool capturing(cudaStream_t s) {
    cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
    return cudaStreamIsCapturing(s, &st) != cudaSuccess || st != cudaStreamCaptureStatusNone;
}

/* Ordinary host memory: an asynchronous copy from it has read it when the call
 * returns, while one from page-locked, managed or device memory reads it when
 * the stream gets there, after what earlier work on the stream writes to it. */
bool pageable(const void *p) {
    cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, p) == cudaSuccess) return a.type == cudaMemoryTypeUnregistered;
    cudaGetLastError();
    return false; /* unknown: the plain copy, waited for */
}

} // namespace

void gc_copy(void *dst, const void *src, size_t bytes) {
    const unsigned hw = std::thread::hardware_concurrency();
    /* a thread costs about 20 us to start, a megabyte 100-300 us to copy */
    const int nt = (int)std::min<size_t>(std::min(hw ? hw : 1u, 8u), bytes >> 20);
    if (nt <= 1) {
        memcpy(dst, src, bytes);
        return;
    }
    const size_t part = (bytes / nt + 4095) & ~(size_t)4095;
    auto work = [&](int t) {
        const size_t a = std::min(bytes, part * t), b = t == nt - 1 ? bytes : std::min(bytes, part * (t + 1));
        memcpy((char *)dst + a, (const char *)src + a, b - a);
    };
    std::vector<std::thread> pool;
    int started = 1;
    try {
        pool.reserve(nt);
        for (; started < nt; started++) pool.emplace_back(work, started);
    } catch (...) {
        /* no more threads, or no memory for them: this one copies the rest */
        for (int t = started; t < nt; t++) work(t);
    }
    work(0);
    for (auto &th : pool) th.join();
}

int gc_field_upload(float *d, size_t pitch_bytes, const float *h, int nx, int ny, cudaStream_t s) {
    const size_t row = (size_t)nx * sizeof(float), total = row * ny;
    std::unique_lock<std::mutex> lock(g_staging.mu, std::defer_lock);
    int first = -1;
    const bool capture = capturing(s);
    const bool host = pageable(h);
    if (total >= kSmall && row <= kSlot && !capture && host) {
        const int rows = (int)(kSlot / row), pieces = (ny + rows - 1) / rows;
        if (pieces > 2) GC_CUDA_OR_RET(cudaStreamSynchronize(s)); /* the third piece waits for the first copy */
        first = g_staging.take(lock, std::min(pieces, 2), s);
    }
    if (first < 0) {
        GC_CUDA_OR_RET(cudaMemcpy2DAsync(d, pitch_bytes, h, row, row, (size_t)ny, cudaMemcpyHostToDevice, s));
        if (!host && !capture) GC_CUDA_OR_RET(cudaStreamSynchronize(s));
        return GC_OK;
    }
    const int rows = (int)(kSlot / row);
    for (int j = 0, k = first; j < ny; j += rows, k ^= 1) {
        const int n = std::min(rows, ny - j);
        int rc = g_staging.wait(k);
        if (rc != GC_OK) return rc;
        gc_copy(g_staging.slot[k], (const char *)h + (size_t)j * row, (size_t)n * row);
        GC_CUDA_OR_RET(cudaMemcpy2DAsync((char *)d + (size_t)j * pitch_bytes, pitch_bytes, g_staging.slot[k], row, row,
                                         (size_t)n, cudaMemcpyHostToDevice, s));
        rc = g_staging.mark(k, s);
        if (rc != GC_OK) return rc;
    }
    return GC_OK;
}

int gc_field_download(void *h, const void *d, size_t pitch_bytes, int nx, int ny, cudaStream_t s) {
    const size_t row = (size_t)nx * sizeof(float), total = row * ny;
    std::unique_lock<std::mutex> lock(g_staging.mu, std::defer_lock);
    int first = -1;
    if (total >= kSmall && row <= kSlot && !capturing(s) && pageable(h)) {
        GC_CUDA_OR_RET(cudaStreamSynchronize(s));
        first = g_staging.take(lock, 2, s);
    }
    if (first < 0) {
        GC_CUDA_OR_RET(cudaMemcpy2DAsync(h, row, d, pitch_bytes, row, (size_t)ny, cudaMemcpyDeviceToHost, s));
        GC_CUDA_OR_RET(cudaStreamSynchronize(s));
        return GC_OK;
    }
    /* quarter slots at least, so that small fields also overlap */
    const int rows = std::max(1, (int)std::min(kSlot / row, (size_t)(ny + 3) / 4));
    auto fetch = [&](int j, int k) -> int {
        const int n = std::min(rows, ny - j);
        int rc = g_staging.wait(k);
        if (rc != GC_OK) return rc;
        GC_CUDA_OR_RET(cudaMemcpy2DAsync(g_staging.slot[k], row, (const char *)d + (size_t)j * pitch_bytes, pitch_bytes,
                                         row, (size_t)n, cudaMemcpyDeviceToHost, s));
        return g_staging.mark(k, s);
    };
    int rc = fetch(0, 0);
    for (int j = 0, k = 0; j < ny && rc == GC_OK; j += rows, k ^= 1) {
        if (j + rows < ny) rc = fetch(j + rows, k ^ 1);
        if (rc == GC_OK) rc = g_staging.wait(k);
        if (rc == GC_OK)
            gc_copy((char *)h + (size_t)j * row, g_staging.slot[k], (size_t)std::min(rows, ny - j) * row);
    }
    return rc;
}

extern "C" int gc_host_copy(void *dst, const void *src, long long bytes) {
    if (!dst || !src || bytes < 0) return GC_EINVAL;
    gc_copy(dst, src, (size_t)bytes);
    return GC_OK;
}
