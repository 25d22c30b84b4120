/*
 * A CUDA runtime of host memory for tests of host code: the calls the field
 * transfers make, on streams that run what is queued on them only when a test
 * or a wait lets them.  "Device" memory is host memory; page-locked memory is
 * what cudaHostAlloc returned, other kinds come from fake::make; every other
 * pointer is pageable.  Copies from or to pageable memory behave as the
 * runtime documents them: the source has been read, the destination has been
 * written, when the call returns.
 */
#ifndef FAKE_CUDA_RUNTIME_H
#define FAKE_CUDA_RUNTIME_H

#include <stdlib.h>
#include <string.h>

#include <condition_variable>
#include <deque>
#include <functional>
#include <map>
#include <memory>
#include <mutex>
#include <vector>

typedef int cudaError_t;
enum { cudaSuccess = 0, cudaErrorInvalidValue = 1, cudaErrorInvalidResourceHandle = 400, cudaErrorNotReady = 600 };
enum { cudaMemcpyHostToDevice = 1, cudaMemcpyDeviceToHost = 2 };
enum { cudaHostAllocPortable = 1, cudaEventDisableTiming = 2 };
enum cudaStreamCaptureStatus { cudaStreamCaptureStatusNone = 0, cudaStreamCaptureStatusActive = 1 };
enum cudaMemoryType { cudaMemoryTypeUnregistered, cudaMemoryTypeHost, cudaMemoryTypeDevice, cudaMemoryTypeManaged };
struct cudaPointerAttributes { cudaMemoryType type; };
struct int2 { int x, y; };
struct float4 { float x, y, z, w; };

struct FakeStream {
    int device = 0;
    bool open = true; /* a closed stream's work waits until the test opens it */
    long long queued = 0, ran = 0;
    std::deque<std::function<void()>> work;
};
typedef FakeStream *cudaStream_t;
struct FakeEvent {
    int device = 0;
    FakeStream *stream = nullptr;
    long long at = 0;
};
typedef FakeEvent *cudaEvent_t;

namespace fake {
inline std::mutex mu;
inline std::condition_variable cv;
inline std::map<const char *, std::pair<size_t, cudaMemoryType>> known; /* start -> size, kind */
inline thread_local int device = 0;
inline thread_local cudaError_t last = cudaSuccess;
inline int device_callers = 0; /* copies whose caller's side is device memory */

inline cudaMemoryType kind(const void *p) {
    auto it = known.upper_bound((const char *)p);
    if (it == known.begin()) return cudaMemoryTypeUnregistered;
    --it;
    return (const char *)p < it->first + it->second.first ? it->second.second : cudaMemoryTypeUnregistered;
}
inline void *make(size_t n, cudaMemoryType k) {
    std::lock_guard<std::mutex> l(mu);
    char *p = (char *)calloc(n, 1);
    known[p] = {n, k};
    return p;
}
/* runs a stream's work up to item `upto`, waiting for the test to open it */
inline void drain(std::unique_lock<std::mutex> &l, FakeStream *s, long long upto) {
    while (s->ran < upto) {
        cv.wait(l, [&] { return s->open; });
        if (s->ran >= upto) break;
        auto f = s->work.front();
        s->work.pop_front();
        f();
        s->ran++;
    }
}
inline void push(FakeStream *s, std::function<void()> f) {
    s->work.push_back(std::move(f));
    s->queued++;
}
inline void set_open(FakeStream *s, bool open) {
    std::lock_guard<std::mutex> l(mu);
    s->open = open;
    cv.notify_all();
}
} // namespace fake

inline const char *cudaGetErrorString(cudaError_t) { return "fake CUDA error"; }
inline cudaError_t cudaPeekAtLastError() { return fake::last; }
inline cudaError_t cudaGetLastError() {
    const cudaError_t e = fake::last;
    fake::last = cudaSuccess;
    return e;
}
inline cudaError_t cudaGetDevice(int *d) { *d = fake::device; return cudaSuccess; }
inline cudaError_t cudaSetDevice(int d) { fake::device = d; return cudaSuccess; }
inline cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) {
    *p = fake::make(n, cudaMemoryTypeHost);
    return cudaSuccess;
}
inline cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *a, const void *p) {
    std::lock_guard<std::mutex> l(fake::mu);
    a->type = fake::kind(p);
    return cudaSuccess;
}
inline cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus *st) {
    *st = cudaStreamCaptureStatusNone;
    return cudaSuccess;
}
inline cudaError_t cudaStreamGetDevice(cudaStream_t s, int *d) { *d = s->device; return cudaSuccess; }
inline cudaError_t cudaStreamSynchronize(cudaStream_t s) {
    std::unique_lock<std::mutex> l(fake::mu);
    fake::drain(l, s, s->queued);
    return cudaSuccess;
}
inline cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) {
    *e = new FakeEvent{fake::device, nullptr, 0};
    return cudaSuccess;
}
inline cudaError_t cudaEventDestroy(cudaEvent_t e) { delete e; return cudaSuccess; }
inline cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
    if (e->device != s->device) return cudaErrorInvalidResourceHandle;
    std::lock_guard<std::mutex> l(fake::mu);
    e->stream = s;
    e->at = s->queued;
    return cudaSuccess;
}
inline cudaError_t cudaEventQuery(cudaEvent_t e) {
    std::unique_lock<std::mutex> l(fake::mu);
    if (e->stream && e->stream->open) fake::drain(l, e->stream, e->at);
    if (!e->stream || e->stream->ran >= e->at) return cudaSuccess;
    if (fake::last == cudaSuccess) fake::last = cudaErrorNotReady;
    return cudaErrorNotReady;
}
inline cudaError_t cudaEventSynchronize(cudaEvent_t e) {
    std::unique_lock<std::mutex> l(fake::mu);
    if (e->stream) fake::drain(l, e->stream, e->at);
    return cudaSuccess;
}
inline cudaError_t cudaMemcpy2DAsync(void *d, size_t dp, const void *s, size_t sp, size_t w, size_t h, int dir,
                                     cudaStream_t st) {
    auto rows = [=](char *to, size_t tp, const char *from, size_t fp) {
        for (size_t j = 0; j < h; j++) memcpy(to + j * tp, from + j * fp, w);
    };
    std::unique_lock<std::mutex> l(fake::mu);
    const bool up = dir == cudaMemcpyHostToDevice;
    const cudaMemoryType k = fake::kind(up ? s : d);
    fake::device_callers += k == cudaMemoryTypeDevice;
    if (k != cudaMemoryTypeUnregistered) {
        fake::push(st, [=] { rows((char *)d, dp, (const char *)s, sp); });
    } else if (up) {
        auto copy = std::make_shared<std::vector<char>>(w * h);
        rows(copy->data(), w, (const char *)s, sp);
        fake::push(st, [=] { rows((char *)d, dp, copy->data(), w); });
    } else {
        fake::push(st, [=] { rows((char *)d, dp, (const char *)s, sp); });
        fake::drain(l, st, st->queued);
    }
    return cudaSuccess;
}

#endif
