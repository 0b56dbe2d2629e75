/* A stand-in for the parts of the CUDA runtime that host_stage.h uses, for a test
 * without a GPU: streams are queues of copies that run as late as they may (when
 * something behind them is waited for), so a buffer used too early shows. */
#pragma once
#include <cstddef>
#include <cstdlib>
#include <cstring>
#include <deque>
#include <functional>

enum cudaError_t { cudaSuccess = 0, cudaErrorUnknown = 999 };
enum cudaMemcpyKind { cudaMemcpyHostToDevice, cudaMemcpyDeviceToHost };
enum cudaMemoryType { cudaMemoryTypeUnregistered, cudaMemoryTypeHost };
struct cudaPointerAttributes {
    cudaMemoryType type;
};
constexpr unsigned cudaHostAllocDefault = 0, cudaHostAllocMapped = 2, cudaEventDisableTiming = 2;

struct FakeStream {
    std::deque<std::function<void()>> q;
    size_t ran = 0, put = 0;
    void run(size_t upto) {
        for (; ran < upto; ran++) {
            q.front()();
            q.pop_front();
        }
    }
};
struct FakeEvent {
    FakeStream *st = nullptr;
    size_t at = 0;
};
using cudaStream_t = FakeStream *;
using cudaEvent_t = FakeEvent *;

inline int fake_fail_copy_in = -1;             /* the n-th copy from now on fails */
inline const char *fake_locked_lo = nullptr, *fake_locked_hi = nullptr;
inline int fake_direct_copies = 0;             /* copies from or to page-locked user memory */
inline void (*fake_after_sync)() = nullptr;    /* what else may happen at that moment */

inline cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) {
    *p = calloc(1, n);
    return cudaSuccess;
}
inline cudaError_t cudaHostGetDevicePointer(void **d, void *h, unsigned) {
    *d = h;
    return cudaSuccess;
}
inline cudaError_t cudaFreeHost(void *p) {
    free(p);
    return cudaSuccess;
}
inline cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) {
    *e = new FakeEvent();
    return cudaSuccess;
}
inline cudaError_t cudaEventDestroy(cudaEvent_t e) {
    delete e;
    return cudaSuccess;
}
inline cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
    e->st = s;
    e->at = s->put;
    return cudaSuccess;
}
inline cudaError_t cudaEventSynchronize(cudaEvent_t e) {
    if (e->st) e->st->run(e->at);
    if (fake_after_sync) fake_after_sync();
    return cudaSuccess;
}
inline cudaError_t cudaStreamSynchronize(cudaStream_t s) {
    s->run(s->put);
    return cudaSuccess;
}
inline bool fake_locked(const void *p) {
    return (const char *)p >= fake_locked_lo && (const char *)p < fake_locked_hi;
}
inline cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind,
                                   cudaStream_t st) {
    if (fake_fail_copy_in >= 0 && fake_fail_copy_in-- == 0) return cudaErrorUnknown;
    if (fake_locked(d) || fake_locked(s)) fake_direct_copies++;
    st->q.push_back([=] { memcpy(d, s, n); });
    st->put++;
    return cudaSuccess;
}
inline cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *a, const void *p) {
    a->type = fake_locked(p) ? cudaMemoryTypeHost : cudaMemoryTypeUnregistered;
    return cudaSuccess;
}
inline cudaError_t cudaGetLastError() { return cudaSuccess; }
