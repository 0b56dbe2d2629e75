/*
 * host_stage.h — host buffers in and out of the device for the host-pointer
 * entry points.
 *
 * The engine's buffers are plain malloc memory.  Given such a pointer the
 * runtime copies through a staging area of its own, on the calling thread and
 * one piece at a time: 8192 tokens (33.5 MB each way) took 3.4 ms beside a
 * 1.9 ms block.  Here the CPU side of the copy runs on several threads and is
 * overlapped with the DMA of the piece before it, in a ring of page-locked
 * slots that is allocated once and kept (2 x 4 x 1 MiB; no call can grow it).
 * Buffers that are page-locked already are handed to the DMA engine as they are.
 */
#pragma once
#include <cuda_runtime.h>
#include <omp.h>

#include <cstddef>
#include <cstring>

namespace apus {

/* below this a single thread's memcpy is faster than waking others */
constexpr size_t HS_PARALLEL_MIN = 256u << 10;

inline void host_copy(void *dst, const void *src, size_t n) {
    int nt = omp_get_num_procs() / 2;
    if (nt > 8) nt = 8;
    if (n < HS_PARALLEL_MIN || nt < 2) {
        memcpy(dst, src, n);
        return;
    }
    const size_t piece = ((n + (size_t)nt - 1) / (size_t)nt + 4095) & ~(size_t)4095;
#pragma omp parallel for num_threads(nt) schedule(static, 1)
    for (int i = 0; i < nt; i++) {
        const size_t lo = (size_t)i * piece;
        if (lo < n)
            memcpy((char *)dst + lo, (const char *)src + lo, n - lo < piece ? n - lo : piece);
    }
}

struct HostStage {
    static constexpr int SLOTS = 4;
    static constexpr size_t SLOT_BYTES = 1u << 20;
    char *in = nullptr, *out = nullptr;      /* [SLOTS][SLOT_BYTES], page-locked */
    char *out_dev = nullptr;                 /* the same memory as the GPU addresses it */
    cudaEvent_t ein[SLOTS] = {}, eout[SLOTS] = {};
    unsigned n_in = 0;                       /* slots handed to uploads so far */
    bool out_busy[SLOTS] = {};               /* a copy into the slot may be under way */

    cudaError_t init() {
        if (in) return cudaSuccess;
        cudaError_t e = cudaHostAlloc((void **)&in, SLOTS * SLOT_BYTES, cudaHostAllocDefault);
        if (e == cudaSuccess)
            e = cudaHostAlloc((void **)&out, SLOTS * SLOT_BYTES, cudaHostAllocMapped);
        if (e == cudaSuccess) e = cudaHostGetDevicePointer((void **)&out_dev, out, 0);
        for (int i = 0; e == cudaSuccess && i < SLOTS; i++) {
            e = cudaEventCreateWithFlags(&ein[i], cudaEventDisableTiming);
            if (e == cudaSuccess) e = cudaEventCreateWithFlags(&eout[i], cudaEventDisableTiming);
        }
        if (e != cudaSuccess) release();
        return e;
    }
    void release() {
        if (in) cudaFreeHost(in);
        if (out) cudaFreeHost(out);
        for (int i = 0; i < SLOTS; i++) {
            if (ein[i]) cudaEventDestroy(ein[i]);
            if (eout[i]) cudaEventDestroy(eout[i]);
            ein[i] = eout[i] = nullptr;
            out_busy[i] = false;
        }
        in = out = out_dev = nullptr;
        n_in = 0;
    }
    static bool page_locked(const void *p) {
        cudaPointerAttributes at;
        if (cudaPointerGetAttributes(&at, p) != cudaSuccess) {
            cudaGetLastError();
            return false;
        }
        return at.type == cudaMemoryTypeHost;
    }
    /* pieces small enough that the ring overlaps, large enough to amortise */
    static size_t piece_of(size_t bytes) {
        size_t p = (bytes / 4 + 65535) & ~(size_t)65535;
        if (p < (512u << 10)) p = 512u << 10;
        return p < SLOT_BYTES ? p : SLOT_BYTES;
    }
    /* Enqueues host -> device on st; src may be reused as soon as this returns
     * unless it is page-locked. */
    cudaError_t upload(void *dst, const void *src, size_t bytes, cudaStream_t st) {
        if (bytes > SLOT_BYTES / 16 && page_locked(src))
            return cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, st);
        cudaError_t e = init();
        if (e != cudaSuccess) return e;
        const size_t piece = piece_of(bytes);
        for (size_t at = 0; at < bytes; at += piece) {
            const size_t n = bytes - at < piece ? bytes - at : piece;
            const int s = (int)(n_in % SLOTS);
            if (n_in >= SLOTS && (e = cudaEventSynchronize(ein[s])) != cudaSuccess) return e;
            char *slot = in + (size_t)s * SLOT_BYTES;
            host_copy(slot, (const char *)src + at, n);
            e = cudaMemcpyAsync((char *)dst + at, slot, n, cudaMemcpyHostToDevice, st);
            if (e == cudaSuccess) e = cudaEventRecord(ein[s], st);
            if (e != cudaSuccess) return e;
            n_in++;
        }
        return cudaSuccess;
    }
    /* The two halves of a download of at most SLOT_BYTES into pageable memory, for
     * callers with more to enqueue in between; one at a time per slot.  A slot that an
     * abandoned call left with a copy under way (on whatever stream) is waited for. */
    cudaError_t download_begin(int slot, const void *src, size_t bytes, cudaStream_t st) {
        cudaError_t e = init();
        if (e == cudaSuccess && out_busy[slot]) e = out_wait(slot);
        if (e != cudaSuccess) return e;
        e = cudaMemcpyAsync(out + (size_t)slot * SLOT_BYTES, src, bytes, cudaMemcpyDeviceToHost,
                            st);
        if (e != cudaSuccess) return e;
        out_busy[slot] = true;
        return cudaEventRecord(eout[slot], st);
    }
    cudaError_t out_wait(int slot) {
        const cudaError_t e = cudaEventSynchronize(eout[slot]);
        if (e == cudaSuccess) out_busy[slot] = false;
        return e;
    }
    cudaError_t download_end(int slot, void *dst, size_t bytes) {
        const cudaError_t e = out_wait(slot);
        if (e == cudaSuccess) host_copy(dst, out + (size_t)slot * SLOT_BYTES, bytes);
        return e;
    }
    /* Device -> host behind what st holds.  Pageable dst: complete on return.
     * Page-locked dst: enqueued only. */
    cudaError_t download(void *dst, const void *src, size_t bytes, cudaStream_t st) {
        if (bytes > SLOT_BYTES / 16 && page_locked(dst))
            return cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, st);
        cudaError_t e = init();
        if (e != cudaSuccess) return e;
        const size_t piece = piece_of(bytes), count = (bytes + piece - 1) / piece;
        auto len = [&](size_t i) { return i + 1 < count ? piece : bytes - i * piece; };
        auto issue = [&](size_t i) {
            return download_begin((int)(i % SLOTS), (const char *)src + i * piece, len(i), st);
        };
        for (size_t i = 0; i < count && i < SLOTS; i++)
            if ((e = issue(i)) != cudaSuccess) return e;
        for (size_t i = 0; i < count; i++) {
            e = download_end((int)(i % SLOTS), (char *)dst + i * piece, len(i));
            if (e == cudaSuccess && i + SLOTS < count) e = issue(i + SLOTS);
            if (e != cudaSuccess) return e;
        }
        return cudaSuccess;
    }
};

}  // namespace apus
