// readback.cuh -- small results of a call on the host.
//
// Sizes, counts and the arena's error word are copied to a piece of pinned
// memory that the calling thread keeps, and the stream is waited for once: a
// copy to pageable memory waits by itself, about 10 us each, and most calls
// made two or three of them.
#pragma once

#include "internal.h"

namespace ms {

// The calling thread's pinned memory (kReadBackBytes; usable on every device;
// freed when the thread ends), or nullptr.
constexpr size_t kReadBackBytes = 192 * 1024;
void *readback_buffer();

// Error word -> status, clearing it (stream-ordered) when set.
int error_status(unsigned err, ms_arena *a, cudaStream_t st);

class ReadBack {
public:
    ReadBack(ms_arena *arena, cudaStream_t stream) : a(arena), st(stream), p(static_cast<uint8_t *>(readback_buffer())) {}
    // `count` values from device memory; the result is valid after wait()
    template <class T> const T *add(const T *dev, uint64_t count = 1) {
        const uint64_t bytes = align_up(count * sizeof(T), 16);
        if (!p || at + bytes > kReadBackBytes - 16) {
            rc = ms_fail(MS_ERR_NOMEM, "no pinned host memory for results");
            return nullptr;
        }
        T *const h = reinterpret_cast<T *>(p + at);
        at += bytes;
        const cudaError_t e = cudaMemcpyAsync(h, dev, count * sizeof(T), cudaMemcpyDeviceToHost, st);
        if (e != cudaSuccess) rc = ms_fail_cuda(e, "result copy");
        return h;
    }
    // the stream is drained and the arena's error word checked
    int wait() {
        const unsigned *err = add(a->d_err);
        if (rc) return rc;
        MS_CUDA_TRY(cudaStreamSynchronize(st));
        return error_status(*err, a, st);
    }
    // as wait(), without the error word (calls that look at it later)
    int wait_results() {
        if (rc) return rc;
        MS_CUDA_TRY(cudaStreamSynchronize(st));
        return MS_OK;
    }

private:
    ms_arena *a;
    cudaStream_t st;
    uint8_t *p;
    uint64_t at = 0;
    int rc = MS_OK;
};

}  // namespace ms
