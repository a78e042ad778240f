/*
 * eg_pool.cuh -- what solves keep between calls instead of making it each
 * time: device memory, streams with their events, pinned staging buffers.
 *
 * A one-call solve of a small game spent 0.8 of 0.9 ms in cudaMalloc, cudaFree
 * and the creation of its stream and events.  All of it is bounded, shared by
 * threads under a lock, and holds nothing of any game: device memory comes
 * from one stream-ordered pool per device that returns what is beyond
 * kPoolKeep to the system at the next synchronisation (and everything when an
 * allocation fails), idle streams and staging buffers are kept up to a count.
 */
#ifndef EG_POOL_CUH
#define EG_POOL_CUH

#include <cuda_runtime.h>

#include <functional>

#include "eg_internal.h"

namespace eg {

/* Device memory for work on `st` (stream-ordered: free of it on any stream
 * that has waited for its last use). */
cudaError_t pool_alloc(void **p, size_t bytes, int device, cudaStream_t st);
void pool_free(void *p, cudaStream_t st);
/* Bytes that the device's pool holds and nobody uses: free memory that
 * cudaMemGetInfo does not count. */
size_t pool_idle(int device);

/* A stream with timing events and some pinned memory. */
struct Lane {
    int device;
    cudaStream_t st;
    cudaEvent_t ev[6];
    void *page; /* kLanePage bytes, pinned */
};
constexpr size_t kLanePage = 64 << 10;
/* An idle lane of the current device, or a new one; NULL on failure. */
Lane *lane_take(int device);
/* Gives it back; its stream must hold no more than stream-ordered frees. */
void lane_give(Lane *l);

/* Copies between host memory and the device.  Pageable memory goes through
 * pinned staging buffers, large copies by several threads at once (the
 * driver's own staging moved 4 GB/s into memory that was not yet mapped).  To
 * the host: returns when the data are there; to the device: when the host
 * memory may be reused, the copy itself ordered on `st`. */
struct CopyItem {
    void *host, *dev;
    size_t bytes;
};
cudaError_t copy_list(const CopyItem *items, int count, bool to_host, int device, cudaStream_t st);
cudaError_t copy_to_host(void *dst, const void *dev, size_t bytes, int device, cudaStream_t st);
cudaError_t copy_to_device(void *dev, const void *src, size_t bytes, int device, cudaStream_t st);
struct CopyPart {
    const void *src;
    size_t at, bytes;
};
/* Several host arrays to places in one device block (`total`: its end); small
 * ones together in one copy. */
cudaError_t copy_parts_to_device(void *dev, const CopyPart *parts, int count, size_t total, int device, cudaStream_t st);
/* A device block of at most kStageBlock bytes in one copy after what `st`
 * holds; `look` sees it in the staging buffer. */
constexpr size_t kStageBlock = 512 << 10;
cudaError_t copy_block_to_host(const void *dev, size_t bytes, int device, cudaStream_t st,
                               const std::function<void(const char *)> &look);

}  // namespace eg

#endif
