// Copies between the caller's (pageable) host arrays and the device.
#pragma once
#include <cuda_runtime.h>

#include <cstddef>

namespace rmx {

// Host to device on stream s. A pageable src may be reused when the call returns;
// a pinned one is read by the device until the stream has passed the copy. Large
// pageable arrays go through a pinned ring filled by several threads: the
// driver's own staging copies them on one (90 MB: 8.4 ms; with the endpoint
// check on eight threads too, creating a handle from 5.67 million weighted edges
// takes 7.0 ms instead of 14.5).
void upload(void *dst, const void *src, size_t bytes, cudaStream_t s);

// Device to host on stream s. Pages of a fresh array that have not been touched
// are first touched by up to 16 threads: faulted in one by one under the copy
// they took 11.6 of 15.6 ms for 68 MB, by 16 threads 2.1 ms (and 9.5 ms with
// MADV_POPULATE_WRITE, whose callers wait for one another). An array that the
// caller uses again has its pages: starting threads for it only cost time (15 MB
// 1.12 ms, 0.78 without, which a look at 16 of its pages does not change).
void download(void *dst, const void *src, size_t bytes, cudaStream_t s);

// Frees the pinned ring (it is allocated again when next needed).
void release_upload_ring();

}  // namespace rmx
