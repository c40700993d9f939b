// Device blocks, streams and pinned words that outlive one solve.
//
// A solve of a small model takes a few milliseconds; cudaMalloc, cudaFree,
// cudaHostAlloc and stream creation cost up to a millisecond each on a busy
// host, and a call needs about twenty of them.  Objects go back to the pool
// when a solve ends and the next one on the same device takes them.  The pool
// is bounded (kPoolBytes of device memory a device, kPoolObjects of the
// rest); what does not fit is freed, and all of it is freed when an
// allocation fails or the caller asks (hprqp_b200_release_memory).  All functions work on the current device, may be called
// from any thread, and drop what belongs to a context that no longer exists.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>

namespace hpr {

constexpr size_t kPoolBytes = size_t(512) << 20;
constexpr size_t kPoolObjects = 16;
constexpr size_t kPinnedBytes = 1024;

// device memory, not cleared; nullptr when there is none.  Work on a block
// must have ended before it is returned.
void *pool_alloc(size_t bytes);
void pool_free(void *p);

// a non-blocking stream; idle when it is returned
cudaStream_t pool_stream();
void pool_stream_return(cudaStream_t s);

// kPinnedBytes of mapped pinned memory, cleared (host address; *dev: the
// device's)
void *pool_pinned(void **dev);
void pool_pinned_return(void *host);

// free what the pool keeps on a device (objects in use are not the pool's);
// false when the device cannot be reached
bool pool_release(int device);

// identity of the current context; false when there is none (context_id.cpp)
bool current_context_id(unsigned long long *id);

}  // namespace hpr
