// Device memory of graphs and of the temporaries of their uploads.
#pragma once
#include <cuda_runtime.h>

#include <cstddef>

namespace gat {

// Stream-ordered allocation on the current device from the library's own
// memory pool.  The memory is usable on `st` at once and on other streams
// after `st` has been synchronised.
cudaError_t dev_alloc(void **p, size_t bytes, cudaStream_t st);
// Gives back memory of dev_alloc on any device (null is allowed): at once in
// `st`'s order, or, without a stream, when no work that uses it is pending
// (every call that reads a graph returns after its work is done).
cudaError_t dev_free(void *p, cudaStream_t st);
void dev_free(void *p);

// cudaMalloc, once more after the pools' unused pages are given back if the
// device has no room (scratch that an executor keeps).
cudaError_t plain_alloc(void **p, size_t bytes);

// Counts the library's live handles (graphs, executors, batches).  The
// pools keep up to kPoolKeepBytes for the next graph while there is one, and
// give everything back when the last is freed.
constexpr size_t kPoolKeepBytes = size_t(2) << 30;
struct PoolUser {
    PoolUser();
    ~PoolUser();
    PoolUser(const PoolUser &) = delete;
    PoolUser &operator=(const PoolUser &) = delete;
};

}  // namespace gat
