// device_pool.h -- device memory blocks kept for the next call that needs one
// of their size.

#ifndef SNOG_DEVICE_POOL_H
#define SNOG_DEVICE_POOL_H

#include <cuda_runtime.h>

#include <cstddef>

namespace snog {

// A block of at least N bytes on the current device, from the kept ones or
// by cudaMalloc; throws Error (SNOG_ENOMEM, SNOG_ECUDA).
//
// A cudaMalloc or cudaFree takes from a tenth of a millisecond to several, and
// a scene's creation made fifty of each, a ray batch from host memory five
// (200k triangles created, traced and destroyed 29 -> 10.6 ms with kept blocks,
// 300k rays from host memory 3.8 -> 1.2 ms).  Blocks are kept up to kPoolKeep
// bytes, counted over all devices together, and handed out again within a quarter
// of the size asked for; where they are full, those not asked for in a long time
// (kStale) are freed for the next.
constexpr size_t kPoolKeep = size_t(256) << 20;
void *pool_get(size_t n);

// The size of a block for N bytes: N rounded up to an eighth of its power of two,
// at least 4096.
size_t size_class(size_t n);

// Give a block back.  No work that uses it may be running: unlike cudaFree,
// this does not wait for the device.
void pool_put(void *p);

// Free a block of the pool, which waits for the device: for blocks that work may
// still use, because a wait for it failed or was not made.
void pool_free(void *p);

// Free every kept block.
void pool_trim();

// cudaMalloc for what does not come from the pool: where the device is full, the
// kept blocks are freed and it is tried again.
cudaError_t device_malloc(void **p, size_t n);

}  // namespace snog

#endif
