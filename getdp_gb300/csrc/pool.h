// Device memory of the library: a context's pool of scratch memory and the
// allocation that every device buffer goes through.  Host code only.
#pragma once

#include <cuda_runtime_api.h>

#include <cstddef>
#include <mutex>

namespace gb {

// One context's stream-ordered pool (pool null: cudaMalloc).  It belongs to one
// stream: a block is handed out again in that stream's order only.
struct MemPool {
  int device = 0;
  cudaStream_t stream = nullptr;
  cudaMemPool_t pool = nullptr;
};

// memory a pool holds on to (in use or free): several systems of 2.7 M unknowns
// and 229 M entries (2.8 GB each, 4.8 GB of scratch in a solve), a ninth of the
// device; at 8 GB a solve beside two other such systems mapped its scratch anew,
// 14 ms each time
constexpr unsigned long long kPoolKeep = 32ull << 30;

void pool_open(MemPool *m, int device, cudaStream_t stream);
// (what was taken from it stays valid until it is freed)
void pool_close(MemPool *m);

// the pool that device_alloc takes from on this thread (null: cudaMalloc)
extern thread_local MemPool *t_pool;

// Memory from t_pool or by cudaMalloc; *from: the stream it is freed on (null:
// cudaFree).  Where the device has none left, what the pools of all contexts
// on it hold in free blocks is given back first.
cudaError_t device_alloc(void **p, size_t bytes, cudaStream_t *from);
cudaError_t device_malloc(void **p, size_t bytes);  // by cudaMalloc, whatever t_pool

// Held from the begin to the end of a stream capture: giving back memory
// synchronises the streams of all contexts, which would break a capture on one
// of them.
std::unique_lock<std::mutex> hold_capture();

}  // namespace gb
