// Device memory of the library (see pool.h).
#include "pool.h"

#include <algorithm>
#include <vector>

namespace gb {

thread_local MemPool *t_pool = nullptr;

static std::mutex g_pools_mutex, g_capture_mutex;
static std::vector<MemPool *> g_pools;  // of the live contexts

std::unique_lock<std::mutex> hold_capture()
{
  return std::unique_lock<std::mutex>(g_capture_mutex);
}

void pool_open(MemPool *m, int device, cudaStream_t stream)
{
  m->device = device;
  m->stream = stream;
  cudaMemPoolProps props = {};
  props.allocType = cudaMemAllocationTypePinned;
  props.location.type = cudaMemLocationTypeDevice;
  props.location.id = device;
  unsigned long long keep = kPoolKeep;
  if(cudaMemPoolCreate(&m->pool, &props) != cudaSuccess) {
    cudaGetLastError();  // no pool: cudaMalloc instead
    m->pool = nullptr;
    return;
  }
  if(cudaMemPoolSetAttribute(m->pool, cudaMemPoolAttrReleaseThreshold, &keep) != cudaSuccess) {
    cudaGetLastError();
    cudaMemPoolDestroy(m->pool);
    m->pool = nullptr;
    return;
  }
  std::lock_guard<std::mutex> lock(g_pools_mutex);
  g_pools.push_back(m);
}

void pool_close(MemPool *m)
{
  {
    std::lock_guard<std::mutex> lock(g_pools_mutex);
    g_pools.erase(std::remove(g_pools.begin(), g_pools.end(), m), g_pools.end());
  }
  if(m->pool) cudaMemPoolDestroy(m->pool);
  m->pool = nullptr;
}

// the free blocks of all pools on the current device go back to it (a block
// counts as free once its stream has been synchronised after the free)
static void give_back()
{
  int device = 0;
  if(cudaGetDevice(&device) != cudaSuccess) cudaGetLastError();
  const auto no_capture = hold_capture();
  std::lock_guard<std::mutex> lock(g_pools_mutex);
  for(MemPool *m : g_pools)
    if(m->device == device && (cudaStreamSynchronize(m->stream) != cudaSuccess ||
                               cudaMemPoolTrimTo(m->pool, 0) != cudaSuccess))
      cudaGetLastError();
}

// try_alloc, and once more after give_back; a failure leaves no error behind for
// the next call to find
template <typename F> static cudaError_t with_retry(F try_alloc)
{
  cudaError_t e = try_alloc();
  if(e == cudaErrorMemoryAllocation) {
    cudaGetLastError();
    give_back();
    e = try_alloc();
  }
  if(e != cudaSuccess) cudaGetLastError();
  return e;
}

cudaError_t device_malloc(void **p, size_t bytes)
{
  return with_retry([&]() { return cudaMalloc(p, bytes); });
}

cudaError_t device_alloc(void **p, size_t bytes, cudaStream_t *from)
{
  const MemPool *m = t_pool;
  *from = nullptr;
  if(!m || !m->pool) return device_malloc(p, bytes);
  const cudaError_t e =
    with_retry([&]() { return cudaMallocFromPoolAsync(p, bytes, m->pool, m->stream); });
  if(e == cudaSuccess) *from = m->stream;
  return e;
}

}  // namespace gb
