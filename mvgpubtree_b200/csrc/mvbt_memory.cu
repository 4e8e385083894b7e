// Device memory of the library (mvbt_memory.h).
#include "mvbt_memory.h"

#include <mutex>

namespace {

constexpr int kMaxDevices = 64;
cudaMemPool_t g_pools[2][kMaxDevices] = {};
std::mutex g_pools_mu;

// The pool, made on first use; null: there is none (make false, or an error in *err).
cudaMemPool_t pool_of(int dev, int which, bool make, cudaError_t* err = nullptr) {
  if (dev < 0 || dev >= kMaxDevices) {
    if (err) *err = cudaErrorInvalidDevice;
    return nullptr;
  }
  std::lock_guard<std::mutex> lk(g_pools_mu);
  if (g_pools[which][dev] || !make) return g_pools[which][dev];
  cudaMemPoolProps props = {};
  props.allocType        = cudaMemAllocationTypePinned;
  props.location.type    = cudaMemLocationTypeDevice;
  props.location.id      = dev;
  cudaMemPool_t pool     = nullptr;
  cudaError_t e          = cudaMemPoolCreate(&pool, &props);
  uint64_t keep          = mvbt_mem::kPoolKeepBytes;
  if (e == cudaSuccess) e = cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
  if (e != cudaSuccess) {
    if (pool) cudaMemPoolDestroy(pool);
    if (err) *err = e;
    return nullptr;
  }
  return g_pools[which][dev] = pool;
}

}  // namespace

namespace mvbt_mem {

cudaError_t release(int dev) {
  for (int which = 0; which < 2; ++which)
    if (cudaMemPool_t pool = pool_of(dev, which, false)) {
      const cudaError_t e = cudaMemPoolTrimTo(pool, 0);
      if (e != cudaSuccess) return e;
    }
  return cudaSuccess;
}

cudaError_t alloc(void** out, uint64_t bytes) {
  cudaError_t e = cudaMalloc(out, bytes);
  if (e != cudaErrorMemoryAllocation) return e;
  cudaGetLastError();
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || release(dev) != cudaSuccess) return e;
  e = cudaMalloc(out, bytes);
  if (e != cudaSuccess) cudaGetLastError();
  return e;
}

cudaError_t pool_alloc(int dev, pool_kind which, void** out, uint64_t bytes, cudaStream_t s) {
  cudaError_t e            = cudaSuccess;
  const cudaMemPool_t pool = pool_of(dev, which, true, &e);
  if (!pool) return e;
  e = cudaMallocFromPoolAsync(out, bytes, pool, s);
  if (e != cudaErrorMemoryAllocation) return e;
  cudaGetLastError();
  if (release(dev) != cudaSuccess) return e;
  e = cudaMallocFromPoolAsync(out, bytes, pool, s);
  if (e != cudaSuccess) cudaGetLastError();
  return e;
}

}  // namespace mvbt_mem
