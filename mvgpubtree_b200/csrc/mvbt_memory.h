// Device memory of the library: two stream-ordered memory pools per device, one for the sort's scratch and one
// for trees, and plain allocations. Freed pool blocks stay cached for the next call, up to kPoolKeepBytes of
// each pool's live and cached blocks together; they are given back when the device is full (every
// allocation below then frees them and tries again) and by mvbt_release_memory.
// Two pools, because a pool that holds more than it may keep gives back every freed block at the next
// synchronisation: with 5.8 GB of trees in the scratch's pool each sorted call mapped its scratch anew
// (2^25 finds 13 ms instead of 2).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace mvbt_mem {

constexpr uint64_t kPoolKeepBytes = 4ull << 30;
enum pool_kind { kScratch = 0, kTrees = 1 };

// cudaMalloc on the current device.
cudaError_t alloc(void** out, uint64_t bytes);
template <class T>
cudaError_t alloc(T** out, uint64_t bytes) {
  return alloc(reinterpret_cast<void**>(out), bytes);
}

// From a pool of device dev, stream-ordered on s; freed with cudaFreeAsync.
cudaError_t pool_alloc(int dev, pool_kind which, void** out, uint64_t bytes, cudaStream_t s);

// Gives back what both pools of device dev keep and no work still uses.
cudaError_t release(int dev);

}  // namespace mvbt_mem
