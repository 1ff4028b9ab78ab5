// Resident blocks per SM of a kernel, with the launch attribute that its
// dynamic shared memory needs.
#pragma once

#include <cuda_runtime.h>

#include <atomic>
#include <cstddef>

namespace spops {

constexpr int kMaxDevices = 64;

// Resident blocks per SM (at least 1) of `kern` with `smem` bytes of dynamic
// shared memory on the current device, 0 when the attribute cannot be set.
// The attribute belongs to the function on one device, so `cache` (static, one
// per kernel instantiation) holds an entry per device; threads that meet here
// write the same value.
template <typename K>
int blocks_per_sm(K* kern, int threads, size_t smem, std::atomic<int> (&cache)[kMaxDevices]) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 0;
  const bool known = dev >= 0 && dev < kMaxDevices;
  int bps = known ? cache[dev].load(std::memory_order_relaxed) : 0;
  if (bps > 0) return bps;
  const void* f = reinterpret_cast<const void*>(kern);
  if (smem && cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) return 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, f, threads, smem) != cudaSuccess || bps < 1) bps = 1;
  if (known) cache[dev].store(bps, std::memory_order_relaxed);
  return bps;
}

}  // namespace spops
