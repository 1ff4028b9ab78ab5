// blocks_per_sm (csrc/launch_util.h) against a fake CUDA runtime: the shared
// memory attribute is raised once on every device that launches the kernel.
#include <cstdio>
#include <map>

#include "launch_util.h"

namespace {
int device = 0;
bool refuse = false;
std::map<int, int> limit;  // device -> dynamic shared memory allowed
std::map<int, int> raised;
}  // namespace

extern "C" cudaError_t cudaGetDevice(int* d) {
  *d = device;
  return cudaSuccess;
}
extern "C" cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute a, int v) {
  if (refuse || a != cudaFuncAttributeMaxDynamicSharedMemorySize) return cudaErrorInvalidValue;
  limit[device] = v;
  ++raised[device];
  return cudaSuccess;
}
extern "C" cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int* n, const void*, int, size_t smem) {
  if ((int)smem > 48 * 1024 && limit[device] < (int)smem) return cudaErrorInvalidValue;
  *n = 2 + device;
  return cudaSuccess;
}

void kernel(int) {}

int bad = 0;
void check(bool ok, const char* what) {
  if (!ok) {
    std::printf("FAILED: %s\n", what);
    ++bad;
  }
}

int main() {
  static std::atomic<int> cache[spops::kMaxDevices];
  const size_t smem = 51200;
  for (int turn = 0; turn < 2; ++turn)
    for (int d : {0, 1, 7, 63, 64, 70}) {
      device = d;
      check(spops::blocks_per_sm(kernel, 256, smem, cache) == 2 + d, "occupancy of the current device");
      check(limit[d] == (int)smem, "attribute set on the current device");
      if (d < spops::kMaxDevices) check(raised[d] == 1, "set once per device");
    }
  static std::atomic<int> other[spops::kMaxDevices];
  device = 3;
  refuse = true;
  check(spops::blocks_per_sm(kernel, 256, smem, other) == 0, "a refused attribute is reported");
  refuse = false;
  check(spops::blocks_per_sm(kernel, 256, smem, other) == 5, "and tried again by the next call");
  check(spops::blocks_per_sm(kernel, 256, 0, other) == 5, "no shared memory: no attribute");
  std::printf("launch failures %d\n", bad);
  return bad != 0;
}
