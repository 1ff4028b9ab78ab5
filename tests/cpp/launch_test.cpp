// The launch helpers against a fake CUDA runtime: blocks_per_sm
// (csrc/launch_util.h) raises the shared memory attribute once on every device
// that launches the kernel; an OverlapChain (csrc/pdl.cuh) begins with a plain
// launch, and every launch passes its arguments on.
#include <device_launch_parameters.h>

#include <cstdint>
#include <cstdio>
#include <map>
#include <vector>

#include "launch_util.h"
#include "pdl.cuh"

namespace {
int device = 0;
bool refuse = false;
std::map<int, int> limit;  // device -> dynamic shared memory allowed
std::map<int, int> raised;
struct Launch {
  bool overlapped;
  unsigned grid, block;
  size_t smem;
  cudaStream_t st;
  int64_t a;
  const double* b;
};
std::vector<Launch> launches;
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

extern "C" cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void*, void** args) {
  bool overlapped = false;
  for (unsigned i = 0; i < c->numAttrs; ++i)
    overlapped |= c->attrs[i].id == cudaLaunchAttributeProgrammaticStreamSerialization &&
                  c->attrs[i].val.programmaticStreamSerializationAllowed;
  launches.push_back({overlapped, c->gridDim.x, c->blockDim.x, c->dynamicSmemBytes, c->stream,
                      *static_cast<int64_t*>(args[0]), *static_cast<const double**>(args[1])});
  return cudaSuccess;
}

void kernel(int) {}
void pair_kernel(int64_t, const double*) {}

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
  const cudaStream_t st = reinterpret_cast<cudaStream_t>(0x40);
  double x = 0;
  for (int chain = 0; chain < 2; ++chain) {
    spops::OverlapChain c(st);
    for (int q = 0; q < 3; ++q) c.launch(pair_kernel, 10 + q, 64, 128 * q, q, &x);
  }
  spops::launch_overlapped(pair_kernel, 9, 32, 0, st, 3, &x);
  check(launches.size() == 7, "every launch reached the runtime");
  for (int q = 0; q < 6; ++q) {
    const Launch& l = launches[q];
    check(l.overlapped == (q % 3 != 0), "a chain's first launch is plain, the later ones overlap");
    check(l.grid == 10u + q % 3 && l.block == 64 && l.smem == 128u * (q % 3) && l.st == st && l.a == q % 3 && l.b == &x,
          "launch shape and arguments");
  }
  check(launches[6].overlapped && launches[6].a == 3, "a waiting kernel's launch overlaps");
  std::printf("launch failures %d\n", bad);
  return bad != 0;
}
