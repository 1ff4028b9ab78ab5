// Launches that overlap with the end of the kernel before them (programmatic
// dependent launch): the next kernel's blocks are set up while this one still
// runs, and wait on the device instead of in the queue (about 2 us of gap
// between two dependent kernels becomes about 0.5 us).
//
// A kernel launched with launch_overlapped begins with overlap_begin() in
// every thread, before it reads or writes anything: it lets the launch after
// it begin the same way and waits until the kernel before it has ended, with
// its writes visible.  Launched plainly, the call does nothing; and a plain
// launch after such a kernel waits for its end as always.  What may be read
// before the wait is a handle's plan and pattern alone: they were complete
// when the plan's analysis returned and do not change while it is in use.
// Everything else is read after it, by plain loads (ld_gather, or a pointer that
// is not const __restrict__).
#pragma once

#include <cuda_runtime.h>

namespace spops {
namespace {

__device__ __forceinline__ void overlap_let_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void overlap_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// For the kernels of an OverlapChain, which share nothing with one another:
// they call overlap_let_next() first, and at their end overlap_end(), where the
// grid's last block alone waits (a block that waited would keep its place on the
// SM), so that the grid does not end before the one before it.
__device__ __forceinline__ void overlap_end() {
  if (blockIdx.x + 1 == gridDim.x) overlap_wait();
}
__device__ __forceinline__ void overlap_begin() {
  overlap_let_next();
  overlap_wait();
}

template <typename... P>
cudaError_t launch_packed(const cudaLaunchConfig_t* cfg, const void* kern, P... args) {
  void* list[] = {(void*)&args...};
  return cudaLaunchKernelExC(cfg, kern, list);
}

template <typename... P, typename... A>
cudaError_t launch_with(int overlapped, void (*kern)(P...), int64_t grid, int block, size_t smem, cudaStream_t st,
                        A... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3((unsigned)block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = overlapped ? 1 : 0;
  return launch_packed(&cfg, reinterpret_cast<const void*>(kern), static_cast<P>(args)...);
}

template <typename... P, typename... A>
cudaError_t launch_overlapped(void (*kern)(P...), int64_t grid, int block, size_t smem, cudaStream_t st, A... args) {
  return launch_with(1, kern, grid, block, smem, st, args...);
}

// Launches that share nothing with one another and do not wait.  The first is
// a plain one: it begins when all work queued before it has ended, with its
// writes visible (the fills and copies of what the kernels read or add to), and
// since the later ones begin after it has, the same holds for them.
struct OverlapChain {
  cudaStream_t st;
  bool begun = false;
  explicit OverlapChain(cudaStream_t s) : st(s) {}
  template <typename... P, typename... A>
  cudaError_t launch(void (*kern)(P...), int64_t grid, int block, size_t smem, A... args) {
    const int overlapped = begun ? 1 : 0;
    begun = true;
    return launch_with(overlapped, kern, grid, block, smem, st, args...);
  }
};

}  // namespace
}  // namespace spops
