// The sort of the SpGEMM, top-k and LSH kernels: a bitonic network over 32-bit
// keys in registers, R to a lane, blocked (lane L holds sorted positions L*R ..
// L*R+R-1), and its extension over the W warps of a block.
//
// How the products of a SpGEMM use it: for a cluster whose products (pairs of a
// cluster column j and an entry k of B's row j) number P <= 32*R*W, every
// product t (flat (j, k) order: the cluster's columns in order, each B row in
// storage order) becomes one key (output column << tbits | t).  Sorted, a
// column's products are adjacent and in flat order, so their sums depend only
// on the matrices, and the number of distinct columns, their min and max come
// from the same keys, which settles the reference's dense/hash classification
// (src/spgemm_Vlength_mixed.cpp:267-319) and its drop rule without a symbolic
// pass.  B's column count has to fit the key: cols < 2^(32 - tbits), tbits =
// log2(32*R*W), or equal with P < 32*R*W.
#pragma once

#include <cstdint>

namespace spops {
namespace {

// Ascending bitonic sort of 32*R keys, blocked: element e = lane*R + s.
// Stages are instantiated by template recursion so that every partner slot
// index is a compile-time constant and the keys stay in registers.
template <int R, int KK, int JJ>
__device__ __forceinline__ void bitonic_stage(uint32_t (&k)[R], int lane) {
  constexpr int N = 32 * R;
  if constexpr (JJ >= R) {  // partner: lane ^ (JJ / R), same slot
    constexpr int lm = JJ / R;
    const bool lower = (lane & lm) == 0;
    const bool asc = (KK >= N) ? true : ((lane & (KK / R)) == 0);
    const bool keep_min = lower == asc;
#pragma unroll
    for (int s = 0; s < R; ++s) {
      const uint32_t o = __shfl_xor_sync(0xffffffffu, k[s], lm);
      k[s] = keep_min ? min(k[s], o) : max(k[s], o);
    }
  } else {  // partner: slot s ^ JJ of the same lane
    const bool lane_asc = (KK >= N) ? true : ((lane & (KK / R)) == 0);
#pragma unroll
    for (int s = 0; s < R; ++s) {
      const int p = s ^ JJ;
      if (p > s) {
        const bool asc = KK < R ? (s & KK) == 0 : lane_asc;
        const uint32_t a = k[s], b = k[p];
        const uint32_t lo = min(a, b), hi = max(a, b);
        k[s] = asc ? lo : hi;
        k[p] = asc ? hi : lo;
      }
    }
  }
  if constexpr (JJ > 1) bitonic_stage<R, KK, JJ / 2>(k, lane);
}

template <int R, int KK>
__device__ __forceinline__ void bitonic_pass(uint32_t (&k)[R], int lane) {
  bitonic_stage<R, KK, KK / 2>(k, lane);
  if constexpr (KK < 32 * R) bitonic_pass<R, KK * 2>(k, lane);
}

// One warp's bitonic sort of its 32*R keys, R <= 16 (larger sorts run on
// several warps, block_sort_keys).
template <int R>
__device__ __forceinline__ void warp_bitonic_sort(uint32_t (&k)[R], int lane) {
  static_assert(R >= 1 && R <= 16 && (R & (R - 1)) == 0, "R: a power of two up to 16");
  bitonic_pass<R, 2>(k, lane);
}

// Bitonic merge of a bitonic sequence of one warp's 32R keys (blocked), in
// the direction asc: stages JJ = 16R .. 1.
template <int R, int JJ>
__device__ __forceinline__ void warp_merge_stage(uint32_t (&k)[R], int lane, bool asc) {
  if constexpr (JJ >= R) {  // partner: lane ^ (JJ / R), same slot
    constexpr int lm = JJ / R;
    const bool keep_min = ((lane & lm) == 0) == asc;
#pragma unroll
    for (int s = 0; s < R; ++s) {
      const uint32_t o = __shfl_xor_sync(0xffffffffu, k[s], lm);
      k[s] = keep_min ? min(k[s], o) : max(k[s], o);
    }
  } else {  // partner: slot s ^ JJ of the same lane
#pragma unroll
    for (int s = 0; s < R; ++s) {
      const int p = s ^ JJ;
      if (p > s) {
        const uint32_t a = k[s], b = k[p];
        const uint32_t lo = min(a, b), hi = max(a, b);
        k[s] = asc ? lo : hi;
        k[p] = asc ? hi : lo;
      }
    }
  }
  if constexpr (JJ > 1) warp_merge_stage<R, JJ / 2>(k, lane, asc);
}

// Ascending sort of a block's 32*R*W keys (W warps, R keys per lane), blocked:
// warp w, lane L, slot s then holds position w*32R + L*R + s.  Each warp sorts
// its 32R keys (descending for odd warps: the complements ascending), then the
// merge levels above run their cross-warp stages through xk (32*R*W keys of
// shared memory, which every warp is done reading after the first barrier).
template <int R, int W>
__device__ __forceinline__ void block_sort_keys(uint32_t (&key)[R], uint32_t* xk, int w, int lane) {
  if constexpr (W == 1) {
    warp_bitonic_sort<R>(key, lane);
    __syncwarp();
  } else {
    constexpr int NW = 32 * R, N = NW * W;
    const uint32_t flip = (w & 1) ? 0xffffffffu : 0u;
#pragma unroll
    for (int s = 0; s < R; ++s) key[s] ^= flip;
    warp_bitonic_sort<R>(key, lane);
#pragma unroll
    for (int s = 0; s < R; ++s) key[s] ^= flip;
    __syncthreads();  // every warp has its keys in registers
#pragma unroll 1
    for (int kk = 2 * NW; kk <= N; kk <<= 1) {
      const bool asc = kk >= N ? true : ((w & (kk / NW)) == 0);
#pragma unroll 1
      for (int jj = kk >> 1; jj >= NW; jj >>= 1) {  // partner: warp w ^ (jj / NW), same lane and slot
        const int pw = w ^ (jj / NW);
        const bool keep_min = ((w & (jj / NW)) == 0) == asc;
#pragma unroll
        for (int s = 0; s < R; ++s) xk[w * NW + s * 32 + lane] = key[s];
        __syncthreads();
#pragma unroll
        for (int s = 0; s < R; ++s) {
          const uint32_t o = xk[pw * NW + s * 32 + lane];
          key[s] = keep_min ? min(key[s], o) : max(key[s], o);
        }
        __syncthreads();
      }
      warp_merge_stage<R, NW / 2>(key, lane, asc);
    }
  }
}

}  // namespace
}  // namespace spops
