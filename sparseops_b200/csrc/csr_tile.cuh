// CSR tiles of 32 lanes x K consecutive entries: the helpers shared by the
// tile SpMV / SpMM kernels (spmv_csr_tile.cu) and the batch's tile items
// (batched.cu).  See spmv_csr_tile.cu for the plan (flags, tile_row, empty
// rows) and the calibration of rows that cross tiles.
#pragma once

#include <cstdint>
#include <cstring>
#include <type_traits>

#include "device_util.cuh"

namespace spops {
namespace {

// last r in [0, n-1] with rp[r] <= e (the non-empty row holding entry e)
template <typename I>
__device__ __forceinline__ int64_t row_holding(const I* rp, int64_t n, int64_t e) {
  int64_t lo = 0, hi = n;
  while (hi - lo > 1) {
    const int64_t mid = (lo + hi) >> 1;
    if ((int64_t)rp[mid] <= e) lo = mid; else hi = mid;
  }
  return lo;
}

// ---- vector loads of one lane's run (32-byte aligned for 32-byte runs).
// kFixed: of the pattern, which nothing writes while a plan is in use; else plain
// loads, as for ld_gather (a launch before this one may have written the values)
template <int BYTES, bool kFixed>
struct RunLoad;
template <bool kFixed>
struct RunLoad<16, kFixed> {
  static __device__ __forceinline__ void ld(const void* p, uint32_t (&w)[4]) {
    if constexpr (kFixed)
      asm volatile("ld.global.nc.L1::no_allocate.v4.b32 {%0,%1,%2,%3}, [%4];"
                   : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3])
                   : "l"(p));
    else
      asm volatile("ld.global.L1::no_allocate.v4.b32 {%0,%1,%2,%3}, [%4];"
                   : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3])
                   : "l"(p));
  }
};
template <bool kFixed>
struct RunLoad<32, kFixed> {
  static __device__ __forceinline__ void ld(const void* p, uint32_t (&w)[8]) {
    if constexpr (kFixed)
      asm volatile("ld.global.nc.L1::no_allocate.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                   : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]), "=r"(w[4]), "=r"(w[5]), "=r"(w[6]), "=r"(w[7])
                   : "l"(p));
    else
      asm volatile("ld.global.L1::no_allocate.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                   : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]), "=r"(w[4]), "=r"(w[5]), "=r"(w[6]), "=r"(w[7])
                   : "l"(p));
  }
};

// K elements of T from p (aligned to min(32, K*sizeof(T)) bytes) into out:
// indices are the pattern's (or a plan's), floating values are not.
template <typename T, int K>
__device__ __forceinline__ void load_run(const T* __restrict__ p, T (&out)[K]) {
  constexpr int BYTES = K * (int)sizeof(T);
  constexpr bool kFixed = !std::is_floating_point<T>::value;
  static_assert(BYTES == 16 || BYTES % 32 == 0, "run must be 16 bytes or a multiple of 32");
  if constexpr (BYTES == 16) {
    uint32_t w[4];
    RunLoad<16, kFixed>::ld(p, w);
    memcpy(out, w, 16);
  } else {
#pragma unroll
    for (int q = 0; q < BYTES / 32; ++q) {
      uint32_t w[8];
      RunLoad<32, kFixed>::ld(reinterpret_cast<const char*>(p) + 32 * q, w);
      memcpy(reinterpret_cast<char*>(out) + 32 * q, w, 32);
    }
  }
}

// K elements of T to p (32-byte aligned) with 256-bit stores: a lane's run
// is written as whole 32-byte sectors.
template <typename T, int K>
__device__ __forceinline__ void store_run(T* __restrict__ p, const T (&v)[K]) {
  constexpr int BYTES = K * (int)sizeof(T);
  static_assert(BYTES % 32 == 0, "run must be a multiple of 32 bytes");
  unsigned long long w[BYTES / 8];
  memcpy(w, v, BYTES);
#pragma unroll
  for (int q = 0; q < BYTES / 32; ++q)
    asm volatile("st.global.v4.b64 [%0], {%1, %2, %3, %4};" ::"l"(reinterpret_cast<char*>(p) + 32 * q),
                 "l"(w[4 * q]), "l"(w[4 * q + 1]), "l"(w[4 * q + 2]), "l"(w[4 * q + 3])
                 : "memory");
}

// Columns and values of lane `lane`'s run of tile t; entries past nnz read as
// column 0 with value 0.
template <typename I, typename V, int K>
__device__ __forceinline__ void tile_load(const I* __restrict__ ci, const V* __restrict__ val, int64_t nnz, int64_t t,
                                          int lane, I (&c)[K], V (&a)[K]) {
  const int64_t el = t * (32 * K) + (int64_t)lane * K;
  if (el + K <= nnz) {
    load_run<I, K>(ci + el, c);
    load_run<V, K>(val + el, a);
  } else {
#pragma unroll
    for (int b = 0; b < K; ++b) {
      const bool in = el + b < nnz;
      c[b] = in ? ci[el + b] : I(0);
      a[b] = in ? ld_stream(val + el + b) : V(0);
    }
  }
}

// x at the columns of lane `lane`'s run of tile t.  Entries past nnz count 0
// whatever x holds: 0 * x[0] would be NaN where x[0] is infinite.  (One test per
// tile, after the loads are out: loads under a mask, or a test per lane, cost the
// power-law SpMV 1.8 and 0.6 %.)
template <typename I, typename V, int K>
__device__ __forceinline__ void gather_run(const V* __restrict__ x, const I (&c)[K], int64_t nnz, int64_t t, int lane,
                                           V (&xv)[K]) {
#pragma unroll
  for (int b = 0; b < K; ++b) xv[b] = ld_gather(x + c[b]);
  if ((t + 1) * (32 * K) > nnz) {  // the partial last tile
#pragma unroll
    for (int b = 0; b < K; ++b)
      if (t * (32 * K) + (int64_t)lane * K + b >= nnz) xv[b] = V(0);
  }
}

// What is left of a tile when its complete rows have gone to y.
template <typename V>
struct TileEnds {
  bool owner;    // this lane holds the row open at the tile's end
  bool any;      // some row starts in the tile
  int64_t row;   // owner: that row
  V open;        // owner: its sum so far
  V cin;         // the entries before the tile's first row start (all lanes)
};

// Given the products p of the lane's run: rows complete inside the lane go to
// y, the heads combine across lanes.
template <typename I, typename V, int K>
__device__ __forceinline__ TileEnds<V> tile_sums(const I* __restrict__ rp, int64_t n, int64_t nnz, int64_t t, int lane,
                                                 uint32_t flags, int64_t tr, const V (&p)[K], V* __restrict__ y,
                                                 V alpha, V beta, bool bz) {
  const unsigned lt = (1u << lane) - 1u;  // lanes below this one
  const int64_t el = t * (32 * K) + (int64_t)lane * K;
  // ---- row of the lane's first entry
  int64_t row;
  if (tr >= 0) {
    const int cnt = __popc(flags);
    int excl = 0;
#pragma unroll
    for (int bit = 0; bit < 4; ++bit) excl += __popc(__ballot_sync(0xffffffffu, (cnt >> bit) & 1) & lt) << bit;
    const int first0 = (int)(__ballot_sync(0xffffffffu, flags & 1u) & 1u);
    row = tr + excl + (int)(flags & 1u) - first0;
  } else {
    row = row_holding(rp, n, el < nnz ? el : nnz - 1);
  }
  // ---- in-lane segments
  V head = V(0), acc = V(0);
  bool in_head = (flags & 1u) == 0;
#pragma unroll
  for (int b = 0; b < K; ++b) {
    if (b > 0 && ((flags >> b) & 1u)) {
      if (in_head) {
        head = acc;
        in_head = false;
      } else {
        axpby_store(y + row, acc, alpha, beta, bz);
      }
      acc = V(0);
      ++row;
      if (tr < 0)
        while (row + 1 < n && rp[row] == rp[row + 1]) ++row;  // skip empty rows
    }
    acc += p[b];
  }
  V tail = V(0);
  if (in_head) head = acc; else tail = acc;
  // ---- cross-lane: segmented inclusive scan of the heads, a segment
  // starting right after every flagged lane
  const bool has_flag = flags != 0;
  const unsigned fmask = __ballot_sync(0xffffffffu, has_flag);
  const unsigned starts = (fmask << 1) | 1u;  // lane l starts a segment if lane l-1 is flagged (or l == 0)
  V S = head;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const V su = __shfl_up_sync(0xffffffffu, S, o);
    // add lane (l - o)'s sum unless a segment starts in lanes l-o+1 .. l
    const unsigned span = (lane >= o) ? ((2u << lane) - 1u) & ~((2u << (lane - o)) - 1u) : 0u;
    if (lane >= o && !(starts & span)) S += su;
  }
  const unsigned later = fmask & ~((2u << lane) - 1u);  // flagged lanes after this one
  const int m = later ? __ffs(later) - 1 : 31;
  const V Sm = __shfl_sync(0xffffffffu, S, m);
  const int m0 = fmask ? __ffs(fmask) - 1 : 31;
  const V cin = __shfl_sync(0xffffffffu, S, m0);
  if (has_flag && later) axpby_store(y + row, tail + Sm, alpha, beta, bz);
  return TileEnds<V>{has_flag && !later, fmask != 0, row, tail + (lane < 31 ? Sm : V(0)), cin};
}

// The same, the tile's open row (it may continue into the next tile) and carry
// going to the calibrator arrays.
template <typename I, typename V, int K>
__device__ __forceinline__ void tile_finish(const I* __restrict__ rp, int64_t n, int64_t nnz, int64_t t, int lane,
                                            uint32_t flags, int64_t tr, const V (&p)[K], V* __restrict__ y, V alpha,
                                            V beta, bool bz, V* __restrict__ carry_in, V* __restrict__ open_sum,
                                            int64_t* __restrict__ open_row) {
  const TileEnds<V> E = tile_sums<I, V, K>(rp, n, nnz, t, lane, flags, tr, p, y, alpha, beta, bz);
  if (E.owner) {
    open_sum[t] = E.open;
    open_row[t] = E.row;
  }
  if (lane == 0) {
    carry_in[t] = E.cin;
    if (!E.any) open_row[t] = -1;
  }
}

// (The calibrations are set up while the tiles' sums are still being written: the
// three arrays are not __restrict__, so that they are read by plain loads.)
//
// The row open at tile t's end: its sum there and the heads of the following
// tiles, in tile order, up to the first one that starts a row.  A long row's
// tiles are read eight at a time (one at a time its loads were the
// calibration's whole time: 6.4 us for a row over 20 tiles).
template <typename V>
__device__ __forceinline__ V chain_sum(int64_t t, int64_t tiles, const V* carry_in,
                                       const V* open_sum, const int64_t* open_row) {
  V tot = open_sum[t];
  if (t + 1 >= tiles) return tot;
  tot += carry_in[t + 1];
  bool more = open_row[t + 1] < 0;
  for (int64_t u = t + 2; more && u < tiles; u += 8) {
    V c[8];
    int64_t r[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const bool in = u + q < tiles;
      c[q] = in ? carry_in[u + q] : V(0);
      r[q] = in ? open_row[u + q] : 0;
    }
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      if (more) tot += c[q];
      more = more && r[q] < 0;
    }
  }
  return tot;
}

// Calibration of one tile t (t < tiles) or empty row (t - tiles < nempty)
// of a single-vector product: the row open at tile t's end receives the heads
// of the following tiles up to the first one that starts a row.
template <typename V>
__device__ __forceinline__ void spmv_calibrate1(int64_t t, int64_t tiles, const V* carry_in,
                                                const V* open_sum, const int64_t* open_row,
                                                const int64_t* __restrict__ empty, int64_t nempty, V* __restrict__ y,
                                                V alpha, V beta, bool bz) {
  if (t < tiles) {
    const int64_t r = open_row[t];
    if (r < 0) return;
    axpby_store(y + r, chain_sum<V>(t, tiles, carry_in, open_sum, open_row), alpha, beta, bz);
  } else if (t - tiles < nempty) {
    axpby_store(y + empty[t - tiles], V(0), alpha, beta, bz);
  }
}

// ---- multi-RHS with up to 32 columns on the SpMV's tile plan
// (csr_tile_spmm and the batch's tile items)
//
// One warp per tile, G lanes per entry: group q (lanes qG .. qG + G - 1) takes
// the 8G consecutive entries of the plan's lanes qG .. qG + G - 1.  A lane
// holds J columns of the result:
//   kVec   columns 4h .. 4h + 3 of lane h (J = 4), an X row's part in one load
//          of 32 (FP64) or 16 (FP32) bytes: k a multiple of 4, rows aligned
//   else   columns h, h + G, ... (one load each): any k and alignment
// so the group's lanes gather an entry's whole X row together and a row costs
// one L2 request per 128 bytes.  Lanes past k load and store nothing.
//
// kStage: the tile's columns and values come through shared memory (SpmmTile),
// copied there asynchronously a tile ahead.  Not staged, the kernel is bound by
// the latency of dependent loads (column, then X row) at 16 warps per SM, with no
// unit above half its rate; staged, a warp never waits for its entries before
// it can ask for X rows, and the copies take no registers, which leaves room
// for eight entries' X rows per lane, four arriving while four are summed.  L1 is
// then busy for four fifths of the time (k = 12 and 32).
// Below eight lanes per entry or so the staging's own instructions weigh more
// than that: those forms load a lane's eight entries into registers.  Which
// form serves which k was measured (spmm_tiles_k).

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, int bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// A tile's columns and values; a group's share is set 16 bytes apart from the
// next one's, so that the groups' broadcast reads use different banks.
template <typename I, typename V, int G>
struct alignas(16) SpmmTile {
  static constexpr int NG = 32 / G, E = 8 * G;  // groups, entries of each
  static constexpr int kColB = E * (int)sizeof(I) + 16, kValB = E * (int)sizeof(V) + 16;
  unsigned char col[NG * kColB];
  unsigned char val[NG * kValB];

  // Starts the copy of tile t by one warp (entries past nnz come as zeros).
  __device__ __forceinline__ void fetch(const I* __restrict__ ci, const V* __restrict__ v, int64_t nnz, int64_t t,
                                        int lane) {
    const int64_t e0 = t * 256;
    const int64_t left = nnz - e0;
    constexpr int CI = 16 / (int)sizeof(I), CV = 16 / (int)sizeof(V);  // entries per 16 bytes
    const uint32_t dc = (uint32_t)__cvta_generic_to_shared(col), dv = (uint32_t)__cvta_generic_to_shared(val);
#pragma unroll
    for (int q = 0; q < 256 / CI / 32; ++q) {
      const int e = (q * 32 + lane) * CI;
      const int64_t m = left - e;
      const int bytes = m >= CI ? 16 : m > 0 ? (int)m * (int)sizeof(I) : 0;
      cp_async16(dc + (e / E) * kColB + (e % E) * (int)sizeof(I), bytes ? ci + e0 + e : ci, bytes);
    }
#pragma unroll
    for (int q = 0; q < 256 / CV / 32; ++q) {
      const int e = (q * 32 + lane) * CV;
      const int64_t m = left - e;
      const int bytes = m >= CV ? 16 : m > 0 ? (int)m * (int)sizeof(V) : 0;
      cp_async16(dv + (e / E) * kValB + (e % E) * (int)sizeof(V), bytes ? v + e0 + e : v, bytes);
    }
  }
  // four consecutive entries of group g
  __device__ __forceinline__ void cols4(int g, int e, I (&c)[4]) const {
    const uint4* p = reinterpret_cast<const uint4*>(col + g * kColB + e * (int)sizeof(I));
#pragma unroll
    for (int q = 0; q < (int)sizeof(I) / 4; ++q) {
      const uint4 w = p[q];
      memcpy(reinterpret_cast<char*>(c) + 16 * q, &w, 16);
    }
  }
  __device__ __forceinline__ void vals4(int g, int e, V (&a)[4]) const {
    const uint4* p = reinterpret_cast<const uint4*>(val + g * kValB + e * (int)sizeof(V));
#pragma unroll
    for (int q = 0; q < (int)sizeof(V) / 4; ++q) {
      const uint4 w = p[q];
      memcpy(reinterpret_cast<char*>(a) + 16 * q, &w, 16);
    }
  }
};

// A lane's part of an X row.
template <typename V, int G, int J, bool kVec, bool kFull>
__device__ __forceinline__ void ld_xpart(const V* __restrict__ p, int k, int h, V (&r)[J]) {
  if constexpr (kVec) {
    static_assert(J == 4, "vector parts hold four columns");
    if constexpr (sizeof(V) == 8) {
      uint32_t w[8];
      asm volatile("ld.global.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                   : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]), "=r"(w[4]), "=r"(w[5]), "=r"(w[6]), "=r"(w[7])
                   : "l"(p + 4 * h));
      memcpy(r, w, 32);
    } else {
      uint32_t w[4];
      asm volatile("ld.global.v4.b32 {%0,%1,%2,%3}, [%4];"
                   : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3])
                   : "l"(p + 4 * h));
      memcpy(r, w, 16);
    }
  } else {
#pragma unroll
    for (int j = 0; j < J; ++j) r[j] = kFull || h + G * j < k ? ld_gather(p + h + G * j) : V(0);
  }
}

// Row-start flags of the 8G entries of group g of tile t (bit b: entry b).
template <int G>
__device__ __forceinline__ uint64_t spmm_flags(const uint8_t* __restrict__ flags_all, int64_t t, int g) {
  const uint8_t* p = flags_all + t * 32 + g * G;
  if constexpr (G == 8) return *reinterpret_cast<const uint64_t*>(p);
  else if constexpr (G == 4) return *reinterpret_cast<const uint32_t*>(p);
  else if constexpr (G == 2) return *reinterpret_cast<const uint16_t*>(p);
  else return *p;
}

// One tile t whose entries are in S.  The group's row starts are its G lanes'
// flags; the heads combine over the 32/G groups with the segmented scan, and
// the row open at the tile's end goes to the k-wide calibrator (carry_in and
// open_sum hold k values per tile).  Every column is summed in an order fixed
// by the matrix and k.
// kFull: k == G * J, no column of any lane lies past k.
template <typename I, typename V, int G, int J, bool kVec, bool kStage, bool kFull>
__device__ __forceinline__ void spmm_tile_groups(const SpmmTile<I, V, G>* S, uint64_t fl, int64_t tr,
                                                 const I* __restrict__ ci, const V* __restrict__ val,
                                                 const I* __restrict__ rp, int64_t n, int64_t nnz, int64_t t,
                                                 const V* __restrict__ X, int64_t ldx, int k, V* __restrict__ Y,
                                                 int64_t ldy, V alpha, V beta, bool bz, V* __restrict__ carry_in,
                                                 V* __restrict__ open_sum, int64_t* __restrict__ open_row, int lane) {
  constexpr int NG = 32 / G, E = 8 * G;
  static_assert(G == 1 || G == 2 || G == 4 || G == 8, "1, 2, 4 or 8 lanes per entry");
  const int gq = lane / G, h = lane % G;
  const bool active = kFull || (kVec ? 4 * h : h) < k;  // some column of this lane is below k
  const int64_t e0 = t * 256 + (int64_t)gq * E;
  const int real = nnz - e0 >= E ? E : nnz > e0 ? (int)(nnz - e0) : 0;  // entries of the group inside the matrix
  // group flags as an NG-bit mask (bit q: group q holds a row start)
  const unsigned lane_f = __ballot_sync(0xffffffffu, fl != 0 && h == 0);
  unsigned gf = 0;
  if constexpr (G == 1) {
    gf = lane_f;
  } else {
#pragma unroll
    for (int q = 0; q < NG; ++q) gf |= ((lane_f >> (G * q)) & 1u) << q;
  }
  int64_t row;
  if (tr >= 0) {
    const int cnt = __popcll(fl);
    const unsigned below = (1u << (gq * G)) - 1u;  // lanes of earlier groups
    int excl = 0;
#pragma unroll
    for (int bit = 0; (1 << bit) <= E; ++bit)
      excl += __popc(__ballot_sync(0xffffffffu, ((cnt >> bit) & 1) && h == 0) & below) << bit;
    const int first0 = (int)(__ballot_sync(0xffffffffu, fl & 1u) & 1u);
    row = tr + excl + (int)(fl & 1u) - first0;
  } else {
    row = row_holding(rp, n, e0 < nnz ? e0 : nnz - 1);
  }
  auto column = [&](int j) { return kVec ? 4 * h + j : h + G * j; };
  auto has = [&](int j) { return kFull || column(j) < k; };
  V acc[J], head[J];
#pragma unroll
  for (int j = 0; j < J; ++j) acc[j] = head[j] = V(0);
  bool in_head = (fl & 1u) == 0;
  // X rows of four entries (entries past nnz have column 0; they are not added)
  auto gather = [&](const I (&c)[4], V (&x)[4][J]) {
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (active) ld_xpart<V, G, J, kVec, kFull>(X + (int64_t)c[q] * ldx, k, h, x[q]);
  };
  auto add = [&](int e, const V (&a)[4], const V (&x)[4][J]) {
    const unsigned f4 = (unsigned)(fl >> e) & 15u;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      if (((f4 >> q) & 1u) && e + q > 0) {
        if (in_head) {
#pragma unroll
          for (int j = 0; j < J; ++j) head[j] = acc[j];
          in_head = false;
        } else {
#pragma unroll
          for (int j = 0; j < J; ++j)
            if (has(j)) axpby_store(Y + row * ldy + column(j), acc[j], alpha, beta, bz);
        }
#pragma unroll
        for (int j = 0; j < J; ++j) acc[j] = V(0);
        ++row;
        if (tr < 0)
          while (row + 1 < n && rp[row] == rp[row + 1]) ++row;  // skip empty rows
      }
      if (e + q < real) {
#pragma unroll
        for (int j = 0; j < J; ++j) acc[j] += a[q] * x[q][j];
      }
    }
  };
  if constexpr (kStage) {
    V x0[4][J], x1[4][J], a[4];
    I c[4];
    S->cols4(gq, 0, c);
    gather(c, x0);
#pragma unroll 1
    for (int e = 0; e < E; e += 8) {
      S->cols4(gq, e + 4, c);
      gather(c, x1);
      S->vals4(gq, e, a);
      add(e, a, x0);
      if (e + 8 < E) {
        S->cols4(gq, e + 8, c);
        gather(c, x0);
      }
      S->vals4(gq, e + 4, a);
      add(e + 4, a, x1);
    }
  } else {
#pragma unroll 1
    for (int e = 0; e < E; e += 8) {
      I c[8], c4[4];
      V a[8], a4[4], x[4][J];
      tile_load<I, V, 8>(ci, val, nnz, t, gq * G + e / 8, c, a);
#pragma unroll
      for (int half = 0; half < 8; half += 4) {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          c4[q] = c[half + q];
          a4[q] = a[half + q];
        }
        gather(c4, x);
        add(e + half, a4, x);
      }
    }
  }
  V tail[J];
#pragma unroll
  for (int j = 0; j < J; ++j) {
    if (in_head) head[j] = acc[j];
    tail[j] = in_head ? V(0) : acc[j];
  }
  const bool has_flag = fl != 0;
  const unsigned starts = (gf << 1) | 1u;  // group q starts a segment if group q - 1 is flagged (or q == 0)
#pragma unroll
  for (int o = 1; o < NG; o <<= 1) {
    const unsigned span = (gq >= o) ? ((2u << gq) - 1u) & ~((2u << (gq - o)) - 1u) : 0u;
    const bool more = gq >= o && !(starts & span);
#pragma unroll
    for (int j = 0; j < J; ++j) {
      const V su = __shfl_up_sync(0xffffffffu, head[j], G * o);
      if (more) head[j] += su;
    }
  }
  const unsigned later = gf & ~((2u << gq) - 1u);
  const int m = later ? __ffs(later) - 1 : NG - 1;
  const int m0 = gf ? __ffs(gf) - 1 : NG - 1;
  V Sm[J], cin[J];
#pragma unroll
  for (int j = 0; j < J; ++j) {
    Sm[j] = __shfl_sync(0xffffffffu, head[j], G * m + h);
    cin[j] = __shfl_sync(0xffffffffu, head[j], G * m0 + h);
  }
  if (has_flag) {
    if (later) {
#pragma unroll
      for (int j = 0; j < J; ++j)
        if (has(j)) axpby_store(Y + row * ldy + column(j), tail[j] + Sm[j], alpha, beta, bz);
    } else {  // the tile's last row: may continue into the next tile
#pragma unroll
      for (int j = 0; j < J; ++j)
        if (has(j)) open_sum[t * k + column(j)] = tail[j] + (gq < NG - 1 ? Sm[j] : V(0));
      if (h == 0) open_row[t] = row;
    }
  }
  if (gq == 0) {
#pragma unroll
    for (int j = 0; j < J; ++j)
      if (has(j)) carry_in[t * k + column(j)] = cin[j];
    if (h == 0 && !gf) open_row[t] = -1;
  }
}

// Lanes per tile of the k-wide calibration: the power of two from k, at most a
// warp (a lane per column: whole lines of carry_in, open_sum and Y).
__host__ __device__ __forceinline__ int spmm_cal_lanes(int64_t k) {
  int L = 1;
  while (L < 32 && L < k) L <<= 1;
  return L;
}

// Calibration of one tile t (t < tiles) or empty row (t - tiles < nempty)
// of a product with k columns; this lane takes columns sub, sub + L, ...
template <typename V>
__device__ __forceinline__ void spmm_calibrate(int64_t t, int sub, int L, int k, int64_t tiles,
                                               const V* carry_in, const V* open_sum,
                                               const int64_t* open_row,
                                               const int64_t* __restrict__ empty, int64_t nempty, V* __restrict__ Y,
                                               int64_t ldy, V alpha, V beta, bool bz) {
  if (t < tiles) {
    const int64_t r = open_row[t];
    if (r < 0) return;
    for (int c = sub; c < k; c += L) {
      V tot = open_sum[t * k + c];
      for (int64_t u = t + 1; u < tiles; ++u) {
        tot += carry_in[u * k + c];
        if (open_row[u] >= 0) break;
      }
      axpby_store(Y + r * ldy + c, tot, alpha, beta, bz);
    }
  } else if (t - tiles < nempty) {
    for (int c = sub; c < k; c += L) axpby_store(Y + empty[t - tiles] * ldy + c, V(0), alpha, beta, bz);
  }
}

}  // namespace
}  // namespace spops
