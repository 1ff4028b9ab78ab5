// Sort-accumulate numeric phase for the clusters of several rows (and one-row
// clusters of up to 64 products): W warps per cluster, R sorted keys per lane,
// up to 32*R*W products, 32*R*W a power of two from 32 to 8192.
//
// Products are gathered as in row_sort_kernel (spgemm_rows.cuh), but what is
// parked per product is B's value and the cluster column, since each row of
// the cluster has its own A value there.  After the sort (spgemm_sort.cuh) the
// product numbers go to shared memory in sorted order, the starts of the
// columns by rank beside them, and the values of C's slab, [column x row of the
// cluster], are one task each: a lane adds its column's products in flat order
// and writes next to its neighbours, and the A values of one product are read
// side by side; the rows' kept entries are counted on the way.  Before, each
// row of the cluster walked all sorted keys and combined the lanes by a scan,
// with strided writes, and a pass of its own counted: grouped rows, clusters of
// up to 8 rows and 129 - 256 products (FP64, int64), 491 us, now 312 with the
// counts (255 without, and 76 for the pass); 257 - 512 products 67 -> 34 us.
// Bound by the loads of B's rows and of the A values (the largest stall, 4.4 cycles
// an instruction at 44 % of the warps) and by issue (61 % of the slots).
//
// Output goes to the cluster's slab: ccol[soff[c] ..], cval[soff_val[c] ..]
// (room for P columns), columns ascending -- the layout the hash kernels write.
#pragma once

#include <cstdint>

#include "pdl.cuh"
#include "spgemm_sort.cuh"

namespace spops {
namespace {

constexpr int kGroupCols = 1024;  // columns of a cluster
constexpr int kGroupPer = 4;      // clusters per block, W = 1
constexpr int kGroupRows = 32;    // up to this many rows of a cluster are counted on the way

template <typename V, int R, int W>
struct alignas(16) GroupSmem {
  static constexpr int N = 32 * R * W;
  static constexpr int kCols = W == 1 ? 32 : 64;  // columns of the cluster staged at a time
  V val[N];             // per product: B's value
  int64_t base[kCols];  // B row start less the products before the column
  uint32_t key[N];      // keys as built, the cross-warp exchange, the columns by rank, what is kept
  int32_t off[kCols + 1];
  uint32_t w_edge[W];
  int32_t w_cnt[W];
  int32_t kept[kGroupRows];  // entries kept per row of the cluster
  uint16_t col[N];      // per product: column of the cluster
  uint16_t ord[N];      // product at each sorted position
  uint16_t pos[N + 1];  // where each column starts, and P
};

template <typename I, typename V, int R, int W>
__global__ void __launch_bounds__(W == 1 ? 32 * kGroupPer : 32 * W)
    group_sort_kernel(const int64_t* __restrict__ list, int64_t nlist, const int64_t* __restrict__ cptr,
                      const int64_t* __restrict__ cptr_val, const int32_t* __restrict__ colids,
                      const V* __restrict__ avals, const int64_t* __restrict__ offsets,
                      const int64_t* __restrict__ perm, const I* __restrict__ brp, const I* __restrict__ bci, const V* __restrict__ bv, double b_rowdense, double budget,
                      bool sort_output, bool rowwise, const int64_t* __restrict__ soff,
                      const int64_t* __restrict__ soff_val, int64_t* __restrict__ nz, int64_t* __restrict__ cmin,
                      int64_t* __restrict__ cmax, unsigned char* __restrict__ drop_out,
                      unsigned long long* __restrict__ ndense, int32_t* __restrict__ ccol, V* __restrict__ cval,
                      int64_t* __restrict__ rowcnt) {
  using S = GroupSmem<V, R, W>;
  constexpr int N = S::N, NW = 32 * R, U = 4;
  constexpr int kTBits = [] {
    int b = 0;
    while ((1 << b) < N) ++b;
    return b;
  }();
  constexpr uint32_t kNone = 0xffffffffu, kTMask = (uint32_t)N - 1u;
  extern __shared__ __align__(16) unsigned char group_smem[];
  const int lane = threadIdx.x & 31;
  const int w = W == 1 ? 0 : threadIdx.x >> 5, tid = W == 1 ? lane : threadIdx.x;
  S& M = reinterpret_cast<S*>(group_smem)[W == 1 ? threadIdx.x >> 5 : 0];
  auto sync = [] {
    if (W == 1) __syncwarp(); else __syncthreads();
  };
  overlap_let_next();
  const int64_t slot = W == 1 ? blockIdx.x * (int64_t)kGroupPer + (threadIdx.x >> 5) : blockIdx.x;
  if (slot >= nlist) return;  // W == 1: whole warps, which share no barrier, and not the block's first
  const int64_t c = list[slot];
  const int64_t j0 = cptr[c], vbase = cptr_val[c];
  const int nj = (int)(cptr[c + 1] - j0);
  const int64_t rows = offsets[c + 1] - offsets[c];
  const int64_t csz = max(rows, (int64_t)1);  // without rows: no products either
  const bool count = csz <= kGroupRows;
  if (tid < kGroupRows) M.kept[tid] = 0;
  // ---- products: B's value, column of the cluster and key at index t
  int P = 0;
  for (int jb = 0; jb < nj; jb += S::kCols) {
    if (w == 0) {
      int32_t carry = 0;
#pragma unroll
      for (int h = 0; h < S::kCols; h += 32) {
        int32_t len = 0;
        int64_t st = 0;
        if (jb + h + lane < nj) {
          const int64_t r = colids[j0 + jb + h + lane];
          st = brp[r];
          len = (int32_t)((int64_t)brp[r + 1] - st);
        }
        int32_t inc = len;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int32_t u = __shfl_up_sync(0xffffffffu, inc, o);
          if (lane >= o) inc += u;
        }
        M.base[h + lane] = st - (carry + inc - len);
        M.off[h + lane + 1] = carry + inc;
        carry += __shfl_sync(0xffffffffu, inc, 31);
      }
      if (lane == 0) M.off[0] = 0;
    }
    sync();
    const int T = M.off[S::kCols];
    int j = 0;
    if (W > 1) {  // the column holding this thread's first product
      int hi = S::kCols;
      while (hi - j > 1) {
        const int mid = (j + hi) >> 1;
        if (M.off[mid] <= tid) j = mid; else hi = mid;
      }
    }
    for (int t0 = tid; t0 < T; t0 += 32 * W * U) {
      int64_t k[U];
      int at[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int t = t0 + 32 * W * u;
        if (t < T)
          while (M.off[j + 1] <= t) ++j;
        k[u] = M.base[j] + t;
        at[u] = jb + j;
      }
      uint32_t col[U];
      V x[U];
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (t0 + 32 * W * u < T) {
          col[u] = (uint32_t)bci[k[u]];
          x[u] = bv[k[u]];
        }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int t = P + t0 + 32 * W * u;
        if (t0 + 32 * W * u < T) {
          M.val[t] = x[u];
          M.col[t] = (uint16_t)at[u];
          M.key[t] = col[u] << kTBits | (uint32_t)t;
        }
      }
    }
    P += T;
    sync();
  }
  // ---- sort
  uint32_t key[R];
#pragma unroll
  for (int s = 0; s < R; ++s) {
    const int t = (w * R + s) * 32 + lane;
    key[s] = t < P ? M.key[t] : kNone;
  }
  block_sort_keys<R, W>(key, M.key, w, lane);
  // ---- the products in order, and where columns start
  const int p0 = w * NW + lane * R;
  const int nv = min(max(P - p0, 0), R);  // real keys of this lane
  uint32_t before = __shfl_up_sync(0xffffffffu, key[R - 1], 1);
  if (W > 1) {
    if (lane == 31) M.w_edge[w] = key[R - 1];
    __syncthreads();
    if (lane == 0 && w > 0) before = M.w_edge[w - 1];
  }
  uint32_t first = 0;
#pragma unroll
  for (int s = 0; s < R; ++s) {
    first |= ((((s ? key[s - 1] : before) ^ key[s]) >> kTBits) != 0 ? 1u : 0u) << s;
    M.ord[p0 + s] = (uint16_t)(key[s] & kTMask);
  }
  if (p0 == 0) first |= 1u;
  first &= (1u << nv) - 1u;
  const int cnt = __popc(first);
  int incl = cnt;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int u = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += u;
  }
  int n = __shfl_sync(0xffffffffu, incl, 31), rank = incl - cnt;
  if (W > 1) {
    if (lane == 31) M.w_cnt[w] = incl;
    __syncthreads();
    n = 0;
#pragma unroll
    for (int v = 0; v < W; ++v) {
      const int q = M.w_cnt[v];
      if (v < w) rank += q;
      n += q;
    }
  }
#pragma unroll
  for (int s = 0; s < R; ++s)
    if (first >> s & 1u) {
      M.key[rank] = key[s] >> kTBits;
      M.pos[rank++] = (uint16_t)(p0 + s);
    }
  if (tid == 0) M.pos[n] = (uint16_t)P;
  sync();
  // ---- classification (the same arithmetic as classify_kernel)
  const int64_t mn = n ? (int64_t)M.key[0] : 0, mx = n ? (int64_t)M.key[n - 1] : 0;
  bool dense = false;
  if (n > 0) {
    const int64_t range = mx - mn + 1;
    const double density = (double)n / (double)range;
    const size_t b_access = (size_t)((double)nj * b_rowdense * (double)(sizeof(int64_t) + sizeof(V)));
    const size_t dense_bytes = (size_t)range * (size_t)csz * sizeof(V);
    dense = (double)(b_access + dense_bytes) <= budget && density >= 0.15;
  }
  const bool drop = !rowwise && (dense || sort_output);
  if (tid == 0) {
    nz[c] = n;
    cmin[c] = mn;
    cmax[c] = mx;
    drop_out[c] = drop ? 1 : 0;
    if (dense && !rowwise) atomicAdd(ndense, 1ULL);
  }
  // ---- columns, then values: task e = column * csz + row
  const int64_t co = soff[c], cvo = soff_val[c];
  for (int q = tid; q < n; q += 32 * W) ccol[co + q] = (int32_t)M.key[q];
  sync();
  if (drop) {  // from here on key[q]: column q keeps its values
    for (int q = tid; q < n; q += 32 * W) M.key[q] = 0;
    sync();
  }
  const int64_t tasks = (int64_t)n * csz;
  int q = (int)(tid / csz);
  int64_t l = tid - q * csz;
  const int dq = (int)(32 * W / csz);
  const int64_t dl = 32 * W - dq * csz;
  int mine = 0;  // entries this thread keeps of a one-row cluster
  auto keep = [&](V v, int64_t row) {
    if (!rowwise && v == V(0)) return;
    if (csz == 1) ++mine; else if (count) atomicAdd(&M.kept[row], 1);
  };
  for (int64_t e = tid; e < tasks; e += 32 * W) {
    const int to = M.pos[q + 1];
    // flat order, each product fused into the sum (16,384 grouped rows, mean
    // error against exact sums, FP32 | FP64: 2.43e-8 | 4.53e-17 with products
    // rounded on their own, 2.10e-8 | 3.91e-17 so); two products' loads in flight
    auto aval = [&](int t) { return avals[vbase + (int64_t)M.col[t] * csz + l]; };
    int p = M.pos[q];
    V sum = V(0);
    for (; p + 1 < to; p += 2) {
      const int t0 = M.ord[p], t1 = M.ord[p + 1];
      const V a0 = aval(t0), a1 = aval(t1);
      sum = fma(a0, M.val[t0], sum);
      sum = fma(a1, M.val[t1], sum);
    }
    if (p < to) {
      const int t = M.ord[p];
      sum = fma(aval(t), M.val[t], sum);
    }
    // zeroed: a value below 1e-12 of a one-row cluster, a column of which no
    // value reaches 1e-12 otherwise
    if (drop && (csz == 1 ? !(fabs((double)sum) < 1e-12) : fabs((double)sum) >= 1e-12)) M.key[q] = 1;
    cval[cvo + e] = sum;
    if (!drop) keep(sum, l);
    l += dl;
    q += dq;
    if (l >= csz) {
      l -= csz;
      ++q;
    }
  }
  if (drop) {
    sync();  // every task's mark, and its value, written
    q = (int)(tid / csz);
    l = tid - q * csz;
    for (int64_t e = tid; e < tasks; e += 32 * W) {
      if (M.key[q] == 0) cval[cvo + e] = V(0); else keep(cval[cvo + e], l);
      l += dl;
      q += dq;
      if (l >= csz) {
        l -= csz;
        ++q;
      }
    }
  }
  if (csz == 1) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mine += __shfl_down_sync(0xffffffffu, mine, o);
    if (lane == 0) atomicAdd(&M.kept[0], mine);
  }
  sync();
  if (count && tid < rows) rowcnt[perm[offsets[c] + tid]] = M.kept[tid];
  overlap_end();
}

}  // namespace
}  // namespace spops
