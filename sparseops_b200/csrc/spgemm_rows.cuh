// Sort-accumulate numeric phase for the clusters of one row (most of a
// LeSpGEMM and all of a row-wise product): W warps of one block per row of C,
// R sorted keys per lane, up to 32*R*W products.
//
// The method is that of spgemm_sort.cuh: a product's key (output column <<
// tbits | product index t, flat (j, k) order) is sorted by a bitonic network
// in registers, so a column's products are adjacent and in flat order.
// Around the network (two thirds of the instructions, 3,900 a row at R = 16, in
// a kernel that built its keys slot by slot and wrote from the lanes):
//   - products are formed in a compact loop over 32*W-product steps, kRowCols
//     columns of A staged at a time with their values, four steps' loads in
//     flight, keys and values parked in shared memory;
//   - sums run forward along a lane's sorted keys without branches, and a
//     column's total replaces the value of its last product (only the lane
//     that holds a key reads or writes its product's value);
//   - the last key of each column goes to a list by rank, from which columns
//     and totals are written in order, coalesced, with the drop rule and the
//     row's count of kept entries (no separate counting pass);
//   - the staging takes 0.6 - 1.3 KB instead of 3 - 12 KB of shared memory, so
//     more rows are resident per SM.
// Measured on the planted matrix (524,288 rows, 2e8 products, 1.2e8 entries of
// C): rows of 257 - 512 products 1.38 -> 0.80 ms, 513 - 1024 2.19 -> 1.10 ms,
// 1025 - 2048 1.07 -> 0.70 ms (the second figures with the multi-row clusters
// that stay on the other kernels).  Bound by instruction issue and the latency
// of the loads at 24 - 32 resident warps per SM.  (Hash tables in shared
// memory with a sort of the distinct columns alone took 1.17 and 2.49 ms for
// 193 - 384 and 385 - 768 products: 12 KB per warp leaves 13 warps per SM.)
// Sums are in a fixed order: in flat order within a lane's run, the runs of a
// column that spans lanes combined by a fixed tree.
#pragma once

#include <cstdint>

#include "pdl.cuh"
#include "spgemm_sort.cuh"

namespace spops {
namespace {

constexpr int kRowUnroll = 4;

// dynamic shared memory of row_sort_kernel<I, V, R, W>
template <typename V, int R, int W>
struct RowSmem {
  static constexpr int N = 32 * R * W;
  static constexpr int kCols = W == 1 ? 32 : 64;  // columns of A staged at a time
  V val[N];            // per product, then per column at its last product
  V a[kCols];
  V w_sum[W];          // per warp: sum open at its end
  int64_t base[kCols];  // B row start less the products before the column
  uint32_t key[N];     // keys as built, the cross-warp exchange, the output list
  int32_t off[kCols + 1];
  uint32_t w_edge[W];  // per warp: last key; whether its first key starts a column
  int32_t w_cnt[W];
  int32_t w_flag[W];
};

template <typename I, typename V, int R, int W>
__global__ void __launch_bounds__(32 * W)
    row_sort_kernel(const int64_t* __restrict__ list, const int64_t* __restrict__ cptr,
                    const int64_t* __restrict__ cptr_val, const int32_t* __restrict__ colids,
                    const V* __restrict__ avals, const int64_t* __restrict__ offsets,
                    const int64_t* __restrict__ perm, const I* __restrict__ brp, const I* __restrict__ bci,
                    const V* __restrict__ bv, double b_rowdense, double budget, bool sort_output, bool rowwise,
                    const int64_t* __restrict__ soff, const int64_t* __restrict__ soff_val,
                    int64_t* __restrict__ nz, int64_t* __restrict__ cmin, int64_t* __restrict__ cmax,
                    unsigned char* __restrict__ drop_out, unsigned long long* __restrict__ ndense,
                    int32_t* __restrict__ ccol, V* __restrict__ cval, int64_t* __restrict__ rowcnt) {
  using S = RowSmem<V, R, W>;
  constexpr int N = S::N, NW = 32 * R, U = kRowUnroll;
  constexpr int kTBits = [] {
    int b = 0;
    while ((1 << b) < N) ++b;
    return b;
  }();
  constexpr uint32_t kNone = 0xffffffffu;
  extern __shared__ __align__(16) unsigned char row_smem[];
  S& M = *reinterpret_cast<S*>(row_smem);
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  auto sync = [] {
    if (W == 1) __syncwarp(); else __syncthreads();
  };
  overlap_let_next();
  const int64_t c = list[blockIdx.x];
  const int64_t j0 = cptr[c], vbase = cptr_val[c];
  const int nj = (int)(cptr[c + 1] - j0);
  // ---- products: value and key at index t
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
          M.a[h + lane] = avals[vbase + jb + h + lane];
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
      V x[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int t = t0 + 32 * W * u;
        if (t < T)
          while (M.off[j + 1] <= t) ++j;
        k[u] = M.base[j] + t;
        x[u] = M.a[j];
      }
      uint32_t col[U];
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (t0 + 32 * W * u < T) {
          col[u] = (uint32_t)bci[k[u]];
          x[u] *= bv[k[u]];
        }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int t = P + t0 + 32 * W * u;
        if (t0 + 32 * W * u < T) {
          M.val[t] = x[u];
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
  // ---- where columns start and end: position w*32R + lane*R + s
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
  for (int s = 0; s < R; ++s) first |= ((((s ? key[s - 1] : before) ^ key[s]) >> kTBits) != 0 ? 1u : 0u) << s;
  if (p0 == 0) first |= 1u;
  first &= nv >= 32 ? kNone : (1u << nv) - 1u;
  uint32_t after = __shfl_down_sync(0xffffffffu, first & 1u, 1);
  if (W > 1) {
    if (lane == 0) M.w_flag[w] = (int32_t)(first & 1u);
    __syncthreads();
    if (lane == 31) after = w + 1 < W ? (uint32_t)M.w_flag[w + 1] : 0u;
  } else if (lane == 31) {
    after = 0;
  }
  uint32_t last = first >> 1 | after << (R - 1);
  if (nv > 0 && p0 + nv == P) last |= 1u << (nv - 1);
  const int cnt = __popc(last);
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
  // ---- sums along the lane; a total goes to its column's last product
  constexpr uint32_t kTMask = (uint32_t)N - 1u;
  constexpr int B = R < 4 ? R : 4;  // values loaded together
  V run = V(0), head = V(0);
  int head_t = -1;  // last product of a column that started in an earlier lane
#pragma unroll
  for (int s0 = 0; s0 < R; s0 += B) {
    V v[B];
#pragma unroll
    for (int q = 0; q < B; ++q) v[q] = s0 + q < nv ? M.val[key[s0 + q] & kTMask] : V(0);
#pragma unroll
    for (int q = 0; q < B; ++q) {
      const int s = s0 + q;
      run = (first >> s & 1u) ? v[q] : run + v[q];
      if (last >> s & 1u) {
        const int t = (int)(key[s] & kTMask);
        M.key[rank++] = key[s];
        if ((first & ((2u << s) - 1u)) == 0) {
          head = run;
          head_t = t;
        } else {
          M.val[t] = run;
        }
      }
    }
  }
  // sums open at the lanes' ends: inclusive segmented scan, then each lane's
  // carry from the lanes (and warps) before it
  {
    V C = run;
    int f = first != 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const V pc = __shfl_up_sync(0xffffffffu, C, o);
      const int pf = __shfl_up_sync(0xffffffffu, f, o);
      if (lane >= o && !f) {
        C = pc + C;
        f = pf;
      }
    }
    V carry = __shfl_up_sync(0xffffffffu, C, 1);
    int cf = __shfl_up_sync(0xffffffffu, f, 1);
    if (lane == 0) {
      carry = V(0);
      cf = 0;
    }
    if (W > 1) {
      __syncthreads();  // w_flag was read
      if (lane == 31) {
        M.w_sum[w] = C;
        M.w_flag[w] = f;
      }
      __syncthreads();
      if (!cf && w > 0) {
        V X = V(0);
        for (int v = 0; v < w; ++v) X = M.w_flag[v] ? M.w_sum[v] : X + M.w_sum[v];
        carry = X + carry;
      }
    }
    if (head_t >= 0) M.val[head_t] = carry + head;
  }
  sync();
  // ---- classification (the same arithmetic as classify_kernel) and output
  const int64_t mn = n ? (int64_t)(M.key[0] >> kTBits) : 0, mx = n ? (int64_t)(M.key[n - 1] >> kTBits) : 0;
  bool dense = false;
  if (n > 0) {
    const int64_t range = mx - mn + 1;
    const double density = (double)n / (double)range;
    const size_t b_access = (size_t)((double)nj * b_rowdense * (double)(sizeof(int64_t) + sizeof(V)));
    dense = (double)(b_access + (size_t)range * sizeof(V)) <= budget && density >= 0.15;
  }
  const bool drop = !rowwise && (dense || sort_output);
  const int64_t co = soff[c], cvo = soff_val[c];
  int kept = 0;
  for (int p = tid; p < n; p += 32 * W) {
    const uint32_t e = M.key[p];
    V v = M.val[e & kTMask];
    if (drop && fabs((double)v) < 1e-12) v = V(0);
    kept += rowwise || v != V(0);
    ccol[co + p] = (int32_t)(e >> kTBits);
    cval[cvo + p] = v;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) kept += __shfl_down_sync(0xffffffffu, kept, o);
  if (W > 1) {
    if (lane == 0) M.w_cnt[w] = kept;
    __syncthreads();
    if (tid == 0)
      for (int v = 1; v < W; ++v) kept += M.w_cnt[v];
  }
  if (tid == 0) {
    nz[c] = n;
    cmin[c] = mn;
    cmax[c] = mx;
    drop_out[c] = drop ? 1 : 0;
    rowcnt[perm[offsets[c]]] = kept;
    if (dense && !rowwise) atomicAdd(ndense, 1ULL);
  }
  overlap_end();
}

}  // namespace
}  // namespace spops
