// MinHash signatures and LSH candidate pairs on the device.
//
// Replaces minhash_signatures_flat (reference include/spgemm_MinHashLSH.h:119-180)
// and lsh_candidate_pairs_from_flat_vector (427-605), which
// lsh_candidate_pairs_vector (777-791) chains.  Outputs are bit-identical:
//   signatures  sig[r][d] = min over the row's columns c of a_d*c + b_d
//               (mod 2^64), a_d, b_d from the reference's LCG (40-43,
//               134-141); empty rows keep UINT64_MAX.  One warp per row, the
//               row's columns broadcast, each lane owning k/32 hash functions.
//   records     bucket = band hash of the band's r = k/bands values
//               (h = h*0x9e3779b97f4a7c15 + v, 277-283); equal hashes of a band
//               meet in its hash table, the bands in batches of up to 2^24
//               records (the reference sorts by (band, bucket, row)).
//   pairs       each bucket of at least two rows pairs every row with every
//               later row, or -- when constrained and it has more than 256
//               rows -- with its next 16 rows (481-516); the pairs (i < j) of
//               all bands, each once, ascending (544-545).
//   scores      matches / k over the two signatures (183-204), four pairs per
//               warp.
#include <cub/cub.cuh>

#include <algorithm>
#include <vector>

#include "pdl.cuh"
#include "spgemm_sort.cuh"
#include "spops_internal.h"

namespace spops {
namespace {

inline unsigned grid_for(int64_t work, int threads = 256) {
  int64_t g = (work + threads - 1) / threads;
  return (unsigned)(g < 1 ? 1 : g);
}

// a*x + b mod 2^64 for a column x below 2^32: one 32x32->64 multiply-add and
// one 32-bit multiply-add into the high half.
__device__ __forceinline__ uint64_t hash_narrow(uint64_t a, uint32_t x, uint64_t b) {
  const uint64_t lo = (uint64_t)(uint32_t)a * x + b;
  const uint32_t hi = (uint32_t)(lo >> 32) + (uint32_t)(a >> 32) * x;
  return (uint64_t)hi << 32 | (uint32_t)lo;
}

// One warp per row, two hash functions per lane per pass, four columns in
// flight.  Bound by the integer multiply-adds and 64-bit minima of k hashes per
// entry.  NARROW: every column below 2^32, two multiplies per hash instead of
// three.  524,288 rows, k = 64, int64: one column at a time with 64-bit
// multiplies took 222 us (short rows) and 423 us (longer ones), this 187 and
// 416.
template <typename I, bool NARROW>
__global__ void minhash_kernel(const I* __restrict__ rp, const I* __restrict__ ci, int64_t n, int k,
                               const uint64_t* __restrict__ a, const uint64_t* __restrict__ b,
                               uint64_t* __restrict__ sig) {
  const int64_t r = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (r >= n) return;
  const int64_t s = rp[r], e = rp[r + 1];
  for (int d0 = 0; d0 < k; d0 += 64) {
    const int d1 = d0 + lane, d2 = d0 + 32 + lane;
    const uint64_t a1 = d1 < k ? a[d1] : 0, b1 = d1 < k ? b[d1] : 0;
    const uint64_t a2 = d2 < k ? a[d2] : 0, b2 = d2 < k ? b[d2] : 0;
    uint64_t m1 = ~0ULL, m2 = ~0ULL;
    auto take = [&](I x) {
      uint64_t h1, h2;
      if constexpr (NARROW) {
        h1 = hash_narrow(a1, (uint32_t)x, b1);
        h2 = hash_narrow(a2, (uint32_t)x, b2);
      } else {
        h1 = a1 * (uint64_t)(int64_t)x + b1;
        h2 = a2 * (uint64_t)(int64_t)x + b2;
      }
      m1 = h1 < m1 ? h1 : m1;
      m2 = h2 < m2 ? h2 : m2;
    };
    const I* p = ci + s;
    int left = (int)(e - s);
    for (; left >= 4; left -= 4, p += 4) {
      const I x0 = p[0], x1 = p[1], x2 = p[2], x3 = p[3];
      take(x0);
      take(x1);
      take(x2);
      take(x3);
    }
    for (; left > 0; --left) take(*p++);
    if (d1 < k) sig[r * k + d1] = m1;
    if (d2 < k) sig[r * k + d2] = m2;
  }
}

// ---- candidate pairs
// A bucket is a set of rows and a row's pairs are the later members of its
// buckets, each once: per row, the members of its `bands` buckets are gathered,
// sorted in registers and deduplicated, so the pairs come out in their final
// (i, j) order without one sort of every record and one of every pair.
//
// Records (band b, row i) go through these steps, q = b * n + i:
//   lsh_slot_kernel   the band's hash and its slot in the band's
//                     open-addressing table of at least 2n slots (equal values
//                     get equal slots, different values different ones), and a
//                     ticket, the number of earlier arrivals there
//   lsh_base_kernel   room for the members of each slot with two or more rows
//   lsh_member_kernel row i into its bucket's room, at its ticket; the record
//                     becomes (where the members are, how many), 0 for a row
//                     that is alone in its bucket, as most are
//   lsh_pair_kernel   the row's members above i, sorted and made unique
// A constrained bucket of more than 256 rows pairs a row with its next 16 only:
// such buckets' members are sorted first (lsh_big_* and a radix sort of them
// alone) and their records become the next 16 positions.
//
// Sorting all records by bucket and then all pairs, 524,288 rows, 16 bands (8.4
// million records): the hash and table passes took 285 to 330 us, the sort and
// its scans 550, and with 2.3 million different pairs their emission, sort and
// unique 400.  Here lsh_slot_kernel takes 259 to 306 us (the tables' atomics),
// lsh_member_kernel 56 to 73, lsh_base_kernel 35 and lsh_pair_kernel 258 for
// the 2.3 million pairs; the whole clustered product went from 7.16 to 6.49 ms
// (8,849 pairs) and from 4.78 to 4.07 ms (2.3 million).

constexpr int kLenBits = 24;  // of a record: members' count; above it their position
constexpr uint64_t kLenMask = (uint64_t(1) << kLenBits) - 1;
constexpr int kTicketBits = 31;
constexpr int64_t kWindowRows = 256;  // constrained buckets above this pair only
constexpr int64_t kWindow = 16;       // the next 16 rows

struct LshCursor {
  unsigned long long small, big, keys;  // members placed from the front, from the back, keys written
  int err;
};

__global__ void lsh_slot_kernel(const uint64_t* __restrict__ sig, int64_t n, int k, int band0, int nb, int r, int lg,
                                unsigned long long* __restrict__ tabs, uint32_t* __restrict__ cnts, uint64_t mask,
                                uint64_t* __restrict__ rec, LshCursor* __restrict__ cur) {
  // a block takes 256 >> lg rows x 2^lg bands: a row's values of neighbouring
  // bands are read together, and only 2^lg bands' tables are in use at a time
  const int64_t row_blocks = (n * (int64_t)(1 << lg) + 255) >> 8;
  const int64_t group = blockIdx.x / row_blocks;
  const int64_t i = (((blockIdx.x - group * row_blocks) << 8) + threadIdx.x) >> lg;
  int64_t b = (group << lg) + (threadIdx.x & ((1 << lg) - 1));
  const bool live = i < n && b < nb;
  if (!live) b = 0;
  unsigned long long h = ~0ULL;
  if (live) {
    const uint64_t* s = sig + i * k + (band0 + b) * r;
    h = 0;
    for (int t = 0; t < r; ++t) h = h * 0x9e3779b97f4a7c15ULL + s[t];
  }
  unsigned long long* tab = tabs + b * (int64_t)(mask + 2);
  uint64_t slot = mask + 1;  // the value ~0, the table's empty mark, has a slot of its own
  if (h != ~0ULL) {
    unsigned long long x = h ^ (h >> 29);
    x *= 0xbf58476d1ce4e5b9ULL;
    x ^= x >> 32;
    slot = x & mask;
    uint64_t probe = 0;
    for (; probe <= mask; ++probe) {
      const unsigned long long old = atomicCAS(tab + slot, ~0ULL, h);
      if (old == ~0ULL || old == h) break;
      slot = (slot + 1) & mask;
    }
    if (probe > mask) {  // table full: cannot happen with 2n slots
      atomicOr(&cur->err, 1);
      slot = 0;
    }
  }
  __syncwarp();
  const uint64_t id = (uint64_t)b * (mask + 2) + slot;
  // one ticket request per bucket and warp (rows of the same bucket are often
  // neighbours, and rows without entries share one bucket)
  const unsigned same = __match_any_sync(0xffffffffu, live ? (unsigned long long)id : ~0ULL);
  const int lane = threadIdx.x & 31, leader = __ffs(same) - 1;
  uint32_t ticket = 0;
  if (live && lane == leader) ticket = atomicAdd(cnts + id, (uint32_t)__popc(same));
  ticket = __shfl_sync(0xffffffffu, ticket, leader) + __popc(same & ((1u << lane) - 1u));
  if (live) rec[b * n + i] = id << kTicketBits | ticket;
}

// Slots [0, m): the position of the members of slots with at least two rows
// replaces the slot's value; windowed buckets take theirs from the back of the
// members' array (total entries), all others from the front.
__global__ void __launch_bounds__(256)
    lsh_base_kernel(const uint32_t* __restrict__ cnts, int64_t m, bool constrain, int64_t total,
                    unsigned long long* __restrict__ tabs, LshCursor* __restrict__ cur) {
  constexpr int U = 8;
  __shared__ uint32_t s_sum[8];
  __shared__ unsigned long long s_base;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int64_t s0 = blockIdx.x * (int64_t)(256 * U) + threadIdx.x;
  uint32_t c[U], sum = 0;
#pragma unroll
  for (int u = 0; u < U; ++u) c[u] = s0 + u * 256 < m ? cnts[s0 + u * 256] : 0;
#pragma unroll
  for (int u = 0; u < U; ++u) {
    if (c[u] < 2) c[u] = 0;
    if (constrain && c[u] > kWindowRows) {
      const unsigned long long o = atomicAdd(&cur->big, (unsigned long long)c[u]);
      tabs[s0 + u * 256] = (unsigned long long)(total - (int64_t)o - (int64_t)c[u]);
      c[u] = 0;
    }
    sum += c[u];
  }
  uint32_t inc = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t v = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += v;
  }
  if (lane == 31) s_sum[w] = inc;
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t t = 0;
    for (int v = 0; v < 8; ++v) {
      const uint32_t x = s_sum[v];
      s_sum[v] = t;
      t += x;
    }
    s_base = t ? atomicAdd(&cur->small, (unsigned long long)t) : 0;
  }
  __syncthreads();
  unsigned long long base = s_base + s_sum[w] + (inc - sum);
#pragma unroll
  for (int u = 0; u < U; ++u)
    if (c[u]) {
      tabs[s0 + u * 256] = base;
      base += c[u];
    }
}

__global__ void lsh_member_kernel(int64_t n, int nb, const unsigned long long* __restrict__ tabs,
                                  const uint32_t* __restrict__ cnts, uint64_t* __restrict__ rec,
                                  int32_t* __restrict__ members, LshCursor* __restrict__ cur) {
  const int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (q >= n * nb) return;
  const uint64_t v = rec[q], id = v >> kTicketBits;
  const uint64_t c = cnts[id];
  uint64_t info = 0;
  if (c >= 2) {
    const uint64_t base = tabs[id];
    members[base + (v & ((uint64_t(1) << kTicketBits) - 1))] = (int32_t)(q % n);
    if (c >= kLenMask) atomicOr(&cur->err, 2);  // windowed: the length is not read again
    info = base << kLenBits | (c < kLenMask ? c : kLenMask);
  }
  rec[q] = info;
}

// Members of the windowed buckets as keys (position of the bucket's room after
// `start`) << 31 | row, in any order: sorted they lie at their places.
__global__ void lsh_big_key_kernel(const uint64_t* __restrict__ rec, int64_t n, int64_t m, int64_t start,
                                   uint64_t* __restrict__ keys, LshCursor* __restrict__ cur) {
  const int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const uint64_t v = q < m ? rec[q] : 0;
  const bool big = (int64_t)(v & kLenMask) > kWindowRows;
  const unsigned vote = __ballot_sync(0xffffffffu, big);
  if (!vote) return;
  const int lane = threadIdx.x & 31;
  unsigned long long p = 0;
  if (lane == __ffs(vote) - 1) p = atomicAdd(&cur->keys, (unsigned long long)__popc(vote));
  p = __shfl_sync(0xffffffffu, p, __ffs(vote) - 1);
  if (big)
    keys[p + __popc(vote & ((1u << lane) - 1u))] =
        ((v >> kLenBits) - (uint64_t)start) << kTicketBits | (uint64_t)(q % n);
}

__global__ void lsh_big_place_kernel(const uint64_t* __restrict__ keys, int64_t c, int32_t* __restrict__ members) {
  const int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (p < c) members[p] = (int32_t)(keys[p] & ((uint64_t(1) << kTicketBits) - 1));
}

// A windowed bucket's record becomes the next 16 members after the row.
__global__ void lsh_big_window_kernel(uint64_t* __restrict__ rec, int64_t n, int64_t m, int64_t start,
                                      const uint64_t* __restrict__ keys, int64_t c) {
  const int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (q >= m) return;
  const uint64_t v = rec[q];
  if ((int64_t)(v & kLenMask) <= kWindowRows) return;
  const uint64_t bucket = (v >> kLenBits) - (uint64_t)start;
  const uint64_t key = bucket << kTicketBits | (uint64_t)(q % n);  // among them
  int64_t lo = (int64_t)bucket, hi = c - 1;
  while (lo < hi) {
    const int64_t mid = (lo + hi) >> 1;
    if (keys[mid] < key) lo = mid + 1; else hi = mid;
  }
  int64_t len = 0;
  while (len < kWindow && lo + 1 + len < c && keys[lo + 1 + len] >> kTicketBits == bucket) ++len;
  rec[q] = len ? (uint64_t)(start + lo + 1) << kLenBits | (uint64_t)len : 0;
}

constexpr int kPairBins = 9;  // members of a row's buckets <= 64, 128, .. 8192, more

// Members per row, and for rows of the last bin how many lie above the row.
// Rows without any take no bin.
__global__ void lsh_row_kernel(const uint64_t* __restrict__ rec, int64_t n, int bands,
                               const int32_t* __restrict__ members, int64_t* __restrict__ room,
                               int32_t* __restrict__ lists, unsigned long long* __restrict__ counts) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const int lane = threadIdx.x & 31;
  int64_t p = 0;
  int bin = -1;
  if (i < n) {
    for (int b = 0; b < bands; ++b) p += (int64_t)(rec[b * n + i] & kLenMask);
    if (p > 0) {
      bin = 0;
      while (bin < kPairBins - 1 && p > ((int64_t)64 << bin)) ++bin;
    }
    if (bin == kPairBins - 1) {
      p = 0;
      for (int b = 0; b < bands; ++b) {
        const uint64_t v = rec[b * n + i];
        const int32_t* mem = members + (v >> kLenBits);
        for (int64_t t = 0; t < (int64_t)(v & kLenMask); ++t) p += mem[t] > (int32_t)i;
      }
    }
    room[i] = p;
  }
  const unsigned same = __match_any_sync(0xffffffffu, bin);
  const int leader = __ffs(same) - 1;
  unsigned long long pos = 0;
  if (bin >= 0 && lane == leader) pos = atomicAdd(counts + bin, (unsigned long long)__popc(same));
  pos = __shfl_sync(0xffffffffu, pos, leader);
  if (bin >= 0) lists[(int64_t)bin * n + (int64_t)pos + __popc(same & ((1u << lane) - 1u))] = (int32_t)i;
}

template <int R, int W>
struct PairSmem {
  static constexpr int kCols = W == 1 ? 32 : 64;
  int64_t base[kCols];
  uint32_t key[32 * R * W];
  int32_t off[kCols + 1];
  uint32_t w_edge[W];
  int32_t w_cnt[W];
};

// One row of up to 32*R*W members per W warps (four rows per block for W = 1);
// the gather and the sort are row_sort_kernel's (spgemm_rows.cuh).  Members not
// above the row become ~0 and sort behind the others.
template <int R, int W>
__global__ void __launch_bounds__(W == 1 ? 128 : 32 * W)
    lsh_pair_kernel(const int32_t* __restrict__ rows, int64_t nrows, const uint64_t* __restrict__ rec, int64_t n,
                    int bands, const int32_t* __restrict__ members, const int64_t* __restrict__ room,
                    int32_t* __restrict__ part, int64_t* __restrict__ cnt) {
  using S = PairSmem<R, W>;
  constexpr int NW = 32 * R, U = 4;
  constexpr uint32_t kNone = 0xffffffffu;
  extern __shared__ __align__(16) unsigned char pair_smem[];
  const int lane = threadIdx.x & 31;
  const int w = W == 1 ? 0 : threadIdx.x >> 5, tid = W == 1 ? lane : threadIdx.x;
  S& M = reinterpret_cast<S*>(pair_smem)[W == 1 ? threadIdx.x >> 5 : 0];
  auto sync = [] {
    if (W == 1) __syncwarp(); else __syncthreads();
  };
  overlap_let_next();
  const int64_t slot = W == 1 ? blockIdx.x * (int64_t)4 + (threadIdx.x >> 5) : blockIdx.x;
  if (slot >= nrows) return;  // W == 1: whole warps, which share no barrier, and not the block's first
  const int64_t i = rows[slot];
  int P = 0;
  for (int b0 = 0; b0 < bands; b0 += S::kCols) {
    if (w == 0) {
      int32_t carry = 0;
#pragma unroll
      for (int h = 0; h < S::kCols; h += 32) {
        uint64_t v = 0;
        if (b0 + h + lane < bands) v = rec[(int64_t)(b0 + h + lane) * n + i];
        const int32_t len = (int32_t)(v & kLenMask);
        int32_t inc = len;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int32_t u = __shfl_up_sync(0xffffffffu, inc, o);
          if (lane >= o) inc += u;
        }
        M.base[h + lane] = (int64_t)(v >> kLenBits) - (carry + inc - len);
        M.off[h + lane + 1] = carry + inc;
        carry += __shfl_sync(0xffffffffu, inc, 31);
      }
      if (lane == 0) M.off[0] = 0;
    }
    sync();
    const int T = M.off[S::kCols];
    int j = 0;
    if (W > 1) {
      int hi = S::kCols;
      while (hi - j > 1) {
        const int mid = (j + hi) >> 1;
        if (M.off[mid] <= tid) j = mid; else hi = mid;
      }
    }
    for (int t0 = tid; t0 < T; t0 += 32 * W * U) {
      int64_t q[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int t = t0 + 32 * W * u;
        if (t < T)
          while (M.off[j + 1] <= t) ++j;
        q[u] = M.base[j] + t;
      }
      int32_t m[U];
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (t0 + 32 * W * u < T) m[u] = members[q[u]];
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (t0 + 32 * W * u < T) M.key[P + t0 + 32 * W * u] = m[u] > (int32_t)i ? (uint32_t)m[u] : kNone;
    }
    P += T;
    sync();
  }
  uint32_t key[R];
#pragma unroll
  for (int s = 0; s < R; ++s) {
    const int t = (w * R + s) * 32 + lane;
    key[s] = t < P ? M.key[t] : kNone;
  }
  block_sort_keys<R, W>(key, M.key, w, lane);
  uint32_t before = __shfl_up_sync(0xffffffffu, key[R - 1], 1);
  if (W > 1) {
    if (lane == 31) M.w_edge[w] = key[R - 1];
    __syncthreads();
    if (lane == 0 && w > 0) before = M.w_edge[w - 1];
  }
  if (tid == 0) before = kNone;  // the first key is a new one unless it is ~0
  uint32_t first = 0;
#pragma unroll
  for (int s = 0; s < R; ++s)
    first |= (key[s] != kNone && (s ? key[s - 1] : before) != key[s] ? 1u : 0u) << s;
  const int c = __popc(first);
  int incl = c;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int u = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += u;
  }
  int total = __shfl_sync(0xffffffffu, incl, 31), rank = incl - c;
  if (W > 1) {
    if (lane == 31) M.w_cnt[w] = incl;
    __syncthreads();
    total = 0;
#pragma unroll
    for (int v = 0; v < W; ++v) {
      const int q = M.w_cnt[v];
      if (v < w) rank += q;
      total += q;
    }
  }
  int32_t* out = part + room[i];
#pragma unroll
  for (int s = 0; s < R; ++s)
    if (first >> s & 1u) out[rank++] = (int32_t)key[s];
  if (tid == 0) cnt[i] = total;
  overlap_end();
}

// The longest rows' pairs as keys i << 32 | j at room[i] - room of the rows
// before them; one block per row.
__global__ void __launch_bounds__(256)
    lsh_long_key_kernel(const int32_t* __restrict__ rows, const int64_t* __restrict__ key_off,
                        const uint64_t* __restrict__ rec, int64_t n, int bands, const int32_t* __restrict__ members,
                        uint64_t* __restrict__ keys) {
  __shared__ unsigned long long s_pos;
  if (threadIdx.x == 0) s_pos = 0;
  __syncthreads();
  const int64_t i = rows[blockIdx.x], o = key_off[blockIdx.x];
  for (int b = 0; b < bands; ++b) {
    const uint64_t v = rec[(int64_t)b * n + i];
    const int32_t* mem = members + (v >> kLenBits);
    for (int64_t t = threadIdx.x; t < (int64_t)(v & kLenMask); t += 256)
      if (mem[t] > (int32_t)i)
        keys[o + (int64_t)atomicAdd(&s_pos, 1ULL)] = (uint64_t)i << 32 | (uint32_t)mem[t];
  }
}

__global__ void lsh_long_room_kernel(const int32_t* __restrict__ rows, int64_t c, const int64_t* __restrict__ room,
                                     int64_t* __restrict__ len) {
  const int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (q <= c) len[q] = q < c ? room[rows[q]] : 0;
}

// Unique ascending keys into their rows' rooms, and the rows' counts.
__global__ void lsh_long_place_kernel(const uint64_t* __restrict__ keys, const int64_t* __restrict__ count,
                                      const int64_t* __restrict__ room, int32_t* __restrict__ part,
                                      int64_t* __restrict__ cnt) {
  const int64_t m = *count;
  for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < m; p += (int64_t)gridDim.x * blockDim.x) {
    const uint64_t v = keys[p], i = v >> 32;
    int64_t lo = 0, hi = p;  // the row's first key
    while (lo < hi) {
      const int64_t mid = (lo + hi) >> 1;
      if (keys[mid] < i << 32) lo = mid + 1; else hi = mid;
    }
    part[room[i] + (p - lo)] = (int32_t)(uint32_t)v;
    if (p + 1 == m || keys[p + 1] >> 32 != i) cnt[i] = p - lo + 1;
  }
}

// The rows' partners to their final places; 8 lanes per row.
__global__ void lsh_list_kernel(const int32_t* __restrict__ part, const int64_t* __restrict__ room,
                                const int64_t* __restrict__ off, int64_t n, int64_t* __restrict__ pi,
                                int64_t* __restrict__ pj) {
  const int64_t i = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 3;
  if (i >= n) return;
  const int64_t o = off[i], c = off[i + 1] - o;
  const int32_t* from = part + room[i];
  for (int64_t t = threadIdx.x & 7; t < c; t += 8) {
    pi[o + t] = i;
    pj[o + t] = from[t];
  }
}

// Four consecutive pairs per warp, all loads of 32 hash functions in flight
// together; bound by the signatures' reads (one pair per warp took 401 us for
// 2.3 million pairs, k = 64, this 346).
__global__ void score_kernel(const uint64_t* __restrict__ sig, int k, const int64_t* __restrict__ pi,
                             const int64_t* __restrict__ pj, int64_t np, double* __restrict__ score) {
  constexpr int U = 4;
  const int64_t p0 = ((blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5) * U;
  const int lane = threadIdx.x & 31;
  if (p0 >= np) return;
  const uint64_t *si[U], *sj[U];
  int m[U];
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const int64_t p = p0 + u < np ? p0 + u : np - 1;
    si[u] = sig + pi[p] * k;
    sj[u] = sig + pj[p] * k;
    m[u] = 0;
  }
  for (int d0 = 0; d0 < k; d0 += 32) {
    const bool ok = d0 + lane < k;
    uint64_t x[U], y[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      x[u] = ok ? si[u][d0 + lane] : 0;
      y[u] = ok ? sj[u][d0 + lane] : 1;
    }
#pragma unroll
    for (int u = 0; u < U; ++u) m[u] += __popc(__ballot_sync(0xffffffffu, x[u] == y[u]));
  }
  int mine = 0;
#pragma unroll
  for (int u = 0; u < U; ++u) mine = lane == u ? m[u] : mine;
  if (lane < U && p0 + lane < np) score[p0 + lane] = (double)mine / (double)k;
}

template <typename I>
spops_status_t minhash_t(Context* ctx, Matrix* A, int k, uint64_t seed, uint64_t* sig) {
  std::vector<uint64_t> ha((size_t)k), hb((size_t)k);
  uint64_t s = seed;
  for (int d = 0; d < k; ++d) {  // the reference's LCG (spgemm_MinHashLSH.h:40-43, 134-141)
    s = s * 6364136223846793005ULL + 1442695040888963407ULL;
    ha[d] = (s >> 1) * 2 + 1;
    s = s * 6364136223846793005ULL + 1442695040888963407ULL;
    hb[d] = s;
  }
  SPOPS_TRY(ctx->scratch_reserve(2 * (size_t)k * 8 + 512));
  uint64_t* da = ctx->scratch.as<uint64_t>();
  uint64_t* db = da + k;
  SPOPS_CUDA(cudaMemcpyAsync(da, ha.data(), (size_t)k * 8, cudaMemcpyHostToDevice, ctx->stream));
  SPOPS_CUDA(cudaMemcpyAsync(db, hb.data(), (size_t)k * 8, cudaMemcpyHostToDevice, ctx->stream));
  if (A->rows > 0) {  // columns are checked to lie in [0, cols)
    auto kern = A->cols <= ((int64_t)1 << 32) ? minhash_kernel<I, true> : minhash_kernel<I, false>;
    kern<<<grid_for(A->rows * 32), 256, 0, ctx->stream>>>(A->row.as<I>(), A->col.as<I>(), A->rows, k, da, db, sig);
  }
  SPOPS_LAUNCH_CHECK();
  SPOPS_CUDA(cudaStreamSynchronize(ctx->stream));  // da/db live in scratch
  return SPOPS_OK;
}

}  // namespace

spops_status_t minhash_signatures(Context* ctx, Matrix* A, int k, uint64_t seed, uint64_t* sig) {
  if (A->format != SPOPS_FMT_CSR) return fail(SPOPS_ERR_INVALID, "MinHash needs a CSR matrix");
  if (k <= 0) return fail(SPOPS_ERR_INVALID, "MinHash: k must be positive");
  if (!A->plan.ready) SPOPS_TRY(csr_analyse(ctx, A));  // validates the pattern
  return A->itype == SPOPS_INDEX_I32 ? minhash_t<int32_t>(ctx, A, k, seed, sig)
                                     : minhash_t<int64_t>(ctx, A, k, seed, sig);
}

spops_status_t lsh_pairs(Context* ctx, const uint64_t* sig, int64_t n, int k, int bands, bool constrain,
                         PairSet* out) {
  out->release();
  if (n <= 0 || bands <= 0 || k <= 0 || k % bands) return SPOPS_OK;  // the reference returns no pairs
  if (n > INT32_MAX) return fail(SPOPS_ERR_UNSUPPORTED, "LSH: more than 2^31 rows");
  const int r = k / bands;
  cudaStream_t st = ctx->stream;
  Trace tr("lsh");
  ArenaScope scope(ctx);  // this call's temporaries come from the arena
  // the bands go through the tables in batches of up to 2^24 records (or one
  // band); a record itself takes 12 bytes until the end
  const int nb = (int)std::max<int64_t>(1, std::min<int64_t>(bands, ((int64_t)1 << 24) / n));
  uint64_t slots = 1;  // per band
  while (slots < 2 * (uint64_t)n) slots <<= 1;
  const int64_t records = (int64_t)bands * n, nslots = (int64_t)nb * (int64_t)(slots + 1);
  PoolBuf rec(ctx), members(ctx), tab(ctx), cnts(ctx), cur(ctx), tmp(ctx);
  SPOPS_TRY(rec.alloc((size_t)records * 8));
  SPOPS_TRY(members.alloc((size_t)records * 4));
  SPOPS_TRY(cur.alloc(sizeof(LshCursor)));
  SPOPS_CUDA(cudaMemsetAsync(cur.p, 0, sizeof(LshCursor), st));
  SPOPS_TRY(tab.alloc((size_t)nslots * 8));
  SPOPS_TRY(cnts.alloc((size_t)nslots * 4));
  LshCursor* dcur = cur.as<LshCursor>();
  for (int band0 = 0; band0 < bands; band0 += nb) {
    const int nbb = std::min(nb, bands - band0);
    const int64_t mb = (int64_t)nbb * n, ms = (int64_t)nbb * (int64_t)(slots + 1);
    uint64_t* brec = rec.as<uint64_t>() + (int64_t)band0 * n;
    SPOPS_CUDA(cudaMemsetAsync(tab.p, 0xff, (size_t)ms * 8, st));
    SPOPS_CUDA(cudaMemsetAsync(cnts.p, 0, (size_t)ms * 4, st));
    const int lg = nbb >= 4 ? 2 : nbb >= 2 ? 1 : 0;
    lsh_slot_kernel<<<grid_for(n << lg) * (unsigned)((nbb + (1 << lg) - 1) >> lg), 256, 0, st>>>(
        sig, n, k, band0, nbb, r, lg, tab.as<unsigned long long>(), cnts.as<uint32_t>(), slots - 1, brec, dcur);
    lsh_base_kernel<<<grid_for(ms, 2048), 256, 0, st>>>(cnts.as<uint32_t>(), ms, constrain, records,
                                                        tab.as<unsigned long long>(), dcur);
    lsh_member_kernel<<<grid_for(mb), 256, 0, st>>>(n, nbb, tab.as<unsigned long long>(), cnts.as<uint32_t>(), brec,
                                                    members.as<int32_t>(), dcur);
    SPOPS_LAUNCH_CHECK();
  }
  LshCursor h;
  SPOPS_CUDA(cudaMemcpyAsync(&h, cur.p, sizeof(h), cudaMemcpyDeviceToHost, st));
  SPOPS_CUDA(cudaStreamSynchronize(st));
  tr.mark(st, "buckets");
  if (h.err & 1) return fail(SPOPS_ERR_CUDA, "LSH: bucket table full");
  if (h.small + h.big == 0) return SPOPS_OK;
  if (h.big > 0) {  // windowed buckets: members ascending, records their next 16
    const int64_t nbig = (int64_t)h.big, start = records - nbig;
    int end_bit = kTicketBits + 1;
    while (end_bit < 64 && (uint64_t(1) << (end_bit - kTicketBits)) < (uint64_t)nbig) ++end_bit;
    PoolBuf k_in(ctx), k_out(ctx);
    SPOPS_TRY(k_in.alloc((size_t)nbig * 8));
    SPOPS_TRY(k_out.alloc((size_t)nbig * 8));
    lsh_big_key_kernel<<<grid_for(records), 256, 0, st>>>(rec.as<uint64_t>(), n, records, start, k_in.as<uint64_t>(),
                                                          dcur);
    SPOPS_LAUNCH_CHECK();
    size_t sb = 0;
    SPOPS_CUDA(cub::DeviceRadixSort::SortKeys(nullptr, sb, k_in.as<uint64_t>(), k_out.as<uint64_t>(), nbig, 0,
                                              end_bit, st));
    SPOPS_TRY(tmp.alloc(sb + 256));
    SPOPS_CUDA(cub::DeviceRadixSort::SortKeys(tmp.p, sb, k_in.as<uint64_t>(), k_out.as<uint64_t>(), nbig, 0, end_bit,
                                              st));
    lsh_big_place_kernel<<<grid_for(nbig), 256, 0, st>>>(k_out.as<uint64_t>(), nbig, members.as<int32_t>() + start);
    lsh_big_window_kernel<<<grid_for(records), 256, 0, st>>>(rec.as<uint64_t>(), n, records, start,
                                                             k_out.as<uint64_t>(), nbig);
    SPOPS_LAUNCH_CHECK();
  } else if (h.err & 2) {  // unconstrained: 2^47 pairs and more from one bucket
    return fail(SPOPS_ERR_ALLOC, "LSH: a bucket of 2^24 rows or more gives too many pairs");
  }
  // each row's room and bin
  PoolBuf room(ctx), cnt(ctx), lists(ctx), bins(ctx), off(ctx);
  SPOPS_TRY(room.alloc((size_t)(n + 1) * 8));
  SPOPS_TRY(cnt.alloc((size_t)(n + 1) * 8));
  SPOPS_TRY(off.alloc((size_t)(n + 1) * 8));
  SPOPS_TRY(lists.alloc((size_t)kPairBins * (size_t)n * 4));
  SPOPS_TRY(bins.alloc(kPairBins * 8));
  SPOPS_CUDA(cudaMemsetAsync(bins.p, 0, kPairBins * 8, st));
  SPOPS_CUDA(cudaMemsetAsync(cnt.p, 0, (size_t)(n + 1) * 8, st));
  SPOPS_CUDA(cudaMemsetAsync(room.as<int64_t>() + n, 0, 8, st));
  lsh_row_kernel<<<grid_for(n), 256, 0, st>>>(rec.as<uint64_t>(), n, bands, members.as<int32_t>(),
                                              room.as<int64_t>(), lists.as<int32_t>(),
                                              bins.as<unsigned long long>());
  SPOPS_LAUNCH_CHECK();
  size_t sb = 0;
  SPOPS_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, sb, room.as<int64_t>(), off.as<int64_t>(), n + 1, st));
  PoolBuf scan(ctx);
  SPOPS_TRY(scan.alloc(sb + 256));
  int64_t nlong = 0;
  unsigned long long hb[kPairBins];
  SPOPS_CUDA(cudaMemcpyAsync(hb, bins.p, sizeof(hb), cudaMemcpyDeviceToHost, st));
  // the longest rows' keys are laid out by their own rooms, before those become offsets
  SPOPS_CUDA(cub::DeviceScan::ExclusiveSum(scan.p, sb, room.as<int64_t>(), off.as<int64_t>(), n + 1, st));
  int64_t rooms = 0;
  SPOPS_CUDA(cudaMemcpyAsync(&rooms, off.as<int64_t>() + n, 8, cudaMemcpyDeviceToHost, st));
  SPOPS_CUDA(cudaStreamSynchronize(st));
  nlong = (int64_t)hb[kPairBins - 1];
  if (rooms == 0) return SPOPS_OK;
  PoolBuf part(ctx);
  SPOPS_TRY(part.alloc((size_t)rooms * 4));
  tr.mark(st, "rows");
  const int64_t* droom = off.as<int64_t>();
  OverlapChain chain(st);
  auto launch = [&](auto kern, int bin, size_t smem, int warps) -> spops_status_t {
    const int64_t c = (int64_t)hb[bin];
    if (c == 0) return SPOPS_OK;
    const int per = warps == 1 ? 4 : 1;
    SPOPS_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem * per));
    SPOPS_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, 100));
    SPOPS_CUDA(chain.launch(kern, (c + per - 1) / per, warps * per * 32, smem * per,
                            lists.as<int32_t>() + (int64_t)bin * n, c, rec.as<uint64_t>(), n, bands,
                            members.as<int32_t>(), droom, part.as<int32_t>(), cnt.as<int64_t>()));
    return SPOPS_OK;
  };
  SPOPS_TRY(launch(lsh_pair_kernel<16, 16>, 7, sizeof(PairSmem<16, 16>), 16));
  SPOPS_TRY(launch(lsh_pair_kernel<16, 8>, 6, sizeof(PairSmem<16, 8>), 8));
  SPOPS_TRY(launch(lsh_pair_kernel<16, 4>, 5, sizeof(PairSmem<16, 4>), 4));
  SPOPS_TRY(launch(lsh_pair_kernel<16, 2>, 4, sizeof(PairSmem<16, 2>), 2));
  SPOPS_TRY(launch(lsh_pair_kernel<16, 1>, 3, sizeof(PairSmem<16, 1>), 1));
  SPOPS_TRY(launch(lsh_pair_kernel<8, 1>, 2, sizeof(PairSmem<8, 1>), 1));
  SPOPS_TRY(launch(lsh_pair_kernel<4, 1>, 1, sizeof(PairSmem<4, 1>), 1));
  SPOPS_TRY(launch(lsh_pair_kernel<2, 1>, 0, sizeof(PairSmem<2, 1>), 1));
  if (nlong > 0) {  // one sort and one unique of the longest rows' pairs
    const int32_t* rows = lists.as<int32_t>() + (int64_t)(kPairBins - 1) * n;
    PoolBuf klen(ctx), koff(ctx), nsel(ctx), k_in(ctx), k_out(ctx), tmp2(ctx);
    SPOPS_TRY(klen.alloc((size_t)(nlong + 1) * 8));
    SPOPS_TRY(koff.alloc((size_t)(nlong + 1) * 8));
    SPOPS_TRY(nsel.alloc(8));
    lsh_long_room_kernel<<<grid_for(nlong + 1), 256, 0, st>>>(rows, nlong, room.as<int64_t>(), klen.as<int64_t>());
    SPOPS_LAUNCH_CHECK();
    size_t b1 = sb;  // nlong <= n
    SPOPS_CUDA(cub::DeviceScan::ExclusiveSum(scan.p, b1, klen.as<int64_t>(), koff.as<int64_t>(), nlong + 1, st));
    int64_t keys = 0;
    SPOPS_CUDA(cudaMemcpyAsync(&keys, koff.as<int64_t>() + nlong, 8, cudaMemcpyDeviceToHost, st));
    SPOPS_CUDA(cudaStreamSynchronize(st));
    if (keys > 0) {
      SPOPS_TRY(k_in.alloc((size_t)keys * 8));
      SPOPS_TRY(k_out.alloc((size_t)keys * 8));
      lsh_long_key_kernel<<<(unsigned)nlong, 256, 0, st>>>(rows, koff.as<int64_t>(), rec.as<uint64_t>(), n, bands,
                                                           members.as<int32_t>(), k_in.as<uint64_t>());
      SPOPS_LAUNCH_CHECK();
      int kend = 33;  // only the bits of i in use above 32
      while (kend < 64 && (int64_t(1) << (kend - 32)) < n) ++kend;
      size_t b2 = 0, b3 = 0;
      SPOPS_CUDA(cub::DeviceRadixSort::SortKeys(nullptr, b2, k_in.as<uint64_t>(), k_out.as<uint64_t>(), keys, 0, kend,
                                                st));
      SPOPS_CUDA(cub::DeviceSelect::Unique(nullptr, b3, k_out.as<uint64_t>(), k_in.as<uint64_t>(),
                                           nsel.as<int64_t>(), keys, st));
      SPOPS_TRY(tmp2.alloc(std::max(b2, b3) + 256));
      SPOPS_CUDA(cub::DeviceRadixSort::SortKeys(tmp2.p, b2, k_in.as<uint64_t>(), k_out.as<uint64_t>(), keys, 0, kend,
                                                st));
      SPOPS_CUDA(cub::DeviceSelect::Unique(tmp2.p, b3, k_out.as<uint64_t>(), k_in.as<uint64_t>(),
                                           nsel.as<int64_t>(), keys, st));
      lsh_long_place_kernel<<<std::min<unsigned>(grid_for(keys), 8192u), 256, 0, st>>>(
          k_in.as<uint64_t>(), nsel.as<int64_t>(), droom, part.as<int32_t>(), cnt.as<int64_t>());
      SPOPS_LAUNCH_CHECK();
    }
  }
  // final places (room's own values are done with)
  SPOPS_CUDA(cub::DeviceScan::ExclusiveSum(scan.p, sb, cnt.as<int64_t>(), room.as<int64_t>(), n + 1, st));
  int64_t nu = 0;
  SPOPS_CUDA(cudaMemcpyAsync(&nu, room.as<int64_t>() + n, 8, cudaMemcpyDeviceToHost, st));
  SPOPS_CUDA(cudaStreamSynchronize(st));
  tr.mark(st, "pairs");
  if (nu == 0) return SPOPS_OK;
  SPOPS_TRY(out->pi.alloc_cached(ctx, (size_t)nu * 8));
  SPOPS_TRY(out->pj.alloc_cached(ctx, (size_t)nu * 8));
  SPOPS_TRY(out->score.alloc_cached(ctx, (size_t)nu * 8));
  lsh_list_kernel<<<grid_for(n * 8), 256, 0, st>>>(part.as<int32_t>(), droom, room.as<int64_t>(), n,
                                                   out->pi.as<int64_t>(), out->pj.as<int64_t>());
  score_kernel<<<grid_for((nu + 3) / 4 * 32), 256, 0, st>>>(sig, k, out->pi.as<int64_t>(), out->pj.as<int64_t>(), nu,
                                                            out->score.as<double>());
  SPOPS_LAUNCH_CHECK();
  SPOPS_CUDA(cudaStreamSynchronize(st));
  tr.mark(st, "scores");
  out->count = nu;
  return SPOPS_OK;
}

}  // namespace spops
