// ME-TCF conversion on the GPU, one pass over the edges per phase.
//
// Output semantics follow the reference conversion bit for bit
// (DTC-SpMM/DTCSpMM_kernel.cu:107-419, DTC-SpMM/DTCSpMM.cpp:313-359):
//   window w = rows [w*H, min(w*H+H, M)); U_w = sorted distinct columns of w;
//   blockPartition[w] = ceil(|U_w|/W) (0 for empty windows);
//   edgeToColumn[e] = rank of col(e) in U_w; block = rank / W, slot = rank % W;
//   TCblocktileId entries of a block are stored in CSR edge order;
//   SparseAToX[b*W + slot] = column (0 in unused slots).
// The reference computes U_w and the per-block scatter with one thread per
// window (:234-240, :309-329).
//
// A window is the unit here too, but everything that a window needs fits a CTA's shared
// memory, so each phase reads every edge once or twice and writes it once (a global radix
// sort moves 16 bytes per edge and pass: five passes for the ranks and three for the
// blocks, with the passes around them 3.8 ms for R-MAT 2^20, 32 M edges, of which the
// edges' own bytes are 0.13 ms; here 1.0 ms: ranks 0.42, places 0.51). By window:
//   ranks, up to 512 edges: one warp sorts packed (column, edge) keys in registers
//     (bitonic, neighbours by shuffles) and reads the ranks off the order (up to 256 where
//     column and edge need more than 32 bits); up to 2048: the same by 128 threads
//   ranks, larger: 1024 threads mark the columns in a bitmap (2^20 columns per sweep over
//     the window) and count the bits before each (a whole CTA per SM, the longest first);
//     where the columns take many sweeps they sort windows of up to 16384 edges instead
//   places, up to 1024 edges: one warp marks the cells of every block and counts the marks
//     before each; larger: a warp per 128 blocks does so, which finds its part of each row
//     by binary search
//   places where some row's ranks do not ascend (unsorted or repeated columns): the window's
//     edges sorted by (block, edge), by one warp up to 1024, 1024 threads up to 16384, several
//     such CTAs that share out the blocks beyond
//   places in windows of more than 32 rows: a global radix sort
// The lines: a sort of 2048 keys beats clearing and counting a bitmap of 2^20 columns (5 us)
// up to there; further ones beside the code.
// Bound: instruction issue and the latency of dependent loads; DRAM is at a fifth.
#include <algorithm>
#include <cub/cub.cuh>
#include "common.cuh"

namespace dtc {
namespace {

constexpr int kGroup = 128;              // threads of a CTA: four windows, or one middle window
constexpr int kWarpFill = 1024;          // windows up to here: places by one warp
constexpr int kLeftBytes = kWarpFill * 5;  // a warp that sorts such a window: keys, tile ids
constexpr int kThreads = 1024;           // threads of a large window
constexpr int kSweepCols = 1 << 20;      // columns per sweep of a large window's bitmap
constexpr int kSortBits = 14, kSortEdges = 1 << kSortBits;  // edges that a large CTA sorts
constexpr int kMergeWarps = 16;          // warps of it that merge repeated entries
constexpr int kPartBlocks = 8192;        // blocks of a part of a huge window, at most
constexpr int kPartSort = 8192, kPartEdges = 6144;  // edges of a part: sorted at a time, on average
constexpr int kMaxH = 256;               // rows of a window (block_h * block_w <= 256)
constexpr int kUnitH = 32;               // rows up to which a warp takes part of a window

template <typename K>
struct Cap {
  static constexpr int kEdges = 2048;  // ranks by 128 threads
  static constexpr int kBits = 11;
  static constexpr int kWarp = sizeof(K) == 4 ? 512 : 256;  // ranks by one warp (registers)
};
// Bytes of a group: keys, 16-bit ranks and row starts of a middle window, or four
// warps' scratch.
constexpr int kCells = 4160;  // bytes of a warp's cell masks (130 blocks of 256 cells)
constexpr int kWarpBytes = kCells * 3 / 2 + (2 * kUnitH + 1) * 4 + 12;  // masks, places, rows
template <typename K>
constexpr int group_bytes() {
  return std::max(Cap<K>::kEdges * ((int)sizeof(K) + 2) + (kMaxH + 1) * 4 + 60, 4 * kWarpBytes);
}
static_assert(Cap<uint32_t>::kWarp * 2 + (kMaxH + 1) * 4 <= kWarpBytes && kWarpBytes % 16 == 0 &&
              kCells >= (kWarpFill / 8 + 1) * 32, "warp scratch");
constexpr int kPer = 16;      // windows per CTA at most, by one warp each
// Up to kLane edges per window on average, a lane takes a window of up to kLane edges: a warp
// per window waits for memory most of the time. Whole conversion of 2^24 rows of 4 edges, a
// warp / a lane per window: one row per window 33 / 1.9 ms, two 17 / 1.8, four 8.8 / 2.2.
constexpr int kLane = 16;
inline bool tiny_windows(int64_t nnz, int32_t nwin) { return nnz <= (int64_t)kLane * nwin; }
// (count_sorted: its keys, ranks, rows)
constexpr int kLargeBytes =
    kSweepCols / 8 + kSweepCols / 64 * 2 + kSweepCols / 32768 * 4 + (kMaxH + 1) * 4 + 256;

constexpr int log2_of(int n) { return n > 1 ? 1 + log2_of(n / 2) : 0; }
inline int bits_for(uint64_t n) {  // bits to represent values in [0, n)
  int b = 0;
  while (b < 63 && (1ull << b) < n) ++b;
  return b < 1 ? 1 : b;
}

struct Csr {
  const int32_t* col;
  const int32_t* rowptr;
  int32_t M, nwin, H, W;
  int64_t nnz;
  int32_t shift;  // log2 W, or -1
  __device__ __forceinline__ int32_t block(int32_t rank) const {
    return shift >= 0 ? rank >> shift : rank / W;
  }
  __device__ __forceinline__ int32_t slot(int32_t rank) const {
    return shift >= 0 ? rank & (W - 1) : rank % W;
  }
};

__device__ __forceinline__ void window_edges(const Csr& a, int32_t w, int32_t& e0, int32_t& n) {
  const int64_t r0 = (int64_t)w * a.H, r1 = min(r0 + a.H, (int64_t)a.M);
  e0 = __ldg(a.rowptr + r0);
  const int32_t e1 = __ldg(a.rowptr + r1);
  n = e1 - e0;
  if (e0 < 0 || e1 > a.nnz || n < 0) n = 0;  // invalid CSR: reported by k_list
}

// The i-th of the listed windows, those of more than kHuge edges first.
constexpr int kHuge = 16384;
__device__ __forceinline__ int32_t listed(const int32_t* count, const int32_t* list, int32_t room,
                                          int32_t i) {
  const int32_t huge = __ldg(count);
  return __ldg(list + (i < huge ? i : room - 1 - (i - huge)));
}
__device__ __forceinline__ int32_t many_listed(const int32_t* count, int32_t room) {
  return (int32_t)min((int64_t)__ldg(count) + __ldg(count + 1), (int64_t)room);
}

// Lists the windows of more than mid_cap edges (mid_list) and of more than `cap`, those of
// more than kHuge from the front and the others from the back (count[0], count[1]); with `bad`,
// checks the row pointer (rowptr[0] == 0, non-decreasing, rowptr[M] == nnz) and sets its bits.
// In phase 2 (`rwo`) also lists their units of `unit` blocks, (window, first block), and clears
// `mixed`.
__global__ void k_list(const Csr a, int32_t cap, int32_t mid_cap, int32_t* count, int32_t* list,
                       int32_t* mid_count, int32_t* mid_list, int32_t mid_room, uint32_t* bad,
                       int32_t room, const int32_t* rwo, int32_t unit, int32_t* units,
                       int2* unit_list, int64_t unit_room, uint8_t* mixed) {
  const int32_t w = blockIdx.x * blockDim.x + threadIdx.x;
  if (w < a.nwin) {
    if (mixed) mixed[w] = 0;
    int32_t e0, n;
    window_edges(a, w, e0, n);
    if (n > cap) {
      const int32_t at = n > kHuge ? atomicAdd(count, 1) : room - 1 - atomicAdd(count + 1, 1);
      const bool in = at >= 0 && at < room;  // (a valid CSR cannot have more)
      if (in) list[at] = w;
      if (in && rwo) {
        const int32_t nb = rwo[w + 1] - rwo[w], many = unit ? (nb + unit - 1) / unit : 0;
        const int32_t u = atomicAdd(units, many);
        for (int32_t i = 0; i < many && u + i < unit_room; ++i)
          unit_list[u + i] = make_int2(w, i * unit);
      }
    } else if (n > mid_cap) {
      const int32_t at = atomicAdd(mid_count, 1);
      if (at < mid_room) mid_list[at] = w;
    }
  }
  if (bad) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t r = w; r <= a.M; r += stride) {
      const int32_t v = a.rowptr[r];
      if (r == 0 && v != 0) atomicOr(bad, 1u);
      if (r == a.M && v != a.nnz) atomicOr(bad, 2u);
      if (r < a.M && a.rowptr[r + 1] < v) atomicOr(bad, 4u);
    }
  }
}

// mixed[w] = 1 for each window of more than kWarpFill edges where the ranks of some row do
// not ascend (unsorted or repeated columns), and *any: one pass over the edges, eight per thread.
__global__ void k_mixed(const Csr a, const int32_t* __restrict__ e2c,
                        const int32_t* __restrict__ e2r, uint8_t* mixed, int32_t* any) {
  const int64_t e0 = (int64_t)blockIdx.x * blockDim.x * 8 + threadIdx.x;
  int32_t c[8], d[8], r[8], q[8];
#pragma unroll
  for (int v = 0; v < 8; ++v) {
    const int64_t e = e0 + v * blockDim.x;
    const bool in = e > 0 && e < a.nnz;
    c[v] = in ? __ldg(e2c + e - 1) : 0;
    d[v] = in ? __ldg(e2c + e) : 1;
    r[v] = in ? __ldg(e2r + e - 1) : 0;
    q[v] = in ? __ldg(e2r + e) : 1;
  }
  bool found = false;
#pragma unroll
  for (int v = 0; v < 8; ++v)
    if (c[v] >= d[v] && r[v] == q[v]) {
      mixed[q[v] / a.H] = 1;
      found = true;
    }
  // (a store per CTA: one per edge waits for the word in L2)
  if (__syncthreads_or(found) && threadIdx.x == 0) *any = 1;
}

// ------------------------------------------------------------- group helpers
// The last row r of `rows` whose start is at or before local edge i.
__device__ __forceinline__ int row_of(const int32_t* start, int rows, int32_t i) {
  int lo = 0, hi = rows;
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (start[mid] <= i) lo = mid; else hi = mid;
  }
  return lo;
}

// Exclusive sum of x over the group's threads (s: kGroup / 32 words); *total = sum.
__device__ __forceinline__ int group_scan(int x, int t, int32_t* s, int* total) {
  int v = x;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int u = __shfl_up_sync(0xffffffffu, v, o);
    if ((t & 31) >= o) v += u;
  }
  if ((t & 31) == 31) s[t >> 5] = v;
  __syncthreads();
  int before = 0, sum = 0;
#pragma unroll
  for (int i = 0; i < kGroup / 32; ++i) {
    if (i < (t >> 5)) before += s[i];
    sum += s[i];
  }
  *total = sum;
  __syncthreads();
  return before + v - x;
}

// The same over the whole CTA (s: kThreads / 32 words).
__device__ __forceinline__ int cta_scan(int x, int32_t* s, int* total) {
  const int t = threadIdx.x;
  int v = x;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int u = __shfl_up_sync(0xffffffffu, v, o);
    if ((t & 31) >= o) v += u;
  }
  if ((t & 31) == 31) s[t >> 5] = v;
  __syncthreads();
  int before = 0, sum = 0;
#pragma unroll
  for (int i = 0; i < kThreads / 32; ++i) {
    if (i < (t >> 5)) before += s[i];
    sum += s[i];
  }
  *total = sum;
  __syncthreads();
  return before + v - x;
}

// Ascending bitonic sort of 32 E keys per warp over T threads (a warp, or the CTA):
// thread t holds elements t E .. t E + E - 1. Distances below E are between a thread's
// own registers, below 32 E between lanes, the others through `buf` (T E keys).
template <typename K, int E, int T>
__device__ __forceinline__ void reg_bitonic(K (&x)[E], int t, K* buf) {
#pragma unroll
  for (int k = 2; k < E; k <<= 1)
#pragma unroll
    for (int j = k >> 1; j > 0; j >>= 1)
#pragma unroll
      for (int i = 0; i < E; ++i)
        if ((i & j) == 0) {
          const K lo = min(x[i], x[i | j]), hi = max(x[i], x[i | j]);
          x[i] = (i & k) == 0 ? lo : hi;
          x[i | j] = (i & k) == 0 ? hi : lo;
        }
  // (loops from here on: unrolled, the steps of all sizes are beyond the instruction
  // cache, and the kernel took four times as long)
#pragma unroll 1
  for (int k = E; k <= T * E; k <<= 1) {
    const bool up = ((t * E) & k) == 0;  // the run of k ascends
#pragma unroll 1
    for (int d = k / E / 2; d > 0; d >>= 1) {
      const bool keep_min = up == ((t & d) == 0);
      if (T > 32 && d >= 32) {
        __syncthreads();
#pragma unroll
        for (int i = 0; i < E; ++i) buf[i * T + t] = x[i];
        __syncthreads();
#pragma unroll
        for (int i = 0; i < E; ++i) {
          const K y = buf[i * T + (t ^ d)];
          x[i] = (x[i] < y) == keep_min ? x[i] : y;
        }
      } else {
#pragma unroll
        for (int i = 0; i < E; ++i) {
          const K y = __shfl_xor_sync(0xffffffffu, x[i], d);
          x[i] = (x[i] < y) == keep_min ? x[i] : y;
        }
      }
    }
#pragma unroll
    for (int j = E / 2; j > 0; j >>= 1)
#pragma unroll
      for (int i = 0; i < E; ++i)
        if ((i & j) == 0) {
          const K p = x[i], q = x[i | j];
          const bool swap = (q < p) == up;  // (equal keys: none, or two paddings)
          x[i] = swap ? q : p;
          x[i | j] = swap ? p : q;
        }
  }
}

// ------------------------------------------------------------------- phase 1
template <typename K, int E>
__device__ __forceinline__ void count_warp(const Csr& a, int32_t w, int32_t e0, int32_t n,
                                           uint8_t* sm, int lane, int32_t* e2c, int32_t* e2r,
                                           int32_t* bp, uint32_t* bad) {
  constexpr int B = 9;  // bits of an edge's place
  uint16_t* rank = reinterpret_cast<uint16_t*>(sm);
  int32_t* start = reinterpret_cast<int32_t*>(sm + Cap<K>::kWarp * 2);
  const int64_t r0 = (int64_t)w * a.H;
  const int rows = (int)min((int64_t)a.H, a.M - r0);
  for (int r = lane; r < rows; r += 32) start[r] = __ldg(a.rowptr + r0 + r) - e0;
  K x[E];
#pragma unroll
  for (int i = 0; i < E; ++i) {  // (any order will do: loaded coalesced)
    const int e = i * 32 + lane;
    x[i] = (K)~(K)0;
    if (e < n) {
      int32_t c = __ldg(a.col + e0 + e);
      if (c < 0 || c >= a.M) {
        atomicOr(bad, 8u);
        c = 0;
      }
      x[i] = ((K)(uint32_t)c << B) | (K)e;
    }
  }
  reg_bitonic<K, E, 32>(x, lane, nullptr);
  const K before = __shfl_up_sync(0xffffffffu, x[E - 1], 1);
  int mine = 0;
#pragma unroll
  for (int i = 0; i < E; ++i) {
    const bool first = i == 0 && lane == 0;
    mine += lane * E + i < n && (first || (x[i] >> B) != ((i ? x[i ? i - 1 : 0] : before) >> B));
  }
  int s = mine;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int u = __shfl_up_sync(0xffffffffu, s, o);
    if (lane >= o) s += u;
  }
  int r = s - mine - 1;
#pragma unroll
  for (int i = 0; i < E; ++i) {
    const bool first = i == 0 && lane == 0;
    if (lane * E + i < n) {
      r += first || (x[i] >> B) != ((i ? x[i ? i - 1 : 0] : before) >> B);
      rank[(int)(x[i] & (K)((1 << B) - 1))] = (uint16_t)r;
    }
  }
  __syncwarp();
  for (int i = lane; i < n; i += 32) {
    e2c[e0 + i] = rank[i];
    e2r[e0 + i] = (int32_t)(r0 + row_of(start, rows, i));
  }
  if (lane == 31) bp[w] = (s + a.W - 1) / a.W;
  __syncwarp();
}

template <typename K, int E>
__device__ __forceinline__ void count_small(const Csr& a, int32_t w, int32_t e0, int32_t n,
                                            uint8_t* sm, int t, int32_t* e2c, int32_t* e2r,
                                            int32_t* bp, uint32_t* bad) {
  constexpr int B = Cap<K>::kBits;
  static_assert(E * kGroup <= Cap<K>::kEdges, "keys fit");
  K* key = reinterpret_cast<K*>(sm);
  uint16_t* rank = reinterpret_cast<uint16_t*>(key + Cap<K>::kEdges);
  int32_t* start = reinterpret_cast<int32_t*>(rank + Cap<K>::kEdges);
  int32_t* part = start + kMaxH + 1;
  const int64_t r0 = (int64_t)w * a.H;
  const int rows = (int)min((int64_t)a.H, a.M - r0);
  for (int r = t; r < rows; r += kGroup) start[r] = __ldg(a.rowptr + r0 + r) - e0;
  K x[E];
#pragma unroll
  for (int i = 0; i < E; ++i) {
    const int e = i * kGroup + t;
    x[i] = (K)~(K)0;
    if (e < n) {
      int32_t c = __ldg(a.col + e0 + e);
      if (c < 0 || c >= a.M) {
        atomicOr(bad, 8u);
        c = 0;
      }
      x[i] = ((K)(uint32_t)c << B) | (K)e;
    }
  }
  reg_bitonic<K, E, kGroup>(x, t, key);
  __syncthreads();
  key[t] = x[E - 1];  // the last key of each thread, for the next one
  __syncthreads();
  const K before = t ? key[t - 1] : 0;
  int mine = 0;
#pragma unroll
  for (int i = 0; i < E; ++i)
    mine += t * E + i < n &&
            ((i == 0 && t == 0) || (x[i] >> B) != ((i ? x[i ? i - 1 : 0] : before) >> B));
  int total;
  int r = group_scan(mine, t, part, &total) - 1;
#pragma unroll
  for (int i = 0; i < E; ++i)
    if (t * E + i < n) {
      r += (i == 0 && t == 0) || (x[i] >> B) != ((i ? x[i ? i - 1 : 0] : before) >> B);
      rank[(int)(x[i] & (K)((1 << B) - 1))] = (uint16_t)r;
    }
  __syncthreads();
  for (int i = t; i < n; i += kGroup) {
    e2c[e0 + i] = rank[i];
    e2r[e0 + i] = (int32_t)(r0 + row_of(start, rows, i));
  }
  if (t == 0) bp[w] = (total + a.W - 1) / a.W;
  __syncthreads();
}

// A window of up to kThreads * E edges by a whole CTA: sorted by column, as count_small.
template <int E>
__device__ void count_sorted(const Csr& a, int32_t w, int32_t e0, int32_t n, uint8_t* sm,
                             int32_t* e2c, int32_t* e2r, int32_t* bp, uint32_t* bad) {
  constexpr int B = kSortBits;
  uint64_t* key = reinterpret_cast<uint64_t*>(sm);
  uint16_t* rank = reinterpret_cast<uint16_t*>(key + kSortEdges);
  int32_t* start = reinterpret_cast<int32_t*>(rank + kSortEdges);
  int32_t* part = start + kMaxH + 1;
  const int t = threadIdx.x;
  const int64_t r0 = (int64_t)w * a.H;
  const int rows = (int)min((int64_t)a.H, a.M - r0);
  for (int r = t; r < rows; r += kThreads) start[r] = __ldg(a.rowptr + r0 + r) - e0;
  uint64_t x[E];
#pragma unroll
  for (int i = 0; i < E; ++i) {
    const int e = i * kThreads + t;
    x[i] = ~0ull;
    if (e < n) {
      int32_t c = __ldg(a.col + e0 + e);
      if (c < 0 || c >= a.M) {
        atomicOr(bad, 8u);
        c = 0;
      }
      x[i] = (uint64_t)(uint32_t)c << B | (uint32_t)e;
    }
  }
  reg_bitonic<uint64_t, E, kThreads>(x, t, key);
  __syncthreads();
  key[t] = x[E - 1];  // the last key of each thread, for the next one
  __syncthreads();
  const uint64_t before = t ? key[t - 1] : 0;
  uint32_t firsts = 0;
#pragma unroll
  for (int i = 0; i < E; ++i)
    firsts |= (uint32_t)(t * E + i < n && ((i == 0 && t == 0) ||
                                           (x[i] >> B) != ((i ? x[i ? i - 1 : 0] : before) >> B)))
              << i;
  int total;
  const int r = cta_scan(__popc(firsts), part, &total) - 1;
#pragma unroll
  for (int i = 0; i < E; ++i)
    if (t * E + i < n)
      rank[(int)(x[i] & (kSortEdges - 1))] = (uint16_t)(r + __popc(firsts & ((2u << i) - 1)));
  __syncthreads();
  for (int i = t; i < n; i += kThreads) {
    e2c[e0 + i] = rank[i];
    e2r[e0 + i] = (int32_t)(r0 + row_of(start, rows, i));
  }
  if (t == 0) bp[w] = (total + a.W - 1) / a.W;
  __syncthreads();
}

__device__ void count_large(const Csr& a, int32_t w, int32_t e0, int32_t n, uint8_t* sm,
                            int32_t* e2c, int32_t* e2r, int32_t* bp, uint32_t* bad) {
  uint32_t* bm = reinterpret_cast<uint32_t*>(sm);                     // kSweepCols bits
  uint16_t* pre = reinterpret_cast<uint16_t*>(bm + kSweepCols / 32);  // set bits before 64 columns,
  int32_t* sup = reinterpret_cast<int32_t*>(pre + kSweepCols / 64);   // counted from 2^15 columns
  int32_t* start = sup + kSweepCols / 32768;
  int32_t* part = start + kMaxH + 1;
  const int t = threadIdx.x;
  const int64_t r0 = (int64_t)w * a.H;
  const int rows = (int)min((int64_t)a.H, a.M - r0);
  for (int r = t; r < rows; r += kThreads) start[r] = __ldg(a.rowptr + r0 + r) - e0;
  int32_t distinct = 0;
  for (int64_t c0 = 0; c0 < a.M; c0 += kSweepCols) {
    const int32_t cols = (int32_t)min((int64_t)kSweepCols, a.M - c0);
    const int words = (cols + 1023) / 1024 * 32;
    for (int i = t; i < words / 4; i += kThreads)
      reinterpret_cast<uint4*>(bm)[i] = make_uint4(0, 0, 0, 0);
    __syncthreads();
    for (int32_t i = t; i < n; i += 8 * kThreads) {  // eight loads under way per thread
      int32_t c[8];
#pragma unroll
      for (int v = 0; v < 8; ++v)
        c[v] = i + v * kThreads < n ? __ldg(a.col + e0 + i + v * kThreads) : -1;
#pragma unroll
      for (int v = 0; v < 8; ++v) {
        if (i + v * kThreads >= n) break;
        if (c0 == 0 && (c[v] < 0 || c[v] >= a.M)) {
          atomicOr(bad, 8u);
          c[v] = 0;
        }
        const uint32_t x = (uint32_t)(c[v] - (int32_t)c0);
        if (x < (uint32_t)cols) atomicOr(bm + (x >> 5), 1u << (x & 31));
      }
    }
    __syncthreads();
    // (neighbouring threads take neighbouring words: with a run of words per thread every
    // load was a 32-way bank conflict, 35 us per window)
    const int pairs = words / 2;
    for (int q = t; q < pairs; q += kThreads)
      pre[q] = (uint16_t)__popcll(reinterpret_cast<const unsigned long long*>(bm)[q]);
    __syncthreads();
    constexpr int V = kSweepCols / 64 / kThreads;  // counts per thread
    static_assert(V == 16 && kThreads / 32 == kSweepCols / 32768, "a warp per 2^15 columns");
    uint4 g[2] = {make_uint4(0, 0, 0, 0), make_uint4(0, 0, 0, 0)};
    if (t * V < pairs) {
      g[0] = reinterpret_cast<const uint4*>(pre)[2 * t];
      g[1] = reinterpret_cast<const uint4*>(pre)[2 * t + 1];
    }
    uint32_t* const u = reinterpret_cast<uint32_t*>(g);
    int mine = 0;
#pragma unroll
    for (int v = 0; v < V / 2; ++v) mine += (u[v] & 0xffffu) + (u[v] >> 16);
    int total;
    int before = cta_scan(mine, part, &total);
    const int first = __shfl_sync(0xffffffffu, before, 0);  // set bits before the warp's columns
    if ((t & 31) == 0) sup[t >> 5] = distinct + first;
    before -= first;  // (at most 2^15)
#pragma unroll
    for (int v = 0; v < V / 2; ++v) {
      const uint32_t lo = u[v] & 0xffffu, hi = u[v] >> 16;
      u[v] = (uint32_t)before | (uint32_t)(before + lo) << 16;
      before += lo + hi;
    }
    if (t * V < pairs) {
      reinterpret_cast<uint4*>(pre)[2 * t] = g[0];
      reinterpret_cast<uint4*>(pre)[2 * t + 1] = g[1];
    }
    __syncthreads();
    int row = 0;  // of the thread's edge: it only moves on
    for (int32_t i = t; i < n; i += 8 * kThreads) {
      int32_t c[8];
#pragma unroll
      for (int v = 0; v < 8; ++v)
        c[v] = i + v * kThreads < n ? __ldg(a.col + e0 + i + v * kThreads) : -1;
#pragma unroll
      for (int v = 0; v < 8; ++v) {
        const int32_t e = i + v * kThreads;
        if (e >= n) break;
        const uint32_t x = (uint32_t)(c[v] - (int32_t)c0);
        if (x < (uint32_t)cols)
          e2c[e0 + e] = sup[x >> 15] + pre[x >> 6] +
                        __popcll(reinterpret_cast<const unsigned long long*>(bm)[x >> 6] &
                                 ((1ull << (x & 63)) - 1));
        if (c0 == 0) {
          while (row + 1 < rows && start[row + 1] <= e) ++row;
          e2r[e0 + e] = (int32_t)(r0 + row);
        }
      }
    }
    distinct += total;
    __syncthreads();
  }
  if (t == 0) bp[w] = (distinct + a.W - 1) / a.W;
}

// A window of at most kLane edges by one lane: an edge's rank is the number of distinct
// columns below its own, counted over the registers. `most`: edges of the warp's longest.
__device__ __forceinline__ void count_lane(const Csr& a, int32_t w, int32_t e0, int32_t n,
                                           int32_t most, int32_t* e2c, int32_t* e2r, int32_t* bp,
                                           uint32_t* bad) {
  int32_t c[kLane];
  uint32_t firsts = 0;  // edges whose column none before has
#pragma unroll
  for (int j = 0; j < kLane; ++j) {
    c[j] = INT32_MAX;
    if (j < most && j < n) {
      c[j] = __ldg(a.col + e0 + j);
      if (c[j] < 0 || c[j] >= a.M) {
        atomicOr(bad, 8u);
        c[j] = 0;
      }
    }
  }
#pragma unroll
  for (int j = 0; j < kLane; ++j)
    if (j < most) {
      bool first = j < n;
#pragma unroll
      for (int i = 0; i < j; ++i) first &= c[i] != c[j];
      firsts |= (uint32_t)first << j;
    }
  const int64_t r0 = (int64_t)w * a.H;
  const int rows = (int)min((int64_t)a.H, a.M - r0);
  int32_t row = -1, end = e0;  // end of that row
#pragma unroll
  for (int j = 0; j < kLane; ++j)
    if (j < most && j < n) {
      int rank = 0;
#pragma unroll
      for (int i = 0; i < kLane; ++i) rank += (firsts >> i & 1) && c[i] < c[j];
      e2c[e0 + j] = rank;
      while (end <= e0 + j && row + 1 < rows) end = __ldg(a.rowptr + r0 + ++row + 1);
      e2r[e0 + j] = (int32_t)(r0 + row);
    }
  bp[w] = (__popc(firsts) + a.W - 1) / a.W;
}

// Matrices of few edges per window: 32 windows per warp, those of more than kLane edges one
// after the other by all its lanes.
template <typename K>
__global__ void __launch_bounds__(kGroup, 6)
    k_count_tiny(const Csr a, int32_t* __restrict__ e2c, int32_t* __restrict__ e2r,
                 int32_t* __restrict__ bp, uint32_t* bad) {
  __shared__ __align__(16) uint8_t sm[4 * kWarpBytes];
  const int lane = threadIdx.x & 31;
  uint8_t* const wsm = sm + (threadIdx.x / 32) * kWarpBytes;
  const int64_t w = (int64_t)blockIdx.x * kGroup + threadIdx.x;
  int32_t e0 = 0, n = 0;
  if (w < a.nwin) window_edges(a, (int32_t)w, e0, n);
  const int32_t most = __reduce_max_sync(0xffffffffu, n <= kLane ? n : 0);
  if (w < a.nwin && n <= kLane) count_lane(a, (int32_t)w, e0, n, most, e2c, e2r, bp, bad);
  for (uint32_t m = __ballot_sync(0xffffffffu, n > kLane && n <= Cap<K>::kWarp); m; m &= m - 1) {
    const int src = __ffs(m) - 1;
    const int32_t ws = (int32_t)(w - lane + src), es = __shfl_sync(0xffffffffu, e0, src),
                  ns = __shfl_sync(0xffffffffu, n, src);
    if (ns <= 128) count_warp<K, 4>(a, ws, es, ns, wsm, lane, e2c, e2r, bp, bad);
    else if (ns <= 256) count_warp<K, 8>(a, ws, es, ns, wsm, lane, e2c, e2r, bp, bad);
    else if constexpr (sizeof(K) == 4)
      count_warp<K, 16>(a, ws, es, ns, wsm, lane, e2c, e2r, bp, bad);
  }
}

// The first mid_ctas CTAs take the listed middle windows, the others `per` windows each,
// one per warp at a time.
template <typename K>
__global__ void __launch_bounds__(kGroup, 8)
    k_count(const Csr a, const int32_t* __restrict__ mid_count,
            const int32_t* __restrict__ mid_list, int32_t mid_room, int mid_ctas, int per,
            int32_t* __restrict__ e2c, int32_t* __restrict__ e2r, int32_t* __restrict__ bp,
            uint32_t* bad) {
  __shared__ __align__(16) uint8_t sm[group_bytes<K>()];
  __shared__ int next;
  int32_t e0, n;
  const int t = threadIdx.x, lane = t & 31;
  if ((int)blockIdx.x < mid_ctas) {
    const int32_t many = min(__ldg(mid_count), mid_room);
    for (int32_t i = blockIdx.x; i < many; i += mid_ctas) {
      const int32_t w = __ldg(mid_list + i);
      window_edges(a, w, e0, n);
      if (n <= 8 * kGroup)
        count_small<K, 8>(a, w, e0, n, sm, t, e2c, e2r, bp, bad);
      else
        count_small<K, 16>(a, w, e0, n, sm, t, e2c, e2r, bp, bad);
    }
    return;
  }
  uint8_t* const wsm = sm + (t / 32) * kWarpBytes;
  const int64_t w0 = (int64_t)(blockIdx.x - mid_ctas) * per;
  if (t == 0) next = kGroup / 32;
  __syncthreads();
  for (int v = t / 32; v < per && w0 + v < a.nwin;) {
    const int32_t w = (int32_t)(w0 + v);
    window_edges(a, w, e0, n);
    if (n == 0) {
      if (lane == 0) bp[w] = 0;
    } else if (n <= 128) {
      count_warp<K, 4>(a, w, e0, n, wsm, lane, e2c, e2r, bp, bad);
    } else if (n <= 256) {
      count_warp<K, 8>(a, w, e0, n, wsm, lane, e2c, e2r, bp, bad);
    } else if (n <= Cap<K>::kWarp) {
      if constexpr (sizeof(K) == 4)
        count_warp<K, 16>(a, w, e0, n, wsm, lane, e2c, e2r, bp, bad);
    }
    if (lane == 0) v = atomicAdd(&next, 1);
    v = __shfl_sync(0xffffffffu, v, 0);
  }
}

__global__ void __launch_bounds__(kThreads, 1)
    k_count_large(const Csr a, const int32_t* __restrict__ count, const int32_t* __restrict__ list,
                  int32_t room, int32_t* ticket, int32_t* __restrict__ e2c,
                  int32_t* __restrict__ e2r, int32_t* __restrict__ bp, uint32_t* bad) {
  extern __shared__ __align__(16) uint8_t dyn[];
  __shared__ int32_t next;
  const int32_t many = many_listed(count, room);
  for (int32_t i = blockIdx.x; i < many;) {
    int32_t e0, n;
    const int32_t w = listed(count, list, room, i);
    window_edges(a, w, e0, n);
    // (a sweep over the columns takes about 5 us of the SM, the sorts 18, 38 and 80 us)
    const int sweeps = (int)(((int64_t)a.M + kSweepCols - 1) / kSweepCols);
    if (n <= 4 * kThreads && sweeps > 3) count_sorted<4>(a, w, e0, n, dyn, e2c, e2r, bp, bad);
    else if (n <= 8 * kThreads && sweeps > 7) count_sorted<8>(a, w, e0, n, dyn, e2c, e2r, bp, bad);
    else if (n <= 16 * kThreads && sweeps > 15) count_sorted<16>(a, w, e0, n, dyn, e2c, e2r, bp, bad);
    else count_large(a, w, e0, n, dyn, e2c, e2r, bp, bad);
    if (threadIdx.x == 0) next = gridDim.x + atomicAdd(ticket, 1);
    __syncthreads();
    i = next;
    __syncthreads();
  }
}

// rwo = exclusive sum of bp (rwo[nwin] = T), 8192 windows per CTA; each CTA adds up the
// windows before its own (a few coalesced loads per thread from L2) instead of a second
// launch. From kManyWindows on that sum is the longer part (it grows with the square), and it
// is taken over the sums of the CTAs before (k_sums): 2^24 windows 36.6 -> 33.3 ms for the
// whole conversion. out = {T, *bad}.
constexpr int kScan = 8192, kManyWindows = 32 * kScan;
__global__ void __launch_bounds__(1024) k_sums(const int32_t* __restrict__ bp, int32_t nwin,
                                               int32_t* __restrict__ sums) {
  __shared__ int32_t part[32];
  const int64_t i0 = (int64_t)blockIdx.x * kScan;
  int32_t s = 0;
#pragma unroll
  for (int v = 0; v < kScan / 1024; ++v) {
    const int64_t i = i0 + v * 1024 + threadIdx.x;
    s += i < nwin ? __ldg(bp + i) : 0;
  }
  s = __reduce_add_sync(0xffffffffu, s);
  if (threadIdx.x % 32 == 0) part[threadIdx.x / 32] = s;
  __syncthreads();
  if (threadIdx.x < 32) {
    s = __reduce_add_sync(0xffffffffu, part[threadIdx.x]);
    if (threadIdx.x == 0) sums[blockIdx.x] = s;
  }
}
__global__ void __launch_bounds__(1024) k_scan(const int32_t* __restrict__ bp, int32_t nwin,
                                               const int32_t* __restrict__ cta_sums,
                                               int32_t* __restrict__ rwo, const uint32_t* bad,
                                               int32_t* out) {
  __shared__ int32_t sums[33], part[kScan];
  const int t = threadIdx.x;
  const int64_t i0 = (int64_t)blockIdx.x * kScan;
  const int cnt = (int)min((int64_t)kScan, nwin - i0);
  int32_t before = 0;
  const int32_t* const earlier = cta_sums ? cta_sums : bp;
  const int64_t many = cta_sums ? (int64_t)blockIdx.x : i0;
#pragma unroll 8
  for (int64_t i = t; i < many; i += 1024) before += __ldg(earlier + i);
  for (int i = t; i < kScan; i += 1024) part[i] = i < cnt ? __ldg(bp + i0 + i) : 0;
#pragma unroll
  for (int o = 16; o; o >>= 1) before += __shfl_xor_sync(0xffffffffu, before, o);
  if (t == 0) sums[32] = 0;
  __syncthreads();
  if ((t & 31) == 0) atomicAdd(&sums[32], before);
  int32_t mine = 0;  // eight consecutive windows per thread
#pragma unroll
  for (int v = 0; v < 8; ++v) mine += part[8 * t + v];
  int s = mine;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int u = __shfl_up_sync(0xffffffffu, s, o);
    if ((t & 31) >= o) s += u;
  }
  if ((t & 31) == 31) sums[t >> 5] = s;
  __syncthreads();
  if (t < 32) {
    int y = sums[t];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, y, o);
      if (t >= o) y += u;
    }
    sums[t] = y;
  }
  __syncthreads();
  int32_t at = sums[32] + s - mine + (t >= 32 ? sums[(t >> 5) - 1] : 0);
#pragma unroll
  for (int v = 0; v < 8; ++v) {
    const int32_t x = part[8 * t + v];
    part[8 * t + v] = at;
    at += x;
  }
  __syncthreads();
  for (int i = t; i < cnt; i += 1024) rwo[i0 + i] = part[i];
  if (t == 1023 && i0 + kScan >= nwin) {  // (the last CTA's last thread has the whole sum)
    rwo[nwin] = at;
    out[0] = at;
    out[1] = (int32_t)*bad;
  }
}

// ------------------------------------------------------------------- phase 2
struct Fill {
  const int32_t *e2c, *e2r, *rwo;
  const float* values;
  int32_t *rowid, *toff, *s2x;
  uint8_t* tile;
  float* tv;
  int64_t T;
};

// Values of one block in tile order where a (row, column) may occur twice: merged into
// its first occurrence (fp32 sum in CSR order), later ones 0. By one thread. `tile`: the tile
// ids, f.tile or a copy in shared memory (of edge j in [j]).
__device__ void merge_block(const Fill& f, const uint8_t* tile, int32_t j0, int32_t j1) {
  uint32_t seen[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  for (int32_t j = j0; j < j1; ++j) {
    const uint32_t p = tile[j], bit = 1u << (p & 31);
    if (!(seen[p >> 5] & bit)) {
      seen[p >> 5] |= bit;
    } else {
      int32_t x = j0;
      while (tile[x] != p) ++x;
      f.tv[x] += f.tv[j];
      f.tv[j] = 0.0f;
    }
  }
}

// The same by one warp, 32 edges at a time: the first lane of each cell adds up its peers.
struct MergeScratch {
  float sum[256], val[32];
  int32_t first[256];  // edge of each cell that comes first, or -1
};
__device__ void merge_block(const Fill& f, const uint8_t* tile, int32_t j0, int32_t j1,
                            MergeScratch& s, int lane) {
  for (int c = lane; c < 256; c += 32) s.first[c] = -1;
  for (int32_t j = j0 + lane; j - lane < j1; j += 32) {
    const bool in = j < j1;
    const uint32_t p = in ? tile[j] : 256u;
    s.val[lane] = in ? f.tv[j] : 0.0f;
    uint32_t peers = __match_any_sync(0xffffffffu, p);
    __syncwarp();
    if (in && lane == __ffs(peers) - 1) {
      float x;
      if (s.first[p] < 0) {
        s.first[p] = j;
        x = s.val[lane];
        peers &= peers - 1;
      } else {
        x = s.sum[p];
      }
      for (; peers; peers &= peers - 1) x += s.val[__ffs(peers) - 1];
      s.sum[p] = x;
    }
    __syncwarp();
    if (in && s.first[p] != j) f.tv[j] = 0.0f;
  }
  for (int c = lane; c < 256; c += 32)
    if (s.first[c] >= 0) f.tv[s.first[c]] = s.sum[c];
  __syncwarp();
}

// Whether a cell occurs twice among the edges of a block.
__device__ bool has_repeats(const uint8_t* tile, int32_t j0, int32_t j1) {
  uint32_t seen[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  for (int32_t j = j0; j < j1; ++j) {
    const uint32_t p = tile[j], bit = 1u << (p & 31);
    uint32_t old = 0;
#pragma unroll
    for (int q = 0; q < 8; ++q)
      if (p >> 5 == q) {
        old = seen[q];
        seen[q] |= bit;
      }
    if (old & bit) return true;
  }
  return false;
}

// All blocks b0 .. b0 + nb - 1, whose edges end at `last`, by `warps` warps: a lane looks
// through a block; one that repeats a cell is merged by the lane up to 24 edges (a warp's
// blocks wait for memory together), by the warp beyond (a lane takes a step per edge and a
// search per repeated one).
__device__ void merge_blocks(const Fill& f, const uint8_t* tile, int32_t b0, int32_t nb,
                             int32_t last, int warp, int warps, MergeScratch& s, int lane) {
  for (int32_t c = warp * 32; c < nb; c += warps * 32) {
    const int32_t b = c + lane;
    const int32_t j0 = b < nb ? f.toff[b0 + b] : 0, j1 = b + 1 < nb ? f.toff[b0 + b + 1] : last;
    const bool any = b < nb && has_repeats(tile, j0, j1);
    if (any && j1 - j0 <= 24) merge_block(f, tile, j0, j1);
    __syncwarp();
    for (uint32_t m = __ballot_sync(0xffffffffu, any && j1 - j0 > 24); m; m &= m - 1)
      merge_block(f, tile, __shfl_sync(0xffffffffu, j0, __ffs(m) - 1),
                  __shfl_sync(0xffffffffu, j1, __ffs(m) - 1), s, lane);
  }
}

__device__ __forceinline__ void zero_slots(const Csr& a, const Fill& f, int64_t b1, int32_t used,
                                           int t, int n) {  // unused slots of the last block
  for (int s = used % a.W + t; used % a.W && s < a.W; s += n) f.s2x[(b1 - 1) * a.W + s] = 0;
}

// Where the edges of `nb` blocks go: a bit per cell of a block (its tile id) marks the
// edges, so that in a window without repeated columns, whose rows' columns ascend, an
// edge's place in its block is the number of set bits below its own. `pos` holds the
// edges before each word of 32 cells. Scratch of one warp.
struct Marks {
  uint32_t* cell;
  uint16_t* pos;
  int words;  // per block
  __device__ Marks(const Csr& a, uint8_t* sm)
      : cell(reinterpret_cast<uint32_t*>(sm)),
        pos(reinterpret_cast<uint16_t*>(sm + kCells)),
        words((a.H * a.W + 31) / 32) {}
  __device__ __forceinline__ void clear(int nb, int lane) const {
    for (int i = lane; i < nb * words; i += 32) cell[i] = 0;
    __syncwarp();
  }
  __device__ __forceinline__ void set(int b, int id) const {
    atomicOr(cell + b * words + (id >> 5), 1u << (id & 31));
  }
  // Sums up; out(b, edges before block b).
  template <typename F>
  __device__ __forceinline__ void sum(int nb, int lane, F out) const {
    __syncwarp();
    int at = 0;
    for (int c = 0; c < nb; c += 32) {
      const int b = c + lane;
      int mine = 0;
      if (b < nb)
        for (int q = 0; q < words; ++q) mine += __popc(cell[b * words + q]);
      int y = mine;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, y, o);
        if (lane >= o) y += u;
      }
      if (b < nb) {
        int p = at + y - mine;
        out(b, p);
        for (int q = 0; q < words; ++q) {
          pos[b * words + q] = (uint16_t)p;
          p += __popc(cell[b * words + q]);
        }
      }
      at += __shfl_sync(0xffffffffu, y, 31);
    }
    __syncwarp();
  }
  __device__ __forceinline__ int place(int b, int id) const {
    const int x = b * words + (id >> 5);
    return pos[x] + __popc(cell[x] & ((1u << (id & 31)) - 1));
  }
};

// Whether edge e's rank is not above that of the edge before it in its row: a repeated column
// is possible (unsorted ones are too).
__device__ __forceinline__ bool repeats(const Fill& f, int32_t e0, int32_t e, int32_t rk) {
  const int32_t q = e > e0 ? e - 1 : e;  // (no branch: all loads under way together)
  return (e > e0) & (__ldg(f.e2c + q) >= rk) & (__ldg(f.e2r + q) == __ldg(f.e2r + e));
}

// Stable sort of key[0, m), one per edge, by the `bits` bits from kSortBits on, by a whole
// CTA: 7 bits per pass, a run of keys per warp, which counts and places 32 at a time by
// matching their digits (by a ballot per bit: match.any took 45 cycles of the SM for 32 keys).
// Returns where the keys end up (key or other). 16384 keys by two passes 35 us; a window of that
// many edges 65 us in all (105 with the columns and values gathered in sorted order).
constexpr int kDigits = 128, kHist = kDigits * 33;  // (a padded row of a word per warp and digit)
__device__ __forceinline__ uint32_t same_digit(uint32_t d, bool in) {
  uint32_t peers = __ballot_sync(0xffffffffu, in);
#pragma unroll
  for (int b = 0; b < 7; ++b) {
    const uint32_t m = __ballot_sync(0xffffffffu, d >> b & 1);
    peers &= d >> b & 1 ? m : ~m;
  }
  return peers;
}
__device__ __forceinline__ uint32_t* cta_sort(uint32_t* key, uint32_t* other, int32_t* hist,
                                              int32_t* part, int m, int bits) {
  static_assert(kThreads == 1024, "32 warps, four counters per thread");
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const int seg = (m + kThreads - 1) / kThreads * 32, j0 = warp * seg, j1 = min(j0 + seg, m);
  for (int shift = kSortBits; shift < kSortBits + bits; shift += 7) {
    for (int i = t; i < kHist; i += kThreads) hist[i] = 0;
    __syncthreads();
    for (int j = j0 + lane; j - lane < j1; j += 32) {
      const uint32_t d = j < j1 ? key[j] >> shift & (kDigits - 1) : 0;
      const uint32_t peers = same_digit(d, j < j1);
      if (j < j1 && lane == __ffs(peers) - 1) hist[d * 33 + warp] += __popc(peers);
      __syncwarp();
    }
    __syncthreads();
    int32_t* const h = hist + t / 8 * 33 + t % 8 * 4;  // four warps of a digit
    const int c[4] = {h[0], h[1], h[2], h[3]};
    int total;
    int at = cta_scan(c[0] + c[1] + c[2] + c[3], part, &total);
#pragma unroll
    for (int v = 0; v < 4; ++v) {
      h[v] = at;
      at += c[v];
    }
    __syncthreads();
    for (int j = j0 + lane; j - lane < j1; j += 32) {
      const uint32_t k = j < j1 ? key[j] : 0, d = k >> shift & (kDigits - 1);
      const uint32_t peers = same_digit(d, j < j1);
      const int to = j < j1 ? hist[d * 33 + warp] + __popc(peers & ((1u << lane) - 1)) : 0;
      __syncwarp();
      if (j < j1) {
        other[to] = k;
        if (lane == __ffs(peers) - 1) hist[d * 33 + warp] += __popc(peers);
      }
      __syncwarp();
    }
    __syncthreads();
    uint32_t* const x = key;
    key = other;
    other = x;
  }
  return key;
}

// The most columns and whether an edge may repeat another, over the T threads of a warp or CTA.
template <int T>
__device__ __forceinline__ void vote(int& used, bool& dup, int t) {
  used = __reduce_max_sync(0xffffffffu, used);
  if constexpr (T == 32) {
    dup = __any_sync(0xffffffffu, dup);
  } else {
    __shared__ int32_t s_used[T / 32];
    if (t % 32 == 0) s_used[t / 32] = used;
    dup = __syncthreads_or(dup);
#pragma unroll
    for (int i = 0; i < T / 32; ++i) used = max(used, s_used[i]);
  }
}

// A window of up to 32 E edges in any order by a warp: its edges sorted by (block, edge), in
// registers, are in their places.
template <int E>
__device__ __forceinline__ void fill_sorted(const Csr& a, const Fill& f, int32_t w, int32_t e0,
                                            int32_t n, uint8_t* sm, int lane) {
  constexpr int B = log2_of(32 * E);
  static_assert((1 << B) == 32 * E && 2 * B <= 32, "block and edge in a key");
  uint32_t* const key = reinterpret_cast<uint32_t*>(sm);
  uint8_t* const ids = sm + kLeftBytes - kWarpFill;
  const int32_t b0 = __ldg(f.rwo + w), nb = __ldg(f.rwo + w + 1) - b0;
  uint32_t x[E];
  int used = 0;
  bool dup = false;
#pragma unroll
  for (int i = 0; i < E; ++i) {
    const int e = i * 32 + lane;
    x[i] = 0xffffffffu;
    if (e < n) {
      const int32_t rk = __ldg(f.e2c + e0 + e);
      x[i] = (uint32_t)a.block(rk) << B | (uint32_t)e;
      used = max(used, rk + 1);
      if (f.values) dup |= repeats(f, e0, e0 + e, rk);
    }
  }
  reg_bitonic<uint32_t, E, 32>(x, lane, nullptr);
#pragma unroll
  for (int i = 0; i < E; ++i) key[lane * E + i] = x[i];
  vote<32>(used, dup, lane);
  __syncwarp();
  for (int b = lane; b < nb; b += 32) f.rowid[b0 + b] = w;
#pragma unroll 4
  for (int j = lane; j < n; j += 32) {
    const uint32_t k = key[j];
    const int32_t b = b0 + (int32_t)(k >> B), e = e0 + (int32_t)(k & ((1u << B) - 1));
    if (j == 0 || key[j - 1] >> B != k >> B) f.toff[b] = e0 + j;
    const int32_t slot = a.slot(__ldg(f.e2c + e));
    ids[j] = (uint8_t)((__ldg(f.e2r + e) - w * a.H) * a.W + slot);
    f.tile[e0 + j] = ids[j];
    f.s2x[(int64_t)b * a.W + slot] = __ldg(a.col + e);  // duplicates write the same value
    if (f.values) f.tv[e0 + j] = __ldg(f.values + e);
  }
  zero_slots(a, f, b0 + nb, used, lane, 32);
  __threadfence_block();
  __syncwarp();
  if (dup)  // (the keys are done with)
    merge_blocks(f, ids - e0, b0, nb, e0 + n, 0, 1, *reinterpret_cast<MergeScratch*>(sm), lane);
  __syncwarp();
}

// A window of up to kSortEdges edges in any order by a whole CTA. Columns and values go through
// shared memory too: read in the sorted order from memory, a sector each, they took longer than
// the sort.
__device__ void fill_cta(const Csr& a, const Fill& f, int32_t w, int32_t e0, int32_t n, uint8_t* sm) {
  uint32_t* key = reinterpret_cast<uint32_t*>(sm);
  uint32_t* other = key + kSortEdges;
  uint8_t* const sorted_ids = reinterpret_cast<uint8_t*>(other + kSortEdges);
  int32_t* const hist = reinterpret_cast<int32_t*>(sorted_ids + kSortEdges);
  uint8_t* const ids = reinterpret_cast<uint8_t*>(hist + kHist + 64);
  const int t = threadIdx.x;
  const int32_t b0 = __ldg(f.rwo + w), nb = __ldg(f.rwo + w + 1) - b0;
  int used = 0;
  bool dup = false;
#pragma unroll 4
  for (int j = t; j < n; j += kThreads) {
    const int32_t rk = __ldg(f.e2c + e0 + j), row = __ldg(f.e2r + e0 + j) - w * a.H;
    key[j] = (uint32_t)a.block(rk) << kSortBits | (uint32_t)j;
    ids[j] = (uint8_t)(row * a.W + a.slot(rk));
    used = max(used, rk + 1);
    if (f.values) dup |= repeats(f, e0, e0 + j, rk);
  }
  vote<kThreads>(used, dup, t);
  const uint32_t* const sorted = cta_sort(key, other, hist, hist + kHist, n, 32 - __clz(nb - 1));
  int32_t* const staged = reinterpret_cast<int32_t*>(sorted == key ? other : key);  // (free now)
  for (int b = t; b < nb; b += kThreads) f.rowid[b0 + b] = w;
#pragma unroll 4
  for (int j = t; j < n; j += kThreads) staged[j] = __ldg(a.col + e0 + j);
  __syncthreads();
  for (int j = t; j < n; j += kThreads) {
    const uint32_t k = sorted[j], b = k >> kSortBits, e = k & (kSortEdges - 1);
    if (j == 0 || sorted[j - 1] >> kSortBits != b) f.toff[b0 + b] = e0 + j;
    const uint8_t id = ids[e];
    sorted_ids[j] = id;
    f.tile[e0 + j] = id;
    f.s2x[(int64_t)(b0 + b) * a.W + id % (uint32_t)a.W] = staged[e];  // duplicates: the same value
  }
  zero_slots(a, f, b0 + nb, used, t, kThreads);
  __syncthreads();
  if (f.values) {
#pragma unroll 4
    for (int j = t; j < n; j += kThreads) staged[j] = __float_as_int(__ldg(f.values + e0 + j));
    __syncthreads();
    for (int j = t; j < n; j += kThreads)
      f.tv[e0 + j] = __int_as_float(staged[sorted[j] & (kSortEdges - 1)]);
    __threadfence_block();
    __syncthreads();
    if (dup && t / 32 < kMergeWarps)
      merge_blocks(f, sorted_ids - e0, b0, nb, e0 + n, t / 32, kMergeWarps,
                   reinterpret_cast<MergeScratch*>(hist)[t / 32], t & 31);
    __syncthreads();
  }
}

// One warp's window; false (nothing written) where a row's ranks do not ascend or the
__device__ __forceinline__ bool fill_warp(const Csr& a, const Fill& f, int32_t w, int32_t e0,
                                          int32_t n, uint8_t* sm, int lane) {
  const int32_t b0 = __ldg(f.rwo + w), nb = __ldg(f.rwo + w + 1) - b0;
  const Marks m(a, sm);
  if (nb * m.words * 4 > kCells) return false;
  const int32_t r0 = w * a.H;
  m.clear(nb, lane);
  bool mixed = false;
  int used = 0, last_rk = -1, last_row = -1;  // of the edge before this warp's 32
#pragma unroll 2
  for (int i = lane; i - lane < n; i += 32) {
    const bool in = i < n;
    const int rk = in ? __ldg(f.e2c + e0 + i) : 0, row = in ? __ldg(f.e2r + e0 + i) - r0 : -2;
    int prk = __shfl_up_sync(0xffffffffu, rk, 1), prow = __shfl_up_sync(0xffffffffu, row, 1);
    if (lane == 0) { prk = last_rk; prow = last_row; }
    mixed |= in && prow == row && prk >= rk;
    last_rk = __shfl_sync(0xffffffffu, rk, 31);
    last_row = __shfl_sync(0xffffffffu, row, 31);
    if (in) {
      used = max(used, rk + 1);
      m.set(a.block(rk), row * a.W + a.slot(rk));
    }
  }
  if (__any_sync(0xffffffffu, mixed)) return false;
  m.sum(nb, lane, [&](int b, int before) {
    f.toff[b0 + b] = e0 + before;
    f.rowid[b0 + b] = w;
  });
  for (int i = lane; i < n; i += 128) {
    int rk[4], row[4], c[4];
    float x[4];
#pragma unroll
    for (int v = 0; v < 4; ++v) {
      const bool in = i + 32 * v < n;
      const int32_t e = e0 + i + 32 * v;
      rk[v] = in ? __ldg(f.e2c + e) : -1;
      row[v] = in ? __ldg(f.e2r + e) - r0 : 0;
      c[v] = in ? __ldg(a.col + e) : 0;
      x[v] = in && f.values ? __ldg(f.values + e) : 0.0f;
    }
#pragma unroll
    for (int v = 0; v < 4; ++v)
      if (rk[v] >= 0) {
        const int b = a.block(rk[v]), slot = a.slot(rk[v]), id = row[v] * a.W + slot;
        const int32_t j = e0 + m.place(b, id);
        f.tile[j] = (uint8_t)id;
        f.s2x[(int64_t)(b0 + b) * a.W + slot] = c[v];
        if (f.values) f.tv[j] = x[v];
      }
  }
  used = __reduce_max_sync(0xffffffffu, used);
  zero_slots(a, f, b0 + nb, used, lane, 32);
  __syncwarp();
  return true;
}

// Blocks [p0, p1) of a window of any size in any order by one CTA: it reads all the window's
// ranks, twice, a run of them per warp, and keeps the edges of its blocks, in order, which are
// sorted by (block, edge). Where it keeps more than kPartSort, that many at a time go on from
// each block's place so far. (16 loads under way per lane: 15 us for the ranks of 65,536 edges.)
__device__ void fill_part(const Csr& a, const Fill& f, int32_t w, int32_t e0, int32_t n,
                          int32_t p0, int32_t p1, uint8_t* sm) {
  constexpr int V = kPartSort / 2 / kThreads, L = 16;
  uint32_t* key = reinterpret_cast<uint32_t*>(sm);
  uint32_t* other = key + kPartSort;
  int32_t* edge = reinterpret_cast<int32_t*>(other + kPartSort);  // kept edges
  int32_t* cur = edge + kPartSort;                                // next place of each block
  int32_t* hist = cur + kPartBlocks;
  int32_t* part = hist + kHist;
  __shared__ uint8_t ids[kPartSort];  // tile ids in sorted order, where it keeps them all
  __shared__ uint8_t kept_ids[kPartSort];
  __shared__ int32_t s_used, s_dup, s_before, s_kept[kThreads / 32];
  const int t = threadIdx.x, lane = t & 31, np = p1 - p0;
  const int64_t seg = ((int64_t)n / kThreads + 1) * 32;  // edges of a warp
  const int64_t i0 = t / 32 * seg, i1 = min(i0 + seg, (int64_t)n);
  const int32_t b0 = __ldg(f.rwo + w), nb = __ldg(f.rwo + w + 1) - b0;
  if (t == 0) s_used = s_dup = s_before = 0;
  for (int b = t; b < np; b += kThreads) cur[b] = 0;
  __syncthreads();
  const int32_t rk0 = p0 * a.W, rk1 = p1 * a.W;  // ranks of the blocks
  int used = 0, before = 0, kept = 0;
  bool dup = false;
  for (int64_t i = i0 + lane; i < i1; i += L * 32) {
    int32_t rk[L];
#pragma unroll
    for (int v = 0; v < L; ++v) rk[v] = i + v * 32 < i1 ? __ldg(f.e2c + e0 + i + v * 32) : INT32_MAX;
#pragma unroll
    for (int v = 0; v < L; ++v) {
      before += rk[v] < rk0;
      if (rk[v] >= rk0 && rk[v] < rk1) {
        atomicAdd(cur + (a.block(rk[v]) - p0), 1);
        ++kept;
        used = max(used, rk[v] + 1);
        if (f.values) dup |= repeats(f, e0, (int32_t)(e0 + i + v * 32), rk[v]);
      }
    }
  }
  if (dup) s_dup = 1;
  used = __reduce_max_sync(0xffffffffu, used);
  before = __reduce_add_sync(0xffffffffu, before);
  kept = __reduce_add_sync(0xffffffffu, kept);
  if (lane == 0) {
    atomicMax(&s_used, used);
    atomicAdd(&s_before, before);
    s_kept[t / 32] = kept;
  }
  __syncthreads();
  const int per = (np + kThreads - 1) / kThreads, q0 = min(t * per, np), q1 = min(q0 + per, np);
  int mine = 0;
  for (int q = q0; q < q1; ++q) mine += cur[q];
  int total;
  int at = s_before + cta_scan(mine, part, &total);
  for (int q = q0; q < q1; ++q) {
    const int c = cur[q];
    cur[q] = at;
    f.toff[b0 + p0 + q] = e0 + at;
    f.rowid[b0 + p0 + q] = w;
    at += c;
  }
  __syncthreads();
  auto flush = [&](int m) {
#pragma unroll 4
    for (int j = t; j < m; j += kThreads) {
      const int32_t rk = __ldg(f.e2c + edge[j]), row = __ldg(f.e2r + edge[j]) - w * a.H;
      key[j] = (uint32_t)(a.block(rk) - p0) << kSortBits | (uint32_t)j;
      kept_ids[j] = (uint8_t)(row * a.W + a.slot(rk));
    }
    __syncthreads();
    const uint32_t* const sorted = cta_sort(key, other, hist, part, m, 32 - __clz(np - 1));
    // the first kept edge of block b (from p0) among the m sorted ones
    auto first_of = [&](uint32_t b) {
      int lo = 0, hi = m;
      while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (sorted[mid] >> kSortBits < b) lo = mid + 1; else hi = mid;
      }
      return lo;
    };
#pragma unroll 2
    for (int j = t; j < m; j += kThreads) {
      const uint32_t k = sorted[j], b = k >> kSortBits;
      const int32_t e = edge[k & (kSortEdges - 1)], to = e0 + cur[b] + j - first_of(b);
      const uint8_t id = kept_ids[k & (kSortEdges - 1)];
      f.tile[to] = id;
      if (total <= kPartSort) ids[to - e0 - s_before] = id;
      f.s2x[(int64_t)(b0 + p0 + b) * a.W + id % (uint32_t)a.W] = __ldg(a.col + e);
      if (f.values) f.tv[to] = __ldg(f.values + e);
    }
    __syncthreads();
    for (int b = t; b < np; b += kThreads) cur[b] += first_of(b + 1) - first_of(b);
    __syncthreads();
  };
  int m = 0;
  if (total <= kPartSort) {
    int to = 0;
    for (int i = 0; i < t / 32; ++i) to += s_kept[i];
    for (int64_t i = i0 + lane; i - lane < i1; i += L * 32) {
      int32_t rk[L];
#pragma unroll
      for (int v = 0; v < L; ++v) rk[v] = i + v * 32 < i1 ? __ldg(f.e2c + e0 + i + v * 32) : -1;
#pragma unroll
      for (int v = 0; v < L; ++v) {
        const bool keep = rk[v] >= rk0 && rk[v] < rk1;
        const uint32_t mask = __ballot_sync(0xffffffffu, keep);
        if (keep) edge[to + __popc(mask & ((1u << lane) - 1))] = (int32_t)(e0 + i + v * 32);
        to += __popc(mask);
      }
    }
    m = total;
    __syncthreads();
  } else
  for (int64_t i0 = 0; i0 < n; i0 += V * kThreads) {
    int32_t keep = 0;  // of this thread's V edges, one after the other
#pragma unroll
    for (int v = 0; v < V; ++v) {
      const int64_t i = i0 + t * V + v;
      const int32_t b = i < n ? a.block(__ldg(f.e2c + e0 + i)) : -1;
      keep |= (b >= p0 && b < p1) << v;
    }
    int add;
    int to = m + cta_scan(__popc(keep), part, &add);
#pragma unroll
    for (int v = 0; v < V; ++v)
      if (keep >> v & 1) edge[to++] = (int32_t)(e0 + i0 + t * V + v);
    m += add;
    __syncthreads();
    if (m > kPartSort - V * kThreads) {
      flush(m);
      m = 0;
    }
  }
  if (m) flush(m);
  if (p1 == nb) zero_slots(a, f, b0 + nb, s_used, t, kThreads);
  __shared__ int32_t s_end;
  if (t == 0) s_end = cur[np - 1];  // (its place after the last block's edges)
  if (f.values && s_dup) {
    __threadfence_block();
    __syncthreads();
    merge_blocks(f, total <= kPartSort ? ids - e0 - s_before : f.tile, b0 + p0, np, e0 + s_end,
                 t / 32, kThreads / 32, reinterpret_cast<MergeScratch*>(sm)[t / 32], lane);
  }
  __syncthreads();
}

// Blocks [p0, p0 + unit) of a window whose ranks ascend along every row, by one warp: its
// part of each row is a run of edges.
__device__ __forceinline__ void fill_unit(const Csr& a, const Fill& f, int32_t w, int32_t p0,
                                          int32_t unit, uint8_t* sm, int lane) {
  const int32_t b0 = __ldg(f.rwo + w), nb = __ldg(f.rwo + w + 1) - b0;
  const int np = min(unit, nb - p0);
  const Marks m(a, sm);
  int32_t* first = reinterpret_cast<int32_t*>(sm + kCells * 3 / 2);  // first edge by row, less
  int32_t* pre = first + kUnitH;                                     // the edges of rows before
  const int64_t r0 = (int64_t)w * a.H;
  const int rows = (int)min((int64_t)a.H, a.M - r0);
  auto lower = [&](int32_t lo, int32_t hi, int32_t rk) {
    while (lo < hi) {
      const int32_t mid = lo + ((hi - lo) >> 1);
      if (__ldg(f.e2c + mid) < rk) lo = mid + 1; else hi = mid;
    }
    return lo;
  };
  // both ends of every row's part: at once where two lanes per row suffice
  const bool twice = rows <= 16;
  const int r = twice ? lane & 15 : lane;
  int32_t s = 0, lo = 0, hi = 0;
  if (r < rows) {
    s = __ldg(a.rowptr + r0 + r);
    const int32_t e = __ldg(a.rowptr + r0 + r + 1);
    lo = lower(s, e, (twice && lane >= 16 ? p0 + np : p0) * a.W);
    if (!twice) hi = lower(lo, e, (p0 + np) * a.W);
  }
  if (twice) hi = __shfl_xor_sync(0xffffffffu, lo, 16);
  if (twice && lane >= 16) s = lo = hi = 0;
  const int32_t start = __reduce_add_sync(0xffffffffu, lo - s);  // edges of the blocks before
  int x = hi - lo;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int u = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += u;
  }
  const int n = __shfl_sync(0xffffffffu, x, 31);
  if (lane < rows) first[lane] = lo - (x - (hi - lo));
  if (lane < rows) pre[lane + 1] = x;
  m.clear(np, lane);
  const int32_t e0 = __ldg(a.rowptr + r0);
  int used = 0, row = 0;
  // (four edges per lane at a time: their rows and places first, then all the loads)
  for (int i = lane; i < n; i += 128) {
    int rk[4], id[4];
#pragma unroll
    for (int v = 0; v < 4; ++v)
      if (i + 32 * v < n) {
        while (pre[row + 1] <= i + 32 * v) ++row;  // (pre[rows] = n)
        rk[v] = first[row] + i + 32 * v;
        id[v] = row * a.W;
      }
#pragma unroll
    for (int v = 0; v < 4; ++v) rk[v] = i + 32 * v < n ? __ldg(f.e2c + rk[v]) : -1;
#pragma unroll
    for (int v = 0; v < 4; ++v)
      if (rk[v] >= 0) {
        used = max(used, rk[v] + 1);
        m.set(a.block(rk[v]) - p0, id[v] + a.slot(rk[v]));
      }
  }
  m.sum(np, lane, [&](int b, int before) {
    f.toff[b0 + p0 + b] = e0 + start + before;
    f.rowid[b0 + p0 + b] = w;
  });
  row = 0;
  for (int i = lane; i < n; i += 128) {
    int e[4], rk[4], id[4], c[4];
    float x[4];
#pragma unroll
    for (int v = 0; v < 4; ++v)
      if (i + 32 * v < n) {
        while (pre[row + 1] <= i + 32 * v) ++row;
        e[v] = first[row] + i + 32 * v;
        id[v] = row * a.W;
      }
#pragma unroll
    for (int v = 0; v < 4; ++v) {
      const bool in = i + 32 * v < n;
      rk[v] = in ? __ldg(f.e2c + e[v]) : -1;
      c[v] = in ? __ldg(a.col + e[v]) : 0;
      x[v] = in && f.values ? __ldg(f.values + e[v]) : 0.0f;
    }
#pragma unroll
    for (int v = 0; v < 4; ++v)
      if (rk[v] >= 0) {
        const int b = a.block(rk[v]), slot = a.slot(rk[v]);
        const int32_t j = e0 + start + m.place(b - p0, id[v] + slot);
        f.tile[j] = (uint8_t)(id[v] + slot);
        f.s2x[(int64_t)(b0 + b) * a.W + slot] = c[v];
        if (f.values) f.tv[j] = x[v];
      }
  }
  used = __reduce_max_sync(0xffffffffu, used);
  if (p0 + np == nb) zero_slots(a, f, b0 + nb, used, lane, 32);
  __syncwarp();
}

// A window of at most kLane edges by one lane; `most` as in count_lane.
__device__ __forceinline__ void fill_lane(const Csr& a, const Fill& f, int32_t w, int32_t e0,
                                          int32_t n, int32_t most) {
  const int32_t b0 = __ldg(f.rwo + w), nb = __ldg(f.rwo + w + 1) - b0;
  int32_t id[kLane];  // block << 16 | rank << 8 | row (past the last edge: beyond every block)
  float x[kLane];
  int used = 0;
#pragma unroll
  for (int j = 0; j < kLane; ++j) {
    id[j] = INT32_MAX;
    x[j] = 0.0f;
    if (j < most && j < n) {
      const int32_t rk = __ldg(f.e2c + e0 + j);
      id[j] = a.block(rk) << 16 | rk << 8 | (__ldg(f.e2r + e0 + j) - w * a.H);
      used = max(used, rk + 1);
      if (f.values) x[j] = __ldg(f.values + e0 + j);
    }
  }
  for (int b = 0; b < nb; ++b) {
    int before = 0;
#pragma unroll
    for (int j = 0; j < kLane; ++j) before += id[j] >> 16 < b;
    f.toff[b0 + b] = e0 + before;
    f.rowid[b0 + b] = w;
  }
#pragma unroll
  for (int j = 0; j < kLane; ++j)
    if (j < most && j < n) {
      const int b = id[j] >> 16, slot = a.slot(id[j] >> 8 & 0xff);
      int place = 0;
      bool again = false;  // a repeated (row, column): its value goes to the first one
      float s = x[j];
#pragma unroll
      for (int i = 0; i < kLane; ++i) {
        place += id[i] >> 16 < b || (i < j && id[i] >> 16 == b);
        again |= i < j && id[i] == id[j];
        if (i > j && id[i] == id[j]) s += x[i];
      }
      f.tile[e0 + place] = (uint8_t)((id[j] & 0xff) * a.W + slot);
      f.s2x[(int64_t)(b0 + b) * a.W + slot] = __ldg(a.col + e0 + j);
      if (f.values) f.tv[e0 + place] = again ? 0.0f : s;
    }
  zero_slots(a, f, b0 + nb, used, 0, 1);
}

// Matrices of few edges per window: as k_count_tiny.
__global__ void __launch_bounds__(kGroup, 5)
    k_fill_tiny(const Csr a, const Fill f, int32_t* left, int32_t* __restrict__ left_list) {
  __shared__ __align__(16) uint8_t sm[4 * kWarpBytes];
  const int t = threadIdx.x, lane = t & 31;
  const int64_t w = (int64_t)blockIdx.x * kGroup + t;
  int32_t e0 = 0, n = 0;
  if (w < a.nwin) window_edges(a, (int32_t)w, e0, n);
  if (w == 0) f.toff[f.T] = (int32_t)a.nnz;
  const int32_t most = __reduce_max_sync(0xffffffffu, n <= kLane ? n : 0);
  if (n > 0 && n <= kLane) fill_lane(a, f, (int32_t)w, e0, n, most);
  for (uint32_t m = __ballot_sync(0xffffffffu, n > kLane && n <= kWarpFill); m; m &= m - 1) {
    const int src = __ffs(m) - 1;
    const int32_t v = (int32_t)(w - lane + src);
    if (!fill_warp(a, f, v, __shfl_sync(0xffffffffu, e0, src), __shfl_sync(0xffffffffu, n, src),
                   sm + (t / 32) * kWarpBytes, lane) && lane == 0)
      left_list[atomicAdd(left, 1)] = v;
  }
}

// Warps first take the units of the listed windows (more than kWarpFill edges), then a
// window each. Windows that they cannot do are left to k_fill_mixed.
__global__ void __launch_bounds__(kGroup, 8)
    k_fill(const Csr a, const Fill f, const int32_t* __restrict__ units,
           const int2* __restrict__ unit_list, const uint8_t* __restrict__ mixed, int unit,
           int64_t unit_room, int unit_ctas, int per, int32_t* left,
           int32_t* __restrict__ left_list) {
  __shared__ __align__(16) uint8_t sm[4 * kWarpBytes];
  __shared__ int next;
  const int t = threadIdx.x;
  if ((int)blockIdx.x < unit_ctas) {
    const int32_t many = (int32_t)min((int64_t)__ldg(units), unit_room);
    for (int32_t i = blockIdx.x * 4 + t / 32; i < many; i += unit_ctas * 4) {
      const int2 u = __ldg(unit_list + i);
      if (!__ldg(mixed + u.x))
        fill_unit(a, f, u.x, u.y, unit, sm + (t / 32) * kWarpBytes, t & 31);
    }
    return;
  }
  int32_t e0, n;
  const int64_t w0 = (int64_t)(blockIdx.x - unit_ctas) * per;
  if (w0 == 0 && t == 0) f.toff[f.T] = (int32_t)a.nnz;
  if (t == 0) next = kGroup / 32;
  __syncthreads();
  for (int v = t / 32; v < per && w0 + v < a.nwin;) {
    window_edges(a, (int32_t)(w0 + v), e0, n);
    if (n > 0 && n <= kWarpFill &&
        !fill_warp(a, f, (int32_t)(w0 + v), e0, n, sm + (t / 32) * kWarpBytes, t & 31) &&
        (t & 31) == 0)
      left_list[atomicAdd(left, 1)] = (int32_t)(w0 + v);
    if ((t & 31) == 0) v = atomicAdd(&next, 1);
    v = __shfl_sync(0xffffffffu, v, 0);
  }
}

// Windows whose edges a sort has to place. Listed ones of more than kHuge edges (the list's
// first) by parts, part p of the i-th by CTA (p + 91 i) % G; the other listed ones by a CTA
// each; then those that k_fill left over, by a warp each.
__global__ void __launch_bounds__(kThreads, 1)
    k_fill_mixed(const Csr a, const Fill f, const int32_t* __restrict__ count,
                 const int32_t* __restrict__ list, const uint8_t* __restrict__ mixed,
                 int32_t room, const int32_t* __restrict__ any, const int32_t* __restrict__ left,
                 const int32_t* __restrict__ left_list) {
  extern __shared__ __align__(16) uint8_t dyn[];
  const int G = gridDim.x, c = blockIdx.x, t = threadIdx.x;
  const int32_t rest = __ldg(left);
  int32_t e0, n;
  if (__ldg(any)) {
    const int32_t many = many_listed(count, room), huge = min(__ldg(count), many);
    for (int32_t i = 0; i < huge; ++i) {
      const int32_t w = listed(count, list, room, i);
      if (!__ldg(mixed + w)) continue;
      window_edges(a, w, e0, n);
      const int32_t nb = __ldg(f.rwo + w + 1) - __ldg(f.rwo + w);
      const int parts = max(min((n + kPartEdges - 1) / kPartEdges, G), (nb + kPartBlocks - 1) / kPartBlocks);
      int p = (int)((c - 91 * (int64_t)i) % G);
      for (p = p < 0 ? p + G : p; p < parts; p += G)
        fill_part(a, f, w, e0, n, (int32_t)((int64_t)nb * p / parts),
                  (int32_t)((int64_t)nb * (p + 1) / parts), dyn);
    }
    for (int32_t i = huge + c; i < many; i += G) {
      const int32_t w = listed(count, list, room, i);
      if (!__ldg(mixed + w)) continue;
      window_edges(a, w, e0, n);
      fill_cta(a, f, w, e0, n, dyn);
    }
    __syncthreads();
  }
  for (int32_t i = c * (kThreads / 32) + t / 32; i < rest; i += G * (kThreads / 32)) {
    const int32_t w = __ldg(left_list + i);
    window_edges(a, w, e0, n);
    uint8_t* const sm = dyn + t / 32 * kLeftBytes;
    if (n <= 128) fill_sorted<4>(a, f, w, e0, n, sm, t & 31);
    else if (n <= 512) fill_sorted<16>(a, f, w, e0, n, sm, t & 31);
    else fill_sorted<32>(a, f, w, e0, n, sm, t & 31);
  }
}

Csr make_csr(const int32_t* col, const int32_t* rowptr, int32_t M, int32_t nwin, int32_t H,
             int32_t W, int64_t nnz) {
  const int32_t b = bits_for((uint64_t)W);
  return {col, rowptr, M, nwin, H, W, nnz, W == 1 ? 0 : (1 << b) == W ? b : -1};
}

struct Layout {
  size_t head, list, mid, mixed, units, sums, left, tall, sort, total;  // head: see Head
  int64_t room, mid_room, unit_room;                 // entries of the lists
  bool wide;
};

// Words of the workspace's head, zero at the start of a phase.
enum Head { kCount = 0, kBad = 2, kOut = 3, kUnits = 5, kTicket = 6, kMid = 7, kAny = 8, kLeft = 9, kHead = 10 };

constexpr int kUnit = 128;  // blocks per unit of a large window
static_assert(kUnit * 8 * 4 <= kCells, "a unit's masks fit");

Layout layout(int32_t M, int64_t nnz, int32_t H) {
  Layout L{};
  L.wide = bits_for((uint64_t)(M > 0 ? M : 1)) + Cap<uint32_t>::kBits > 32;
  const size_t large = (size_t)nnz / (kWarpFill + 1) + 1;  // listed windows, at most
  L.room = (int64_t)large;
  L.unit_room = H > kUnitH ? 0 : nnz / kUnit + (int64_t)large;
  L.head = 0;
  L.list = 256;
  L.mid_room = nnz / (Cap<uint64_t>::kWarp + 1) + 1;
  L.mid = align_up(L.list + large * 4, 256);
  L.mixed = align_up(L.mid + (size_t)L.mid_room * 4, 256);
  L.units = align_up(L.mixed + ((size_t)M + H - 1) / H, 256);
  L.sums = align_up(L.units + (size_t)L.unit_room * 8, 256);
  L.left = align_up(L.sums + (((size_t)M + H - 1) / H / kScan + 1) * 4, 256);
  L.tall = align_up(L.left + ((size_t)M + H - 1) / H * 4, 256);
  L.sort = L.total = L.tall;
  if (H > kUnitH) {
    size_t bytes = 0;
    cub::DeviceRadixSort::SortPairs(nullptr, bytes, (uint32_t*)nullptr, (uint32_t*)nullptr,
                                    (int32_t*)nullptr, (int32_t*)nullptr, nnz > 0 ? nnz : 1, 0, 32);
    L.sort = align_up(L.tall + (size_t)nnz * 16, 256);
    L.total = align_up(L.sort + bytes, 256);
  }
  return L;
}

static_assert(kHuge <= kSortEdges, "fill_cta takes every window that is not huge");
constexpr int kSortBytes =
    kSortEdges * 9 + std::max(kHist * 4 + 256 + kSortEdges, kMergeWarps * (int)sizeof(MergeScratch));
static_assert(kThreads / 32 * (int)sizeof(MergeScratch) <= kPartSort * 12 && kPartSort <= kSortEdges &&
              kPartSort * 12 + kPartBlocks * 4 + kHist * 4 + 256 <= kSortBytes, "fill_part fits");
static_assert(kThreads / 32 * kLeftBytes <= kSortBytes && sizeof(MergeScratch) <= kWarpFill * 4,
              "fill_sorted, by every warp");

// CTAs for the windows of more than `cap` edges: no more than there can be, one per SM.
int large_ctas(int64_t nnz, int cap) {
  const int64_t most = nnz / (cap + 1), want = num_sms();
  return (int)(most < want ? most : want);
}

// Windows per CTA: kPer share out uneven windows among its warps, fewer where that would
// leave SMs idle.
int windows_per_cta(int32_t nwin) {
  const int64_t p = nwin / (8 * (int64_t)num_sms());
  return p < 4 ? 4 : p > kPer ? kPer : (int)p;
}

template <typename K>
dtc_status count_impl(const Csr& a, char* ws, const Layout& L, int32_t* e2c, int32_t* e2r,
                      int32_t* bp, cudaStream_t st) {
  int32_t* count = (int32_t*)(ws + L.head) + kCount;
  int32_t* list = (int32_t*)(ws + L.list);
  uint32_t* bad = (uint32_t*)(ws + L.head) + kBad;
  int32_t* mid_count = (int32_t*)(ws + L.head) + kMid;
  int32_t* mid_list = (int32_t*)(ws + L.mid);
  k_list<<<(a.nwin + 255) / 256, 256, 0, st>>>(a, Cap<K>::kEdges, Cap<K>::kWarp, count, list,
                                               mid_count, mid_list, (int32_t)L.mid_room, bad,
                                               (int32_t)L.room, nullptr, 0, nullptr, nullptr, 0, nullptr);
  const int large = large_ctas(a.nnz, Cap<K>::kEdges);
  if (large) {
    DTC_CUDA(cudaFuncSetAttribute(k_count_large, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  kLargeBytes));
    k_count_large<<<large, kThreads, kLargeBytes, st>>>(a, count, list, (int32_t)L.room,
                                                        (int32_t*)(ws + L.head) + kTicket, e2c,
                                                        e2r, bp, bad);
  }
  const int64_t most = a.nnz / (Cap<K>::kWarp + 1), want = 8 * (int64_t)num_sms();
  const int mid_ctas = (int)(most < want ? most : want), per = windows_per_cta(a.nwin);
  const bool tiny = tiny_windows(a.nnz, a.nwin);
  const int64_t ctas = tiny ? 0 : ((int64_t)a.nwin + per - 1) / per;
  if (mid_ctas + ctas)
    k_count<K><<<(unsigned)(mid_ctas + ctas), kGroup, 0, st>>>(
        a, mid_count, mid_list, (int32_t)L.mid_room, mid_ctas, per, e2c, e2r, bp, bad);
  if (tiny)
    k_count_tiny<K><<<(unsigned)(((int64_t)a.nwin + kGroup - 1) / kGroup), kGroup, 0, st>>>(
        a, e2c, e2r, bp, bad);
  return DTC_OK;
}

// Windows of more than kUnitH rows (block shapes of 64 x 4 and taller): all edges sorted by
// block, with a global radix sort. A warp finds its part of a row by search; with that many
// rows the searches cost more than the sort's passes.
__global__ void k_tall_keys(const Csr a, const Fill f, uint32_t* __restrict__ key,
                            int32_t* __restrict__ edge, int32_t* any) {
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  bool found = false;
  if (e < a.nnz) {
    const int32_t rk = __ldg(f.e2c + e);
    key[e] = (uint32_t)(__ldg(f.rwo + __ldg(f.e2r + e) / a.H) + a.block(rk));
    edge[e] = (int32_t)e;
    found = repeats(f, 0, (int32_t)e, rk);
  }
  if (__syncthreads_or(found) && threadIdx.x == 0) *any = 1;
}
__global__ void k_tall_emit(const Csr a, const Fill f, const uint32_t* __restrict__ key,
                            const int32_t* __restrict__ edge) {
  const int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= a.nnz) return;
  const uint32_t b = __ldg(key + j);
  const int32_t e = __ldg(edge + j), row = __ldg(f.e2r + e), w = row / a.H;
  const int32_t slot = a.slot(__ldg(f.e2c + e));
  if (j == 0) f.toff[f.T] = (int32_t)a.nnz;
  if (j == 0 || __ldg(key + j - 1) != b) {
    f.toff[b] = (int32_t)j;
    f.rowid[b] = w;
  }
  f.tile[j] = (uint8_t)((row - w * a.H) * a.W + slot);
  f.s2x[(int64_t)b * a.W + slot] = __ldg(a.col + e);
  if (f.values) f.tv[j] = __ldg(f.values + e);
}
__global__ void __launch_bounds__(kGroup) k_tall_merge(const Csr a, const Fill f, const int32_t* any) {
  __shared__ MergeScratch s[kGroup / 32];
  if (*any)
    merge_blocks(f, f.tile, 0, (int32_t)f.T, (int32_t)a.nnz, blockIdx.x * (kGroup / 32) + threadIdx.x / 32,
                 gridDim.x * (kGroup / 32), s[threadIdx.x / 32], threadIdx.x & 31);
}
dtc_status fill_tall(const Csr& a, const Fill& f, char* ws, const Layout& L, cudaStream_t st) {
  uint32_t *kin = (uint32_t*)(ws + L.tall), *kout = kin + a.nnz;
  int32_t *ein = (int32_t*)(kout + a.nnz), *eout = ein + a.nnz;
  int32_t* any = (int32_t*)(ws + L.head) + kAny;
  const unsigned g = (unsigned)((a.nnz + 255) / 256);
  DTC_CUDA(cudaMemsetAsync(f.s2x, 0, (size_t)f.T * a.W * 4, st));
  k_tall_keys<<<g, 256, 0, st>>>(a, f, kin, ein, any);
  size_t bytes = L.total - L.sort;
  DTC_CUDA(cub::DeviceRadixSort::SortPairs(ws + L.sort, bytes, kin, kout, ein, eout, a.nnz, 0,
                                           bits_for((uint64_t)f.T), st));
  k_tall_emit<<<g, 256, 0, st>>>(a, f, kout, eout);
  if (f.values) k_tall_merge<<<8 * num_sms(), kGroup, 0, st>>>(a, f, any);
  return DTC_OK;
}

dtc_status fill_impl(const Csr& a, const Fill& f, char* ws, const Layout& L, cudaStream_t st) {
  int32_t* head = (int32_t*)(ws + L.head);
  int32_t *list = (int32_t*)(ws + L.list), *left_list = (int32_t*)(ws + L.left);
  int2* unit_list = (int2*)(ws + L.units);
  uint8_t* mixed = (uint8_t*)(ws + L.mixed);
  int unit_ctas = 0;
  if (a.nnz > kWarpFill) {
    k_list<<<(a.nwin + 255) / 256, 256, 0, st>>>(a, kWarpFill, INT32_MAX, head + kCount, list, nullptr,
                                                 nullptr, 0, nullptr, (int32_t)L.room, f.rwo, kUnit,
                                                 head + kUnits, unit_list, L.unit_room, mixed);
    k_mixed<<<(unsigned)((a.nnz + 2047) / 2048), 256, 0, st>>>(a, f.e2c, f.e2r, mixed, head + kAny);
    // a warp per unit up to eight CTAs per SM
    unit_ctas = (int)std::min<int64_t>((L.unit_room + 3) / 4, 8 * num_sms());
  }
  const int per = windows_per_cta(a.nwin);
  const bool tiny = tiny_windows(a.nnz, a.nwin);
  const int64_t ctas = tiny ? 0 : ((int64_t)a.nwin + per - 1) / per;
  if (unit_ctas + ctas)
    k_fill<<<(unsigned)(unit_ctas + ctas), kGroup, 0, st>>>(a, f, head + kUnits, unit_list, mixed, kUnit,
                                                          L.unit_room, unit_ctas, per, head + kLeft,
                                                          left_list);
  if (tiny)
    k_fill_tiny<<<(unsigned)(((int64_t)a.nwin + kGroup - 1) / kGroup), kGroup, 0, st>>>(
        a, f, head + kLeft, left_list);
  // a CTA per SM, fewer where there are not the edges
  const int mixed_ctas = (int)std::min<int64_t>(a.nnz / 512 + 1, num_sms());
  DTC_CUDA(cudaFuncSetAttribute(k_fill_mixed, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                kSortBytes));
  k_fill_mixed<<<mixed_ctas, kThreads, kSortBytes, st>>>(a, f, head + kCount, list, mixed,
                                                         (int32_t)L.room, head + kAny, head + kLeft,
                                                         left_list);
  return DTC_OK;
}

}  // namespace
}  // namespace dtc

using namespace dtc;

extern "C" dtc_status dtc_convert_workspace_bytes(int32_t num_nodes, int64_t nnz, int32_t block_h,
                                                  int32_t block_w, size_t* bytes) {
  DTC_REQUIRE(bytes != nullptr, "bytes is null");
  DTC_REQUIRE(num_nodes >= 0 && nnz >= 0 && block_h > 0 && block_w > 0,
              "negative sizes or non-positive block shape");
  DTC_REQUIRE((int64_t)block_h * block_w <= 256, "block_h * block_w must be <= 256 (u8 tile ids)");
  DTC_REQUIRE(nnz < (int64_t)INT32_MAX, "nnz must fit in int32 (reference index type)");
  *bytes = layout(num_nodes, nnz, block_h).total;
  return DTC_OK;
}

extern "C" dtc_status dtc_convert_count(const int32_t* d_col, const int32_t* d_rowptr,
                                        int32_t num_nodes, int64_t nnz, int32_t block_h,
                                        int32_t block_w, int32_t* d_blockPartition,
                                        int32_t* d_edgeToColumn, int32_t* d_edgeToRow,
                                        int32_t* d_rowWindowOffset, void* d_workspace,
                                        size_t workspace_bytes, int64_t* num_blocks,
                                        dtc_stream_t stream) {
  size_t need = 0;
  dtc_status s = dtc_convert_workspace_bytes(num_nodes, nnz, block_h, block_w, &need);
  if (s != DTC_OK) return s;
  DTC_REQUIRE(num_blocks != nullptr, "num_blocks is null");
  DTC_REQUIRE(d_rowptr && d_blockPartition && d_rowWindowOffset, "null device pointer");
  DTC_REQUIRE(nnz == 0 || (d_col && d_edgeToColumn && d_edgeToRow), "null device pointer");
  if (workspace_bytes < need || d_workspace == nullptr) {
    set_error("conversion workspace too small");
    return DTC_ERR_WORKSPACE_TOO_SMALL;
  }
  cudaStream_t st = (cudaStream_t)stream;
  const int32_t nwin = (int32_t)(((int64_t)num_nodes + block_h - 1) / block_h);
  const Layout L = layout(num_nodes, nnz, block_h);
  char* ws = (char*)d_workspace;
  const Csr a = make_csr(d_col, d_rowptr, num_nodes, nwin, block_h, block_w, nnz);
  DTC_CUDA(cudaMemsetAsync(ws + L.head, 0, kHead * 4, st));
  uint32_t* bad = (uint32_t*)(ws + L.head) + kBad;
  if (nwin > 0) {
    s = L.wide ? count_impl<uint64_t>(a, ws, L, d_edgeToColumn, d_edgeToRow, d_blockPartition, st)
               : count_impl<uint32_t>(a, ws, L, d_edgeToColumn, d_edgeToRow, d_blockPartition, st);
    if (s != DTC_OK) return s;
  } else {
    k_list<<<1, 32, 0, st>>>(a, 0, 0, nullptr, nullptr, nullptr, nullptr, 0, bad, 0,
                             nullptr, 0, nullptr, nullptr, 0, nullptr);
  }
  int32_t* out = (int32_t*)(ws + L.head) + kOut;
  const int32_t ctas = nwin ? (int32_t)(((int64_t)nwin + kScan - 1) / kScan) : 1;
  int32_t* sums = nwin > kManyWindows ? (int32_t*)(ws + L.sums) : nullptr;
  if (sums) k_sums<<<ctas, 1024, 0, st>>>(d_blockPartition, nwin, sums);
  k_scan<<<ctas, 1024, 0, st>>>(d_blockPartition, nwin, sums, d_rowWindowOffset, bad, out);
  DTC_CUDA(cudaGetLastError());
  int32_t hostv[2] = {0, 0};
  DTC_CUDA(cudaMemcpyAsync(hostv, out, 8, cudaMemcpyDeviceToHost, st));
  DTC_CUDA(cudaStreamSynchronize(st));
  if (hostv[1] != 0) {
    set_error("invalid CSR input (flags " + std::to_string(hostv[1]) +
              "): need rowptr[0]==0, non-decreasing rowptr, rowptr[M]==nnz, 0<=col<M");
    return DTC_ERR_INVALID_ARGUMENT;
  }
  *num_blocks = hostv[0];
  return DTC_OK;
}

extern "C" dtc_status dtc_convert_fill(const int32_t* d_col, const int32_t* d_rowptr,
                                       int32_t num_nodes, int64_t nnz, int32_t block_h,
                                       int32_t block_w, const int32_t* d_edgeToColumn,
                                       const int32_t* d_edgeToRow,
                                       const int32_t* d_rowWindowOffset, int64_t num_blocks,
                                       int32_t* d_tcblockRowid, uint8_t* d_tileId,
                                       int32_t* d_tcblockOffset, int32_t* d_sparseAToX,
                                       const float* d_values, float* d_tcValues,
                                       void* d_workspace, size_t workspace_bytes,
                                       dtc_stream_t stream) {
  size_t need = 0;
  dtc_status s = dtc_convert_workspace_bytes(num_nodes, nnz, block_h, block_w, &need);
  if (s != DTC_OK) return s;
  DTC_REQUIRE(num_blocks >= 0 && num_blocks <= nnz, "num_blocks out of range");
  DTC_REQUIRE(d_tcblockOffset != nullptr, "null tcblockOffset");
  DTC_REQUIRE((d_values == nullptr) == (d_tcValues == nullptr),
              "values and tcValues must both be set or both be null");
  if (workspace_bytes < need || d_workspace == nullptr) {
    set_error("conversion workspace too small");
    return DTC_ERR_WORKSPACE_TOO_SMALL;
  }
  cudaStream_t st = (cudaStream_t)stream;
  if (num_blocks == 0 || nnz == 0) {
    DTC_CUDA(cudaMemsetAsync(d_tcblockOffset, 0, 4, st));
    return DTC_OK;
  }
  const int32_t nwin = (int32_t)(((int64_t)num_nodes + block_h - 1) / block_h);
  const Layout L = layout(num_nodes, nnz, block_h);
  char* ws = (char*)d_workspace;
  const Csr a = make_csr(d_col, d_rowptr, num_nodes, nwin, block_h, block_w, nnz);
  const Fill f{d_edgeToColumn, d_edgeToRow, d_rowWindowOffset, d_values, d_tcblockRowid,
               d_tcblockOffset, d_sparseAToX, d_tileId, d_tcValues, num_blocks};
  DTC_CUDA(cudaMemsetAsync(ws + L.head, 0, kHead * 4, st));
  s = block_h > kUnitH ? fill_tall(a, f, ws, L, st) : fill_impl(a, f, ws, L, st);
  if (s != DTC_OK) return s;
  DTC_CUDA(cudaGetLastError());
  return DTC_OK;
}
