// CSR relabelling on the GPU: symmetric row/column permutation (applying a
// TCA-style reorder) and transposition (the Aᵀ operand of a backward SpMM).
//
// The reference applies a reorder in Python (reordering/TCA_reorder.py:308-326:
// reorder[i_new] = i_old, d[old] = new, src' = d[src], dst' = d[dst]) and
// rebuilds CSR with scipy (scripts/DTCSpMM/dataset.py:38-44: coo_matrix(...)
// .tocsr(), which sorts the columns of each row and sums duplicate entries).
// Both operations here produce that canonical CSR: the edges are radix-sorted by their
// new row and column, values carried along, and one pass over the sorted edges writes the
// columns, the values and the row pointer. A transposition sorts by the old column only
// (32-bit keys, three passes for 2^19 columns where row and column took five passes of
// 64-bit keys): edges come in row order and the sort is stable. Equal pairs are merged by
// summing their values in input CSR order; as a canonical input has none, the pass assumes
// so, and only where it meets one a second, merging pass follows.
// Bound: DRAM and the sort, 24 bytes per edge and pass. R-MAT 2^19 (16.0 M edges)
// transposed with values: 0.67 ms, of it 0.46 the sort (1.38 ms with a row search per edge,
// 64-bit keys, values gathered through edge numbers and separate passes for flags, scan,
// output and row pointer).
#include <algorithm>
#include <cub/cub.cuh>
#include "common.cuh"

namespace dtc {
namespace {

constexpr int kThreads = 256;

inline unsigned grid_for(int64_t n) {
  int64_t g = (n + kThreads - 1) / kThreads;
  if (g < 1) g = 1;
  if (g > (1 << 30)) g = 1 << 30;
  return (unsigned)g;
}

inline int bits_for(uint64_t n) {
  int b = 0;
  while (b < 63 && (1ull << b) < n) ++b;
  return b < 1 ? 1 : b;
}

// inv[perm[i]] = i; marks bad[0] when perm is not a permutation of [0, M).
__global__ void k_invert(const int32_t* __restrict__ perm, int32_t M, int32_t* __restrict__ inv,
                         int32_t* __restrict__ seen, uint32_t* bad) {
  int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < M; i += stride) {
    const int32_t o = perm[i];
    if (o < 0 || o >= M) { atomicOr(bad, 1u); continue; }
    if (atomicAdd(seen + o, 1) != 0) { atomicOr(bad, 1u); continue; }
    inv[o] = (int32_t)i;
  }
}

// The edges in sorted order. Transposition: key = new row (the old column), `row` the old
// row of each edge, alone or (pair) with its value; otherwise key = new row << colbits |
// new column and `val` the values.
template <bool kT>
struct Sorted {
  const uint32_t* key32;
  const uint64_t* key64;
  const uint32_t* row;
  const uint2* pair;
  const float* val;
  int colbits;
  __device__ __forceinline__ uint2 at(int64_t i) const {  // (new row, new column)
    if constexpr (kT) return make_uint2(__ldg(key32 + i), pair ? __ldg(&pair[i].x) : __ldg(row + i));
    const uint64_t k = __ldg(key64 + i);
    return make_uint2((uint32_t)(k >> colbits), (uint32_t)(k & ((1ull << colbits) - 1)));
  }
  __device__ __forceinline__ uint2 at(int64_t i, float& x) const {  // and, of pairs, the value
    if constexpr (kT) {
      const uint2 v = pair ? __ldg(pair + i) : make_uint2(__ldg(row + i), __float_as_uint(1.0f));
      x = __uint_as_float(v.y);
      return make_uint2(__ldg(key32 + i), v.x);
    }
    return at(i);
  }
  __device__ __forceinline__ float value(int64_t i) const {
    if constexpr (kT) return pair ? __uint_as_float(__ldg(&pair[i].y)) : 1.0f;
    return val ? __ldg(val + i) : 1.0f;
  }
};

// The last r in [0, M) with rowptr[r] <= e, found by a warp, 32 probes at a time. Probes
// stay in rowptr[1, M) for any contents.
__device__ __forceinline__ int32_t row_at(const int32_t* __restrict__ rowptr, int32_t M, int64_t e) {
  int32_t lo = 0, hi = M;
  while (hi - lo > 1) {
    const int32_t step = (hi - lo) / 33 + 1;
    const int64_t p = lo + (int64_t)(threadIdx.x % 32 + 1) * step;
    const int before = __popc(__ballot_sync(0xffffffffu, p < hi && __ldg(rowptr + p) <= e));
    lo += before * step;
    hi = (int32_t)min((int64_t)hi, (int64_t)lo + step);
  }
  return lo;
}

// Checks the input (CSR: rowptr[0] == 0, non-decreasing, rowptr[M] == nnz; 0 <= col < K;
// COO, mode 2: 0 <= row < M) and writes the keys and what they carry. A CTA takes 2048
// edges: it marks the places where rows start and a maximum scan gives every edge its row
// (a search per edge took 19 dependent loads, 211 us for R-MAT 2^19; a warp per row walks
// each hub row alone). mode 0: permutation (inv applied to row and column), 1: transpose,
// 2: identity. Bad inputs are clamped: they stay in bounds until the host reads the error.
constexpr int kTile = 2048;
__global__ void __launch_bounds__(kThreads)
    k_expand(const int32_t* __restrict__ rowptr, const int32_t* __restrict__ col,
             const float* __restrict__ val, const int32_t* __restrict__ inv, int32_t M, int32_t K,
             int64_t nnz, int mode, int colbits, uint32_t* __restrict__ key32,
             uint64_t* __restrict__ key64, uint32_t* __restrict__ row_pay,
             uint2* __restrict__ pair_pay, uint32_t* bad) {
  __shared__ int32_t row[kTile], warp_max[kThreads / 32], ends[2];
  const int t = threadIdx.x;
  const int64_t t0 = (int64_t)blockIdx.x * kTile;
  if (mode != 2)
    for (int64_t r = (int64_t)blockIdx.x * kThreads + t; r < M; r += (int64_t)gridDim.x * kThreads) {
      const int32_t e0 = __ldg(rowptr + r), e1 = __ldg(rowptr + r + 1);
      if (e1 < e0 || (r == 0 && e0 != 0) || (r == M - 1 && e1 != nnz)) atomicOr(bad, 2u);
    }
  if (t0 >= nnz) return;
  const int cnt = (int)min((int64_t)kTile, nnz - t0);
  constexpr int V = kTile / kThreads;
  int32_t c[V], r[V];
  float x[V];
#pragma unroll
  for (int v = 0; v < V; ++v) {  // (under way while the rows are found)
    const int i = v * kThreads + t;
    c[v] = i < cnt ? __ldg(col + t0 + i) : 0;
    x[v] = i < cnt && pair_pay ? __ldg(val + t0 + i) : 0.0f;
    r[v] = i < cnt && mode == 2 ? __ldg(rowptr + t0 + i) : 0;
  }
  if (mode != 2) {
    if (t < 64) {
      const int32_t r = row_at(rowptr, M, t < 32 ? t0 : t0 + cnt - 1);
      if (t % 32 == 0) ends[t / 32] = r;
    }
    for (int i = t; i < kTile; i += kThreads) row[i] = 0;
    __syncthreads();
    const int32_t r0 = ends[0], r1 = ends[1];
    for (int32_t r = r0 + 1 + t; r <= r1; r += kThreads) {
      const int64_t at = __ldg(rowptr + r) - t0;
      if (at >= 0 && at < kTile) atomicMax(row + at, r);  // (the last of rows that start here)
    }
    __syncthreads();
    int32_t y[V];  // eight neighbours per thread
#pragma unroll
    for (int v = 0; v < V; ++v) {
      y[v] = row[t * V + v];
      if (v) y[v] = max(y[v], y[v - 1]);
    }
    int32_t m = y[V - 1];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int32_t u = __shfl_up_sync(0xffffffffu, m, o);
      if ((t & 31) >= o) m = max(m, u);
    }
    if ((t & 31) == 31) warp_max[t >> 5] = m;
    __syncthreads();
    int32_t before = __shfl_up_sync(0xffffffffu, m, 1);
    if ((t & 31) == 0) before = 0;
    before = max(before, r0);
    for (int i = 0; i < (t >> 5); ++i) before = max(before, warp_max[i]);
#pragma unroll
    for (int v = 0; v < V; ++v) row[t * V + v] = max(y[v], before);
    __syncthreads();
#pragma unroll
    for (int v = 0; v < V; ++v) r[v] = row[v * kThreads + t];
  }
#pragma unroll
  for (int v = 0; v < V; ++v) {
    if (v * kThreads + t < cnt && (c[v] < 0 || c[v] >= K || r[v] < 0 || r[v] >= M)) {
      atomicOr(bad, 2u);
      c[v] = c[v] < 0 ? 0 : (c[v] >= K ? max(K - 1, 0) : c[v]);
      r[v] = r[v] < 0 ? 0 : (r[v] >= M ? M - 1 : r[v]);
    }
    if (mode == 0 && v * kThreads + t < cnt) {
      r[v] = __ldg(inv + r[v]);
      c[v] = __ldg(inv + c[v]);
    }
  }
#pragma unroll
  for (int v = 0; v < V; ++v) {
    const int64_t e = t0 + v * kThreads + t;
    if (e >= nnz) break;
    if (mode != 1) {
      key64[e] = (uint64_t)(uint32_t)r[v] << colbits | (uint32_t)c[v];
    } else {
      key32[e] = (uint32_t)c[v];
      if (pair_pay) pair_pay[e] = make_uint2((uint32_t)r[v], __float_as_uint(x[v]));
      else row_pay[e] = (uint32_t)r[v];
    }
  }
}

// rowptr[first .. end) = value by each thread of a warp; long runs (rows without entries) by all
// of its lanes, one after the other. A thread alone wrote 8 M rows in 30 to 160 ms.
__device__ __forceinline__ void fill_rows(int32_t* __restrict__ rowptr, uint32_t first,
                                          uint32_t end, int32_t value) {
  const bool far = end > first && end - first > 32;
  if (!far)
    for (uint32_t r = first; r < end; ++r) rowptr[r] = value;
  for (uint32_t m = __ballot_sync(0xffffffffu, far); m; m &= m - 1) {
    const int src = __ffs(m) - 1;
    const uint32_t r1 = __shfl_sync(0xffffffffu, end, src);
    const int32_t x = __shfl_sync(0xffffffffu, value, src);
    for (int64_t r = (int64_t)__shfl_sync(0xffffffffu, first, src) + threadIdx.x % 32; r < r1; r += 32)
      rowptr[r] = x;
  }
}

// Writes the result where all pairs differ (bad[1] = 1 where some do not): edge i is entry
// i; the first edge of a row also fills the row pointer since the row before. Writes nothing
// for an invalid input (bad[0]), whose call leaves the outputs as they are; once an equal pair
// was met, the rest is left to the merging pass, which writes all of it again.
template <bool kT>
__global__ void __launch_bounds__(kThreads)
    k_emit(const Sorted<kT> in, int64_t nnz, int32_t rows, int32_t* __restrict__ rowptr,
           int32_t* __restrict__ col_out, float* __restrict__ val_out, uint32_t* bad) {
  constexpr int V = kTile / kThreads;
  const int64_t t0 = (int64_t)blockIdx.x * kTile + threadIdx.x;
  uint2 k[V], p[V];
  float x[V];
#pragma unroll
  for (int v = 0; v < V; ++v) {
    const int64_t i = t0 + v * kThreads;
    k[v] = i < nnz ? in.at(i, x[v]) : make_uint2((uint32_t)rows, 0);
    p[v] = i > 0 && i <= nnz ? in.at(i - 1) : make_uint2(i > nnz ? (uint32_t)rows : 0xffffffffu, 0);
  }
  // (one thread asks: the words are one place in L2, 16 requests per CTA took 0.1 ms)
  if (__syncthreads_or(threadIdx.x == 0 && *(volatile uint64_t*)bad != 0)) return;
  bool equal = false;
#pragma unroll
  for (int v = 0; v < V; ++v) {
    const int64_t i = t0 + v * kThreads;
    fill_rows(rowptr, p[v].x + 1, k[v].x + 1, (int32_t)i);
    if (i >= nnz) continue;
    equal |= p[v].x == k[v].x && p[v].y == k[v].y;
    col_out[i] = (int32_t)k[v].y;
    if (val_out) val_out[i] = kT ? x[v] : in.value(i);
  }
  if (__any_sync(0xffffffffu, equal) && threadIdx.x % 32 == 0) bad[1] = 1;  // (a store per pair: 0.15 ms)
}

// counts[b] = first edges of equal pairs among the edges of tile b; 0 past the last one.
template <bool kT>
__global__ void __launch_bounds__(kThreads)
    k_firsts(const Sorted<kT> in, int64_t nnz, int32_t* __restrict__ counts) {
  __shared__ int32_t sum;
  const int64_t t0 = (int64_t)blockIdx.x * kTile + threadIdx.x;
  if (threadIdx.x == 0) sum = 0;
  int mine = 0;
#pragma unroll
  for (int v = 0; v < kTile / kThreads; ++v) {
    const int64_t i = t0 + v * kThreads;
    if (i >= nnz) continue;
    const uint2 k = in.at(i), p = i > 0 ? in.at(i - 1) : make_uint2(0xffffffffu, 0);
    mine += k.x != p.x || k.y != p.y;
  }
  mine = __reduce_add_sync(0xffffffffu, mine);
  __syncthreads();
  if (threadIdx.x % 32 == 0) atomicAdd(&sum, mine);
  __syncthreads();
  if (threadIdx.x == 0) counts[blockIdx.x] = sum;
}

// The result with equal pairs merged: the first edge of each sums up the values (input CSR
// order) and writes its entry, the number of first edges before it: `before` its tile
// (k_firsts, summed up), and in it by a scan over the CTA. A flag and a sum per edge in memory
// instead cost 16 bytes per edge more.
template <bool kT>
__global__ void __launch_bounds__(kThreads)
    k_emit_merged(const Sorted<kT> in, const int32_t* __restrict__ before, int64_t nnz,
                  int32_t rows, int32_t* __restrict__ rowptr, int32_t* __restrict__ col_out,
                  float* __restrict__ val_out) {
  __shared__ int32_t part[kTile / 32];
  constexpr int V = kTile / kThreads;
  const int lane = threadIdx.x % 32, warp = threadIdx.x / 32;
  const int64_t t0 = (int64_t)blockIdx.x * kTile + threadIdx.x;
  uint2 k[V], p[V];
  uint32_t firsts[V];  // of the 32 edges of this warp's v-th load
#pragma unroll
  for (int v = 0; v < V; ++v) {
    const int64_t i = t0 + v * kThreads;
    k[v] = i < nnz ? in.at(i) : make_uint2((uint32_t)rows, 0);
    p[v] = i > 0 && i <= nnz ? in.at(i - 1) : make_uint2(i > nnz ? (uint32_t)rows : 0xffffffffu, 0);
    firsts[v] = __ballot_sync(0xffffffffu, i < nnz && (k[v].x != p[v].x || k[v].y != p[v].y));
    if (lane == 0) part[v * (kThreads / 32) + warp] = __popc(firsts[v]);
  }
  __syncthreads();
  if (warp == 0) {  // sums before each 32 edges, two per lane
    static_assert(kTile / 32 == 64, "two per lane");
    const int a = part[2 * lane], b = part[2 * lane + 1];
    int y = a + b;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, y, o);
      if (lane >= o) y += u;
    }
    part[2 * lane] = y - a - b;
    part[2 * lane + 1] = y - b;
  }
  __syncthreads();
  const int32_t base = before[blockIdx.x];
#pragma unroll
  for (int v = 0; v < V; ++v) {
    const int64_t i = t0 + v * kThreads;
    const int32_t o =
        base + part[v * (kThreads / 32) + warp] + __popc(firsts[v] & ((1u << lane) - 1));
    fill_rows(rowptr, p[v].x + 1, k[v].x + 1, o);
    if (!(firsts[v] >> lane & 1)) continue;
    col_out[o] = (int32_t)k[v].y;
    if (val_out) {
      float s = in.value(i);
      for (int64_t j = i + 1; j < nnz; ++j) {
        const uint2 q = in.at(j);
        if (q.x != k[v].x || q.y != k[v].y) break;
        s += in.value(j);
      }
      val_out[o] = s;
    }
  }
}

struct Layout {
  size_t inv, seen, keys_in, keys_out, pay_in, pay_out, bad, sort, scan;
  size_t total;
  int colbits, endbit;
};

// Workspace of a mode; the merging pass's counts per tile and their sums take the place of
// the unsorted keys and what they carried (at least 4 bytes per edge each, and one more).
Layout layout(int32_t rows_in, int32_t cols_in, int64_t nnz, int mode, bool with_val) {
  Layout L{};
  const int32_t rows_out = mode == 1 ? cols_in : rows_in;
  const int32_t cols_out = mode == 1 ? rows_in : cols_in;
  const int rowbits = bits_for((uint64_t)(rows_out > 0 ? rows_out : 1));
  L.colbits = mode == 1 ? 0 : bits_for((uint64_t)(cols_out > 0 ? cols_out : 1));
  L.endbit = L.colbits + rowbits;
  const size_t n = (size_t)(nnz > 0 ? nnz : 1);
  const size_t m = (size_t)(rows_in > 0 ? rows_in : 1);
  const size_t key = mode == 1 ? 4 : 8, pay = mode == 1 && with_val ? 8 : 4;
  size_t off = 0;
  auto take = [&](size_t bytes) { size_t o = off; off = align_up(off + bytes, 256); return o; };
  L.inv = take(mode == 0 ? m * 4 : 0);
  L.seen = take(mode == 0 ? m * 4 : 0);
  L.keys_in = take((n + 1) * key);
  L.keys_out = take(n * key);
  L.pay_in = take((n + 1) * pay);
  L.pay_out = take(n * pay);
  L.bad = take(16);
  size_t s1 = 0, s2 = 0;
  if (mode == 1 && with_val)
    cub::DeviceRadixSort::SortPairs(nullptr, s1, (uint32_t*)nullptr, (uint32_t*)nullptr,
                                    (uint64_t*)nullptr, (uint64_t*)nullptr, (int64_t)n, 0, L.endbit);
  else if (mode == 1)
    cub::DeviceRadixSort::SortPairs(nullptr, s1, (uint32_t*)nullptr, (uint32_t*)nullptr,
                                    (uint32_t*)nullptr, (uint32_t*)nullptr, (int64_t)n, 0, L.endbit);
  else if (with_val)
    cub::DeviceRadixSort::SortPairs(nullptr, s1, (uint64_t*)nullptr, (uint64_t*)nullptr,
                                    (uint32_t*)nullptr, (uint32_t*)nullptr, (int64_t)n, 0, L.endbit);
  else
    cub::DeviceRadixSort::SortKeys(nullptr, s1, (uint64_t*)nullptr, (uint64_t*)nullptr, (int64_t)n,
                                   0, L.endbit);
  cub::DeviceScan::ExclusiveSum(nullptr, s2, (int32_t*)nullptr, (int32_t*)nullptr,
                                (int64_t)n / kTile + 2);
  L.sort = take(s1);
  L.scan = take(s2);
  L.total = off;
  return L;
}

// From the sorted edges to the result; reads the input's error word on the way.
template <bool kT>
dtc_status emit(const Sorted<kT>& in, int64_t nnz, int32_t rows_out, int32_t* rowptr_out,
                int32_t* col_out, float* val_out, int32_t* counts, int32_t* before, uint32_t* bad,
                void* scan, size_t scan_bytes, uint32_t* hbad, int64_t* nnz_out, cudaStream_t st) {
  k_emit<kT><<<(unsigned)(nnz / kTile + 1), kThreads, 0, st>>>(in, nnz, rows_out, rowptr_out,
                                                              col_out, val_out, bad);
  DTC_CUDA(cudaGetLastError());
  DTC_CUDA(cudaMemcpyAsync(hbad, bad, 8, cudaMemcpyDeviceToHost, st));
  DTC_CUDA(cudaStreamSynchronize(st));
  if (hbad[0]) return DTC_OK;  // (the caller reports it)
  *nnz_out = nnz;
  if (!hbad[1]) return DTC_OK;
  const int64_t tiles = nnz / kTile + 1;  // (the last one has the end of the row pointer)
  k_firsts<kT><<<(unsigned)tiles, kThreads, 0, st>>>(in, nnz, counts);
  // (the sums of one tile more: the last is the number of entries)
  DTC_CUDA(cudaMemsetAsync(counts + tiles, 0, 4, st));
  DTC_CUDA(cub::DeviceScan::ExclusiveSum(scan, scan_bytes, counts, before, tiles + 1, st));
  k_emit_merged<kT><<<(unsigned)tiles, kThreads, 0, st>>>(in, before, nnz, rows_out, rowptr_out,
                                                         col_out, val_out);
  DTC_CUDA(cudaGetLastError());
  int32_t hn = 0;
  DTC_CUDA(cudaMemcpyAsync(&hn, before + tiles, 4, cudaMemcpyDeviceToHost, st));
  DTC_CUDA(cudaStreamSynchronize(st));
  *nnz_out = hn;
  return DTC_OK;
}

dtc_status relabel(int mode, const int32_t* rowptr, const int32_t* col, const float* val,
                   int32_t M, int32_t K, int64_t nnz, const int32_t* perm, int32_t* rowptr_out,
                   int32_t* col_out, float* val_out, int64_t* nnz_out, void* ws, size_t wsb,
                   cudaStream_t st) {
  DTC_REQUIRE(M >= 0 && K >= 0 && nnz >= 0, "negative sizes");
  DTC_REQUIRE(M > 0 || nnz == 0, "a matrix without rows has no entries");
  DTC_REQUIRE(nnz < (int64_t)INT32_MAX, "nnz must fit in int32");
  DTC_REQUIRE(nnz_out != nullptr, "nnz_out is null");
  DTC_REQUIRE((rowptr || (mode == 2 && nnz == 0)) && rowptr_out, "null device pointer");
  DTC_REQUIRE(nnz == 0 || (col && col_out), "null device pointer");
  DTC_REQUIRE(mode != 0 || perm || M == 0, "perm is null");
  const bool with_val = val != nullptr && val_out != nullptr;
  const Layout L = layout(M, K, nnz, mode, with_val);
  if (!ws || wsb < L.total) {
    set_error("relabel workspace too small");
    return DTC_ERR_WORKSPACE_TOO_SMALL;
  }
  char* w = (char*)ws;
  int32_t* inv = (int32_t*)(w + L.inv);
  int32_t* seen = (int32_t*)(w + L.seen);
  void *kin = w + L.keys_in, *kout = w + L.keys_out, *pin = w + L.pay_in, *pout = w + L.pay_out;
  uint32_t* bad = (uint32_t*)(w + L.bad);  // error bits; 1 where two pairs are equal
  const int32_t rows_out = mode == 1 ? K : M;
  DTC_CUDA(cudaMemsetAsync(bad, 0, 8, st));
  if (mode == 0 && M > 0) {
    DTC_CUDA(cudaMemsetAsync(inv, 0, (size_t)M * 4, st));  // (in range for a bad perm too)
    DTC_CUDA(cudaMemsetAsync(seen, 0, (size_t)M * 4, st));
    k_invert<<<grid_for(M), kThreads, 0, st>>>(perm, M, inv, seen, bad);
  }
  if (M > 0) {
    const int64_t tiles = (nnz + kTile - 1) / kTile;
    const int64_t rows = mode == 2 ? 1 : std::min<int64_t>(((int64_t)M + kThreads - 1) / kThreads, 2048);
    k_expand<<<(unsigned)std::max(tiles, rows), kThreads, 0, st>>>(
        rowptr, col, val, inv, M, K, nnz, mode, L.colbits, (uint32_t*)kin, (uint64_t*)kin,
        (uint32_t*)pin, mode == 1 && with_val ? (uint2*)pin : nullptr, bad);
    DTC_CUDA(cudaGetLastError());
  }
  uint32_t hbad[2] = {0, 0};
  dtc_status s = DTC_OK;
  if (nnz == 0) {
    DTC_CUDA(cudaMemcpyAsync(hbad, bad, 4, cudaMemcpyDeviceToHost, st));
    DTC_CUDA(cudaStreamSynchronize(st));
  } else {
    size_t sb = L.scan - L.sort;
    const size_t cb = L.total - L.scan;
    if (mode == 1 && with_val)
      DTC_CUDA(cub::DeviceRadixSort::SortPairs(w + L.sort, sb, (uint32_t*)kin, (uint32_t*)kout,
                                               (uint64_t*)pin, (uint64_t*)pout, nnz, 0, L.endbit, st));
    else if (mode == 1)
      DTC_CUDA(cub::DeviceRadixSort::SortPairs(w + L.sort, sb, (uint32_t*)kin, (uint32_t*)kout,
                                               (uint32_t*)pin, (uint32_t*)pout, nnz, 0, L.endbit, st));
    else if (with_val)
      DTC_CUDA(cub::DeviceRadixSort::SortPairs(w + L.sort, sb, (uint64_t*)kin, (uint64_t*)kout,
                                               (const uint32_t*)val, (uint32_t*)pout, nnz, 0,
                                               L.endbit, st));
    else
      DTC_CUDA(cub::DeviceRadixSort::SortKeys(w + L.sort, sb, (uint64_t*)kin, (uint64_t*)kout, nnz, 0,
                                              L.endbit, st));
    if (mode == 1)
      s = emit(Sorted<true>{(uint32_t*)kout, nullptr, (uint32_t*)pout,
                            with_val ? (uint2*)pout : nullptr, nullptr, 0},
               nnz, rows_out, rowptr_out, col_out, val_out, (int32_t*)kin, (int32_t*)pin, bad,
               w + L.scan, cb, hbad, nnz_out, st);
    else
      s = emit(Sorted<false>{nullptr, (uint64_t*)kout, nullptr, nullptr,
                             with_val ? (float*)pout : nullptr, L.colbits},
               nnz, rows_out, rowptr_out, col_out, val_out, (int32_t*)kin, (int32_t*)pin, bad,
               w + L.scan, cb, hbad, nnz_out, st);
    if (s != DTC_OK) return s;
  }
  if (hbad[0] & 1u) {
    set_error("perm is not a permutation of [0, num_nodes)");
    return DTC_ERR_INVALID_ARGUMENT;
  }
  if (hbad[0] & 2u) {
    set_error(mode == 2 ? "invalid COO (a coordinate out of range)"
                        : "invalid CSR (rowptr not monotone from 0 to nnz, or a column out of range)");
    return DTC_ERR_INVALID_ARGUMENT;
  }
  if (nnz == 0) {
    DTC_CUDA(cudaMemsetAsync(rowptr_out, 0, ((size_t)rows_out + 1) * 4, st));
    *nnz_out = 0;
  }
  return DTC_OK;
}

}  // namespace
}  // namespace dtc

using namespace dtc;

extern "C" {

dtc_status dtc_relabel_workspace_bytes(int32_t num_rows, int32_t num_cols, int64_t nnz,
                                       size_t* bytes) {
  DTC_REQUIRE(bytes != nullptr, "bytes is null");
  DTC_REQUIRE(num_rows >= 0 && num_cols >= 0 && nnz >= 0, "negative sizes");
  *bytes = 0;
  for (int mode = 0; mode < 2; ++mode)  // (a COO input needs no more than a permutation)
    for (bool with_val : {false, true})
      *bytes = std::max(*bytes, layout(num_rows, num_cols, nnz, mode, with_val).total);
  return DTC_OK;
}

dtc_status dtc_permute_csr(const int32_t* d_rowptr, const int32_t* d_col, const float* d_val,
                           int32_t num_nodes, int64_t nnz, const int32_t* d_perm,
                           int32_t* d_rowptr_out, int32_t* d_col_out, float* d_val_out,
                           int64_t* nnz_out, void* d_workspace, size_t workspace_bytes,
                           dtc_stream_t stream) {
  return relabel(0, d_rowptr, d_col, d_val, num_nodes, num_nodes, nnz, d_perm, d_rowptr_out,
                 d_col_out, d_val_out, nnz_out, d_workspace, workspace_bytes,
                 (cudaStream_t)stream);
}

dtc_status dtc_transpose_csr(const int32_t* d_rowptr, const int32_t* d_col, const float* d_val,
                             int32_t num_rows, int32_t num_cols, int64_t nnz,
                             int32_t* d_rowptr_out, int32_t* d_col_out, float* d_val_out,
                             int64_t* nnz_out, void* d_workspace, size_t workspace_bytes,
                             dtc_stream_t stream) {
  return relabel(1, d_rowptr, d_col, d_val, num_rows, num_cols, nnz, nullptr, d_rowptr_out,
                 d_col_out, d_val_out, nnz_out, d_workspace, workspace_bytes,
                 (cudaStream_t)stream);
}

dtc_status dtc_coo_to_csr(const int32_t* d_src, const int32_t* d_dst, const float* d_val,
                          int32_t num_rows, int32_t num_cols, int64_t nnz, int32_t* d_rowptr_out,
                          int32_t* d_col_out, float* d_val_out, int64_t* nnz_out,
                          void* d_workspace, size_t workspace_bytes, dtc_stream_t stream) {
  return relabel(2, d_src, d_dst, d_val, num_rows, num_cols, nnz, nullptr,
                 d_rowptr_out, d_col_out, d_val_out, nnz_out, d_workspace, workspace_bytes,
                 (cudaStream_t)stream);
}

}  // extern "C"
