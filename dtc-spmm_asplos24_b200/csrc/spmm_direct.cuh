// TC-block SpMM with register fragments (mma.sync): every warp runs its own range of
// TC blocks, from the gather of the dense rows to the stores of C. The narrow widths,
// the odd ones and the forms that rebuild their operand rows run here; the others on
// tcgen05 (spmm_umma.cuh; the rule is in spmm_run).
//
// Why warp-level instructions. A TC block is 16 x 8 (32 x 8, 16 x 16) with 9-20
// nonzeros: as a tcgen05 operand it uses K = 8 and N = 16 of the 128-row
// instruction, of which an SM takes one per 40-56 cycles, and at up to 64 features
// half of its rows are empty. m16n8k8 has the block's own shape (window rows = M,
// slots = K; 2 cycles per instruction and SM, measured), a lane's B fragment is the
// 16 bytes it loads, and no warp waits for another one.
//
// Fragments. Lane l = 4 gr + gc of an m16n8k8 holds B[k = gc and gc + 4][n = gr].
// The order of the k rows and of the n columns is free. k = gc and gc + 4 are slots
// 2 gc and 2 gc + 1; fp32: a lane loads 4 features of a slot (16 bytes) for the four
// instructions of a group of 32 features; bf16: ldmatrix gives the pairs of slots of
// 8 features. The gather itself copies a whole 128-byte line with 8 lanes: with the
// fragment order instead (4 lines per 8 lanes) L2 returned twice the bytes and
// R-MAT 2^20, N = 128 took 3.8 ms instead of 1.7.
//
// Pipeline of one warp. A step is 8 slots (a block of width 16 is two), a group four
// steps; the loop runs the four phases of a group with compile-time places and
// leaves it at a window's end. Step i of group g sits in slot i of the warp's ring
// and its copies start when step i of group g - 1 is consumed: three to four steps
// (4 KB each at 128 fp32 features) are in flight. SparseAToX of a step is loaded two
// groups ahead, TCblockoffset three, tile ids and values one; the A values are
// scattered to one 512-byte tile per step, and zeroed by the lane that reads them.
// What bounds it: instruction latency of about 150 instructions per step with 12-16
// warps per SM (registers: the accumulators), not bytes: without the gather the same
// loop takes 0.80 of the time (R-MAT 2^19, N = 128: 0.60 of 0.75 ms), and 0.42 ms are
// enough for the gather alone.
// Measured on a B200 (tcgen05 pipeline before / this), R-MAT 2^19, 16 x 8 blocks:
// fp32 N = 64 1.42 / 0.46 ms, N = 128 1.29 / 0.73 ms; SPLIT24 N = 128 2.32 / 1.18 ms;
// FP8 N = 128 2.27 / 0.90 ms; fp32 N = 41, R-MAT 2^17: 6.9 ms (one CTA per window,
// no prefetch) / 0.3 ms.
//
// Work split (both kernels). The TC blocks are cut into G chunks, one CTA each (the
// hardware scheduler balances them), and here a chunk into one range per warp. A
// boundary that falls into a window of at most `lmax` blocks (chunks) or half a range
// (ranges) moves to the window's start; larger windows are cut there. Inside a CTA
// the pieces of a cut window are added right to left (the warp on the right stores
// its piece, sets a flag, the warp to its left adds its own). A window cut by a chunk
// boundary leaves its first piece in C and each later chunk's piece in that chunk's
// slot of the workspace; k_add_slots adds them in chunk order. Without a workspace
// (SEQ) clusters of kTeam CTAs take the chunks: see kTeam.
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp8.h>
#include <type_traits>
#include "common.cuh"
#include "impl.h"

namespace dtc {
enum { kF32 = 0, kF32Odd = 1, kBF16X2 = 2, kSplit24 = 3, kBF16 = 4, kFP8 = 5 };

struct DirectParams {
  const int32_t* rwo;        // RowWindowOffset [nwin+1]
  const int32_t* toff;       // TCblockoffset [T+1]
  const int32_t* s2x;        // SparseAToX [T*W]
  const uint8_t* tile;       // TCblocktileId [nnz]
  const float* vals;         // tile-order values or null (A = 1)
  const void* b0;            // B: fp32 rows / bf16 (hi) plane / e4m3 plane
  const void* b1;            // second plane: bf16 lo / u8 extension / fp32 row scales
  float* C;                  // [M x N]
  float* slots;              // [G x H x N] pieces of windows cut by chunk boundaries, or null
  uint32_t* err;
  uint64_t* stamps;          // per-CTA timer records or null
  int32_t stamp_cap;
  const float* bias;         // epilogue bias [N] or null
  int32_t relu;
  int32_t M, nwin, N, G, H;
  int32_t G1;                // chunks of the first three quarters (0: all chunks alike)
  int32_t lmax;              // windows of more blocks are cut at chunk boundaries
  int32_t wf;                // feature slices (warps side by side) per CTA (mma.sync kernel)
  int32_t T;
};

// The products of each B form (one translation unit per pair of forms).
dtc_status direct_f32(DirectParams& p, int W, cudaStream_t st);
dtc_status direct_f32_odd(DirectParams& p, int W, cudaStream_t st);
dtc_status direct_bf16x2(DirectParams& p, int W, bool four, cudaStream_t st);
dtc_status direct_split24(DirectParams& p, int W, bool four, cudaStream_t st);
dtc_status direct_bf16(DirectParams& p, int W, cudaStream_t st);
dtc_status direct_fp8(DirectParams& p, int W, cudaStream_t st);
dtc_status umma_f32(DirectParams& p, int W, cudaStream_t st);
dtc_status umma_bf16x2(DirectParams& p, int W, bool four, cudaStream_t st);
dtc_status umma_bf16(DirectParams& p, int W, cudaStream_t st);
constexpr int kNW = 4;  // warps per CTA

namespace {

__device__ __forceinline__ float finish(const DirectParams& p, float x, int f) {
  if (p.bias) x += __ldg(p.bias + f);
  return p.relu ? fmaxf(x, 0.0f) : x;
}

// ---------------------------------------------------------------- work split
// First index in [lo, hi) with a[i] >= x (hi if none), for two searches at once:
// lanes 0-15 and 16-31 each probe 16-ary, all lanes return both answers.
__device__ __forceinline__ int2 search2(const int32_t* a, int32_t lo0, int32_t hi0, int32_t x0,
                                        int32_t lo1, int32_t hi1, int32_t x1, int lane) {
  const int half = lane >> 4, l = lane & 15;
  int32_t lo = half ? lo1 : lo0, hi = half ? hi1 : hi0;
  const int32_t x = half ? x1 : x0;
  while (__any_sync(0xffffffffu, lo < hi)) {
    const int32_t step = (hi - lo + 15) >> 4;
    const int32_t at = lo + l * step;
    const bool ge = at < hi ? __ldg(a + at) >= x : true;
    const uint32_t m = (__ballot_sync(0xffffffffu, ge) >> (16 * half)) & 0xffffu;
    const int j = m ? __ffs(m) - 1 : 16;
    const int32_t nhi = min(lo + j * step, hi);
    if (j > 0) lo = lo + (j - 1) * step + 1;
    hi = nhi;
  }
  return make_int2(__shfl_sync(0xffffffffu, lo, 0), __shfl_sync(0xffffffffu, lo, 16));
}

// A place where the blocks are cut: its block, the window there (the last one
// that starts at or before it) and whether that window starts earlier.
struct Cut {
  int32_t pos, win;
  bool open;
};

// The cut of block c, where `i` is the answer of a search for c + 1. A table that starts at 0
// and ends at T holds c in window i - 1 even where it is not ascending (made from a caller's
// invalid window ids): the search has seen rwo[i - 1] <= c < rwo[i]. The clamps are for a table
// that the caller made.
__device__ __forceinline__ Cut cut_at(const DirectParams& p, int32_t c, int32_t i, int32_t most) {
  const int32_t w = max(i - 1, 0);
  const int32_t ws = min(max(__ldg(p.rwo + w), 0), p.T), we = __ldg(p.rwo + w + 1);
  Cut b;
  b.win = w;
  b.open = ws < c && we - ws > most;
  b.pos = b.open ? c : ws;
  return b;
}

__device__ __forceinline__ int32_t chunk_start(const DirectParams& p, int32_t k) {
  // the first G1 chunks hold the first three quarters of the blocks, the others (a
  // quarter as long) the rest: the last CTAs to start are short
  const int32_t big = (int32_t)((int64_t)p.T * 3 / 4), G1 = p.G1, G2 = p.G - p.G1;
  return k <= G1 && G1 > 0 ? (int32_t)((int64_t)k * big / G1)
                           : (int32_t)(big * (G1 > 0) + (int64_t)(k - G1) * (p.T - big * (G1 > 0)) / G2);
}

// Both ends of chunk k.
__device__ __forceinline__ void chunk_cuts(const DirectParams& p, int32_t k, int lane, Cut& b0,
                                           Cut& b1) {
  const int32_t x0 = chunk_start(p, k), x1 = chunk_start(p, k + 1);
  const int2 i = search2(p.rwo, 0, p.nwin, x0 + 1, 0, p.nwin, min(x1, p.T - 1) + 1, lane);
  b0 = cut_at(p, x0, i.x, p.lmax);
  if (x1 >= p.T) {
    b1.pos = p.T;
    b1.win = max(i.y - 1, 0);
    b1.open = false;
  } else {
    b1 = cut_at(p, x1, i.y, p.lmax);
  }
}

// Chunks without a workspace. A cluster of kTeam CTAs runs kTeam chunks in a row, one each, and
// keeps their pieces of cut windows in shared memory, where the cluster adds them to the first
// piece (in C), in chunk order: the same sums and bits as k_add_slots. A cut window belongs to
// the cluster whose chunks hold its start. Where it goes on beyond the cluster's last chunk the
// cluster runs its pieces of the next kTeam chunks, round after round, up to its end; those
// chunks' own clusters leave these pieces out. (One CTA for all chunks of windows that follow
// each other without an uncut boundary: R-MAT 2^20, N = 128, fp32 8.7 ms, this 2.4; with a
// workspace 1.44.)
constexpr int kTeam = 8;
// The boundaries base .. base + kTeam of chunks, by all warps of a CTA.
__device__ __forceinline__ void team_cuts(const DirectParams& p, int32_t base, Cut* s, int warp,
                                          int warps, int lane) {
  for (int i = 2 * warp; i <= kTeam; i += 2 * warps) {
    const int32_t x0 = base + i < p.G ? chunk_start(p, base + i) : p.T;
    const int32_t x1 = base + i + 1 < p.G ? chunk_start(p, base + i + 1) : p.T;
    const int2 a = search2(p.rwo, 0, p.nwin, min(x0, p.T - 1) + 1, 0, p.nwin, min(x1, p.T - 1) + 1, lane);
    if (lane == 0) {
      s[i] = x0 < p.T ? cut_at(p, x0, a.x, p.lmax) : Cut{p.T, max(a.x - 1, 0), false};
      if (i < kTeam) s[i + 1] = x1 < p.T ? cut_at(p, x1, a.y, p.lmax) : Cut{p.T, max(a.y - 1, 0), false};
    }
  }
}
// A round of a cluster: the first one (of its own chunks), or of window `only`'s next chunks.
struct Round {
  int32_t only, foreign;  // -1: none; foreign: the window that an earlier cluster adds up
  __device__ __forceinline__ Round(const Cut* cut, int32_t only_)
      : only(only_), foreign(only_ < 0 && cut[0].open ? cut[0].win : -1) {}
  // whether a piece that starts at boundary c is one of the round's
  __device__ __forceinline__ bool has(const Cut& c) const {
    return c.open && (only >= 0 ? c.win == only : c.win != foreign);
  }
  // member `rank`'s part of chunk k: the windows from c0 on, up to block hi
  __device__ __forceinline__ void part(const DirectParams& p, const Cut* cut, int rank, int32_t k,
                                       int lane, Cut& c0, int32_t& hi) const {
    c0 = cut[rank];
    hi = cut[rank + 1].pos;
    if (only >= 0) {
      hi = has(c0) ? min(hi, min(max(__ldg(p.rwo + only + 1), 0), p.T)) : c0.pos;
    } else if (c0.open && c0.win == foreign) {  // what comes after it
      const int32_t at = min(max(__ldg(p.rwo + c0.win + 1), 0), p.T - 1);
      const int2 i = search2(p.rwo, 0, p.nwin, at + 1, 0, 0, 0, lane);
      c0 = Cut{min(max(__ldg(p.rwo + c0.win + 1), 0), p.T), max(i.x - 1, 0), false};
    }
  }
  __device__ __forceinline__ int32_t next(const Cut* cut) const {  // the next round's window
    return has(cut[kTeam]) ? cut[kTeam].win : -1;
  }
  __device__ __forceinline__ uint32_t pieces(const Cut* cut) const {  // members that have one
    uint32_t m = 0;
    for (int r = 0; r < kTeam; ++r) m |= (uint32_t)has(cut[r]) << r;
    return m;
  }
};
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}
__device__ __forceinline__ float ld_peer(uint32_t addr, int rank) {  // a peer's shared memory
  uint32_t a;
  float v;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(addr), "r"(rank));
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
  return v;
}
// The end of a round: adds up its pieces, H x width floats each at `tile` of the members' shared
// memory, columns from col0 on. Returns the next round's window, -1: the CTA is done (a member
// without a piece need not wait for the others then). Called by all threads.
__device__ __forceinline__ int32_t end_round(const DirectParams& p, const Cut* cut, const Round& round,
                                             const float* tile, int width, int col0, int rank, int t,
                                             int threads) {
  const uint32_t at = smem_u32(tile), pieces = round.pieces(cut);
  const int32_t next = round.next(cut);
  if (pieces == 0 || (next < 0 && !(pieces >> rank & 1))) return next;
  const uint32_t who = next < 0 ? pieces : (1u << kTeam) - 1;  // members that add
  cluster_sync();  // every member's pieces are there
  t += __popc(who & ((1u << rank) - 1)) * threads;
  threads *= __popc(who);
  for (int r = 0; r < kTeam;) {
    if (!round.has(cut[r])) {
      ++r;
      continue;
    }
    const int32_t w = cut[r].win;
    int e = r + 1;  // pieces r .. e - 1 are of one window
    while (e < kTeam && cut[e].open && cut[e].win == w) ++e;
    const bool ends = !(cut[e].open && cut[e].win == w);
    const int64_t row0 = (int64_t)w * p.H;
    const int rows = (int)min((int64_t)p.H, p.M - row0);
    for (int x = t; x < rows * width; x += threads) {
      const int f = col0 + x % width;
      if (f >= p.N) continue;
      float* const c = p.C + (row0 + x / width) * p.N + f;
      float acc = *c;
      for (int q = r; q < e; ++q) acc += ld_peer(at + x * 4, q);
      *c = ends ? finish(p, acc, f) : acc;
    }
    r = e;
  }
  cluster_sync();  // the pieces are read, and what they were added to is written
  return next;
}

// Adds the pieces of every window that chunk boundaries cut to the first piece (in C), in
// chunk order, and applies the epilogue. A CTA looks at kAddCuts boundaries, a warp each
// (most cut no window, and finding that out is a chain of dependent loads: with a CTA per
// boundary it took 90 us for the 7615 of R-MAT 2^20 in 32-row windows, now 28), then all
// its threads add up the windows found.
constexpr int kAddThreads = 256, kAddCuts = 4;
__global__ void __launch_bounds__(kAddThreads) k_add_slots(const DirectParams p) {
  __shared__ int3 found[kAddCuts];  // window, first and last chunk; -1: none
  const int32_t lane = threadIdx.x & 31, wr = threadIdx.x >> 5;
  if (wr < kAddCuts) {
    const int32_t k = blockIdx.x * kAddCuts + wr + 1;
    int3 f = make_int3(-1, 0, 0);
    if (k < p.G) {
      const int32_t c = chunk_start(p, k);
      const int2 i = search2(p.rwo, 0, p.nwin, c + 1, 0, 0, 0, lane);
      const Cut b = cut_at(p, c, i.x, p.lmax);
      const int32_t ws = __ldg(p.rwo + b.win), we = __ldg(p.rwo + b.win + 1);
      if (b.open && !(k > 1 && chunk_start(p, k - 1) > ws)) {  // else an earlier one has it
        f = make_int3(b.win, k, k);
        while (f.z + 1 < p.G && chunk_start(p, f.z + 1) < we) ++f.z;
      }
    }
    if (lane == 0) found[wr] = f;
  }
  __syncthreads();
  const int64_t tile = (int64_t)p.H * p.N;
  const bool vec = p.N % 4 == 0 && (((uintptr_t)p.slots | (uintptr_t)p.C) & 15) == 0;
  for (int u = 0; u < kAddCuts; ++u) {
    const int3 f = found[u];
    if (f.x < 0) continue;
    const int64_t row0 = (int64_t)f.x * p.H;
    const int32_t n = (int32_t)min((int64_t)p.H, p.M - row0) * p.N;
    float* const C = p.C + row0 * p.N;
    const float* const s = p.slots + f.y * tile;
    if (vec) {
      for (int32_t x = threadIdx.x * 4; x < n; x += kAddThreads * 4) {
        float4 acc = *reinterpret_cast<const float4*>(C + x);
#pragma unroll 4
        for (int32_t j = 0; j <= f.z - f.y; ++j) {
          const float4 v = __ldcs(reinterpret_cast<const float4*>(s + j * tile + x));
          acc = make_float4(acc.x + v.x, acc.y + v.y, acc.z + v.z, acc.w + v.w);
        }
        const int32_t c = x % p.N;
        *reinterpret_cast<float4*>(C + x) =
            make_float4(finish(p, acc.x, c), finish(p, acc.y, c + 1), finish(p, acc.z, c + 2),
                        finish(p, acc.w, c + 3));
      }
    } else {
      for (int32_t x = threadIdx.x; x < n; x += kAddThreads) {
        float acc = C[x];
#pragma unroll 4
        for (int32_t j = 0; j <= f.z - f.y; ++j) acc += __ldcs(s + j * tile + x);
        C[x] = finish(p, acc, x % p.N);
      }
    }
  }
}
inline unsigned add_ctas(const DirectParams& p) { return (p.G - 1 + kAddCuts - 1) / kAddCuts; }

// -------------------------------------------------------------- instructions
// Copies to shared memory; `none`: zeros instead, the source is not read.
__device__ __forceinline__ void cp16(uint32_t dst, const void* src, bool none) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %2, 0;\n\t"
      "cp.async.cg.shared.global [%0], [%1], 16, p;\n\t}" ::"r"(dst), "l"(src), "r"((int)none)
      : "memory");
}
__device__ __forceinline__ void cp8(uint32_t dst, const void* src, bool none) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %2, 0;\n\t"
      "cp.async.ca.shared.global [%0], [%1], 8, p;\n\t}" ::"r"(dst), "l"(src), "r"((int)none)
      : "memory");
}
__device__ __forceinline__ void cp4(uint32_t dst, const void* src, bool none) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %2, 0;\n\t"
      "cp.async.ca.shared.global [%0], [%1], 4, p;\n\t}" ::"r"(dst), "l"(src), "r"((int)none)
      : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
// Four 8 x 8 tiles of 16-bit elements, transposed: lane (gr, gc) gets elements
// (2 gc, gr) and (2 gc + 1, gr) of tile i in v[i]; lane l gives the address of row
// l % 8 of tile l / 8.
__device__ __forceinline__ void ldsm4t(uint32_t (&v)[4], uint32_t a) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3])
               : "r"(a)
               : "memory");
}
__device__ __forceinline__ uint32_t rna_tf32(float x) {
  uint32_t r;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ void mma_tf32_k8(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2,
                                            uint32_t a3, uint32_t b0, uint32_t b1) {
  asm(
      "mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void mma_bf16_k16(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2,
                                             uint32_t a3, uint32_t b0, uint32_t b1) {
  asm(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, "
      "{%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void mma_bf16_k8(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t b0) {
  asm(
      "mma.sync.aligned.m16n8k8.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5}, {%6}, "
      "{%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a0), "r"(a1), "r"(b0));
}

// ------------------------------------------------------------------- shapes
// NF features per warp, MH 16-row halves of the window, SUB steps per block
// (block width 8 SUB), NW warps per CTA, P steps per group (= ring slots).
template <int FORM, int NF, int MH, int SUB, int NW, int P>
struct Shape {
  static constexpr bool kFp32 = FORM == kF32 || FORM == kF32Odd;
  static constexpr bool kLdsm = FORM == kBF16X2 || FORM == kBF16;  // fragments by ldmatrix
  static constexpr int kQF = kFp32 ? 32 : 64;       // features of one 16-byte copy per row
  static constexpr int kQ = NF / kQF;
  static constexpr int kJ = kFp32 ? 4 : 8;          // instructions per group of kQF features
  // bytes per step: 16-byte pieces, then 8-byte pieces, then 4-byte ones, lane by lane
  static constexpr int kPlanes16 = FORM == kBF16X2 ? 2 : FORM == kFP8 ? 0 : 1;
  static constexpr int kPieces16 = 2 * kPlanes16 * kQ;
  static constexpr int kPieces8 = (FORM == kSplit24 || FORM == kFP8) ? 2 * kQ : 0;
  static constexpr int kPieces4 = FORM == kFP8 ? 1 : 0;
  static constexpr int kOff8 = kPieces16 * 512;
  static constexpr int kOff4 = kOff8 + kPieces8 * 256;
  static constexpr int kStep = kOff4 + kPieces4 * 128;
  static constexpr int kA = P * MH * 512;           // A tiles of a group
  static constexpr int kWarp = P * kStep + kA;
  static constexpr int kAcc = kQ * kJ * MH * 4;     // accumulators per lane
  static constexpr int kSmem = NW * kWarp;
  static constexpr int PB = P / SUB;                // blocks per group
  static_assert(P == 4 && P % SUB == 0, "four phases");
};

constexpr int kPre = 4;  // tile ids / values per lane loaded one group ahead (128 entries)

template <int FORM, bool FOUR, int NF, int MH, int SUB, int NW, int P, int CTAS, bool SEQ>
__global__ void __launch_bounds__(NW * 32, CTAS) k_spmm_direct(const DirectParams p) {
  using S = Shape<FORM, NF, MH, SUB, NW, P>;
  constexpr int BW = 8 * SUB, PB = S::PB, Q = S::kQ, J = S::kJ;
  extern __shared__ __align__(128) uint8_t smem[];
  __shared__ volatile uint32_t flags[NW];  // pieces handed over by each warp's left neighbour rule
  const uint64_t t_entry = p.stamps ? global_timer_ns() : 0;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int gr = lane >> 2, gc = lane & 3;
  const int wr = warp / p.wf, nranges = NW / p.wf;
  const int col0 = (blockIdx.y * p.wf + warp % p.wf) * NF;
  const bool full = col0 + NF <= p.N;  // every feature of the slice exists
  if (threadIdx.x < NW) flags[threadIdx.x] = 0;
  __syncthreads();

  uint8_t* const ringp = smem + warp * S::kWarp;  // this warp's ring, then its A tiles
  const uint32_t ring = smem_u32(ringp);
  uint8_t* const abuf = ringp + P * S::kStep;
  auto lds16 = [](const uint8_t* a) { return *reinterpret_cast<const uint4*>(a); };
  auto lds8 = [](const uint8_t* a) { return *reinterpret_cast<const uint2*>(a); };
  const int32_t cta_col0 = blockIdx.y * p.wf * NF;
  float* const piece = reinterpret_cast<float*>(smem + S::kSmem);  // (SEQ) H x tw floats
  const int tw = p.wf * NF;
  float acc[Q][J][MH][4];
  // Copies: 8 lanes read one row's 128 (64) consecutive bytes, lane l chunk l % 8 of rows
  // 2 (l / 8) and the next. Places of chunk c, chosen so that neither the copies nor the
  // fragment loads have a bank conflict:
  //   fp32: chunk c of rows 2 r (then of rows 2 r + 1) at 16-byte place c ^ r of 128 bytes;
  //         lane (gr, gc) loads chunk gr / 2 + 4 (gr % 2) of rows 2 gc and 2 gc + 1, which
  //         puts the C elements of a row's four lanes side by side for each 16-byte store
  //   bf16: chunk c of row r at place c ^ r; ldmatrix, or 16-byte loads of chunk gr
  //   ext / fp8 bytes: chunk c of rows 2 r (2 r + 1) at 8-byte place c ^ 4 (r / 2) of 64
  const int lc = lane & 7;
  const int lr = FORM == kF32Odd ? gc : lane >> 3;  // this lane copies rows 2 lr and 2 lr + 1
  constexpr int E = S::kFp32 ? 4 : 2;               // bytes per element of the 16-byte pieces
  const uint32_t a_at = (gr * BW + 2 * gc) * 4;     // this lane's A fragments in a block's tile
  uint32_t bad = 0;                                 // an out-of-range tile id leaves a high bit
  uint32_t puta, putb, geta, getb;
  if constexpr (FORM == kF32Odd) {  // (each lane reads back what it copied)
    puta = geta = lane * 16;
    putb = getb = Q * 512 + lane * 16;
  } else if constexpr (FORM == kF32) {
    puta = lr * 128 + ((lc ^ lr) << 4);
    geta = gc * 128 + ((((gr >> 1) + 4 * (gr & 1)) ^ gc) << 4);
    putb = Q * 512 + puta;
    getb = Q * 512 + geta;
  } else {
    puta = 2 * lr * 128 + ((lc ^ (2 * lr)) << 4);
    putb = (2 * lr + 1) * 128 + ((lc ^ (2 * lr + 1)) << 4);
    geta = 2 * gc * 128 + ((gr ^ (2 * gc)) << 4);
    getb = (2 * gc + 1) * 128 + ((gr ^ (2 * gc + 1)) << 4);
  }
  constexpr int kPart = S::kFp32 ? 512 : 1024;      // bytes of a group of features per plane
  constexpr int kPlane = Q * kPart;                 // (bf16) bytes of one plane
  const uint32_t put8 = (lane >> 3) * 64 + ((lc ^ (4 * (lane >> 4))) << 3);
  const uint32_t get8 = gc * 64 + ((gr ^ (4 * (gc >> 1))) << 3);
  // ldmatrix: row l % 8 of tile l / 8; tiles: hi and lo of two chunks (two planes) or four
  // chunks (one plane). The chunks of the next load are 2 (4) further: an XOR of the place.
  const uint32_t mrow = (lane & 7) * 128;
  const uint32_t mplane = FORM == kBF16X2 ? ((lane >> 3) & 1) * kPlane : 0;
  const uint32_t mchunk = FORM == kBF16X2 ? lane >> 4 : lane >> 3;

  auto clear_acc = [&]() {
#pragma unroll
    for (int q = 0; q < Q; ++q)
#pragma unroll
      for (int j = 0; j < J; ++j)
#pragma unroll
        for (int h = 0; h < MH; ++h)
#pragma unroll
          for (int x = 0; x < 4; ++x) acc[q][j][h][x] = 0.0f;
  };
  // Visits the lane's C elements: 4 consecutive floats at a time (single ones for
  // the odd widths) as fn(row of the window, first feature, pointers to acc).
  auto each4 = [&](auto&& fn) {
#pragma unroll
    for (int q = 0; q < Q; ++q)
#pragma unroll
      for (int h = 0; h < MH; ++h)
#pragma unroll
        for (int hh = 0; hh < 2; ++hh)
#pragma unroll
          for (int e = 0; e < 2; ++e)
#pragma unroll
            for (int k = 0; k < J / 4; ++k) {
              const int row = h * 16 + hh * 8 + gr;
              const int chunk = S::kFp32 ? gc + 4 * e : 2 * gc + e;
              const int f = col0 + q * S::kQF + chunk * J + 4 * k;
              fn(row, f, acc[q][4 * k][h][2 * hh + e], acc[q][4 * k + 1][h][2 * hh + e],
                 acc[q][4 * k + 2][h][2 * hh + e], acc[q][4 * k + 3][h][2 * hh + e]);
            }
  };
  auto each1 = [&](auto&& fn) {
#pragma unroll
    for (int q = 0; q < Q; ++q)
#pragma unroll
      for (int h = 0; h < MH; ++h)
#pragma unroll
        for (int x = 0; x < 4; ++x)
#pragma unroll
          for (int j = 0; j < J; ++j)
            fn(h * 16 + (x >> 1) * 8 + gr, col0 + q * 32 + j * 8 + 2 * gc + (x & 1),
               acc[q][j][h][x]);
  };
  auto each2 = [&](auto&& fn) {  // (ldmatrix forms) pairs of floats
#pragma unroll
    for (int h = 0; h < MH; ++h)
#pragma unroll
      for (int hh = 0; hh < 2; ++hh)
#pragma unroll
        for (int q = 0; q < Q; ++q)
#pragma unroll
          for (int j = 0; j < J; ++j)
            fn(h * 16 + hh * 8 + gr, col0 + q * 64 + j * 8 + 2 * gc, acc[q][j][h][2 * hh],
               acc[q][j][h][2 * hh + 1]);
  };
  // acc += the tile at `t` (rows of N floats, `rows` of them valid); `slot`: a piece's place
  auto add_tile = [&](const float* t, int rows, bool slot) {
    const size_t ld = SEQ && slot ? tw : p.N;
    if constexpr (FORM == kF32Odd) {
      each1([&](int r, int f, float& x) {
        if (r < rows && f < p.N) x += t[r * ld + f];
      });
    } else if constexpr (S::kLdsm) {
      each2([&](int r, int f, float& x, float& y) {
        if (r < rows && f < p.N) {
          const float2 v = *reinterpret_cast<const float2*>(t + r * ld + f);
          x += v.x; y += v.y;
        }
      });
    } else {
      each4([&](int r, int f, float& x, float& y, float& z, float& w) {
        if (r < rows && f < p.N) {
          const float4 v = *reinterpret_cast<const float4*>(t + r * ld + f);
          x += v.x; y += v.y; z += v.z; w += v.w;
        }
      });
    }
  };
  auto store_tile = [&](float* t, int rows, bool epi, bool slot) {
    const size_t ld = SEQ && slot ? tw : p.N;
    if constexpr (FORM == kF32Odd) {
      each1([&](int r, int f, float& x) {
        if (r < rows && f < p.N) t[r * ld + f] = epi ? finish(p, x, f) : x;
      });
    } else if constexpr (S::kLdsm) {
      each2([&](int r, int f, float& x, float& y) {
        if (r < rows && f < p.N)
          *reinterpret_cast<float2*>(t + r * ld + f) =
              epi && (p.bias || p.relu) ? make_float2(finish(p, x, f), finish(p, y, f + 1))
                                        : make_float2(x, y);
      });
    } else {
      each4([&](int r, int f, float& x, float& y, float& z, float& w) {
        if (r < rows && f < p.N) {
          float4 v = make_float4(x, y, z, w);
          if (epi && (p.bias || p.relu))
            v = make_float4(finish(p, x, f), finish(p, y, f + 1), finish(p, z, f + 2),
                            finish(p, w, f + 3));
          *reinterpret_cast<float4*>(t + r * ld + f) = v;
        }
      });
    }
  };
  constexpr int H = 16 * MH;
  auto rows_of = [&](int32_t w) {  // (at most 0 past the last window)
    const int64_t left = p.M - (int64_t)w * H;
    return left < H ? (int)left : H;
  };
  auto c_rows = [&](int32_t w) { return p.C + (int64_t)w * H * p.N; };
  auto zero_window = [&](int32_t w) {
    const int rows = rows_of(w);
    for (int f = col0 + lane; f < col0 + NF && f < p.N; f += 32)
      for (int r = 0; r < rows; ++r) c_rows(w)[(size_t)r * p.N + f] = finish(p, 0.0f, f);
  };

  __shared__ Cut cuts[SEQ ? kTeam + 1 : 1];
  const int rank = SEQ ? blockIdx.x % kTeam : 0;
  int32_t k = blockIdx.x, only = -1;
  for (uint32_t mark = 1;; ++mark) {  // (SEQ: rounds)
    Cut c0, c1, from;
    int32_t hi = 0;
    if constexpr (SEQ) {
      team_cuts(p, k - rank, cuts, warp, NW, lane);
      __syncthreads();
      c0 = cuts[rank];
      c1 = cuts[rank + 1];
      Round(cuts, only).part(p, cuts, rank, k, lane, from, hi);
    } else {
      chunk_cuts(p, k, lane, c0, c1);
    }
    // (c1.win < c0.win: only with invalid window ids)
    const int32_t len = c1.win < c0.win ? 0 : c1.pos - c0.pos;
    float* const slot = SEQ ? piece - cta_col0 : p.slots + (size_t)k * H * p.N;
    const int nr = min(nranges, max(1, len >> 2));  // ranges of at least 4 blocks
    if (len > 0 && wr < nr && col0 < p.N) {
      // this warp's range
      const int32_t x0 = c0.pos + (int32_t)((int64_t)len * wr / nr);
      const int32_t x1 = c0.pos + (int32_t)((int64_t)len * (wr + 1) / nr);
      const int32_t most = max(len / nr / 2, 1);
      const int32_t wtop = min(c1.win + 1, p.nwin);
      const int2 si = search2(p.rwo, c0.win, wtop, x0 + 1, c0.win, wtop, min(x1, p.T - 1) + 1, lane);
      Cut r0 = wr == 0 ? c0 : cut_at(p, x0, si.x, most);
      Cut r1 = wr == nr - 1 ? c1 : cut_at(p, x1, si.y, most);
      if constexpr (SEQ) {  // (the ranges of the whole chunk: the same sums)
        if (r0.pos < from.pos) r0 = from;
        if (r1.pos > hi) r1 = Cut{hi, 0, false};
      }
      const int32_t nblk = r1.pos - r0.pos;
      if (nblk > 0) {
        const int32_t nst = nblk * SUB;
        const int32_t cutw = c0.open ? c0.win : -1;  // the window that started before the chunk
        const int32_t* s2x = p.s2x + (int64_t)r0.pos * BW + 2 * lr;
        const int32_t* toff = p.toff + r0.pos;
        auto load_rows = [&](int32_t st) -> int2 {  // SparseAToX of this lane's two rows
          const int32_t* a = s2x + 8 * min(st, nst - 1);
          if constexpr (FORM == kF32Odd) return make_int2(__ldg(a), __ldg(a + 1));
          return __ldg(reinterpret_cast<const int2*>(a));
        };
        auto load_offs = [&](int32_t g) -> int32_t {
          return __ldg(toff + min(PB * g + lane, nblk));  // (lanes past PB: unused)
        };
        // Copies of a step into ring slot i (`half`: of a 16-wide block). Columns ascend in
        // a block, so row 0 past a block's first slot is padding; its rows are zeros.
        auto gather = [&](int2 r, int i, int half) {
          const uint32_t slot = ring + i * S::kStep;
          const bool na = r.x == 0 && (lr > 0 || half > 0), nb = r.y == 0;
          // bytes of a B row in the plane of the 16-byte (8-byte) pieces; this lane's place in it
          const uint32_t rb16 = (uint32_t)p.N * E, rb8 = (uint32_t)p.N;
          const uint64_t oa = (uint64_t)(uint32_t)r.x * rb16, ob = (uint64_t)(uint32_t)r.y * rb16;
          const uint8_t* p0 = reinterpret_cast<const uint8_t*>(p.b0) + (col0 * E + lc * 16);
          const uint8_t* p1 = reinterpret_cast<const uint8_t*>(p.b1) + (col0 * E + lc * 16);
          if constexpr (FORM == kF32Odd) {
            const float* s0 = reinterpret_cast<const float*>(p.b0);
            const int64_t ea = (int64_t)r.x * p.N, eb = (int64_t)r.y * p.N;
#pragma unroll
            for (int q = 0; q < Q; ++q)
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                const int f = col0 + q * 32 + j * 8 + gr;
                const bool out = f >= p.N;
                cp4(slot + puta + q * 512 + j * 4, s0 + ea + f, out || na);
                cp4(slot + putb + q * 512 + j * 4, s0 + eb + f, out || nb);
              }
          } else {
#pragma unroll
            for (int q = 0; q < Q; ++q) {
              // (a slice that ends inside a group of features: zeros past column N)
              const bool out = !full && col0 + q * S::kQF + lc * (S::kQF / 8) >= p.N;
              if constexpr (S::kPlanes16 > 0) {
                cp16(slot + puta + q * kPart, p0 + oa + q * 128, na || out);
                cp16(slot + putb + q * kPart, p0 + ob + q * 128, nb || out);
              }
              if constexpr (FORM == kBF16X2) {
                cp16(slot + kPlane + puta + q * kPart, p1 + oa + q * 128, na || out);
                cp16(slot + kPlane + putb + q * kPart, p1 + ob + q * 128, nb || out);
              }
              if constexpr (S::kPieces8 > 0) {
                const uint8_t* p8 = reinterpret_cast<const uint8_t*>(FORM == kFP8 ? p.b0 : p.b1) +
                                    (col0 + lc * 8) + q * 64;
                cp8(slot + S::kOff8 + put8 + q * 256, p8 + (uint64_t)(uint32_t)r.x * rb8,
                    na || out);
                cp8(slot + S::kOff8 + put8 + (Q + q) * 256, p8 + (uint64_t)(uint32_t)r.y * rb8,
                    nb || out);
              }
            }
          }
          if constexpr (FORM == kFP8) {  // the row scales, one lane per slot
            if (lc < 2)
              cp4(slot + S::kOff4 + (2 * lr + lc) * 4,
                  reinterpret_cast<const float*>(p.b1) + (lc ? r.y : r.x), lc ? nb : na);
          }
        };
        // Tile ids and values of a group: 32 kPre entries ahead of time (lane l holds the
        // l-th of each 32), the rest when they are scattered.
        uint32_t pt[kPre];
        float pv[kPre];
        auto load_entries = [&](int32_t offs) {
          const int32_t e0 = __shfl_sync(0xffffffffu, offs, 0);
          const int32_t n = __shfl_sync(0xffffffffu, offs, PB) - e0;
          const uint8_t* t = p.tile + e0 + lane;
          const float* v = p.vals + e0 + lane;
#pragma unroll
          for (int c = 0; c < kPre; ++c)
            if (32 * c < n) {
              const bool in = 32 * c + lane < n;
              pt[c] = in ? __ldg(t + 32 * c) : 0u;
              pv[c] = in ? (p.vals ? __ldg(v + 32 * c) : 1.0f) : 0.0f;
            }
        };
        // A values of zero are skipped, among them the later ones of merged duplicates.
        auto put = [&](uint32_t pos, float v, uint8_t* at) {
          uint32_t word;
          if constexpr (S::kFp32) {
            word = rna_tf32(v);
          } else {
            const __nv_bfloat16 hi = __float2bfloat16_rn(v);
            const __nv_bfloat16 lo = __float2bfloat16_rn(v - __bfloat162float(hi));
            word = ((uint32_t)__bfloat16_as_ushort(hi) << 16) | __bfloat16_as_ushort(lo);
          }
          bad |= pos;
          if (v != 0.0f && pos < H * BW) *reinterpret_cast<uint32_t*>(at + pos * 4) = word;
        };
        auto scatter = [&](int32_t offs) {
          int32_t o[PB + 1];
#pragma unroll
          for (int i = 0; i <= PB; ++i) o[i] = __shfl_sync(0xffffffffu, offs, i);
          const int32_t n = o[PB] - o[0];
          auto at_of = [&](int32_t e) {  // the tile of entry e's block
            uint8_t* at = abuf;
#pragma unroll
            for (int i = 1; i < PB; ++i) at += e >= o[i] - o[0] ? H * BW * 4 : 0;
            return at;
          };
#pragma unroll
          for (int c = 0; c < kPre; ++c)
            if (32 * c < n) put(pt[c], pv[c], at_of(32 * c + lane));
#pragma unroll 1
          for (int32_t e = 32 * kPre + lane; e < n; e += 32)
            put(__ldg(p.tile + o[0] + e), p.vals ? __ldg(p.vals + o[0] + e) : 1.0f, at_of(e));
        };

        const int32_t offs_0 = load_offs(0);
        int32_t offs_n = load_offs(1);
        int2 rows[P];  // SparseAToX of the next group, one step each
#pragma unroll
        for (int i = 0; i < P; ++i) rows[i] = load_rows(i);
#pragma unroll
        for (int i = 0; i < P; ++i) {
          if (i < nst) gather(rows[i], i, i % SUB);
          cp_commit();
          rows[i] = load_rows(P + i);
        }
        load_entries(offs_0);
        // windows: ends of the 32 windows from wb on, the next 32 loaded ahead
        int32_t w = r0.win, wb = r0.win;
        auto load_ends = [&](int32_t b) { return __ldg(p.rwo + min(b + 1 + lane, p.nwin)); };
        int32_t ends = load_ends(wb), ends_n = load_ends(wb + 32);
#pragma unroll
        for (int i = 0; i < P * MH; ++i)
          *reinterpret_cast<uint4*>(abuf + (i * 32 + lane) * 16) = make_uint4(0, 0, 0, 0);
        __syncwarp();
        scatter(offs_0);
        int32_t offs_e = offs_n;  // of the group whose entries are held
        load_entries(offs_e);
        offs_n = load_offs(2);
        bool head = r0.open;  // the current window started left of this range
        if (!head) {          // empty windows that start with this range
          int32_t e = w;
          while (true) {
            const int32_t i = e - 1 - lane;
            const bool same = i >= 0 && __ldg(p.rwo + i) == r0.pos;
            const uint32_t m = __ballot_sync(0xffffffffu, same);
            const int n = m == 0xffffffffu ? 32 : __ffs(~m) - 1;
            e -= n;
            if (n < 32) break;
          }
          for (; e < w; ++e) zero_window(e);
        }
        int32_t wend = __shfl_sync(0xffffffffu, ends, 0) - r0.pos;  // relative to the range
        clear_acc();

        int32_t st = 0;
        int32_t run = min(wend, nblk) * SUB;  // steps up to the end of this window or range
        // One step: ring slot and A tile i of the group.
        auto step = [&](auto phase) {
            constexpr int i = decltype(phase)::value;
            cp_wait<P - 1>();
            __syncwarp();  // every lane's copies and scattered values are here
            // A fragments: slots 2 gc and 2 gc + 1 of rows gr + 8 t. Their places are zeroed
            // for the next group.
            uint2 af[2 * MH];
            uint8_t* const at = abuf + (i / SUB) * (H * BW * 4) + (i % SUB) * 32 + a_at;
#pragma unroll
            for (int t = 0; t < 2 * MH; ++t) {
              af[t] = lds8(at + t * 8 * BW * 4);
              *reinterpret_cast<uint2*>(at + t * 8 * BW * 4) = make_uint2(0, 0);
            }
            const uint8_t* const slot = ringp + i * S::kStep;
            if constexpr (S::kFp32) {
#pragma unroll
              for (int q = 0; q < Q; ++q) {
                uint4 x = lds16(slot + geta + q * 512), y = lds16(slot + getb + q * 512);
                if constexpr (FORM == kF32Odd) {  // the odd widths round B to nearest
                  x = make_uint4(rna_tf32(__uint_as_float(x.x)), rna_tf32(__uint_as_float(x.y)),
                                 rna_tf32(__uint_as_float(x.z)), rna_tf32(__uint_as_float(x.w)));
                  y = make_uint4(rna_tf32(__uint_as_float(y.x)), rna_tf32(__uint_as_float(y.y)),
                                 rna_tf32(__uint_as_float(y.z)), rna_tf32(__uint_as_float(y.w)));
                }
#pragma unroll
                for (int h = 0; h < MH; ++h) {
                  const uint2 a = af[2 * h], b = af[2 * h + 1];
                  mma_tf32_k8(acc[q][0][h], a.x, b.x, a.y, b.y, x.x, y.x);
                  mma_tf32_k8(acc[q][1][h], a.x, b.x, a.y, b.y, x.y, y.y);
                  mma_tf32_k8(acc[q][2][h], a.x, b.x, a.y, b.y, x.z, y.z);
                  mma_tf32_k8(acc[q][3][h], a.x, b.x, a.y, b.y, x.w, y.w);
                }
              }
            } else {
              uint32_t ah[MH][2], al[MH][2];
#pragma unroll
              for (int h = 0; h < MH; ++h)
#pragma unroll
                for (int t = 0; t < 2; ++t) {
                  ah[h][t] = __byte_perm(af[2 * h + t].x, af[2 * h + t].y, 0x7632);
                  al[h][t] = __byte_perm(af[2 * h + t].x, af[2 * h + t].y, 0x5410);
                }
              if constexpr (S::kLdsm) {
                const uint32_t mb = ring + i * S::kStep + mplane + mrow;
                constexpr int T = FORM == kBF16X2 ? 2 : 4;  // chunks per load
#pragma unroll
                for (int q = 0; q < Q; ++q)
#pragma unroll
                  for (int c = 0; c < 8; c += T) {
                    uint32_t v[4];
                    ldsm4t(v, mb + q * kPart + (((mchunk ^ (lane & 7)) ^ c) << 4));
                    if constexpr (FORM == kBF16X2) {
#pragma unroll
                      for (int j = 0; j < 2; ++j)
#pragma unroll
                        for (int h = 0; h < MH; ++h)
                          mma_bf16_k16(acc[q][c + j][h], ah[h][0], ah[h][1], ah[h][0], ah[h][1],
                                       v[2 * j], v[2 * j + 1]);
#pragma unroll
                      for (int j = 0; j < 2; ++j)
#pragma unroll
                        for (int h = 0; h < MH; ++h)
                          if constexpr (FOUR)
                            mma_bf16_k16(acc[q][c + j][h], al[h][0], al[h][1], al[h][0], al[h][1],
                                         v[2 * j], v[2 * j + 1]);
                          else
                            mma_bf16_k8(acc[q][c + j][h], al[h][0], al[h][1], v[2 * j]);
                    } else {
#pragma unroll
                      for (int j = 0; j < 4; ++j)
#pragma unroll
                        for (int h = 0; h < MH; ++h)  // lo = 0
                          mma_bf16_k16(acc[q][c + j][h], ah[h][0], ah[h][1], al[h][0], al[h][1],
                                       v[j], v[j]);
                    }
                  }
              } else {
              float2 sc = make_float2(0.0f, 0.0f);
              if constexpr (FORM == kFP8) {
                const uint2 v = lds8(slot + S::kOff4 + gc * 8);
                sc = make_float2(__uint_as_float(v.x), __uint_as_float(v.y));
              }
#pragma unroll
              for (int q = 0; q < Q; ++q) {
                uint32_t xh[4], yh[4], xl[4], yl[4];  // rows 2 gc, 2 gc + 1: hi and lo words
                const uint8_t* const s8 = slot + S::kOff8 + get8;
                if constexpr (S::kPlanes16 > 0) {
                  const uint4 x = lds16(slot + geta + q * kPart), y = lds16(slot + getb + q * kPart);
                  xh[0] = x.x; xh[1] = x.y; xh[2] = x.z; xh[3] = x.w;
                  yh[0] = y.x; yh[1] = y.y; yh[2] = y.z; yh[3] = y.w;
                }
                if constexpr (FORM == kSplit24) {
                  // lo = b24 - hi, exact in bf16: the hi bits on top of an fp32
                  // word, the extension byte under them, one subtraction
                  const uint2 ex = lds8(s8 + q * 256), ey = lds8(s8 + (Q + q) * 256);
                  auto lo_words = [](const uint32_t (&h)[4], const uint2& e, uint32_t (&o)[4]) {
#pragma unroll
                    for (int z = 0; z < 4; ++z) {
                      const uint32_t ew = z < 2 ? e.x : e.y;
                      const uint32_t h0 = h[z] << 16, h1 = h[z] & 0xFFFF0000u;
                      const uint32_t b0 = __byte_perm(h0, ew, z & 1 ? 0x3260 : 0x3240);
                      const uint32_t b1 = __byte_perm(h1, ew, z & 1 ? 0x3270 : 0x3250);
                      o[z] = __byte_perm(
                          __float_as_uint(__uint_as_float(b0) - __uint_as_float(h0)),
                          __float_as_uint(__uint_as_float(b1) - __uint_as_float(h1)), 0x7632);
                    }
                  };
                  lo_words(xh, ex, xl);
                  lo_words(yh, ey, yl);
                }
                if constexpr (FORM == kFP8) {
                  const uint2 ex = lds8(s8 + q * 256), ey = lds8(s8 + (Q + q) * 256);
                  auto words = [](const uint2& e, float s, uint32_t (&o)[4]) {
#pragma unroll
                    for (int z = 0; z < 4; ++z) {
                      const uint16_t q2 = (uint16_t)((z < 2 ? e.x : e.y) >> ((z & 1) * 16));
                      const __half2_raw hr =
                          __nv_cvt_fp8x2_to_halfraw2((__nv_fp8x2_storage_t)q2, __NV_E4M3);
                      const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&hr));
                      const __nv_bfloat162 b2 = __floats2bfloat162_rn(f.x * s, f.y * s);
                      o[z] = *reinterpret_cast<const uint32_t*>(&b2);
                    }
                  };
                  words(ex, sc.x, xh);
                  words(ey, sc.y, yh);
                }
                // every instruction's second product comes after the first ones of all, so
                // that no instruction waits for the one before it
                uint32_t bh[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                  const uint32_t sel = j & 1 ? 0x7632 : 0x5410;
                  bh[j] = __byte_perm(xh[j >> 1], yh[j >> 1], sel);
                  if constexpr (FORM == kFP8) {  // lo = 0
#pragma unroll
                    for (int h = 0; h < MH; ++h)
                      mma_bf16_k16(acc[q][j][h], ah[h][0], ah[h][1], al[h][0], al[h][1], bh[j],
                                   bh[j]);
                  } else {
                    const uint32_t bl = __byte_perm(xl[j >> 1], yl[j >> 1], sel);
#pragma unroll
                    for (int h = 0; h < MH; ++h) {
                      mma_bf16_k16(acc[q][j][h], ah[h][0], ah[h][1], ah[h][0], ah[h][1], bh[j],
                                   bl);
                      if constexpr (FOUR)
                        mma_bf16_k16(acc[q][j][h], al[h][0], al[h][1], al[h][0], al[h][1], bh[j],
                                     bl);
                    }
                  }
                }
                if constexpr (FORM == kSplit24 && !FOUR) {
#pragma unroll
                  for (int j = 0; j < 8; ++j)
#pragma unroll
                    for (int h = 0; h < MH; ++h)
                      mma_bf16_k8(acc[q][j][h], al[h][0], al[h][1], bh[j]);
                }
              }
              }
            }
            __syncwarp();  // every lane has read the slot (and, at a group's end, its A tiles)
            if (st + P < nst) gather(rows[i], i, i % SUB);
            cp_commit();
            rows[i] = load_rows(st + 2 * P);
            if constexpr (i == P - 1) {
              scatter(offs_e);  // (the next group's)
              offs_e = offs_n;
              load_entries(offs_e);
              offs_n = load_offs(st / P + 3);
            }
            ++st;
        };
        int phase = 0;
        while (true) {
          switch (phase) {  // (each phase runs on into the next one)
            case 0:
              step(std::integral_constant<int, 0>{});
              phase = 1;
              if (st >= run) break;
              [[fallthrough]];
            case 1:
              step(std::integral_constant<int, 1>{});
              phase = 2;
              if (st >= run) break;
              [[fallthrough]];
            case 2:
              step(std::integral_constant<int, 2>{});
              phase = 3;
              if (st >= run) break;
              [[fallthrough]];
            default:
              step(std::integral_constant<int, 3>{});
              phase = 0;
              if (st < run) continue;
          }
          if (wend > nblk) break;
          {  // the window is complete
            const int rows = rows_of(w);
            float* out = c_rows(w);
            if (head) {
              const bool cut = wr == 0 || w == cutw;
              store_tile(cut ? slot : out, cut ? H : rows, false, cut);
              if (wr > 0) {  // the left neighbour adds its piece
                __threadfence_block();
                __syncwarp();
                if (lane == 0) flags[warp] = mark;
              }
              head = false;
            } else {
              store_tile(out, rows, true, false);
            }
            if (wend >= nblk) {
              if (r1.pos == p.T)  // windows without blocks at the very end
                for (++w; w < p.nwin; ++w) zero_window(w);
              break;
            }
            clear_acc();
            const int32_t was = wend;
            while (true) {  // on to the next window with blocks
              ++w;
              if (w - wb == 32) {
                wb += 32;
                ends = ends_n;
                ends_n = load_ends(wb + 32);
              }
              wend = __shfl_sync(0xffffffffu, ends, w - wb) - r0.pos;
              if (wend > was || w >= p.nwin) break;
              zero_window(w);
            }
            if (wend <= was) break;  // (only with invalid offsets)
            run = min(wend, nblk) * SUB;
          }
        }
        if (bad >= (uint32_t)(H * BW)) atomicOr(p.err, kErrBadIndex);
        cp_wait<0>();
        if (wend > nblk) {  // the last window goes on to the right
          const int rows = rows_of(w);
          float* out = c_rows(w);
          const bool cut = w == cutw;
          if (wr + 1 < nr) {
            const int nb = warp + p.wf;
            if (lane == 0) {
              const uint64_t t0 = global_timer_ns();
              while (flags[nb] != mark) {
                __nanosleep(64);
                if (global_timer_ns() - t0 > 2000000000ull) {
                  atomicOr(p.err, kErrWaitTimeout);
                  break;
                }
              }
            }
            __syncwarp();
            __threadfence_block();
            add_tile(cut ? slot : out, cut ? H : rows, cut);
          }
          // does the window end inside the chunk?
          const bool ends_here = wend + r0.pos <= c1.pos;
          if (head) {
            const bool own = wr == 0 || cut;
            store_tile(own ? slot : out, own ? H : rows, false, own);
            __threadfence_block();
            __syncwarp();
            if (wr > 0 && lane == 0) flags[warp] = mark;
          } else {
            store_tile(out, rows, ends_here, false);
          }
        }
      }
      // a warp that handed nothing over: its left neighbour waits for it all the same where
      // invalid window ids make a window run on into a range that does not start inside it
      __syncwarp();
      if (lane == 0) flags[warp] = mark;
    }
    if constexpr (!SEQ) {
      // (Always, as there are slots; written as the end of a loop where the compiler orders the body
      // better with one. us, without / with: R-MAT 2^17, fp32 N = 41 319 / 311; R-MAT 2^18, FP8 N = 128
      // 16 x 16 4 % less with, BF16 32 x 8 N = 64 6 %, fp32 N = 128 16 x 8 3 %; fp32 N = 32 2 % more,
      // SPLIT24 32 x 8 5 % more.)
      constexpr bool kLoop = FORM == kF32Odd || ((NF == 128 || MH == 2) && FORM != kSplit24);
      if (!kLoop || p.slots) break;
    } else {
      only = end_round(p, cuts, Round(cuts, only), piece, tw, cta_col0, rank, threadIdx.x, NW * 32);
      if (only < 0) break;
      __syncthreads();  // (the next round's cuts)
      k += kTeam;
    }
  }
  if (p.stamps) {
    __syncthreads();
    const int c = blockIdx.x + gridDim.x * blockIdx.y;
    if (threadIdx.x == 0 && c < p.stamp_cap) {
      uint32_t smid;
      asm volatile("mov.u32 %0, %%smid;" : "=r"(smid));
      uint64_t* s = p.stamps + 4 * (size_t)c;
      s[0] = t_entry;
      s[1] = global_timer_ns();
      s[2] = smid;
      s[3] = 1;
    }
  }
}

constexpr int kP = 4;

// A kernel on clusters of kTeam CTAs along x (SEQ), or on single ones.
template <bool SEQ>
dtc_status launch_ctas(void (*fn)(DirectParams), const DirectParams& p, unsigned slices, int threads,
                       int smem, int most, cudaStream_t st, bool (&attr_set)[64]) {
  int dev = 0;
  cudaGetDevice(&dev);
  if (!attr_set[dev & 63]) {
    DTC_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
    attr_set[dev & 63] = true;
  }
  if constexpr (SEQ) {
    cudaLaunchConfig_t c = {};
    cudaLaunchAttribute a;
    a.id = cudaLaunchAttributeClusterDimension;
    a.val.clusterDim.x = kTeam;
    a.val.clusterDim.y = a.val.clusterDim.z = 1;
    c.gridDim = dim3((unsigned)((p.G + kTeam - 1) / kTeam * kTeam), slices);
    c.blockDim = dim3(threads);
    c.dynamicSmemBytes = smem;
    c.stream = st;
    c.attrs = &a;
    c.numAttrs = 1;
    DTC_CUDA(cudaLaunchKernelEx(&c, fn, p));
  } else {
    fn<<<dim3((unsigned)p.G, slices), threads, smem, st>>>(p);
  }
  DTC_CUDA(cudaGetLastError());
  return DTC_OK;
}

// `slices`: feature slices of the form with a workspace, which set the ranges per chunk.
template <int FORM, bool FOUR, int NF, int MH, int SUB, int CTAS, bool SEQ>
dtc_status launch_form(DirectParams& p, int slices, cudaStream_t st) {
  using S = Shape<FORM, NF, MH, SUB, kNW, kP>;
  constexpr int kPiece = 16 * MH * NF * 4;  // per slice of features
  static_assert(S::kSmem + 4 * kPiece <= 232448 - 2048, "shared memory per CTA");
  static bool attr_set[64] = {};
  p.wf = slices >= 4 ? 4 : slices >= 2 ? 2 : 1;
  slices = (p.N + NF - 1) / NF;
  return launch_ctas<SEQ>(k_spmm_direct<FORM, FOUR, NF, MH, SUB, kNW, kP, CTAS, SEQ>, p,
                          (unsigned)((slices + p.wf - 1) / p.wf), kNW * 32,
                          S::kSmem + (SEQ ? p.wf * kPiece : 0), S::kSmem + (SEQ ? 4 * kPiece : 0), st,
                          attr_set);
}

template <int FORM, bool FOUR, int NF, int MH, int SUB, int CTAS>
dtc_status launch(DirectParams& p, cudaStream_t st) {
  // (SEQ: the pieces' place in shared memory would leave room for two CTAs of 128 features)
  const int slices = (p.N + NF - 1) / NF;
  const dtc_status s =
      p.slots ? launch_form<FORM, FOUR, NF, MH, SUB, CTAS, false>(p, slices, st)
              : launch_form<FORM, FOUR, NF == 128 ? 64 : NF, MH, SUB, NF == 128 ? 4 : CTAS, true>(
                    p, slices, st);
  if (s != DTC_OK) return s;
  if (p.slots && p.G > 1) {
    k_add_slots<<<add_ctas(p), kAddThreads, 0, st>>>(p);
    DTC_CUDA(cudaGetLastError());
  }
  return DTC_OK;
}

template <int FORM, bool FOUR, int MH, int SUB>
dtc_status by_width(DirectParams& p, cudaStream_t st) {
  // (32 features of acc at 5 CTAs, 64 at 4 and 128 at 3: what the registers allow, but for 4 to
  // 28 bytes that a dozen of the instances spill)
  if constexpr (FORM == kF32 || FORM == kF32Odd) {
    if (p.N <= 32) return launch<FORM, FOUR, 32, MH, SUB, MH == 2 ? 4 : 5>(p, st);
  }
  constexpr bool wide = MH == 1 && FORM != kBF16X2;  // forms that reach this kernel beyond 64
  if constexpr (wide) {
    if (p.N > 64) return launch<FORM, FOUR, 128, MH, SUB, 3>(p, st);
  }
  return launch<FORM, FOUR, 64, MH, SUB, MH == 2 ? 3 : 4>(p, st);
}

template <int FORM, bool FOUR>
dtc_status by_block(DirectParams& p, int W, cudaStream_t st) {
  if (p.H == 32) return by_width<FORM, FOUR, 2, 1>(p, st);
  if (W == 16) return by_width<FORM, FOUR, 1, 2>(p, st);
  return by_width<FORM, FOUR, 1, 1>(p, st);
}

}  // namespace
}  // namespace dtc
