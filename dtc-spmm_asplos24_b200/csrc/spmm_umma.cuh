// TC-block SpMM on tcgen05: several small pipelines per SM, each a CTA of ten
// warps that runs one chunk of TC blocks through a ring in shared memory.
//
// Product mapping. tcgen05 needs M in {64, 128}, so the product is transposed:
//     C_w^T [features x WH] += B_b^T [features x 8] * A_b^T [8 x WH]
// UMMA M = 128 features, N = WH window rows (2 WH columns, A_hi^T | A_lo^T, for the
// bf16 forms), K = 8 slots (16: the hi and the lo rows). The gathered B rows are
// the MN-major operand (fp32: 128-byte swizzle with 32-byte granules; bf16:
// 128-byte swizzle), the densified TC block the K-major one.
//
// What bounds it. An SM's tensor pipe takes one of these narrow instructions per
// 40-46 cycles and one thread issues at most one per ~93, while a gathered 4 KB
// block needs 64 cycles of the SM's 64-byte L2 port. One pipeline per SM spent
// ~125-290 cycles per block on the round trip of its ring slots (wait, issue,
// commit, wait, gather); three pipelines per SM overlap theirs.
//   warps 0-3   epilogue: tcgen05.ld of a finished window (features are TMEM lanes,
//               so a warp's row of C is 128 consecutive bytes), bias, ReLU, stores
//   warps 4-5   loaders: 16-byte cp.async gathers of every second block
//   warps 6-8   tile builders: the A values of every third block (apart from the
//               loaders: their fence to the async proxy would wait for the copies)
//   warp 9      issuer: waits for a block, issues its instructions, commits the slots
// Work split, cut windows and the order of their pieces: spmm_direct.cuh.
#pragma once
#include "spmm_direct.cuh"

namespace dtc {
namespace {

// One arrival on `bar` when this thread's copies so far have landed (part of its count).
__device__ __forceinline__ void cp_async_arrive_noinc(uint64_t* bar) {
  asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(bar))
               : "memory");
}

constexpr int kLoaders = 2, kTilers = 3;
constexpr int kLoad0 = 4, kTile0 = kLoad0 + kLoaders, kIssuer = kTile0 + kTilers;
constexpr int kUmmaThreads = 32 * (kIssuer + 1);

template <int FORM, int NT, int WH, int SUB, int R>
struct UShape {
  static constexpr bool kTf32 = FORM == kF32;
  static constexpr int kXTile = 4096;                       // 8 slots x 128 features (hi + lo)
  static constexpr int kX = NT * SUB * kXTile;              // one block's gathered rows
  static constexpr int kYHalf = kTf32 ? WH * 32 : WH * 64;  // 8 slots' A^T tile
  static constexpr int kY = SUB * kYHalf;
  static constexpr int kBlocks = 4 / (SUB * NT);            // blocks per stage
  static constexpr int kStageX = kBlocks * kX, kStageY = kBlocks * kY;
  static constexpr int kCols = (kTf32 ? WH : 2 * WH) * NT;  // TMEM columns of one accumulator
  static constexpr int kNacc = kCols * 4 <= 128 ? 4 : 2;
  static constexpr uint32_t kTmem = kCols * kNacc <= 64 ? 64 : kCols * kNacc <= 128 ? 128
                                    : kCols * kNacc <= 256 ? 256 : 512;
  static constexpr int kBars = (2 * R + 2 * kNacc + 1) * 8;
  static constexpr int kSmem = R * (kStageX + kStageY) + kBars + 16 + 1024;
  static constexpr int kPre = WH * SUB > 16 ? 2 : 1;
  static_assert(kCols * kNacc <= 512, "TMEM");
  // A slot's parity wait may be one phase ahead, not two: the warp that fills stage h has
  // filled h - T before, which proves that stage h - T - R is consumed; h - 2R has to be.
  static_assert(kLoaders <= R && kTilers <= R, "warps that fill stages");
};

// The windows a chunk meets, in order: empty ones, and those with blocks with the
// part [.., end) that lies in the chunk. All lanes of a warp walk together.
struct WindowWalk {
  const DirectParams& p;
  int lane;
  int32_t w, wb, ends, ends_n, end, base, nblk;
  __device__ __forceinline__ int32_t load(int32_t b) const {
    return __ldg(p.rwo + min(b + 1 + lane, p.nwin));
  }
  __device__ __forceinline__ WindowWalk(const DirectParams& p_, int lane_, int32_t w0, int32_t base_,
                                        int32_t nblk_)
      : p(p_), lane(lane_), w(w0), wb(w0), base(base_), nblk(nblk_) {
    ends = load(wb);
    ends_n = load(wb + 32);
    end = max(__shfl_sync(0xffffffffu, ends, 0) - base, 1);  // (less: only with invalid offsets)
  }
  // On to the next window with blocks; `empty` is called for each one without.
  template <typename F>
  __device__ __forceinline__ void next(F&& empty) {
    const int32_t was = end;
    while (true) {
      ++w;
      if (w - wb == 32) {
        wb += 32;
        ends = ends_n;
        ends_n = load(wb + 32);
      }
      end = __shfl_sync(0xffffffffu, ends, w - wb) - base;
      if (end > was || w >= p.nwin) break;
      empty(w);
    }
    if (end <= was) end = 0x7fffffff;  // (only with invalid offsets: ends the walk)
  }
};

template <int FORM, bool FOUR, int NT, int WH, int SUB, int R, int CTAS, bool SEQ>
__global__ void __launch_bounds__(kUmmaThreads, CTAS)
    k_spmm_umma(const __grid_constant__ DirectParams p) {
  using S = UShape<FORM, NT, WH, SUB, R>;
  constexpr int BW = 8 * SUB, PB = S::kBlocks, NA = S::kNacc;
  const uint64_t t_entry = p.stamps ? global_timer_ns() : 0;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* const smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint8_t* const xring = smem;
  uint8_t* const yring = smem + R * S::kStageX;
  uint64_t* const full = reinterpret_cast<uint64_t*>(yring + R * S::kStageY);
  uint64_t* const empty = full + R;           // [R] the issuer's commits
  uint64_t* const acc_full = empty + R;    // [NA]
  uint64_t* const acc_empty = acc_full + NA;    // [NA]
  uint64_t* const drain = acc_empty + NA;
  uint32_t* const tmem_slot = reinterpret_cast<uint32_t*>(drain + 1);
  volatile uint32_t* const abort_flag = tmem_slot + 1;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int col0 = blockIdx.y * NT * 128;
  float* const piece = reinterpret_cast<float*>(smem + S::kSmem - 1024);  // (SEQ) WH x NT * 128 floats

  if (threadIdx.x == 0) {
    for (int i = 0; i < R; ++i) mbar_init(full + i, 32 + 1);  // 32 lanes' copies, the A values
    for (int i = 0; i < R; ++i) mbar_init(empty + i, 1);
    for (int i = 0; i < NA; ++i) {
      mbar_init(acc_full + i, 1);
      mbar_init(acc_empty + i, 4);
    }
    mbar_init(drain, 1);
    *abort_flag = 0;
    fence_mbar_init();
  }
  if constexpr (FORM == kBF16) {  // the lo rows stay zero
    for (int i = threadIdx.x; i < R * PB * NT * SUB * 128; i += kUmmaThreads)
      *reinterpret_cast<uint4*>(xring + (i / 128) * S::kXTile + 2048 + (i % 128) * 16) =
          make_uint4(0, 0, 0, 0);
    fence_proxy_async_smem();
  }
  if (warp == kIssuer) {
    tmem_alloc(tmem_slot, S::kTmem);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  uint32_t n = 0;    // stages of the CTA so far (over its chunks)
  uint32_t acq = 0;  // windows with blocks so far
  bool ok = true;
  __shared__ Cut cuts[SEQ ? kTeam + 1 : 1];
  const int rank = SEQ ? blockIdx.x % kTeam : 0;
  // (SEQ: rounds. Without them one pass; for 32-row windows a loop all the same, that is left
  // after it: the compiler's order of the body is better then, R-MAT 2^20, N = 128, BF16X2 1.90 ms,
  // 2.03 without; for 16-row windows it is worse, 1.90 and 1.85.)
  constexpr bool kLoop = !SEQ && WH == 32;
  int32_t only = -1;
  for (int32_t k = blockIdx.x; !kLoop || ok; k += kLoop ? 1 : 0) {
    Cut c0, c1;
    if constexpr (SEQ) {
      team_cuts(p, k - rank, cuts, warp, kUmmaThreads / 32, lane);
      __syncthreads();
      Round(cuts, only).part(p, cuts, rank, k, lane, c0, c1.pos);
      if (!ok) c1.pos = c0.pos;
    } else {
      chunk_cuts(p, k, lane, c0, c1);
    }
    const int32_t nblk = c1.pos - c0.pos;
    if (nblk > 0) {
      if (warp >= kLoad0 && warp < kTile0) {
        // --------------------------------------------------------- loaders
        const int j = warp - kLoad0;
        const int lr = lane >> 3, lc = lane & 7;  // copies chunk lc of rows 2 lr and 2 lr + 1
        constexpr int E = S::kTf32 ? 4 : 2, Q = S::kTf32 ? 4 : 2;  // 128-byte pieces of a tile's row
        auto place = [&](int r) -> uint32_t {
          if constexpr (S::kTf32)
            return (r >> 2) * 512 + (r & 3) * 128 + (((((lc >> 1) ^ (r & 3)) << 1) | (lc & 1)) << 4);
          else
            return r * 128 + ((lc ^ r) << 4);
        };
        const uint32_t puta = place(2 * lr), putb = place(2 * lr + 1);
        const bool fullw = col0 + NT * 128 <= p.N;
        const int32_t* const s2x = p.s2x + (int64_t)c0.pos * BW + 2 * lr;
        auto load_rows = [&](int32_t b, int u) -> int2 {
          return __ldg(reinterpret_cast<const int2*>(s2x + min(b, nblk - 1) * BW + 8 * u));
        };
        auto gather = [&](int2 r, uint32_t slot, int half) {
          // columns ascend in a block: row 0 past its first slot is padding, zeros
          const bool na = r.x == 0 && (lr > 0 || half > 0), nb = r.y == 0;
          const uint32_t rb = (uint32_t)p.N * E;
          const uint64_t oa = (uint64_t)(uint32_t)r.x * rb, ob = (uint64_t)(uint32_t)r.y * rb;
          const uint8_t* p0 = reinterpret_cast<const uint8_t*>(p.b0) + (col0 * E + lc * 16);
          const uint8_t* p1 = reinterpret_cast<const uint8_t*>(p.b1) + (col0 * E + lc * 16);
          if (fullw) {
#pragma unroll
            for (int t = 0; t < NT; ++t)
#pragma unroll
              for (int q = 0; q < Q; ++q) {
                const uint32_t d = slot + t * SUB * S::kXTile + q * 1024;
                cp16(d + puta, p0 + oa + (t * Q + q) * 128, na);
                cp16(d + putb, p0 + ob + (t * Q + q) * 128, nb);
                if constexpr (FORM == kBF16X2) {
                  cp16(d + 2048 + puta, p1 + oa + (t * Q + q) * 128, na);
                  cp16(d + 2048 + putb, p1 + ob + (t * Q + q) * 128, nb);
                }
              }
          } else {  // a slice that ends inside a tile: zeros past column N
#pragma unroll 1
            for (int x = 0; x < NT * Q; ++x) {
              const bool out = col0 + x * (128 / E) + lc * (16 / E) >= p.N;
              const uint32_t d = slot + (x / Q) * SUB * S::kXTile + (x % Q) * 1024;
              cp16(d + puta, p0 + oa + x * 128, na || out);
              cp16(d + putb, p0 + ob + x * 128, nb || out);
              if constexpr (FORM == kBF16X2) {
                cp16(d + 2048 + puta, p1 + oa + x * 128, na || out);
                cp16(d + 2048 + putb, p1 + ob + x * 128, nb || out);
              }
            }
          }
        };
        const int32_t nstage = (nblk + PB - 1) / PB;
        int2 rows[PB * SUB];  // SparseAToX of the next own stage, 8 slots each
#pragma unroll
        for (int i = 0; i < PB * SUB; ++i) rows[i] = load_rows(j * PB + i / SUB, i % SUB);
        for (int32_t st = j; ok && st < nstage; st += kLoaders) {
          const uint32_t g = n + st, s = g % R;
          ok = mbar_wait(empty + s, ((g / R) & 1) ^ 1, p.err);
          if (!__all_sync(0xffffffffu, ok) || *abort_flag) {
            *abort_flag = 1;
            ok = false;
            break;
          }
          const uint32_t x = smem_u32(xring + s * S::kStageX);
#pragma unroll
          for (int i = 0; i < PB * SUB; ++i) {
            if (st * PB + i / SUB < nblk)
              gather(rows[i], x + (i / SUB) * S::kX + (i % SUB) * S::kXTile, i % SUB);
            rows[i] = load_rows((st + kLoaders) * PB + i / SUB, i % SUB);
          }
          cp_async_arrive_noinc(full + s);
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
      } else if (warp >= kTile0 && warp < kIssuer) {
        // --------------------------------------------------- tile builders
        const int j = warp - kTile0;
        const int32_t* const toff = p.toff + c0.pos;
        uint32_t bad = 0;
        auto load_offs = [&](int32_t b) -> int32_t { return __ldg(toff + min(b + lane, nblk)); };
        // A values of zero are skipped, among them the later ones of merged duplicates.
        auto put = [&](uint32_t pos, float v, uint8_t* y) {
          bad |= pos;
          if (v == 0.0f || pos >= WH * BW) return;
          const uint32_t r = pos / BW, s = pos % 8;
          y += (pos % BW) / 8 * S::kYHalf;
          if constexpr (S::kTf32) {
            *reinterpret_cast<uint32_t*>(y + (r & 7) * 16 + (r >> 3) * 256 + (s >> 2) * 128 +
                                         (s & 3) * 4) = rna_tf32(v);
          } else {
            const __nv_bfloat16 hi = __float2bfloat16_rn(v);
            const __nv_bfloat16 lo = __float2bfloat16_rn(v - __bfloat162float(hi));
            uint8_t* const h = y + (r & 7) * 16 + (r >> 3) * 256 + s * 2;  // column r, K row s
            *reinterpret_cast<__nv_bfloat16*>(h) = hi;
            *reinterpret_cast<__nv_bfloat16*>(h + 128) = hi;
            *reinterpret_cast<__nv_bfloat16*>(h + WH * 32) = lo;             // column WH + r
            if constexpr (FOUR) *reinterpret_cast<__nv_bfloat16*>(h + WH * 32 + 128) = lo;
          }
        };
        const int32_t nstage = (nblk + PB - 1) / PB;
        // entries of the next own stage, offsets of the one after it
        uint32_t pt[PB][S::kPre];
        float pv[PB][S::kPre];
        auto load_entries = [&](int32_t offs) {
#pragma unroll
          for (int i = 0; i < PB; ++i) {
            const int32_t e0 = __shfl_sync(0xffffffffu, offs, i);
            const int32_t e1 = __shfl_sync(0xffffffffu, offs, i + 1);
#pragma unroll
            for (int c = 0; c < S::kPre; ++c) {
              const int32_t e = e0 + 32 * c + lane;
              pt[i][c] = e < e1 ? __ldg(p.tile + e) : 0u;
              pv[i][c] = e < e1 ? (p.vals ? __ldg(p.vals + e) : 1.0f) : 0.0f;
            }
          }
        };
        int32_t offs = load_offs(j * PB), offs_n = load_offs((j + kTilers) * PB);
        load_entries(offs);
        for (int32_t st = j; ok && st < nstage; st += kTilers) {
          const uint32_t g = n + st, s = g % R;
          const int32_t offs_nn = load_offs((st + 2 * kTilers) * PB);
          ok = mbar_wait(empty + s, ((g / R) & 1) ^ 1, p.err);
          if (!__all_sync(0xffffffffu, ok) || *abort_flag) {
            *abort_flag = 1;
            ok = false;
            break;
          }
          uint8_t* const y = yring + s * S::kStageY;
#pragma unroll
          for (int z = 0; z < S::kStageY / 512; ++z)
            *reinterpret_cast<uint4*>(y + (z * 32 + lane) * 16) = make_uint4(0, 0, 0, 0);
          __syncwarp();
#pragma unroll
          for (int i = 0; i < PB; ++i) {
#pragma unroll
            for (int c = 0; c < S::kPre; ++c) put(pt[i][c], pv[i][c], y + i * S::kY);
            const int32_t e1 = __shfl_sync(0xffffffffu, offs, i + 1);
            for (int32_t e = __shfl_sync(0xffffffffu, offs, i) + 32 * S::kPre + lane; e < e1; e += 32)
              put(__ldg(p.tile + e), p.vals ? __ldg(p.vals + e) : 1.0f, y + i * S::kY);
          }
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) mbar_arrive(full + s);
          offs = offs_n;
          offs_n = offs_nn;
          load_entries(offs);
        }
        if (bad >= (uint32_t)(WH * BW)) atomicOr(p.err, kErrBadIndex);
      } else if (warp == kIssuer) {
        // ---------------------------------------------------------- issuer
        constexpr uint32_t idesc = S::kTf32 ? umma_idesc(2, 128, WH, 1, 0)
                                            : umma_idesc(1, 128, 2 * WH, 1, 0);
        const uint64_t xd = S::kTf32 ? umma_desc(smem_u32(xring), 1024, 512, 1)
                                     : umma_desc(smem_u32(xring), 1024, 2048, 2);
        const uint64_t yd = umma_desc(smem_u32(yring), 128, 256, 0);
        const uint32_t xlo = (uint32_t)xd, xhi = (uint32_t)(xd >> 32);
        const uint32_t ylo = (uint32_t)yd, yhi = (uint32_t)(yd >> 32);
        WindowWalk win(p, lane, c0.win, c0.pos, nblk);
        int32_t b = 0;
        while (ok) {
          const int a = (int)(acq % NA);
          const uint32_t d = tmem + (uint32_t)(a * S::kCols);
          const int32_t run = min(win.end, nblk);
          if (lane == 0) {
            ok = mbar_wait(acc_empty + a, ((acq / NA) & 1) ^ 1, p.err);
            tc_fence_after();
            uint32_t accum = 0;
            while (b < run) {
              const uint32_t g = n + b / PB, s = g % R;
              const int32_t i0 = b % PB, i1 = min(PB, i0 + run - b);
              if (i0 == 0) {  // the stage's first block: its copies and A values are here
                ok = mbar_wait(full + s, (g / R) & 1, p.err);
                if (!ok) break;
                fence_proxy_async_smem();  // the copies (generic proxy) before the UMMA reads
                tc_fence_after();
              }
              const uint32_t x = xlo + ((s * S::kStageX) >> 4), y = ylo + ((s * S::kStageY) >> 4);
#pragma unroll
              for (int i = 0; i < PB; ++i)
                if (i >= i0 && i < i1) {
#pragma unroll
                  for (int u = 0; u < SUB; ++u)
#pragma unroll
                    for (int t = 0; t < NT; ++t) {
                      const uint64_t ad =
                          desc_at(x + ((i * S::kX + (t * SUB + u) * S::kXTile) >> 4), xhi);
                      const uint64_t bd = desc_at(y + ((i * S::kY + u * S::kYHalf) >> 4), yhi);
                      const uint32_t dt = d + t * (S::kCols / NT);
                      if constexpr (S::kTf32) mma_tf32(dt, ad, bd, idesc, u == 0 ? accum : 1u);
                      else mma_f16(dt, ad, bd, idesc, u == 0 ? accum : 1u);
                    }
                  accum = 1;
                }
              b += i1 - i0;
              if (b % PB == 0 || b == nblk) tc_commit(empty + s);
            }
          }
          b = run;
          __syncwarp();
          ok = __all_sync(0xffffffffu, ok) && !*abort_flag;
          if (!ok) {
            *abort_flag = 1;
            break;
          }
          if (lane == 0) tc_commit(acc_full + a);
          ++acq;
          if (win.end >= nblk) break;
          win.next([](int32_t) {});
        }
        __syncwarp();
      } else {
        // -------------------------------------------------------- epilogue
        const int64_t tile = (int64_t)WH * p.N;
        auto zero_window = [&](int32_t w) {
          for (int f = col0 + warp * 32 + lane; f < col0 + NT * 128 && f < p.N; f += 128)
            for (int r = 0; r < WH && (int64_t)w * WH + r < p.M; ++r)
              p.C[(int64_t)w * tile + (int64_t)r * p.N + f] = finish(p, 0.0f, f);
        };
        if (!c0.open) {  // empty windows that start with this chunk
          int32_t e = c0.win;
          while (true) {
            const int32_t i = e - 1 - lane;
            const bool same = i >= 0 && __ldg(p.rwo + i) == c0.pos;
            const uint32_t m = __ballot_sync(0xffffffffu, same);
            const int c = m == 0xffffffffu ? 32 : __ffs(~m) - 1;
            e -= c;
            if (c < 32) break;
          }
          for (; e < c0.win; ++e) zero_window(e);
        }
        WindowWalk win(p, lane, c0.win, c0.pos, nblk);
        bool head = c0.open;
        while (true) {
          const int a = (int)(acq % NA);
          ok = mbar_wait(acc_full + a, (acq / NA) & 1, p.err);
          if (!__all_sync(0xffffffffu, ok) || *abort_flag) {
            *abort_flag = 1;
            ok = false;
            break;
          }
          tc_fence_after();
          // a piece of a cut window: to the chunk's slot; the first piece, and a whole window, to C
          const bool raw = win.end > nblk, slot = head;
          float* const out = !slot ? p.C + (int64_t)win.w * tile
                             : SEQ ? piece - col0
                                   : p.slots + (int64_t)k * tile;
          const int32_t ld = SEQ && slot ? NT * 128 : p.N;
          const int rows = slot ? WH : (int)min((int64_t)WH, p.M - (int64_t)win.w * WH);
#pragma unroll 1
          for (int t = 0; t < NT; ++t) {
            const int f = col0 + t * 128 + warp * 32 + lane;
#pragma unroll 1
            for (int h = 0; h < WH / 16; ++h) {
              uint32_t v[16];
              const uint32_t at = tmem + ((uint32_t)(warp * 32) << 16) + a * S::kCols +
                                  t * (S::kCols / NT) + h * 16;
              tmem_ld16(at, v);
              if constexpr (!S::kTf32) {
                uint32_t u[16];
                tmem_ld16(at + WH, u);
                tmem_ld_wait();
#pragma unroll
                for (int r = 0; r < 16; ++r)
                  v[r] = __float_as_uint(__uint_as_float(v[r]) + __uint_as_float(u[r]));
              } else {
                tmem_ld_wait();
              }
              if (t == NT - 1 && h == WH / 16 - 1) {
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(acc_empty + a);
              }
              if (f < p.N) {
#pragma unroll
                for (int r = 0; r < 16; ++r) {
                  if (h * 16 + r < rows) {
                    float* const o = out + (int64_t)(h * 16 + r) * ld + f;
                    const float x = __uint_as_float(v[r]);
                    *o = slot || raw ? x : finish(p, x, f);
                  }
                }
              }
            }
          }
          ++acq;
          head = false;
          if (win.end >= nblk) {
            if (c1.pos == p.T && win.end == nblk)  // windows without blocks at the very end
              for (int32_t w = win.w + 1; w < p.nwin; ++w) zero_window(w);
            break;
          }
          win.next(zero_window);
        }
      }
      n += (uint32_t)((nblk + PB - 1) / PB);
    }
    if constexpr (!SEQ) {
      if (!kLoop || p.slots) break;
    } else {
      __syncthreads();
      only = end_round(p, cuts, Round(cuts, only), piece, NT * 128, col0, rank, threadIdx.x,
                       kUmmaThreads);
      if (only < 0) break;
      __syncthreads();  // (the next round's cuts)
      k += kTeam;
      ok = ok && !*abort_flag;
    }
  }
  if (warp == kIssuer && lane == 0) {  // every MMA has finished before the TMEM is freed
    tc_commit(drain);
    mbar_wait(drain, 0, p.err);
  }
  tc_fence_before();
  __syncthreads();
  if (p.stamps && threadIdx.x == 0) {
    const int c = blockIdx.x + gridDim.x * blockIdx.y;
    if (c < p.stamp_cap) {
      uint32_t smid;
      asm volatile("mov.u32 %0, %%smid;" : "=r"(smid));
      uint64_t* s = p.stamps + 4 * (size_t)c;
      s[0] = t_entry;
      s[1] = global_timer_ns();
      s[2] = smid;
      s[3] = 1;
    }
  }
  if (warp == kIssuer) {
    tc_fence_after();
    tmem_dealloc(tmem, S::kTmem);
  }
}

template <int FORM, bool FOUR, int NT, int WH, int SUB, int R, int CTAS, bool SEQ>
dtc_status launch_umma_form(DirectParams& p, cudaStream_t st) {
  using S = UShape<FORM, NT, WH, SUB, R>;
  constexpr int smem = S::kSmem + (SEQ ? WH * NT * 128 * 4 : 0);
  static_assert(smem <= 232448 - 1024 && S::kTmem * CTAS <= 512, "per-SM budget");
  static bool attr_set[64] = {};
  return launch_ctas<SEQ>(k_spmm_umma<FORM, FOUR, NT, WH, SUB, R, CTAS, SEQ>, p,
                          (unsigned)((p.N + NT * 128 - 1) / (NT * 128)), kUmmaThreads, smem, smem, st,
                          attr_set);
}

template <int FORM, bool FOUR, int NT, int WH, int SUB, int R, int CTAS>
dtc_status launch_umma(DirectParams& p, cudaStream_t st) {
  const dtc_status s = p.slots ? launch_umma_form<FORM, FOUR, NT, WH, SUB, R, CTAS, false>(p, st)
                               : launch_umma_form<FORM, FOUR, NT, WH, SUB, 3, CTAS, true>(p, st);  // (room for the pieces)
  if (s != DTC_OK) return s;
  if (p.slots && p.G > 1) {
    k_add_slots<<<add_ctas(p), kAddThreads, 0, st>>>(p);
    DTC_CUDA(cudaGetLastError());
  }
  return DTC_OK;
}

template <int FORM, bool FOUR>
dtc_status umma_by_block(DirectParams& p, int W, cudaStream_t st) {
  constexpr int R = FORM == kF32 ? 4 : 3;
  if (p.N > 128) {
    if (p.H == 32) return launch_umma<FORM, FOUR, 2, 32, 1, FORM == kF32 ? 3 : 5, FORM == kF32 ? 3 : 2>(p, st);
    if (W == 16) return launch_umma<FORM, FOUR, 2, 16, 2, R, 3>(p, st);
    return launch_umma<FORM, FOUR, 2, 16, 1, R, 3>(p, st);
  }
  if (p.H == 32) return launch_umma<FORM, FOUR, 1, 32, 1, 3, 3>(p, st);
  if (W == 16) return launch_umma<FORM, FOUR, 1, 16, 2, R, 3>(p, st);
  return launch_umma<FORM, FOUR, 1, 16, 1, R, 3>(p, st);
}

}  // namespace
}  // namespace dtc
