// Host side of the TC-block SpMM (kernels in spmm_direct.cuh): argument checks,
// chunk counts, workspace sizes, and the fp32 forms' kernels.
#include <algorithm>
#include "spmm_direct.cuh"

namespace dtc {
namespace {

constexpr int kWavesPerSm = 16;  // chunks per SM of the required partials region

// rwo[w] = first block of window w, from the sorted window id of every block.
// Ids come from the caller: an id outside [0, nwin) or a descending pair is
// reported through kErrBadIndex, and the written range is clamped to the
// (nwin + 1)-entry table, so a bad id never writes outside it. The table starts at 0
// and ends at T whatever the ids are: the kernels rely on it to find a window that
// holds a given block (cut_at).
__global__ void k_rowid_to_rwo(const int32_t* __restrict__ rowid, int64_t T, int32_t nwin,
                               int32_t* __restrict__ rwo, uint32_t* err) {
  int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t b = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; b <= T; b += stride) {
    const int32_t prev = (b == 0) ? -1 : __ldg(rowid + b - 1);
    const int32_t cur = (b == T) ? nwin : __ldg(rowid + b);
    const bool bad = (b < T && (cur < 0 || cur >= nwin)) || cur < prev;
    if (bad) atomicOr(err, kErrBadIndex);
    const int32_t lo = prev < -1 ? -1 : (prev > nwin ? nwin : prev);
    const int32_t hi = cur < -1 ? -1 : (cur > nwin ? nwin : cur);
    for (int32_t w = max(lo + 1, 1); w <= min(hi, nwin - 1); ++w) rwo[w] = (int32_t)b;
    if (b == 0) rwo[0] = 0;
    if (b == T) rwo[nwin] = (int32_t)T;
  }
}

// C of a matrix without blocks: the epilogue of 0, a warp per row.
__global__ void __launch_bounds__(256) k_no_blocks(const DirectParams p) {
  for (int64_t r = blockIdx.x * 8ll + threadIdx.x / 32; r < p.M; r += gridDim.x * 8ll)
    for (int f = threadIdx.x % 32; f < p.N; f += 32) p.C[r * p.N + f] = finish(p, 0.0f, f);
}

}  // namespace

dtc_status direct_f32(DirectParams& p, int W, cudaStream_t st) {
  return by_block<kF32, false>(p, W, st);
}

int64_t spmm_partials(int64_t T, int grid) {
  int64_t G = grid > 0 ? grid : kWavesPerSm * num_sms();
  if (G > T) G = T > 0 ? T : 1;
  return 2 * G;
}

size_t spmm_partials_bytes(int64_t T, int32_t N, int grid, int H) {
  return (size_t)spmm_partials(T, grid) * H * (size_t)N * sizeof(float);
}

dtc_status rowid_to_rwo(const int32_t* rowid, int64_t T, int32_t nwin, int32_t* rwo,
                        cudaStream_t st) {
  int64_t n = T + 1;
  unsigned g = (unsigned)((n + 255) / 256);
  if (g > 65535u * 16) g = 65535u * 16;
  k_rowid_to_rwo<<<g, 256, 0, st>>>(rowid, T, nwin, rwo, device_error_word());
  DTC_CUDA(cudaGetLastError());
  return DTC_OK;
}

// Chunks of the TC-block range when no workspace limits them.
//   up to 1024 blocks: chunks of 8; then 128 of them until they have 32
//   chunks of 32 blocks up to three per SM (one wave), then these until they have 64
//   beyond, chunks of a third of an SM's share until that is kNW * 80 blocks, of that size until
//   it is a fifteenth of a share, then up to kNW * 192 blocks; the last quarter of the blocks in
//   chunks a quarter as long, so that the last CTAs to start are short (R-MAT 2^19, N = 128 on
//   tcgen05: 1.10 -> 0.87 ms): 5.25 and 26 chunks per SM in all
// A chunk costs its pipeline's start and, where it cuts a window, a piece in the workspace; too few
// leave SMs idle. us, before / with the line in question: 302 blocks, fp32 N = 256 20.7 (chunks of 32)
// / 13.1; 24,059 blocks, fp32 N = 256 57 (3.1 per SM: a second wave) / 40; 27-point stencil 40^3,
// BF16, 32-row windows 117 (15 alike per SM) / 69, R-MAT 2^15 133 / 94; R-MAT 2^18 with the 15 per SM
// 502, with 3 580.
// kMaxChunks bounds the workspace (a tile of H x N floats each), not the speed: beyond 7 M blocks
// there are more than 60 per SM all the same.
constexpr int64_t kMaxChunks = 16384;
struct Chunks {
  int64_t g, g1;  // all chunks; those of the first three quarters (0: all alike)
};
Chunks chunks_of(int64_t T) {
  const int64_t sms = num_sms(), wave = 3 * sms;
  if (T / (wave * kNW) < 16)
    return {std::max<int64_t>({1, std::min<int64_t>(T / 8, 128), std::min(T / 32, wave)}), 0};
  int64_t q = std::max(std::min<int64_t>(T / (wave * kNW), 80), T / (5 * wave * kNW));
  q = std::max(std::min<int64_t>(q, 192), T / (kMaxChunks * 4 / 7 * kNW) + 1);
  const int64_t g = T / (q * kNW);
  return {g * 3 / 4 + g, g * 3 / 4};
}
int direct_chunks(int64_t T) { return (int)chunks_of(T).g; }

size_t direct_slots_bytes(int64_t T, int32_t N, int H) {
  return align_up((size_t)direct_chunks(T) * H * (size_t)N * sizeof(float), 256);
}

dtc_status spmm_run(const int32_t* rwo, const uint8_t* tile, const int32_t* toff,
                    const int32_t* s2x, const float* vals, int32_t M, int32_t nwin, int64_t T,
                    int bformat, const void* b0, const void* b1, int32_t N, int precision, float* C,
                    cudaStream_t st, Epilogue epi, int H, int W, float* slots, int64_t nslots) {
  DTC_REQUIRE(M >= 0 && N >= 1 && T >= 0, "bad sizes");
  DTC_REQUIRE(T < ((int64_t)1 << 31), "more than 2^31 - 1 TC blocks");
  DTC_REQUIRE(H == 16 || H == 32, "window height must be 16 or 32");
  DTC_REQUIRE(W == 8 || (W == 16 && H == 16),
              "block width must be 8, or 16 at window height 16 (tile ids are bytes)");
  DTC_REQUIRE(nwin == (M + (int64_t)H - 1) / H,
              "num_windows must be ceil(num_nodes / window height)");
  if (bformat == DTC_B_F32 && precision == DTC_PREC_TF32) {
    if (N % 4 == 0) {
      DTC_REQUIRE(((uintptr_t)b0 & 15) == 0, "B must be 16-byte aligned");
      DTC_REQUIRE(((uintptr_t)s2x & 15) == 0, "SparseAToX must be 16-byte aligned");
    }
  } else {
    DTC_REQUIRE(bformat == DTC_B_SPLIT24 || bformat == DTC_B_BF16 || bformat == DTC_B_FP8 ||
                    bformat == DTC_B_BF16X2,
                "split kernels take SPLIT24, BF16, FP8 or BF16X2 B");
    DTC_REQUIRE(precision == DTC_PREC_SPLIT3 || precision == DTC_PREC_SPLIT4,
                "split kernels take precision SPLIT3 or SPLIT4");
    DTC_REQUIRE(N % 16 == 0, "split forms need N % 16 == 0 (16-byte row segments of every plane)");
    DTC_REQUIRE(bformat == DTC_B_BF16 || b1 != nullptr, "second B plane missing");
    DTC_REQUIRE(((uintptr_t)b0 & 15) == 0 && ((uintptr_t)b1 & 15) == 0,
                "planes must be 16-byte aligned");
    DTC_REQUIRE(((uintptr_t)s2x & 15) == 0, "SparseAToX must be 16-byte aligned");
  }
  if (!is_sm100()) {
    set_error("the SpMM kernels need an sm_100 device");
    return DTC_ERR_UNSUPPORTED;
  }
  if (M == 0) return DTC_OK;
  DirectParams p{};
  p.rwo = rwo; p.toff = toff; p.s2x = s2x; p.tile = tile; p.vals = vals;
  p.b0 = b0; p.b1 = b1; p.C = C; p.err = device_error_word();
  p.stamps = cta_timer_buffer(&p.stamp_cap);
  p.bias = epi.bias; p.relu = epi.relu;
  p.M = M; p.nwin = nwin; p.N = N; p.H = H; p.T = (int32_t)T;
  if (T == 0) {
    if (epi.bias) {
      k_no_blocks<<<(unsigned)std::min<int64_t>(((int64_t)M + 7) / 8, 8 * num_sms()), 256, 0, st>>>(p);
      DTC_CUDA(cudaGetLastError());
    } else {  // (ReLU of 0 is 0)
      DTC_CUDA(cudaMemsetAsync(C, 0, (size_t)M * N * sizeof(float), st));
    }
    return DTC_OK;
  }
  if (N % 4 == 0) DTC_REQUIRE(((uintptr_t)C & 15) == 0, "C must be 16-byte aligned");
  // tcgen05 (spmm_umma.cuh) beyond 128 features, where an instruction fills its 128
  // rows twice per gathered block, and from 65 on where the mma.sync kernel needs twice
  // the instructions per block (32-row windows; the two planes of BF16X2). ms, mma.sync /
  // tcgen05, B200: R-MAT 2^19 N = 128, 16 x 8: fp32 0.73 / 0.87, BF16X2 0.99 / 0.97, BF16
  // 0.84 / 0.91; 32 x 8: fp32 1.25 / 0.90, BF16X2 1.63 / 1.03, BF16 1.27 / 0.96; stencil
  // 100^3 N = 256, 16 x 8: fp32 1.45 / 1.19, BF16X2 1.60 / 1.24, BF16 1.22 / 1.03.
  const bool umma = N > 128 || (N > 64 && (H == 32 || bformat == DTC_B_BF16X2));
  // Fewer slots than chunks: as many chunks as there are slots. So few that the product leaves SMs
  // idle are left alone: R-MAT 2^18, 2 per SM / none, ms: fp32 N = 128 0.56 / 0.68; on tcgen05 (a
  // pipeline per CTA) N = 256 1.96 / 0.98, BF16X2 N = 128 1.26 / 0.67. R-MAT 2^20, fp32 N = 128, 32
  // per SM 1.5 / 2.4.
  const Chunks c = chunks_of(T);
  if (slots && c.g > nslots && nslots < (umma ? 8 : 2) * num_sms()) slots = nullptr;
  const bool limited = slots && c.g > nslots;
  p.slots = slots;
  p.G = (int)(limited ? nslots : c.g);
  p.G1 = limited ? 0 : (int)c.g1;
  // Windows of more blocks are cut at chunk boundaries: of more than a chunk has, and than a common
  // window of small graphs (4096 rows of 8 edges, 32-row windows of about 32 blocks, N = 512 fp32: half
  // of them cut 44 us, none 27).
  p.lmax = (int32_t)(p.G1 ? T * 3 / 4 / p.G1 + 1
                          : std::max<int64_t>((T + p.G - 1) / p.G, H == 32 ? 48 : 32));
  const bool four = precision == DTC_PREC_SPLIT4;
  switch (bformat) {
    case DTC_B_F32:
      if (N % 4) return direct_f32_odd(p, W, st);
      return umma ? umma_f32(p, W, st) : direct_f32(p, W, st);
    case DTC_B_SPLIT24:
      return direct_split24(p, W, four, st);
    case DTC_B_BF16X2:
      return umma ? umma_bf16x2(p, W, four, st) : direct_bf16x2(p, W, four, st);
    case DTC_B_BF16:
      return umma ? umma_bf16(p, W, st) : direct_bf16(p, W, st);
    default:
      return direct_fp8(p, W, st);
  }
}

}  // namespace dtc
