// Dense-operand storage forms ("B formats"), produced once and reused by
// every SpMM over the same B:
//   SPLIT24 : fp32 rounded to nearest-even at 16 significant bits and stored
//             as a bf16 "hi" plane plus a u8 "extension" plane (the next 8
//             mantissa bits). 3 bytes/element. In-kernel, lo = b24 - hi is
//             exact in bf16, so (hi, lo) reproduces b24 exactly.
//   BF16    : round-to-nearest-even bf16, 2 bytes/element.
//   FP8     : e4m3 (satfinite, RNE) of B[r,:] / s_r with s_r = max|B[r,:]|/448,
//             plus the fp32 per-row scale s_r. 1 byte/element + 4 bytes/row.
//   BF16X2  : hi = bf16_rn(b), lo = bf16_rn(b - hi) (b - hi is exact in fp32;
//             lo = 0 where hi is not finite), two bf16 planes: 4 bytes/element,
//             hi + lo carries ~16 significant bits and needs no rebuild.
#include <type_traits>
#include <cuda_bf16.h>
#include <cuda_fp8.h>
#include "common.cuh"

namespace dtc {
namespace {

__device__ __forceinline__ uint32_t round_to_b24(uint32_t u) {
  const uint32_t e = (u >> 23) & 0xFF;
  if (e == 0xFF) return (u & 0x7FFFFF) ? 0x7FC00000u : u;  // NaN -> canonical, Inf kept
  uint32_t r = u + 0x7Fu + ((u >> 8) & 1u);                // RNE at bit 8
  return r & 0xFFFFFF00u;
}

__device__ __forceinline__ uint32_t bf16_bits(float x) {
  return __bfloat16_as_ushort(__float2bfloat16_rn(x));
}

// One element to its planes: low 16 bits to plane 0 and, for two planes, the next to plane 1.
struct Split24 {
  using Second = uint8_t;
  __device__ __forceinline__ static uint32_t pack(float b) {
    const uint32_t r = round_to_b24(__float_as_uint(b));
    return (r >> 16) | (r >> 8 & 0xffu) << 16;
  }
};
struct Bf16 {
  using Second = void;
  __device__ __forceinline__ static uint32_t pack(float b) { return bf16_bits(b); }
};
struct Bf16x2 {
  using Second = uint16_t;
  __device__ __forceinline__ static uint32_t pack(float b) {
    const __nv_bfloat16 h = __float2bfloat16_rn(b);
    const float hf = __bfloat162float(h);
    return __bfloat16_as_ushort(h) | bf16_bits(isfinite(hf) ? b - hf : 0.0f) << 16;
  }
};

// Bound: DRAM (every element once in, once out). Where the base addresses allow (kVec: all
// aligned to 16 bytes) a thread takes 8 elements: two
// 16-byte loads, a 16-byte store to plane 0 and 16 or 8 bytes to plane 1. 2^20 x 128, an
// element per thread / this: BF16X2 189 / 170 us, SPLIT24 176 / 148, BF16 142 / 125.
template <typename F, bool kVec>
__global__ void __launch_bounds__(256)
    k_pack(const float* __restrict__ B, int64_t n, uint16_t* __restrict__ p0, void* __restrict__ p1) {
  constexpr bool kTwo = !std::is_void_v<typename F::Second>;
  constexpr bool kWide = std::is_same_v<typename F::Second, uint16_t>;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  int64_t done = 0;
  if constexpr (kVec) {
    done = n / 8 * 8;
    for (int64_t i = t; i < n / 8; i += stride) {
      const float4 x = __ldcs(reinterpret_cast<const float4*>(B) + 2 * i);
      const float4 y = __ldcs(reinterpret_cast<const float4*>(B) + 2 * i + 1);
      const uint32_t u[8] = {F::pack(x.x), F::pack(x.y), F::pack(x.z), F::pack(x.w),
                             F::pack(y.x), F::pack(y.y), F::pack(y.z), F::pack(y.w)};
      uint32_t a[4], b[4];
#pragma unroll
      for (int v = 0; v < 4; ++v) {
        a[v] = __byte_perm(u[2 * v], u[2 * v + 1], 0x5410);
        b[v] = __byte_perm(u[2 * v], u[2 * v + 1], kWide ? 0x7632 : 0x0062);
      }
      reinterpret_cast<uint4*>(p0)[i] = make_uint4(a[0], a[1], a[2], a[3]);
      if constexpr (kWide)
        reinterpret_cast<uint4*>(p1)[i] = make_uint4(b[0], b[1], b[2], b[3]);
      else if constexpr (kTwo)
        reinterpret_cast<uint2*>(p1)[i] = make_uint2(__byte_perm(b[0], b[1], 0x5410),
                                                     __byte_perm(b[2], b[3], 0x5410));
    }
  }
  for (int64_t i = done + t; i < n; i += stride) {
    const uint32_t u = F::pack(B[i]);
    p0[i] = (uint16_t)u;
    if constexpr (kTwo) reinterpret_cast<typename F::Second*>(p1)[i] = (typename F::Second)(u >> 16);
  }
}

// One warp per row: scale = max|x| / 448, q = e4m3(x / scale). kVec (N a multiple of 4,
// 16-byte aligned rows): four elements per lane and load. 2^20 x 128: 166 us, 209 us with
// one element per load and store.
__device__ __forceinline__ uint32_t e4m3(float x) {
  return (uint32_t)(uint8_t)__nv_cvt_float_to_fp8(x, __NV_SATFINITE, __NV_E4M3);
}
template <bool kVec>
__global__ void k_pack_fp8(const float* __restrict__ B, int64_t rows, int32_t N,
                           uint8_t* __restrict__ q, float* __restrict__ scale) {
  int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  int lane = threadIdx.x & 31;
  int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t r = warp; r < rows; r += nw) {
    const float* x = B + r * N;
    float m = 0.f;
    if constexpr (kVec) {
      for (int j = lane; j < N / 4; j += 32) {
        const float4 v = __ldg(reinterpret_cast<const float4*>(x) + j);
        m = fmaxf(fmaxf(m, fmaxf(fabsf(v.x), fabsf(v.y))), fmaxf(fabsf(v.z), fabsf(v.w)));
      }
    } else {
      for (int j = lane; j < N; j += 32) m = fmaxf(m, fabsf(x[j]));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    const float s = (m > 0.f && isfinite(m)) ? m / 448.0f : 1.0f;
    if (lane == 0) scale[r] = s;
    if constexpr (kVec) {
      for (int j = lane; j < N / 4; j += 32) {
        const float4 v = __ldg(reinterpret_cast<const float4*>(x) + j);
        reinterpret_cast<uint32_t*>(q + r * N)[j] =
            e4m3(v.x / s) | e4m3(v.y / s) << 8 | e4m3(v.z / s) << 16 | e4m3(v.w / s) << 24;
      }
    } else {
      for (int j = lane; j < N; j += 32) q[r * N + j] = (uint8_t)e4m3(x[j] / s);
    }
  }
}

inline unsigned grid_for(int64_t n) {
  int64_t g = (n + 255) / 256;
  if (g < 1) g = 1;
  if (g > 148 * 64) g = 148 * 64;
  return (unsigned)g;
}

template <typename F>
void pack(const float* B, int64_t n, void* p0, void* p1, cudaStream_t st) {
  if (((uintptr_t)B | (uintptr_t)p0 | (uintptr_t)p1) % 16 == 0)
    k_pack<F, true><<<grid_for((n + 7) / 8), 256, 0, st>>>(B, n, (uint16_t*)p0, p1);
  else
    k_pack<F, false><<<grid_for(n), 256, 0, st>>>(B, n, (uint16_t*)p0, p1);
}

}  // namespace

dtc_status bformat_bytes_impl(int fmt, int64_t rows, int32_t N, size_t* b0, size_t* b1) {
  DTC_REQUIRE(b0 && b1, "null size pointer");
  DTC_REQUIRE(rows >= 0 && N >= 1, "bad sizes");
  size_t n = (size_t)rows * N;
  switch (fmt) {
    case DTC_B_F32: *b0 = n * 4; *b1 = 0; return DTC_OK;
    case DTC_B_SPLIT24: *b0 = n * 2; *b1 = n; return DTC_OK;
    case DTC_B_BF16: *b0 = n * 2; *b1 = 0; return DTC_OK;
    case DTC_B_FP8: *b0 = n; *b1 = (size_t)rows * 4; return DTC_OK;
    case DTC_B_BF16X2: *b0 = n * 2; *b1 = n * 2; return DTC_OK;
  }
  set_error("unknown B format");
  return DTC_ERR_INVALID_ARGUMENT;
}

dtc_status pack_b_impl(int fmt, const float* B, int64_t rows, int32_t N, void* p0, void* p1,
                       cudaStream_t st) {
  DTC_REQUIRE(B && p0, "null device pointer");
  DTC_REQUIRE(rows >= 0 && N >= 1, "bad sizes");
  int64_t n = rows * (int64_t)N;
  if (n == 0) return DTC_OK;
  switch (fmt) {
    case DTC_B_F32:
      DTC_CUDA(cudaMemcpyAsync(p0, B, (size_t)n * 4, cudaMemcpyDeviceToDevice, st));
      return DTC_OK;
    case DTC_B_SPLIT24:
      DTC_REQUIRE(p1, "SPLIT24 needs two planes");
      pack<Split24>(B, n, p0, p1, st);
      break;
    case DTC_B_BF16:
      pack<Bf16>(B, n, p0, nullptr, st);
      break;
    case DTC_B_BF16X2:
      DTC_REQUIRE(p1, "BF16X2 needs two planes");
      pack<Bf16x2>(B, n, p0, p1, st);
      break;
    case DTC_B_FP8:
      DTC_REQUIRE(p1, "FP8 needs the scale plane");
      if (N % 4 == 0 && (uintptr_t)B % 16 == 0 && (uintptr_t)p0 % 4 == 0)
        k_pack_fp8<true><<<grid_for(rows * 32), 256, 0, st>>>(B, rows, N, (uint8_t*)p0, (float*)p1);
      else
        k_pack_fp8<false><<<grid_for(rows * 32), 256, 0, st>>>(B, rows, N, (uint8_t*)p0, (float*)p1);
      break;
    default:
      set_error("unknown B format");
      return DTC_ERR_INVALID_ARGUMENT;
  }
  DTC_CUDA(cudaGetLastError());
  return DTC_OK;
}

}  // namespace dtc
