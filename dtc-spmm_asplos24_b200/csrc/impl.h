// Internal entry points shared between the library's translation units (not
// part of the C ABI).
#pragma once
#include "common.cuh"

namespace dtc {

// Epilogue applied to every C element the SpMM writes: C = act(A*B + bias[col]),
// act = ReLU when relu != 0 (the GCN layer's bias + activation).
struct Epilogue {
  const float* bias = nullptr;  // [N] or null
  int relu = 0;
};

// C = act(A B + bias) on ME-TCF arrays of block shape H x W. `slots`: workspace for
// the pieces of windows that chunk boundaries cut, H x N floats for each of
// `nslots` chunks, or null (clusters of CTAs then add the pieces up, with the same bits).
dtc_status spmm_run(const int32_t* rwo, const uint8_t* tile, const int32_t* toff,
                    const int32_t* s2x, const float* vals, int32_t M, int32_t nwin, int64_t T,
                    int bformat, const void* b0, const void* b1, int32_t N, int precision, float* C,
                    cudaStream_t st, Epilogue epi, int H, int W, float* slots, int64_t nslots);
// Chunks spmm_run cuts T blocks into when `nslots` does not limit them, and the
// bytes of that many slots.
int direct_chunks(int64_t T);
size_t direct_slots_bytes(int64_t T, int32_t N, int H);
// The tiles of a required region of `n` of them from its first 16-byte boundary on (the widths
// that are multiples of 4 are written 8 and 16 bytes at a time): one less off that boundary.
float* aligned_tiles(void* region, int32_t N, int64_t* n);
// The slots at byte `offset` of a caller workspace: `n` of them, a slot per chunk or as many
// as fit; null when none does.
float* slot_region(void* ws, size_t bytes, size_t offset, int64_t T, int32_t N, int H, int64_t* n);
// Tiles of the partials region that strict balance requires for `grid` chunks
// (0 = 16 per SM), and its bytes.
int64_t spmm_partials(int64_t T, int grid);
size_t spmm_partials_bytes(int64_t T, int32_t N, int grid, int H = 16);
dtc_status rowid_to_rwo(const int32_t* rowid, int64_t T, int32_t nwin, int32_t* rwo,
                        cudaStream_t st);
dtc_status spmm_mma_sync_impl(const int32_t* rwo, const uint8_t* tile, const int32_t* toff,
                              const int32_t* s2x, const float* vals, int32_t M, int32_t nwin,
                              const float* B, int32_t N, float* C, cudaStream_t st);
dtc_status pack_b_impl(int fmt, const float* B, int64_t rows, int32_t N, void* p0, void* p1,
                       cudaStream_t st);
dtc_status bformat_bytes_impl(int fmt, int64_t rows, int32_t N, size_t* b0, size_t* b1);

}  // namespace dtc
