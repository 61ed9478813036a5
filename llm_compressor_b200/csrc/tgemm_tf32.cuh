// Interface of the float32-accurate tensor-core GEMM (implementation: tgemm_tf32.cu).
#pragma once

#include "common.cuh"

#include <cuda_runtime.h>

namespace b200q {
namespace tgemm {

constexpr int kTile = 128;      // rows of a tile
constexpr int kMaxDepth = 512;  // largest contraction of one launch
// Chunks of 32 terms that one tensor-core accumulation runs over, before float32 additions take the sums up.  The tensor
// core cuts off at every addition, always downwards, so a long run drifts.  Relative error of a batch's factors against
// float64, 2048 columns of 8192 tokens: 5.6e-7 with four chunks, 1.5e-7 with one; elimination by float32 multiply-adds has
// 1.7e-7 (768 columns of 4096: 3.5e-7, 1.1e-7, 1.5e-7).  Half a chunk gives 1.4e-7.  64 factors of K = 2048 take 8.3, 9.0
// and 10.1 ms with four, one and half a chunk, 32 of K = 768 0.65, 0.68 and 0.71.  The single problem keeps four (K = 14336:
// 11.3 ms, 15.5 with one): 4.2e-7 where rank-128 updates had 6.1e-7.
constexpr int kLongSlice = 4, kShortSlice = 1;

// One side of a product: float32 values x as hi = tf32_rn(x), lo = tf32_rn(x - hi), K-major (row r holds
// the values of output row / column r), zero-padded to `ld`.  `rows`: rows the two arrays hold, reads
// beyond give zeros.  Problem b of a batch starts at row b * batch_rows.
struct Operand {
  const float* hi;
  const float* lo;
  int64_t ld;
  int64_t rows;
  int64_t batch_rows;
  int row0;            // operand row of output row / column 0
};

inline int64_t split_ld(int64_t cols) { return (cols + 31) / 32 * 32; }

// One half of an operand split: x rounded to nearest even on 10 mantissa bits, as a float32 word
// whose low 13 mantissa bits are zero.
__device__ __forceinline__ float tf32_rn(float x) {
  uint32_t b = __float_as_uint(x);
  b = (b + 0xFFFu + ((b >> 13) & 1u)) & 0xFFFFE000u;
  return __uint_as_float(b);
}

// Which tiles of the output a launch computes:
//   kAll    every tile
//   kLower  tiles that hold something on or below the diagonal
//   kPanel  all columns of every row outside [skip0, skip1)
//   kBulk   rows from row_begin on: columns below skip0 for rows below skip1, else everything on or below the diagonal
//   kLowerBlocks   as kLower, and nothing outside the 128 x 128 blocks on or below the diagonal: tiles no larger than these
enum TileSet { kAll = 0, kLower = 1, kPanel = 2, kBulk = 3, kLowerBlocks = 4 };

struct Job {
  Operand A, B;
  int M, N, Kd;                 // extent of the output (row and column limits) and of the contraction
  int set = kAll, row_begin = 0, skip0 = 0, skip1 = 0;
  int batch = 1;
  const int32_t* b_index = nullptr;   // device: problem b multiplies with operand B of problem b_index[b]
  float alpha = 1.0f, beta = 0.0f;
  // output: C = beta * C + alpha * product, with beta = 0 for columns in [fresh0, fresh1) ...
  float* C = nullptr;           // problem b: C + b * c_batch, or c_table[b] + c_offset
  float* const* c_table = nullptr;
  int64_t c_offset = 0, c_batch = 0, ldc = 0;
  int fresh0 = 0, fresh1 = 0;
  // ... or (out_hi set) the operand form of alpha * product, and for rows below xt_rows also
  // X[column][row] = alpha * product in float32
  float* out_hi = nullptr;
  float* out_lo = nullptr;
  int64_t out_ld = 0, out_batch = 0;
  int out_row0 = 0;
  float* X = nullptr;
  int64_t x_batch = 0, ldx = 0;
  int xt_rows = 0;
  int* status = nullptr;        // problem b: status + b * status_stride
  int status_stride = 0;
  int max_ctas = 0;             // 0: the whole GPU
  int slice = kLongSlice;       // chunks that one tensor-core accumulation runs over
};
int launch(const Job& j, cudaStream_t st);

// src [rows][cols] -> hi/lo [rows][split_ld(cols)]
int split(const float* src, int64_t ld_src, int rows, int cols, float* hi, float* lo, cudaStream_t st);
// src [rows][cols] -> hi/lo [cols][ld_dst], row c = column c of src zero-padded; `batch` problems given by a device
// table of pointers (src + src_offset each) or, without one, a single matrix
int split_transposed(const float* src, const float* const* table, int64_t src_offset, int64_t ld_src, int rows, int cols,
                     float* hi, float* lo, int64_t ld_dst, int64_t dst_batch, int batch, cudaStream_t st);

// A helper stream of the calling host thread (same priority as `like`), with events, for the look-ahead of the
// blocked solves: the bulk of an update runs there while the caller's stream goes on with the next block.
// Created once per device and caller stream; null on failure.
struct SideStream {
  cudaStream_t stream = nullptr;
  cudaEvent_t ready = nullptr;   // recorded on the caller's stream: operands of the bulk update exist
  cudaEvent_t next = nullptr;    // recorded on the caller's stream: the part that goes first is done
  cudaEvent_t done = nullptr;    // recorded on the helper: bulk update finished
};
SideStream* side_stream(cudaStream_t like);

}  // namespace tgemm
}  // namespace b200q
