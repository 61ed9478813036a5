// Interface of the float32-accurate tensor-core GEMM (implementation: tgemm_tf32.cu).
#pragma once

#include "common.cuh"

#include <cuda_runtime.h>

namespace b200q {
namespace tgemm {

constexpr int kTile = 128;      // rows of a tile
constexpr int kMaxDepth = 512;  // largest contraction of one launch
// How long one tensor-core accumulation runs before float32 additions take the sums up, in k-steps (an MMA each: 8 terms of
// tf32, 16 of halves).  The tensor core cuts off at every addition, always downwards, so a long run drifts.
//   tf32: relative error of a batch's factors against float64, 2048 columns of 8192 tokens: 5.6e-7 with 16 steps, 1.5e-7 with
//   four; elimination by float32 multiply-adds has 1.7e-7.  64 factors of K = 2048 take 8.3 and 9.0 ms.  The single problem
//   keeps 16 (K = 14336: 11.3 ms, 15.5 with four).
//   halves: the factor's update with eight steps leaves 3.3e-7 where tf32 with 16 left 5.0e-7 (K = 2048, 4873 tokens; 4096:
//   3.6e-7 and 5.8e-7), 14336 columns take 10.1 ms instead of 11.3; the sweep's products 2.9e-7 instead of 5.4e-7 (last of
//   4096 columns).  In a batch's factors four steps are 1 to 2 % worse than tf32 with four, two are not.
constexpr int kLongSlice = 16, kShortSlice = 4;
constexpr int kLongSlice16 = 8, kShortSlice16 = 4, kShortestSlice16 = 2;

// One side of a product: float32 values x as hi = tf32_rn(x), lo = tf32_rn(x - hi), K-major (row r holds
// the values of output row / column r), zero-padded to `ld`.  `rows`: rows the two arrays hold, reads
// beyond give zeros.  Problem b of a batch starts at row b * batch_rows.
// Or (`scale` set, on both sides) as halves: x * 2^k = hi + lo, eleven bits each like tf32, at half the bytes and twice
// the rate of the tensor cores; scale[row] = 2^-k brings the row's largest value below 2^15, so that values down to 2^-18
// of it keep all 22 bits and smaller ones are off by 2^-40 of it at most.  That is as good as tf32 unless the contraction
// index is graded in opposite directions on the two sides by more than that: whoever makes such operands evens it out
// (pivot_power below).
struct Operand {
  const void* hi;
  const void* lo;
  int64_t ld;
  int64_t rows;
  int64_t batch_rows;
  int row0;            // operand row of output row / column 0
  const float* scale = nullptr;
};

inline int64_t split_ld(int64_t cols) { return (cols + 31) / 32 * 32; }

// 2^k for a row whose largest magnitude is `largest`, and its inverse
__device__ __forceinline__ void row_scale(float largest, float& scale, float& inverse) {
  int k = 141 - (int)(__float_as_uint(largest) >> 23);
  k = min(max(k, -112), 126);
  scale = __uint_as_float((uint32_t)(127 + k) << 23);
  inverse = __uint_as_float((uint32_t)(127 - k) << 23);
}
// the hi halves of two neighbours and their lo halves
__device__ __forceinline__ void split_pair(float a, float b, uint32_t& hi, uint32_t& lo) {
  const __half2 h = __floats2half2_rn(a, b);
  const float2 f = __half22float2(h);
  const __half2 l = __floats2half2_rn(a - f.x, b - f.y);
  hi = *reinterpret_cast<const uint32_t*>(&h);
  lo = *reinterpret_cast<const uint32_t*>(&l);
}

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
  // ... or (out_hi set) the operand form of alpha * product (out_lo null: its float32 values, from row xt_rows on), and
  // for rows below xt_rows also X[column][row] = alpha * product in float32
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
  int slice = kLongSlice;       // k-steps that one tensor-core accumulation runs over
};
int launch(const Job& j, cudaStream_t st);

// src [rows][cols] -> hi/lo [rows][split_ld(cols)]
int split(const float* src, int64_t ld_src, int rows, int cols, float* hi, float* lo, cudaStream_t st);
// src [rows][cols] -> hi/lo [cols][ld_dst], row c = column c of src zero-padded
int split_transposed(const float* src, int64_t ld_src, int rows, int cols, float* hi, float* lo, int64_t ld_dst, cudaStream_t st);

// The sweep's products are sums over p of an error (w - q) / U[p,p] and U[p,j], one scale per row on either side.  Where the
// activations of column p have size s_p, pivots are of size 1 / s_p, rows of U as even as the correlations (with H = S R S,
// U is that of R times S^-1: columns are graded, and a column has its own scale), and errors go as (w - q) s_p.  With even
// weights it is the rows U[p,:] / U[p,p] that carry the grading and w - q that are even; with weights that go as 1 / s_p, or
// where clamping lets the errors grow, the errors are even and U is.  Half of the grading goes to each side: errors are taken
// times a power of two near the root of the pivot, rows of U times its inverse, and both keep all 22 bits in either
// case, and for rows of U in any sizes, while the sizes of a superblock's columns lie within 2^36 of one another
// (damping by 1 % of the mean diagonal alone keeps them within 10 sqrt(K)).
// Error of the last column of a sweep with all codes zero, 1001 x 1160, sizes 2^-18 .. 2^18: even weights 4.4e-7, weights
// that go as 1 / s_p 2.3e-7, rows of U in any sizes 2.3e-7 (2.4e-2, 2.2e-2 and 2.1e-7 with the whole grading on U's side);
// equal sizes 2.1e-7 either way.
// With w - q in place of the errors and -V U_bb in place of U it is the other way round: V is R's factor with its rows times
// s_p, so w - q are taken times the root's inverse and the rows times the root.
// (The factor needs none of this: in A - P P^T, P D and P X the contraction index has the columns of L = S L', whose rows
// are graded, and the rows of L^-1, whose columns are; what is left are the pivots of L', the factor of a matrix with unit
// diagonal, and where one of these is below 2^-12 float32 elimination fails.)
__device__ __forceinline__ int pivot_exponent(float reciprocal) {   // of its root, biased
  return 127 + ((min(max((int)(__float_as_uint(reciprocal) >> 23) & 255, 1), 253) - 127) >> 1);
}
__device__ __forceinline__ float pivot_power(float reciprocal) { return __uint_as_float((uint32_t)pivot_exponent(reciprocal) << 23); }
__device__ __forceinline__ float pivot_inverse(float reciprocal) {
  return __uint_as_float((uint32_t)(254 - pivot_exponent(reciprocal)) << 23);
}

// Operands of halves, rows of LD = 512 or 256 zero-padded beyond `cols`.
// Rows of src (src2 set: src + src2) -> hi / lo [rows][LD], scale[row], by CTA `cta` of `ctas` (256 threads): a warp takes a row,
// kept in registers between the search for its largest value and the split.  `columns` (optional): factors of the columns,
// `inverse`: powers of two whose inverses are.
template <int LD>
__device__ __forceinline__ void split_rows16(const float* __restrict__ src, const float* __restrict__ src2, int64_t ld_src,
                                             int64_t rows, int cols, __half* hi, __half* lo, float* scale,
                                             const float* __restrict__ columns, bool inverse, int64_t cta, int64_t ctas) {
  constexpr int kParts = LD / 128;
  const int lane = threadIdx.x & 31;
  float4 f[kParts];
#pragma unroll
  for (int i = 0; i < kParts; ++i) {
    f[i] = columns ? *reinterpret_cast<const float4*>(columns + i * 128 + lane * 4) : make_float4(1.f, 1.f, 1.f, 1.f);
    if (inverse) f[i] = make_float4(__frcp_rn(f[i].x), __frcp_rn(f[i].y), __frcp_rn(f[i].z), __frcp_rn(f[i].w));
  }
  for (int64_t r = cta * 8 + (threadIdx.x >> 5); r < rows; r += ctas * 8) {
    float4 x[kParts], y[kParts];
#pragma unroll
    for (int i = 0; i < kParts; ++i) x[i] = *reinterpret_cast<const float4*>(src + r * ld_src + i * 128 + lane * 4);
#pragma unroll
    for (int i = 0; i < kParts; ++i)
      y[i] = src2 ? *reinterpret_cast<const float4*>(src2 + r * ld_src + i * 128 + lane * 4) : make_float4(0.f, 0.f, 0.f, 0.f);
    float largest = 0.0f;
#pragma unroll
    for (int i = 0; i < kParts; ++i) {
      x[i].x = (x[i].x + y[i].x) * f[i].x; x[i].y = (x[i].y + y[i].y) * f[i].y;
      x[i].z = (x[i].z + y[i].z) * f[i].z; x[i].w = (x[i].w + y[i].w) * f[i].w;
      float* e = &x[i].x;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        if (i * 128 + lane * 4 + k >= cols) e[k] = 0.0f;
        largest = fmaxf(largest, fabsf(e[k]));
      }
    }
    largest = warp_max(largest);
    float to, back;
    row_scale(largest, to, back);
    if (lane == 0) scale[r] = back;
#pragma unroll
    for (int i = 0; i < kParts; ++i) {
      uint2 h, l;
      split_pair(x[i].x * to, x[i].y * to, h.x, l.x);
      split_pair(x[i].z * to, x[i].w * to, h.y, l.y);
      *reinterpret_cast<uint2*>(hi + r * LD + i * 128 + lane * 4) = h;
      *reinterpret_cast<uint2*>(lo + r * LD + i * 128 + lane * 4) = l;
    }
  }
}
// Columns 32 `cta` .. + 31 of src [rows][cols] -> operand rows of those numbers, by a CTA of 256 threads with
// split_columns16_smem(LD) bytes of shared memory.  Entries whose column is above `diagonal` + their row count as zero.
// `pivots`: row p is taken times pivot_power, or its inverse, of the pivot `rows` columns before src[p, p].
enum Pivots { kNoPivots = 0, kPowers = 1, kInverses = 2 };
constexpr size_t split_columns16_smem(int ld) { return 32 * (ld + 2) * sizeof(float); }
template <int LD>
__device__ __forceinline__ void split_columns16(const float* __restrict__ src, int64_t ld_src, int rows, int64_t cols,
                                                int64_t diagonal, __half* hi, __half* lo, float* scale, int pivots,
                                                int64_t cta, float* stage) {   // stage [32][LD + 2]
  __shared__ float s_max[8][32];
  __shared__ float s_power[LD];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t c = cta * 32 + lane, last = c < cols ? c : cols - 1;
  float v[LD / 8], largest = 0.0f;
  // (no load depends on a condition: they go out together)
#pragma unroll
  for (int i = 0; i < LD / 8; ++i) v[i] = src[(int64_t)min(warp + i * 8, rows - 1) * ld_src + last];
  if (pivots) {
    for (int p = threadIdx.x; p < LD; p += 256) {
      const float reciprocal = p < rows ? __frcp_rn(src[(int64_t)p * ld_src + p - rows]) : 1.0f;
      s_power[p] = pivots == kInverses ? pivot_inverse(reciprocal) : pivot_power(reciprocal);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < LD / 8; ++i) {
    const int p = warp + i * 8;
    if (p >= rows || c >= cols || c > diagonal + p) v[i] = 0.0f;
    if (pivots) v[i] *= s_power[p];
    largest = fmaxf(largest, fabsf(v[i]));
  }
  s_max[warp][lane] = largest;
  __syncthreads();
#pragma unroll
  for (int k = 0; k < 8; ++k) largest = fmaxf(largest, s_max[k][lane]);
  float to, back;
  row_scale(largest, to, back);
  if (warp == 0 && c < cols) scale[c] = back;
#pragma unroll
  for (int i = 0; i < LD / 8; ++i) stage[lane * (LD + 2) + warp + i * 8] = v[i] * to;
  __syncthreads();
  for (int k = warp; k < 32; k += 8) {
    if (cta * 32 + k >= cols) break;
    uint32_t* h = reinterpret_cast<uint32_t*>(hi + (cta * 32 + k) * LD);
    uint32_t* l = reinterpret_cast<uint32_t*>(lo + (cta * 32 + k) * LD);
#pragma unroll
    for (int i = 0; i < LD / 64; ++i) {
      const float2 x = *reinterpret_cast<const float2*>(stage + k * (LD + 2) + i * 64 + lane * 2);
      uint32_t a, b;
      split_pair(x.x, x.y, a, b);
      h[i * 32 + lane] = a;
      l[i * 32 + lane] = b;
    }
  }
}
// src [rows][ld_src] -> operand; `batch` problems src_batch, dst_rows apart, problem b with the column factors (ld of them)
// (or the inverses of these) at columns + columns_batch * index[b] (null: b)
int split_rows16(const float* src, int64_t ld_src, int64_t src_batch, int64_t rows, int cols, __half* hi, __half* lo, float* scale,
                 int ld, int64_t dst_rows, int batch, const float* columns, bool inverse, int64_t columns_batch, const int32_t* index,
                 cudaStream_t st);
// The operand of an update of the factor: rows [0, end) are the columns of the block row `row` [n][end] (its last n columns
// lower triangular), rows [end, end + first) f_hi + f_lo, then `rows` rows of p.
struct UpdateOperand {
  const float* row; int64_t row_ld, row_batch; int n; int64_t end;
  const float *f_hi, *f_lo; int64_t f_batch, first;
  const float* p; int64_t p_batch, rows;
  __half *hi, *lo; float* scale; int64_t dst_rows;
};
int split_update16(const UpdateOperand& u, int batch, cudaStream_t st);

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
