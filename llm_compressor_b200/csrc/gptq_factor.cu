// GPTQ solve: the factor U (upper) with U^T U = H^-1, on device in fp32, for one Hessian or a batch of equal size.
//
// Let J be the index reversal.  If J H J = L L^T (ordinary lower Cholesky) then H = V V^T with V = J L J upper
// triangular, hence H^-1 = V^-T V^-1 and the wanted factor is U = V^-1 = J L^-1 J (upper, positive diagonal, so it
// equals the upper Cholesky factor of H^-1).  That is one Cholesky and one triangular inverse (2/3 K^3 flops)
// instead of Cholesky, Cholesky-inverse and a second Cholesky (4/3 K^3).
//
// The chain of dependent steps, not the arithmetic, is what a factorisation waits for, so the matrix is worked on in
// two levels.  The outer level takes 512 columns at a time: the 512 x 512 square on the diagonal is replaced by the
// inverse D of its Cholesky factor, everything else takes rank-512 products with D and with the panels on the tensor
// cores (tgemm).  Only the square is on the chain: four 128-column steps of one small kernel each for the diagonal
// block, the panel inside the square and the square's own update.  (With rank-128 steps over the whole matrix the
// chain was ten launches and 115 us per 128 columns, and every step moved all of the trailing matrix through HBM.)
//
// Storage during the pass, A = J H J (lower part): block columns left of the current outer block hold, in the rows
// below it, S[i,j] = -sum_m L[i,m] X[m,j] of the forward substitution for X = L^-1, block columns right of it the
// Schur complement.  Outer step o with D = L_oo^-1:
//     X[o,:o] = D S[o,:o]      P = A[below,o] D^T (= L[below,o])      S[below,o] = -P D
//     S[i,:o] -= P_i X[o,:o]   and   A[i,j] -= P_i P_j^T (o < j <= i)
// The last three are one launch: the rows of its second operand are X[o,:o]^T, D^T and P, indexed by absolute column.
//
// A pivot <= 0 (or NaN) sets the problem's status; the host then takes the reference's identity fallback.
#include "common.cuh"
#include "tgemm_tf32.cuh"

namespace b200q {
namespace factor {

constexpr int NB = 128;          // inner block
constexpr int OB = 512;          // outer block
constexpr int kThreads = 256;
constexpr int LD = NB + 4;       // shared-memory stride: 16-byte rows, float4 accesses of 8 consecutive rows conflict-free

struct Mat {                     // the batch's work matrices and status words
  float* A; int64_t batch, lda;
  int* status;
};

__device__ __forceinline__ uint64_t pack2(float a, float b) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void fma2(uint64_t& d, uint64_t a, uint64_t b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}
__device__ __forceinline__ float sum2(uint64_t v) {
  float a, b;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
  return a + b;
}
// 32-deep dot products of R rows and C columns of shared memory, both with the contraction contiguous; packed
// float32 pairs along the contraction, so that a float4 load feeds two FFMA2 without shuffling
template <int R, int C>
__device__ __forceinline__ void dots(const float* (&row)[R], const float* (&col)[C], int depth, uint64_t (&acc)[R][C]) {
#pragma unroll
  for (int r = 0; r < R; ++r)
#pragma unroll
    for (int c = 0; c < C; ++c) acc[r][c] = 0;
#pragma unroll 2
  for (int m = 0; m < depth; m += 4) {
    ulonglong2 a[R], b[C];
#pragma unroll
    for (int r = 0; r < R; ++r) a[r] = *reinterpret_cast<const ulonglong2*>(row[r] + m);
#pragma unroll
    for (int c = 0; c < C; ++c) b[c] = *reinterpret_cast<const ulonglong2*>(col[c] + m);
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int c = 0; c < C; ++c) { fma2(acc[r][c], a[r].x, b[c].x); fma2(acc[r][c], a[r].y, b[c].y); }
  }
}

// ---------------------------------------------------------------------------------------
// Diagonal block: L^-1 of the n x n (n <= 128) block at (k0, k0), over the block itself.
//
// One CTA on the critical path, so the design is about latency.  The identity is appended below the block, which
// turns the triangular inverse into more rows of the same elimination (a row e_i ends as row i of L^-T): at every
// 32-column step exactly four 32-row blocks take part, one per warp.  A step:
//   warp 0 factors the 32 x 32 diagonal block in registers, a lane per row, about 95 cycles a column: the next pivot
//          is formed by its own lane and broadcast before the other columns are updated; meanwhile the other seven
//          warps finish the update by the step before
//   four warps substitute their 32 rows, a lane per row, against the transposed block in shared memory
//   all warps bring the next diagonal block up to date
// 11 us for 128 columns; the register-tiled version with a barrier per column that this replaces took 58.
constexpr int kCholSmemFloats = 2 * NB * LD + 32 * 36 + 32;

__global__ void __launch_bounds__(kThreads, 1) chol_diag_kernel(Mat mt, int k0, int n) {
  extern __shared__ __align__(16) float sm[];
  float* R = sm;                    // rows 0..127: the block, then L; rows 128..255: the identity, then L^-T
  float* Lt = R + 2 * NB * LD;      // [32][36] transposed diagonal block of the step
  float* rinv = Lt + 32 * 36;       // [32]
  float* A = mt.A + blockIdx.x * mt.batch + (int64_t)k0 * mt.lda + k0;
  int* status = mt.status + 4 * blockIdx.x;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
#pragma unroll 4
  for (int idx = tid; idx < NB * NB / 4; idx += kThreads) {
    const int r = idx >> 5, c = (idx & 31) << 2;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    float* e = &v.x;
    if (r < n && c <= r) {
      if (c + 3 < n) v = *reinterpret_cast<const float4*>(A + (int64_t)r * mt.lda + c);
      else
        for (int k = 0; k < 4; ++k)
          if (c + k < n) e[k] = A[(int64_t)r * mt.lda + c + k];
    }
    float4 id = make_float4(0.f, 0.f, 0.f, 0.f);
    float* d = &id.x;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      if (c + k > r) e[k] = 0.0f;
      if (c + k == r) { d[k] = 1.0f; if (r >= n) e[k] = 1.0f; }   // identity padding beyond n
    }
    *reinterpret_cast<float4*>(R + r * LD + c) = v;
    *reinterpret_cast<float4*>(R + (NB + r) * LD + c) = id;
  }
  __syncthreads();
  for (int kb = 0; kb < 4; ++kb) {
    const int c0 = kb * 32;
    if (warp == 0) {
      float a[32];
      const float* src = R + (c0 + lane) * LD + c0;
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const float4 v = *reinterpret_cast<const float4*>(src + 4 * q);
        a[4 * q] = v.x; a[4 * q + 1] = v.y; a[4 * q + 2] = v.z; a[4 * q + 3] = v.w;
      }
      float piv = __shfl_sync(0xffffffffu, a[0], 0);
#pragma unroll
      for (int j = 0; j < 32; ++j) {
        if (!(piv > 0.0f)) {   // also true for NaN; uniform
          if (lane == 0 && atomicCAS(status, 0, B200Q_NOT_POSITIVE_DEFINITE) == 0) status[1] = k0 + c0 + j + 1;
          piv = 1.0f;
        }
        float r = rsqrtf(piv);
        r = fmaf(0.5f * r, fmaf(-piv * r, r, 1.0f), r);   // one Newton step: within an ulp of 1 / sqrt
        const float l = (lane == j) ? piv * r : a[j] * r;
        if (j + 1 < 32) piv = __shfl_sync(0xffffffffu, fmaf(-l, l, a[j + 1]), j + 1);
        a[j] = l;
        if (lane == j) rinv[j] = r;
#pragma unroll
        for (int c = j + 1; c < 32; ++c) a[c] = fmaf(-l, __shfl_sync(0xffffffffu, l, c), a[c]);
      }
#pragma unroll
      for (int j = 0; j < 32; ++j) Lt[j * 36 + lane] = (j <= lane) ? a[j] : 0.0f;
    } else if (kb > 0) {
      // the rest of the update by step kb - 1: every active row block x the columns from c0 on, but the next
      // diagonal block, which is done already.  A warp per 32 x 32 block, 8 rows x 4 columns a lane.
      const int p0 = c0 - 32, nc = 4 - kb;
      for (int t = warp - 1; t < 4 * nc - 1; t += 7) {
        const int u = t + 1;                                  // task 0 is the diagonal block
        const int rb = (kb + u / nc) & 3, cb = kb + u % nc;   // row blocks kb, kb+1, ... wrapping to the identity rows
        const int r0 = (rb >= kb ? rb * 32 : NB + rb * 32) + (lane >> 3) * 8, cc = cb * 32 + (lane & 7);
        if (rb >= kb && cb > rb) continue;                    // above the diagonal
        const float *row[8], *col[4];
#pragma unroll
        for (int i = 0; i < 8; ++i) row[i] = R + (r0 + i) * LD + p0;
#pragma unroll
        for (int i = 0; i < 4; ++i) col[i] = R + (cc + 8 * i) * LD + p0;
        uint64_t acc[8][4];
        dots<8, 4>(row, col, 32, acc);
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
          for (int q = 0; q < 4; ++q) R[(r0 + i) * LD + cc + 8 * q] -= sum2(acc[i][q]);
      }
    }
    __syncthreads();
    if (warp < 4) {
      // block s: identity rows up to kb (their inverse is being born), rows of the matrix after it
      float* row = R + ((warp <= kb ? NB : 0) + warp * 32 + lane) * LD + c0;
      float a[32];
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const float4 v = *reinterpret_cast<const float4*>(row + 4 * q);
        a[4 * q] = v.x; a[4 * q + 1] = v.y; a[4 * q + 2] = v.z; a[4 * q + 3] = v.w;
      }
#pragma unroll
      for (int j = 0; j < 32; ++j) {
        const float y = a[j] * rinv[j];
        a[j] = y;
#pragma unroll
        for (int q = (j + 1) / 4; q < 8; ++q) {
          const float4 l = *reinterpret_cast<const float4*>(Lt + j * 36 + 4 * q);
          if (4 * q > j) a[4 * q] = fmaf(-y, l.x, a[4 * q]);
          if (4 * q + 1 > j) a[4 * q + 1] = fmaf(-y, l.y, a[4 * q + 1]);
          if (4 * q + 2 > j) a[4 * q + 2] = fmaf(-y, l.z, a[4 * q + 2]);
          if (4 * q + 3 > j) a[4 * q + 3] = fmaf(-y, l.w, a[4 * q + 3]);
        }
      }
#pragma unroll
      for (int q = 0; q < 8; ++q)
        *reinterpret_cast<float4*>(row + 4 * q) = make_float4(a[4 * q], a[4 * q + 1], a[4 * q + 2], a[4 * q + 3]);
    }
    __syncthreads();
    if (kb < 3) {   // next diagonal block: a lane per row, four columns a warp
      const int d0 = c0 + 32;
      const float* row[1] = {R + (d0 + lane) * LD + c0};
      const float* col[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) col[i] = R + (d0 + warp * 4 + i) * LD + c0;
      uint64_t acc[1][4];
      dots<1, 4>(row, col, 32, acc);
      float* o = R + (d0 + lane) * LD + d0 + warp * 4;
      float4 v = *reinterpret_cast<float4*>(o);
      v.x -= sum2(acc[0][0]); v.y -= sum2(acc[0][1]); v.z -= sum2(acc[0][2]); v.w -= sum2(acc[0][3]);
      *reinterpret_cast<float4*>(o) = v;
      __syncthreads();
    }
  }
  // D[j][i] = (L^-T)[i][j]: a lane reads four columns of its row i, the lanes of a store hold consecutive i
#pragma unroll 4
  for (int idx = tid; idx < NB * NB / 4; idx += kThreads) {
    const int i = idx & 127, j = (idx >> 7) << 2;
    const float4 v = *reinterpret_cast<const float4*>(R + (NB + i) * LD + j);
    const float e[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (j + k < n && i < n) A[(int64_t)(j + k) * mt.lda + i] = (i <= j + k) ? e[k] : 0.0f;
  }
}

// ---------------------------------------------------------------------------------------
// Inside the square at K0 (n columns), step k: everything the diagonal block's inverse D multiplies.  A CTA owns 16
// "vectors" of 128: rows r below the block (P[r] = A[r, blk] D^T, into the scratch P), then columns c left of it
// (X[blk, c] = D S[blk, c], in place).  D is triangular, so output j needs only the first j + 1 terms.
constexpr int kVec = 16;
constexpr int kPanelSmemFloats = (NB + kVec) * LD;

__global__ void __launch_bounds__(kThreads) panel_kernel(Mat mt, float* P0, int K0, int n, int k) {
  extern __shared__ __align__(16) float sm[];
  float* D = sm;                 // [128][LD]
  float* V = D + NB * LD;        // [16][LD] the CTA's vectors, contraction contiguous
  float* A = mt.A + blockIdx.y * mt.batch + (int64_t)K0 * mt.lda + K0;
  float* P = P0 + (int64_t)blockIdx.y * OB * NB;
  const int tid = threadIdx.x, b0 = k * NB, bn = n - b0 < NB ? n - b0 : NB, below = n - b0 - bn;
  const int below_ctas = (below + kVec - 1) / kVec;
  const bool rows = (int)blockIdx.x < below_ctas;
  const int v0 = rows ? b0 + bn + blockIdx.x * kVec : ((int)blockIdx.x - below_ctas) * kVec;
  const float* Dk = A + (int64_t)b0 * mt.lda + b0;
#pragma unroll 8
  for (int idx = tid; idx < NB * NB / 4; idx += kThreads) {
    const int r = idx >> 5, c = (idx & 31) << 2;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (r < bn && c <= r) {
      if (c + 3 < bn) v = *reinterpret_cast<const float4*>(Dk + (int64_t)r * mt.lda + c);
      else {
        float* e = &v.x;
        for (int q = 0; q < 4; ++q)
          if (c + q < bn) e[q] = Dk[(int64_t)r * mt.lda + c + q];
      }
    }
    *reinterpret_cast<float4*>(D + r * LD + c) = v;
  }
  for (int idx = tid; idx < kVec * NB; idx += kThreads) {
    const int v = rows ? idx >> 7 : idx & 15, m = rows ? idx & 127 : idx >> 4;
    float x = 0.0f;
    if (m < bn && (rows ? v0 + v < n : true))
      x = rows ? A[(int64_t)(v0 + v) * mt.lda + b0 + m] : A[(int64_t)(b0 + m) * mt.lda + v0 + v];
    V[v * LD + m] = x;
  }
  __syncthreads();
  // outputs 4 vectors x 2 entries of D's rows per thread; a warp's rows of D are 32 consecutive ones
  const int warp = tid >> 5, lane = tid & 31;
  const int vq = lane & 3, j0 = (warp & 3) * 32 + (lane >> 2), jh = (warp >> 2) * 16;
  const float *row[4], *col[2];
#pragma unroll
  for (int i = 0; i < 4; ++i) row[i] = V + (vq + 4 * i) * LD;
#pragma unroll
  for (int i = 0; i < 2; ++i) col[i] = D + (j0 + jh + 8 * i) * LD;
  uint64_t acc[4][2];
  dots<4, 2>(row, col, (warp & 3) * 32 + 32, acc);
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const int v = v0 + vq + 4 * i, j = j0 + jh + 8 * q;
      const float x = sum2(acc[i][q]);
      if (j >= bn) continue;
      if (rows) { if (v < n) P[(int64_t)v * NB + j] = x; }
      else A[(int64_t)(b0 + j) * mt.lda + v] = x;
    }
}

// Inside the square, step k: rows below the block take -P times X (columns left), D (the block's own columns, which
// start from zero) and P^T (columns right, on and below the diagonal).  A CTA owns a 32 x 32 tile.
constexpr int kUpdSmemFloats = 2 * 32 * LD;

__global__ void __launch_bounds__(kThreads) square_update_kernel(Mat mt, const float* P0, int K0, int n, int k) {
  extern __shared__ __align__(16) float sm[];
  float* Ps = sm;                // [32][LD]
  float* Qs = Ps + 32 * LD;      // [32][LD] second operand, contraction contiguous
  float* A = mt.A + blockIdx.y * mt.batch + (int64_t)K0 * mt.lda + K0;
  const float* P = P0 + (int64_t)blockIdx.y * OB * NB;
  const int tid = threadIdx.x, b0 = k * NB, r_begin = b0 + NB;
  // tile list: row tile i (32 rows from r_begin on) has r_begin / 32 + i + 1 column tiles
  const int base = r_begin / 32;
  int i = 0, t = blockIdx.x;
  while (t >= base + i + 1) { t -= base + i + 1; ++i; }
  const int r0 = r_begin + i * 32, c0 = t * 32;
  const bool right = c0 >= r_begin, own = !right && c0 >= b0;
#pragma unroll 4
  for (int idx = tid; idx < 32 * NB / 4; idx += kThreads) {
    const int r = idx >> 5, m = (idx & 31) << 2;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (r0 + r < n) v = *reinterpret_cast<const float4*>(P + (int64_t)(r0 + r) * NB + m);
    *reinterpret_cast<float4*>(Ps + r * LD + m) = v;
  }
  if (right) {
#pragma unroll 4
    for (int idx = tid; idx < 32 * NB / 4; idx += kThreads) {
      const int r = idx >> 5, m = (idx & 31) << 2;
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
      if (c0 + r < n) v = *reinterpret_cast<const float4*>(P + (int64_t)(c0 + r) * NB + m);
      *reinterpret_cast<float4*>(Qs + r * LD + m) = v;
    }
  } else {
    // X or D of block row k (all 128 rows exist: there are rows below): four rows of one column per float4
#pragma unroll 4
    for (int idx = tid; idx < 32 * NB / 4; idx += kThreads) {
      const int c = idx & 31, m = (idx >> 5) << 2;
      const float* src = A + (int64_t)(b0 + m) * mt.lda + c0 + c;
      *reinterpret_cast<float4*>(Qs + c * LD + m) =
          make_float4(src[0], src[mt.lda], src[2 * mt.lda], src[3 * mt.lda]);
    }
  }
  __syncthreads();
  const int warp = tid >> 5, lane = tid & 31;
  const int r = (warp & 3) * 8 + (lane >> 3) * 2, c = (warp >> 2) * 16 + (lane & 7);
  const float* row[2] = {Ps + r * LD, Ps + (r + 1) * LD};
  const float* col[2] = {Qs + c * LD, Qs + (c + 8) * LD};
  float old[2][2];
#pragma unroll
  for (int y = 0; y < 2; ++y)
#pragma unroll
    for (int x = 0; x < 2; ++x)
      old[y][x] = (!own && r0 + r + y < n && c0 + c + 8 * x < n) ? A[(int64_t)(r0 + r + y) * mt.lda + c0 + c + 8 * x] : 0.0f;
  uint64_t acc[2][2];
  dots<2, 2>(row, col, NB, acc);
#pragma unroll
  for (int y = 0; y < 2; ++y)
#pragma unroll
    for (int x = 0; x < 2; ++x)
      if (r0 + r + y < n && c0 + c + 8 * x < n)
        A[(int64_t)(r0 + r + y) * mt.lda + c0 + c + 8 * x] = old[y][x] - sum2(acc[y][x]);
}

// ---------------------------------------------------------------------------------------
// Operand forms.  D (the square's inverse, zero above the diagonal) as rows, and D^T as the rows K0.. of the
// update's second operand.
__global__ void __launch_bounds__(256) split_square_kernel(Mat mt, int K0, int n, float* d_hi, float* d_lo,
                                                           float* t_hi, float* t_lo, int64_t t_batch) {
  __shared__ float tile[32][33];
  const float* A = mt.A + blockIdx.y * mt.batch + (int64_t)K0 * mt.lda + K0;
  const int64_t db = (int64_t)blockIdx.y * OB * OB, tb = blockIdx.y * t_batch + (int64_t)K0 * OB;
  const int tr = blockIdx.x >> 4, tc = blockIdx.x & 15, tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int r = tr * 32 + ty + 8 * i, c = tc * 32 + tx;
    const float x = (r < n && c <= r) ? A[(int64_t)r * mt.lda + c] : 0.0f;
    const float h = tgemm::tf32_rn(x);
    d_hi[db + (int64_t)r * OB + c] = h;
    d_lo[db + (int64_t)r * OB + c] = tgemm::tf32_rn(x - h);
    tile[ty + 8 * i][tx] = x;
  }
  if (!t_hi) return;
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int c = tc * 32 + ty + 8 * i, r = tr * 32 + tx;
    const float x = tile[tx][ty + 8 * i];
    const float h = tgemm::tf32_rn(x);
    t_hi[tb + (int64_t)c * OB + r] = h;
    t_lo[tb + (int64_t)c * OB + r] = tgemm::tf32_rn(x - h);
  }
}

// Rows [r0, r1) of the panel A[:, K0 : K0 + n] as they are, and columns [0, tcols) of the block row S[K0 : K0 + n, :]
// transposed; operand row = matrix row or column, zero-padded to 32.
__global__ void __launch_bounds__(256) split_panel_kernel(Mat mt, int K0, int n, int r0, int r1, int tcols, float* hi,
                                                          float* lo, int64_t dst_batch) {
  __shared__ float tile[32][33];
  const float* A = mt.A + blockIdx.y * mt.batch;
  hi += blockIdx.y * dst_batch;
  lo += blockIdx.y * dst_batch;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const int depth = (n + 31) / 32, direct = (r1 - r0 + 31) / 32 * depth, all = direct + tcols / 32 * depth;
  for (int t = blockIdx.x; t < all; t += gridDim.x) {
    const bool rows = t < direct;
    const int u = rows ? t : t - direct, line = u / depth, m0 = (u - line * depth) * 32;
    float x[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int y = ty + 8 * i;
      const int r = rows ? r0 + line * 32 + y : K0 + m0 + y, c = rows ? K0 + m0 + tx : line * 32 + tx;
      const bool in = rows ? (r < r1 && m0 + tx < n) : (m0 + y < n);
      x[i] = in ? A[(int64_t)r * mt.lda + c] : 0.0f;
    }
    if (!rows) {
#pragma unroll
      for (int i = 0; i < 4; ++i) tile[ty + 8 * i][tx] = x[i];
      __syncthreads();
#pragma unroll
      for (int i = 0; i < 4; ++i) x[i] = tile[tx][ty + 8 * i];
      __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int row = (rows ? r0 : 0) + line * 32 + ty + 8 * i;
      if (rows && row >= r1) continue;
      const float h = tgemm::tf32_rn(x[i]);
      hi[(int64_t)row * OB + m0 + tx] = h;
      lo[(int64_t)row * OB + m0 + tx] = tgemm::tf32_rn(x[i] - h);
    }
  }
}

// Index reversal: the lower part of A = J H J in, U = J X J with a zeroed lower part out.  A block takes rows; the
// half that is not needed is neither read nor (on the way in) written.
__global__ void __launch_bounds__(256) reverse_in_kernel(const float* H0, float* const* Hs, int64_t K, int64_t ldh, Mat mt) {
  const float* H = Hs ? Hs[blockIdx.y] : H0;
  float* A = mt.A + blockIdx.y * mt.batch;
  for (int64_t r = blockIdx.x; r < K; r += gridDim.x)
    for (int64_t c = threadIdx.x; c <= r; c += 256) A[r * mt.lda + c] = H[(K - 1 - r) * ldh + (K - 1 - c)];
}
__global__ void __launch_bounds__(256) reverse_out_kernel(float* H0, float* const* Hs, int64_t K, int64_t ldh, Mat mt) {
  float* U = Hs ? Hs[blockIdx.y] : H0;
  const float* A = mt.A + blockIdx.y * mt.batch;
  for (int64_t r = blockIdx.x; r < K; r += gridDim.x)
    for (int64_t c = threadIdx.x; c < K; c += 256)
      U[r * ldh + c] = (c >= r) ? A[(K - 1 - r) * mt.lda + (K - 1 - c)] : 0.0f;
}

static int64_t round_up(int64_t v, int64_t m) { return (v + m - 1) / m * m; }

// floats of workspace per problem: the matrix, the scratch panel of the square, the square's operand form and (for
// more than one outer block) three operand panels with a row per matrix row
static int64_t problem_floats(int64_t K) {
  const int64_t rows = round_up(K, NB);
  return K * round_up(K, 32) + OB * NB + (K > OB ? 2 * OB * OB + 6 * rows * OB : 0);
}

// SMs the bulk of an update leaves to the chain beside it: the square's kernels are small (24 to 120 CTAs of which
// several fit an SM), and while the matrix is narrow the chain is the longer of the two
static int chain_reserve(int64_t K) { return K <= 6144 ? 40 : 20; }

static int factor(float* H, float* const* Hs, int batch, int64_t K, int64_t ldh, float* ws, int* status, bool lookahead,
                  cudaStream_t st) {
  using tgemm::Job;
  using tgemm::Operand;
  int rc;
#define B200Q_RC(expr) do { rc = (expr); if (rc != B200Q_OK) return rc; } while (0)
  const int64_t lda = round_up(K, 32), rows = round_up(K, NB);
  Mat mt;
  mt.A = ws; mt.batch = K * lda; mt.lda = lda; mt.status = status;
  float* P = ws + (int64_t)batch * K * lda;
  float* d_hi = P + (int64_t)batch * OB * NB;
  float* d_lo = d_hi + (int64_t)batch * OB * OB;
  float* a_hi = d_lo + (int64_t)batch * OB * OB;          // panel before its product with D, and S[o,:o]^T
  const int64_t cap = (int64_t)batch * rows * OB, pb = rows * OB;
  float* a_lo = a_hi + cap;
  float* q_base = a_lo + cap;                             // the update's second operand, two copies used in turn
  const size_t chol_smem = kCholSmemFloats * sizeof(float), panel_smem = kPanelSmemFloats * sizeof(float);
  B200Q_TRY(cudaFuncSetAttribute(chol_diag_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)chol_smem));
  B200Q_TRY(cudaFuncSetAttribute(panel_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)panel_smem));
  auto grid = [&](int64_t x, int64_t cap_x) { return dim3((unsigned)(x < cap_x ? x : cap_x), (unsigned)batch, 1); };
  const int64_t row_ctas = batch > 8 ? 2 * kNumSMs / batch + 1 : 8 * kNumSMs;

  reverse_in_kernel<<<grid(K, row_ctas), 256, 0, st>>>(H, Hs, K, ldh, mt);
  B200Q_LAUNCH_CHECK();
  // Look-ahead: the chain (caller's stream) works on the next square while the products of this step that the next
  // square does not need run on a helper stream.  Arithmetic and its order do not depend on it.
  tgemm::SideStream* side = lookahead && K > 2 * OB ? tgemm::side_stream(st) : nullptr;
  cudaStream_t bulk = side ? side->stream : st;
  bool side_busy = false;
  for (int64_t K0 = 0, step = 0; K0 < K; K0 += OB, ++step) {
    const int n = (int)(K - K0 < OB ? K - K0 : OB), blocks = (n + NB - 1) / NB;
    const int64_t K1 = K0 + n;
    const bool last = K1 >= K;
    for (int k = 0; k < blocks; ++k) {
      const int bn = n - k * NB < NB ? n - k * NB : NB, below = n - k * NB - bn;
      chol_diag_kernel<<<batch, kThreads, chol_smem, st>>>(mt, (int)K0 + k * NB, bn);
      B200Q_LAUNCH_CHECK();
      const int vec_ctas = (below + kVec - 1) / kVec + k * NB / kVec;
      if (vec_ctas) {
        panel_kernel<<<dim3(vec_ctas, batch), kThreads, panel_smem, st>>>(mt, P, (int)K0, n, k);
        B200Q_LAUNCH_CHECK();
      }
      if (below > 0) {
        const int rt = (below + 31) / 32, base = (k + 1) * (NB / 32);
        square_update_kernel<<<dim3(rt * base + rt * (rt + 1) / 2, batch), kThreads, kUpdSmemFloats * sizeof(float), st>>>(
            mt, P, (int)K0, n, k);
        B200Q_LAUNCH_CHECK();
      }
    }
    if (K0 == 0 && last) break;
    float* q_hi = q_base + (step & 1) * 2 * cap;
    float* q_lo = q_hi + cap;
    const Operand D{d_hi, d_lo, OB, (int64_t)batch * OB, OB, 0}, Pan{a_hi, a_lo, OB, (int64_t)batch * rows, rows, 0},
        Q{q_hi, q_lo, OB, (int64_t)batch * rows, rows, 0};
    const int n2 = last ? 0 : (int)(K - K1 < OB ? K - K1 : OB);
    if (side_busy) B200Q_TRY(cudaStreamWaitEvent(st, side->done, 0));   // products of the step before
    split_square_kernel<<<dim3(OB / 32 * (OB / 32), batch), 256, 0, st>>>(mt, (int)K0, n, d_hi, d_lo, last ? nullptr : q_hi,
                                                                          q_lo, pb);
    B200Q_LAUNCH_CHECK();
    auto split_panel = [&](int64_t r0, int64_t r1, int64_t tcols, cudaStream_t on) -> int {
      const int64_t tiles = ((r1 - r0 + 31) / 32 + tcols / 32) * ((n + 31) / 32);
      if (tiles == 0) return B200Q_OK;
      split_panel_kernel<<<grid(tiles, row_ctas), 256, 0, on>>>(mt, (int)K0, n, (int)r0, (int)r1, (int)tcols, a_hi, a_lo, pb);
      B200Q_LAUNCH_CHECK();
      return B200Q_OK;
    };
    Job j;
    j.A = Pan; j.B = D; j.Kd = n; j.N = n; j.batch = batch; j.status = status + 2; j.status_stride = 4;
    j.out_ld = OB; j.out_batch = pb;
    if (!last) {
      // the next block's rows of P and its square: all the chain needs
      B200Q_RC(split_panel(K1, K1 + n2, 0, st));
      if (side) {
        B200Q_TRY(cudaEventRecord(side->ready, st));
        B200Q_TRY(cudaStreamWaitEvent(bulk, side->ready, 0));
      }
      Job f = j;
      f.A.row0 = (int)K1; f.M = n2; f.out_hi = q_hi; f.out_lo = q_lo; f.out_row0 = (int)K1;
      B200Q_RC(tgemm::launch(f, st));
      if (side) B200Q_TRY(cudaEventRecord(side->next, st));
      Job d;
      d.A = d.B = Q; d.A.row0 = d.B.row0 = (int)K1; d.M = d.N = n2; d.Kd = n; d.set = tgemm::kLower; d.batch = batch;
      d.alpha = -1.0f; d.beta = 1.0f; d.C = mt.A + K1 * (lda + 1); d.c_batch = mt.batch; d.ldc = lda;
      d.status = status + 2; d.status_stride = 4;
      B200Q_RC(tgemm::launch(d, st));
    } else {
      bulk = st;
    }
    // the other rows of P, and X[o,:o] with its transpose
    B200Q_RC(split_panel(K1 + n2, K, K0, bulk));
    Job r = j;
    r.set = tgemm::kPanel; r.skip0 = (int)K0; r.skip1 = (int)(K1 + n2); r.M = (int)K;
    if (!last) { r.out_hi = q_hi; r.out_lo = q_lo; }
    r.X = mt.A + K0 * lda; r.x_batch = mt.batch; r.ldx = lda; r.xt_rows = (int)K0;
    r.max_ctas = side && !last ? kNumSMs - chain_reserve(K) : 0;
    B200Q_RC(tgemm::launch(r, bulk));
    if (last) break;
    if (side) B200Q_TRY(cudaStreamWaitEvent(bulk, side->next, 0));
    // S[below,o] = -P D, S[i,:o] -= P_i X[o,:o], A[i,j] -= P_i P_j^T, without the next square
    Job u;
    u.A = Q; u.B = Q; u.A.row0 = 0; u.M = u.N = (int)K; u.Kd = n; u.set = tgemm::kBulk; u.batch = batch;
    u.row_begin = (int)K1; u.skip0 = (int)K1; u.skip1 = (int)(K1 + n2);
    u.alpha = -1.0f; u.beta = 1.0f; u.C = mt.A; u.c_batch = mt.batch; u.ldc = lda; u.fresh0 = (int)K0; u.fresh1 = (int)K1;
    u.status = status + 2; u.status_stride = 4; u.max_ctas = r.max_ctas;
    B200Q_RC(tgemm::launch(u, bulk));
    if (side) {
      B200Q_TRY(cudaEventRecord(side->done, bulk));
      side_busy = true;
    }
  }
#undef B200Q_RC
  reverse_out_kernel<<<grid(K, row_ctas), 256, 0, st>>>(H, Hs, K, ldh, mt);
  B200Q_LAUNCH_CHECK();
  return B200Q_OK;
}

}  // namespace factor
}  // namespace b200q

using namespace b200q;

extern "C" {

size_t b200q_gptq_factor_workspace_bytes(int64_t K) {
  return K <= 0 ? 0 : (size_t)factor::problem_floats(K) * sizeof(float);
}

int b200q_gptq_factor(float* H, int64_t K, int64_t ldh, void* workspace, int* status, void* stream) {
  if (!H || !workspace || !status || K <= 0 || ldh < K || K > (1 << 24)) return B200Q_ERR_ARG;
  return factor::factor(H, nullptr, 1, K, ldh, (float*)workspace, status, true, (cudaStream_t)stream);
}

size_t b200q_gptq_factor_batched_workspace_bytes(int64_t K, int count) {
  if (K <= 0 || count <= 0) return 0;
  return (size_t)K * (size_t)K * sizeof(float) * (size_t)count;
}

size_t b200q_gptq_factor_many_workspace_bytes(int64_t K, int count) {
  return K <= 0 || count <= 0 ? 0 : (size_t)factor::problem_floats(K) * sizeof(float) * (size_t)count;
}

int b200q_gptq_factor_many(float* const* H, int count, int64_t K, int64_t ldh, void* workspace, int* status, void* stream) {
  if (!H || !workspace || !status || count <= 0 || count > 65535 || K <= 0 || ldh < K) return B200Q_ERR_ARG;
  if (K > 4096) return B200Q_ERR_UNSUPPORTED;
  cudaStream_t st = (cudaStream_t)stream;
  B200Q_TRY(cudaMemsetAsync(status, 0, sizeof(int) * 4 * (size_t)count, st));
  return factor::factor(nullptr, H, count, K, ldh, (float*)workspace, status, false, st);
}

int b200q_gptq_factor_batched(float* const* H, float* const* scratch, int count, int64_t K, int64_t ldh, int* status,
                              void* stream) {
  if (!H || !scratch || !status || count <= 0 || K <= 0 || ldh < K) return B200Q_ERR_ARG;
  if (K > 4096) return B200Q_ERR_UNSUPPORTED;
  // the scratch this entry point is given (K * K floats a problem) is smaller than the workspace in use now
  void* ws = nullptr;
  cudaStream_t st = (cudaStream_t)stream;
  B200Q_TRY(cudaMallocAsync(&ws, b200q_gptq_factor_many_workspace_bytes(K, count), st));
  const int rc = b200q_gptq_factor_many(H, count, K, ldh, ws, status, stream);
  B200Q_TRY(cudaFreeAsync(ws, st));
  return rc;
}

}  // extern "C"
