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
// The last three are one launch on halves with a scale per row: the rows of its second operand are X[o,:o]^T, D^T and P,
// indexed by absolute column.
//
// The blocked form is what the sweep of a single weight needs and half of the work: the squares of U on the diagonal, and
// beside them S as step o leaves it, -V[:o,o] U_oo, which no later step touches.  Then neither X[o,:o] nor S[i,:o] -= P_i X
// is computed, 1/3 K^3 instead of 2/3 K^3 (gptq_sweep.cu: products across superblocks take w - q in place of the errors).
// Its squares are the superblocks of the sweep, so the short one comes first, and the matrix begins with as many rows of the
// identity as make its order a multiple of 32.  K = 14336: 6.2 ms (U: 9.7), 4096: 1.04 (1.10), 2048: 0.50 (0.53),
// 1160: 0.31 (0.34).
//
// A pivot <= 0 (or NaN) sets the problem's status; the host then takes the reference's identity fallback.
#include <type_traits>

#include "common.cuh"
#include "tgemm_tf32.cuh"

namespace b200q {
namespace factor {

constexpr int NB = 128;          // inner block
constexpr int OB = 512;          // outer block
constexpr int kThreads = 256;
constexpr int LD = NB + 4;       // shared-memory stride: 16-byte rows, float4 accesses of 8 consecutive rows conflict-free

constexpr int64_t kScratchFloats = 2LL * OB * NB;   // of the square: P [512][128] and X [128][512]

struct Mat {                     // the batch's work matrices and status words
  float* A; int64_t batch, lda;
  int* status;
  int pad;                       // rows of the identity before the matrix
};

__device__ __forceinline__ void cp_async16(float* dst, const float* src, int src_bytes) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(src_bytes) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Products inside the square: warp-level 16 x 8 x 8 tf32 MMAs on operands in shared memory, three per product of
// hi / lo splits as in tgemm.  Tiles of 16 are too small for tcgen05 (its operands would have to be rewritten in
// swizzled form between two steps of the chain); measured here, these MMAs retire 512 multiply-adds a cycle and SM,
// 170 of float32 accuracy, and need a sixth of the shared-memory loads of a register-tiled FFMA2 product.
__device__ __forceinline__ uint32_t tf32_bits(float x) { return (__float_as_uint(x) + 0x1000u) & 0xFFFFE000u; }
template <int N>
__device__ __forceinline__ void split_frag(const float (&x)[N], uint32_t (&hi)[N], uint32_t (&lo)[N]) {
#pragma unroll
  for (int i = 0; i < N; ++i) {
    hi[i] = tf32_bits(x[i]);
    lo[i] = tf32_bits(x[i] - __uint_as_float(hi[i]));
  }
}
__device__ __forceinline__ void mma_tf32(float (&c)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
  asm(
      "mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}
// acc[j] = A[16 x depth] B_j[8 x depth]^T, B_j = rows 8 j .. 8 j + 7 of B.  Lane (g, t) = (lane / 4, lane % 4) ends
// with rows g, g + 8 and columns 2 t, 2 t + 1.  A: contraction contiguous, row stride lda; B: element (n, k) at
// n * sn + k * sk.
// An MMA's addition to its accumulator cuts off instead of rounding, so the large products run over 16 terms at most and
// the runs are added by float32 additions (all 128 in one accumulator: relative error of the factor 3.5e-7 at K = 256
// and 4.4e-7 at 512 against 1.9e-7 and 2.1e-7).
template <int NT, int UNROLL>
__device__ __forceinline__ void mma_block(const float* A, int lda, const float* B, int sn, int sk, int depth, int lane,
                                          float (&acc)[NT][4]) {
  const float* a0 = A + (lane >> 2) * lda + (lane & 3);
  const float* b0 = B + (lane >> 2) * sn + (lane & 3) * sk;
  // the three products accumulate apart: a warp issues in order, and an MMA whose accumulator the one before it
  // still has stalls everything behind it for some 35 cycles
  float part[2][NT][4] = {}, run[NT][4] = {}, sum[NT][4] = {};
#pragma unroll UNROLL
  for (int k = 0; k < depth; k += 8) {
    const float x[4] = {a0[k], a0[k + 8 * lda], a0[k + 4], a0[k + 8 * lda + 4]};
    float y[NT][2];
#pragma unroll
    for (int j = 0; j < NT; ++j) { y[j][0] = b0[j * 8 * sn + k * sk]; y[j][1] = b0[j * 8 * sn + (k + 4) * sk]; }
    uint32_t ah[4], al[4], bh[NT][2], bl[NT][2];
    split_frag(x, ah, al);
#pragma unroll
    for (int j = 0; j < NT; ++j) split_frag(y[j], bh[j], bl[j]);
#pragma unroll
    for (int j = 0; j < NT; ++j) mma_tf32(run[j], ah, bh[j]);
#pragma unroll
    for (int j = 0; j < NT; ++j) mma_tf32(part[0][j], ah, bl[j]);
#pragma unroll
    for (int j = 0; j < NT; ++j) mma_tf32(part[1][j], al, bh[j]);
    if (depth > 16 && (k & 8)) {
#pragma unroll
      for (int j = 0; j < NT; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) { sum[j][e] += run[j][e]; run[j][e] = 0.0f; }
    }
  }
#pragma unroll
  for (int j = 0; j < NT; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      acc[j][e] = run[j][e] + (part[0][j][e] + part[1][j][e]);
      if (depth > 16) acc[j][e] += sum[j][e];
    }
}

// ---------------------------------------------------------------------------------------
// Diagonal block: L^-1 of the n x n (n <= 128) block at (k0, k0), over the block itself.
//
// One CTA on the critical path, so the design is about latency.  The identity is appended below the block, which
// turns the triangular inverse into more rows of the same elimination (a row e_i ends as row i of L^-T): at every
// 16-column step exactly eight 16-row blocks take part.  A step:
//   warp 0 brings the 16 x 16 diagonal block up to date and factors it in registers, a lane per row: the next pivot
//          is formed by its own lane and broadcast before the other columns are updated, no branches.  Meanwhile the
//          others apply the step before to everything else.
//   four warps substitute the 128 active rows, a row a lane
//
// Sixteen warps.  The elimination and what follows it in the same step are the chain; the update of the step before has to
// be through in that time, and warps on the eliminating warp's scheduler slow it down, so the twelve on the other three
// take it.  Cycles, clocks read in the kernel: 2700 until the block is there, steps of 2600 to 3200 (the diagonal block's
// update 330, its elimination 1270 to 1500, substitution and operands 800; in the longer steps 400 until the others are
// through), 1900 out; 28700 in all, 32200 with eight warps and tf32 pairs.
constexpr int W16 = 16;
constexpr int kCholThreads = 512;
// A step's 128 active rows as operands: 16 hi and 16 lo halves and a power of two per row (tgemm::Operand), in rows of 80 bytes,
// which ldmatrix reads without bank conflicts.  The rows are written once and read by up to ten products: split by every
// reader into tf32 pairs, the update of a step took 3300 cycles, longer than the chain beside it.
constexpr int kOpBytes = 80;
constexpr int CLD = NB + 8;   // stride of the diagonal block's rows: a tile's pairs of columns conflict-free
constexpr int kCholSmemFloats = 2 * NB * CLD + W16 * 20 + W16 + NB * kOpBytes / 4 + NB;

__device__ __forceinline__ void ldmatrix4(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void mma_f16(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// o[16 x 8 NT] -= A B^T over 16 terms, A the operand rows from ra on, B those from rb on; column tiles from `tiles` on are left
// out.  Lane (g, t) has rows g, g + 8 and columns 2 t, 2 t + 1 of every tile; o points at its first.
template <int NT>
__device__ __forceinline__ void subtract_product(float* o, uint32_t op, const float* scale, int ra, int rb, int tiles, int lane) {
  float2 old[NT][2];   // (all of them before the products: loads cannot pass the stores below)
#pragma unroll
  for (int j = 0; j < NT; ++j)
#pragma unroll
    for (int h = 0; h < 2; ++h)
      if (j < tiles) old[j][h] = *reinterpret_cast<float2*>(o + h * 8 * CLD + 8 * j);
  uint32_t ah[4], al[4], bh[NT / 2][4], bl[NT / 2][4];
  const uint32_t a = op + (ra + (lane & 15)) * kOpBytes + (lane >> 4) * 16;
  const uint32_t b = op + (rb + (lane & 7) + (lane >> 4) * 8) * kOpBytes + ((lane >> 3) & 1) * 16;
  ldmatrix4(a, ah);
  ldmatrix4(a + 32, al);
#pragma unroll
  for (int j = 0; j < NT / 2; ++j) {
    if (2 * j >= tiles) break;
    ldmatrix4(b + j * 16 * kOpBytes, bh[j]);
    ldmatrix4(b + j * 16 * kOpBytes + 32, bl[j]);
  }
  const float s0 = scale[ra + (lane >> 2)], s1 = scale[ra + (lane >> 2) + 8];
#pragma unroll
  for (int j = 0; j < NT; ++j) {
    if (j >= tiles) break;
    float x[4] = {0.f, 0.f, 0.f, 0.f}, y[4] = {0.f, 0.f, 0.f, 0.f};
    const int e = 2 * (j & 1);
    mma_f16(y, ah, bl[j / 2][e], bl[j / 2][e + 1]);
    mma_f16(x, ah, bh[j / 2][e], bh[j / 2][e + 1]);
    mma_f16(y, al, bh[j / 2][e], bh[j / 2][e + 1]);
    const float2 sc = *reinterpret_cast<const float2*>(scale + rb + 8 * j + 2 * (lane & 3));
    *reinterpret_cast<float2*>(o + 8 * j) = make_float2(fmaf(-(x[0] + y[0]) * s0, sc.x, old[j][0].x), fmaf(-(x[1] + y[1]) * s0, sc.y, old[j][0].y));
    *reinterpret_cast<float2*>(o + 8 * CLD + 8 * j) = make_float2(fmaf(-(x[2] + y[2]) * s1, sc.x, old[j][1].x), fmaf(-(x[3] + y[3]) * s1, sc.y, old[j][1].y));
  }
}

// active row block s (0..7) of step kb: identity rows up to kb, whose inverse is being born, matrix rows after it
__device__ __forceinline__ float* active_row(float* R, int ar, int kb) {
  return R + ((ar >> 4) <= kb ? NB + ar : ar) * CLD;
}

__global__ void __launch_bounds__(kCholThreads, 1) chol_diag_kernel(Mat mt, int k0, int n) {
  extern __shared__ __align__(16) float sm[];
  float* R = sm;                    // rows 0..127: the block, then L; rows 128..255: the identity, then L^-T
  float* Lt = R + 2 * NB * CLD;      // [16][20] transposed diagonal block of the step
  float* rinv = Lt + W16 * 20;      // [16]
  float* scale = rinv + W16;        // [128] inverse powers of the operand rows
  unsigned char* rows_op = reinterpret_cast<unsigned char*>(scale + NB);
  const uint32_t op = (uint32_t)__cvta_generic_to_shared(rows_op);
  float* A = mt.A + blockIdx.x * mt.batch + (int64_t)k0 * mt.lda + k0;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  // (nothing reads what is above the diagonal of a matrix row or left of an identity row's block)
  for (int idx = tid; idx < NB * NB / 4; idx += kCholThreads) {
    const int r = idx >> 5, c = (idx & 31) << 2;
    const float4 id = make_float4(c == r ? 1.f : 0.f, c + 1 == r ? 1.f : 0.f, c + 2 == r ? 1.f : 0.f, c + 3 == r ? 1.f : 0.f);
    if (c <= r && r >= n) *reinterpret_cast<float4*>(R + r * CLD + c) = id;   // identity padding beyond n
    if (c >= (r & ~(W16 - 1))) *reinterpret_cast<float4*>(R + (NB + r) * CLD + c) = id;
  }
  chain_wait();
#pragma unroll
  for (int i = 0; i < NB * NB / 4 / kCholThreads; ++i) {
    const int idx = tid + i * kCholThreads, r = idx >> 5, c = (idx & 31) << 2;
    if (c <= r && r < n) cp_async16(R + r * CLD + c, A + (int64_t)r * mt.lda + c, 16);   // (rows are padded to 32)
  }
  cp_async_wait_all();
  __syncthreads();
  int bad = 0;   // first pivot that is not positive, + 1
#pragma unroll 1
  for (int kb = 0; kb < 8; ++kb) {
    const int c0 = kb * W16, p0 = c0 - W16;
    if (warp == 0) {
      if (kb > 0) {   // the diagonal block takes the step before
        subtract_product<2>(R + (c0 + (lane >> 2)) * CLD + c0 + 2 * (lane & 3), op, scale, c0, c0, 2, lane);
        __syncwarp();
      }
      float a[W16], ri;
      const float* src = R + (c0 + (lane & 15)) * CLD + c0;
      // the first pivot that `Exact` does not accept, + 1: the quick form takes positive normal numbers, the exact one
      // (rare, so out of the way) everything above zero.  Garbage from that pivot on.
      auto eliminate = [&](auto Exact) -> int {
        int first = 0;
        ri = 0.0f;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const float4 v = *reinterpret_cast<const float4*>(src + 4 * q);
          a[4 * q] = v.x; a[4 * q + 1] = v.y; a[4 * q + 2] = v.z; a[4 * q + 3] = v.w;
        }
        // Column j reaches column j + 1 by one shuffle, and the pivot there, t - x^2, is formed by every lane for itself; the
        // columns behind take it from shared memory a column later, four a load.  (A shuffle for each of them: they and the
        // other warps' loads share a pipe, 1300 to 2100 cycles
        // for the 16 columns; now 1270 to 1500.)
        float t = __shfl_sync(0xffffffffu, a[0], 0), l = 0.0f;
#pragma unroll
        for (int j = 0; j < W16; ++j) {
          const float x = j ? __shfl_sync(0xffffffffu, l, j) : 0.0f;
          const float piv = fmaf(-x, x, t);
          a[j] = fmaf(-l, x, a[j]);
          float root;   // 1 / sqrt(piv)
          if constexpr (Exact) {
            first = (!(piv > 0.0f) && first == 0) ? j + 1 : first;
            root = __fdiv_rn(1.0f, __fsqrt_rn(piv));
            l = a[j] * root;
          } else {
            first = (!(piv >= 1.17549435e-38f) && first == 0) ? j + 1 : first;
            float r;
            asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(piv));
            // one Newton step r (1.5 - piv r^2 / 2), within an ulp of 1 / sqrt, folded into the column's scaling
            const float u = fmaf(-(0.5f * piv) * r, r, 1.5f);
            l = (a[j] * r) * u;
            root = r * u;
          }
          a[j] = l;
          ri = (lane == j) ? root : ri;
          if (j + 2 < W16) {
            Lt[j * 20 + (lane & 15)] = l;
            __syncwarp();
#pragma unroll
            for (int q = (j + 2) / 4; q < 4; ++q) {
              const float4 v = *reinterpret_cast<const float4*>(Lt + j * 20 + 4 * q);
              const float e[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
              for (int k = 0; k < 4; ++k)
                if (4 * q + k >= j + 2) a[4 * q + k] = fmaf(-l, e[k], a[4 * q + k]);
            }
          }
          // (of the next column's own row, without this column yet)
          if (j + 1 < W16) t = __shfl_sync(0xffffffffu, a[j + 1], j + 1);
        }
        return first;
      };
      if (eliminate(std::false_type())) {
        const int first = eliminate(std::true_type());
        bad = (first && bad == 0) ? c0 + first : bad;
      }
      if (lane < W16) {
#pragma unroll
        for (int j = 0; j < W16; ++j) Lt[j * 20 + lane] = (j <= lane) ? a[j] : 0.0f;
        rinv[lane] = ri;
      }
    } else if (kb > 0 && (warp & 3)) {
      // everything else takes the step before: the eight row blocks that were active then x the columns from c0 on,
      // on and below the diagonal.  A warp takes 16 rows x 32 columns at a time.
      // Task list: kb identity row blocks with `wide` pairs of column blocks each, then matrix row blocks r = 0, 1, ...
      // (s = kb + r) with r / 2 + 1 pairs.  (Counted out in closed form: a loop over all tasks that skips the other
      // warps' costs 180 cycles a skip, mostly instruction fetch.  From a table the first task of a step begins 300 cycles
      // sooner and takes 460 longer: what the tasks wait for is one another's loads, stores and products.)
      const int wide = (9 - kb) / 2, left = kb * wide, half = (8 - kb) / 2;
      const int all = left + half * (half + 1) + (kb & 1) * (half + 1);
      for (int t = (warp >> 2) * 3 + (warp & 3) - 1; t < all; t += 12) {
        int s, g;
        if (t < left) {
          s = t / wide; g = t - s * wide;
        } else {
          const int u = t - left, q = (u >= 2) + (u >= 6) + (u >= 12);
          g = u - q * (q + 1); s = kb + 2 * q;
          if (g > q) { g -= q + 1; ++s; }
        }
        const bool matrix = s >= kb;
        const int cc = c0 + g * 32, last = matrix ? s * W16 : NB - W16;   // first column of the last block of 16 to take
        // (the diagonal block itself is the first warp's)
        const int tiles = matrix && s == kb ? 0 : min(4, (last + W16 - cc) / 8);
        subtract_product<4>(R + ((matrix ? 0 : NB) + s * W16 + (lane >> 2)) * CLD + cc + 2 * (lane & 3), op, scale, s * W16, cc,
                            tiles, lane);
      }
    }
    __syncthreads();
    if (warp < 4) {
      float a[W16];
      const int ar = warp * 32 + lane;
      float* row = active_row(R, ar, kb) + c0;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const float4 v = *reinterpret_cast<const float4*>(row + 4 * q);
        a[4 * q] = v.x; a[4 * q + 1] = v.y; a[4 * q + 2] = v.z; a[4 * q + 3] = v.w;
      }
#pragma unroll
      for (int j = 0; j < W16; ++j) {
        const float y = a[j] * rinv[j];
        a[j] = y;
#pragma unroll
        for (int q = (j + 1) / 4; q < 4; ++q) {
          const float4 l4 = *reinterpret_cast<const float4*>(Lt + j * 20 + 4 * q);
          const float l[4] = {l4.x, l4.y, l4.z, l4.w};
#pragma unroll
          for (int k = 0; k < 4; ++k)
            if (4 * q + k > j) a[4 * q + k] = fmaf(-y, l[k], a[4 * q + k]);
        }
      }
      float largest[4] = {0.f, 0.f, 0.f, 0.f}, to, back;
#pragma unroll
      for (int j = 0; j < W16; ++j) largest[j & 3] = fmaxf(largest[j & 3], fabsf(a[j]));
      tgemm::row_scale(fmaxf(fmaxf(largest[0], largest[1]), fmaxf(largest[2], largest[3])), to, back);
      scale[ar] = back;
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        uint32_t hi[4], lo[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) tgemm::split_pair(a[8 * q + 2 * k] * to, a[8 * q + 2 * k + 1] * to, hi[k], lo[k]);
        *reinterpret_cast<uint4*>(rows_op + ar * kOpBytes + q * 16) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
        *reinterpret_cast<uint4*>(rows_op + ar * kOpBytes + 32 + q * 16) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
      }
#pragma unroll
      for (int q = 0; q < 4; ++q)   // (of the matrix rows nothing reads these any more)
        if ((ar >> 4) <= kb) *reinterpret_cast<float4*>(row + 4 * q) = make_float4(a[4 * q], a[4 * q + 1], a[4 * q + 2], a[4 * q + 3]);
    }
    __syncthreads();
  }
  chain_go();
  if (tid == 0 && bad) {
    int* status = mt.status + 4 * blockIdx.x;
    if (atomicCAS(status, 0, B200Q_NOT_POSITIVE_DEFINITE) == 0) status[1] = k0 + bad - mt.pad;
  }
  // D[j][i] = (L^-T)[i][j] in the 16 x 16 blocks on and below the diagonal, zero above it (whoever reads beyond these blocks
  // takes zeros by himself); a thread turns 4 x 4 entries round
#pragma unroll
  for (int it = 0; it < NB * NB / 16 / kCholThreads; ++it) {
    const int u = it * 16 + warp, i = (lane & 1) * 4 + (u & 15) * 8, j = (lane >> 1) * 4 + (u >> 4) * 64;
    if (i / W16 > j / W16) continue;
    float v[4][4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const float4 q = *reinterpret_cast<const float4*>(R + (NB + i + k) * CLD + j);
      v[k][0] = q.x; v[k][1] = q.y; v[k][2] = q.z; v[k][3] = q.w;
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      if (j + k >= n) continue;
      float* o = A + (int64_t)(j + k) * mt.lda + i;
#pragma unroll
      for (int e = 0; e < 4; ++e)
        if (i + e > j + k) v[e][k] = 0.0f;
      if (i + 3 < n) *reinterpret_cast<float4*>(o) = make_float4(v[0][k], v[1][k], v[2][k], v[3][k]);
      else
        for (int e = 0; e < 4; ++e)
          if (i + e < n) o[e] = v[e][k];
    }
  }
}

// ---------------------------------------------------------------------------------------
// Inside the square at K0 (n columns), step k: everything the diagonal block's inverse D multiplies.  Two CTAs own 16
// "vectors" of 128, each 64 of their outputs: rows r below the block (P[r] = A[r, blk] D^T, into the scratch P), then
// columns c left of it (X[blk, c] = D S[blk, c], into the scratch X; the update kernel puts them in their place).  D is
// triangular, so output j needs only the first j + 1 terms.  The time is that of fetching D from L2.
constexpr int kVec = 16;
constexpr int kPanelSmemFloats = (NB / 2 + kVec) * LD;

__global__ void __launch_bounds__(kThreads) panel_kernel(Mat mt, float* P0, int K0, int n, int k) {
  chain_wait();
  extern __shared__ __align__(16) float sm[];
  float* D = sm;                   // [64][LD] rows of D
  float* V = D + NB / 2 * LD;      // [16][LD] the vectors, contraction contiguous
  const float* A = mt.A + blockIdx.y * mt.batch + (int64_t)K0 * mt.lda + K0;
  float* P = P0 + (int64_t)blockIdx.y * kScratchFloats;
  const int tid = threadIdx.x, b0 = k * NB, bn = n - b0 < NB ? n - b0 : NB, below = n - b0 - bn;
  const int below_ctas = (below + kVec - 1) / kVec, unit = blockIdx.x >> 1, half = (blockIdx.x & 1) * 64;
  const bool rows = unit < below_ctas;
  const int v0 = rows ? b0 + bn + unit * kVec : (unit - below_ctas) * kVec;
  const int depth = half + 64;
  if (half >= bn) return;
  for (int idx = tid; idx < 64 * (depth / 4); idx += kThreads) {
    const int r = idx / (depth / 4), c = (idx - r * (depth / 4)) * 4, j = half + r;
    const int left = (j < bn && c < bn) ? bn - c : 0;
    cp_async16(D + r * LD + c, left ? A + (int64_t)(b0 + j) * mt.lda + b0 + c : A, left >= 4 ? 16 : left * 4);
  }
  if (rows) {
    for (int idx = tid; idx < kVec * (depth / 4); idx += kThreads) {
      const int v = idx / (depth / 4), c = (idx - v * (depth / 4)) * 4;
      const int left = (v0 + v < n && c < bn) ? bn - c : 0;
      cp_async16(V + v * LD + c, left ? A + (int64_t)(v0 + v) * mt.lda + b0 + c : A, left >= 4 ? 16 : left * 4);
    }
  } else {
    float x[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int idx = tid + i * kThreads, v = idx & 15, m = idx >> 4;
      x[i] = (m < bn && m < depth) ? A[(int64_t)(b0 + m) * mt.lda + v0 + v] : 0.0f;
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int idx = tid + i * kThreads;
      V[(idx & 15) * LD + (idx >> 4)] = x[i];
    }
  }
  chain_go();
  cp_async_wait_all();
  __syncthreads();
  // a warp: 16 vectors x 8 outputs
  const int warp = tid >> 5, lane = tid & 31, j0 = warp * 8;
  float acc[1][4];
  mma_block<1, 4>(V, LD, D + j0 * LD, LD, 1, half + j0 + 8, lane, acc);
  const int v = v0 + (lane >> 2), j = half + j0 + 2 * (lane & 3);
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const int vv = v + (e >> 1) * 8, jj = j + (e & 1);
    if (jj >= bn) continue;
    if (rows) { if (vv < n) P[(int64_t)vv * NB + jj] = acc[0][e]; }
    else P[(int64_t)OB * NB + (int64_t)jj * OB + vv] = acc[0][e];
  }
}

// Inside the square, step k: rows below the block take -P times X (columns left), D (the block's own columns, which
// start from zero) and P^T (columns right, on and below the diagonal); the block row itself takes X.  A CTA owns a
// 32 x 32 tile, a warp 16 x 8 of it.
constexpr int kUpdSmemFloats = 32 * LD + NB * 40;

__global__ void __launch_bounds__(kThreads) square_update_kernel(Mat mt, const float* P0, int K0, int n, int k, int tiles) {
  chain_wait();
  extern __shared__ __align__(16) float sm[];
  float* Ps = sm;                // [32][LD]
  float* Qs = Ps + 32 * LD;      // second operand: [32][LD] contraction contiguous, or [128][40] column contiguous
  float* A = mt.A + blockIdx.y * mt.batch + (int64_t)K0 * mt.lda + K0;
  const float* P = P0 + (int64_t)blockIdx.y * kScratchFloats;
  const float* X = P + (int64_t)OB * NB;
  const int tid = threadIdx.x, b0 = k * NB, r_begin = b0 + NB;
  if ((int)blockIdx.x >= tiles) {   // 32 x 32 of X into its place
    const int u = blockIdx.x - tiles, y0 = (u & 3) * 32, x0 = (u >> 2) * 32, y = y0 + (tid >> 3), x = x0 + (tid & 7) * 4;
    if (b0 + y < n)
      *reinterpret_cast<float4*>(A + (int64_t)(b0 + y) * mt.lda + x) = *reinterpret_cast<const float4*>(X + (int64_t)y * OB + x);
    return;
  }
  // tile list: row tile i (32 rows from r_begin on) has r_begin / 32 + i + 1 column tiles
  const int base = r_begin / 32;
  int i = 0, t = blockIdx.x;
  while (t >= base + i + 1) { t -= base + i + 1; ++i; }
  const int r0 = r_begin + i * 32, c0 = t * 32;
  const bool right = c0 >= r_begin, own = !right && c0 >= b0;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int idx = tid + q * kThreads, r = idx >> 5, m = (idx & 31) << 2;
    cp_async16(Ps + r * LD + m, P + (int64_t)(r0 + r < n ? r0 + r : 0) * NB + m, r0 + r < n ? 16 : 0);
  }
  if (right) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int idx = tid + q * kThreads, r = idx >> 5, m = (idx & 31) << 2;
      cp_async16(Qs + r * LD + m, P + (int64_t)(c0 + r < n ? c0 + r : 0) * NB + m, c0 + r < n ? 16 : 0);
    }
  } else {
    // D or X of block row k, which has all its 128 rows: there are rows below
    const float* src = own ? A + (int64_t)b0 * mt.lda + c0 : X + c0;
    const int64_t ld = own ? mt.lda : OB;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int idx = tid + q * kThreads, m = idx >> 3, c = (idx & 7) << 2;
      const bool zero = own && c0 - b0 + c > m;   // above D's diagonal
      cp_async16(Qs + m * 40 + c, zero ? A : src + (int64_t)m * ld + c, zero ? 0 : 16);
    }
  }
  const int warp = tid >> 5, lane = tid & 31, tr = (warp & 1) * 16, tc = (warp >> 1) * 8;
  const int r = r0 + tr + (lane >> 2), c = c0 + tc + 2 * (lane & 3);
  float old[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const int rr = r + (e >> 1) * 8, cc = c + (e & 1);
    old[e] = (!own && rr < n && cc < n) ? A[(int64_t)rr * mt.lda + cc] : 0.0f;
  }
  chain_go();
  cp_async_wait_all();
  __syncthreads();
  float acc[1][4];
  if (right) mma_block<1, 4>(Ps + tr * LD, LD, Qs + tc * LD, LD, 1, NB, lane, acc);
  else mma_block<1, 4>(Ps + tr * LD, LD, Qs + tc, 1, 40, NB, lane, acc);
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const int rr = r + (e >> 1) * 8, cc = c + (e & 1);
    if (rr < n && cc < n) A[(int64_t)rr * mt.lda + cc] = old[e] - acc[0][e];
  }
}

// ---------------------------------------------------------------------------------------
// Rows [r0, r1) of the panel A[:, K0 : K0 + n] as they are, and columns [0, tcols) of the block row S[K0 : K0 + n, :]
// transposed; operand row = matrix row or column, zero-padded to 32.  The first `squares` CTAs, if any, make the operand form
// of D (the square's inverse, zero above the diagonal) as rows instead: what the chain needs before the next block's rows of P,
// in one launch.
constexpr int kSquareCtas = OB / 32 * (OB / 32);
struct SquareForm { float *hi, *lo; int ctas; };
__global__ void __launch_bounds__(256) split_panel_kernel(Mat mt, int K0, int n, int r0, int r1, int tcols, float* hi,
                                                          float* lo, int64_t dst_batch, const SquareForm square) {
  chain_wait();
  chain_go();
  __shared__ float tile[32][33];
  const float* A = mt.A + blockIdx.y * mt.batch;
  if ((int)blockIdx.x < square.ctas) {
    const float* S = A + (int64_t)K0 * mt.lda + K0;
    const int64_t db = (int64_t)blockIdx.y * OB * OB;
    const int tr = blockIdx.x >> 4, tc = blockIdx.x & 15, tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int r = tr * 32 + ty + 8 * i, c = tc * 32 + tx;
      const float x = (r < n && c <= r) ? S[(int64_t)r * mt.lda + c] : 0.0f;
      const float h = tgemm::tf32_rn(x);
      square.hi[db + (int64_t)r * OB + c] = h;
      square.lo[db + (int64_t)r * OB + c] = tgemm::tf32_rn(x - h);
    }
    return;
  }
  hi += blockIdx.y * dst_batch;
  lo += blockIdx.y * dst_batch;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const int depth = (n + 31) / 32, direct = (r1 - r0 + 31) / 32 * depth, all = direct + tcols / 32 * depth;
  for (int t = blockIdx.x - square.ctas; t < all; t += gridDim.x - square.ctas) {
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
// half that is not needed is neither read nor (on the way in) written, but for the rest of a diagonal's four.  Bound by HBM.
// Four columns a thread and step where both sides are aligned (a row's four in reverse order), four steps at a time:
// 14336 columns in 139 us (225 a column a thread and step), out 196 (280), of the blocked form 136.
__device__ __forceinline__ float4 reversed(float4 v) { return make_float4(v.w, v.z, v.y, v.x); }
__device__ __forceinline__ bool quads_ok(const void* p, int64_t ld, int64_t end) {
  return ((uintptr_t)p & 15) == 0 && (ld & 3) == 0 && (end & 3) == 0;
}
__global__ void __launch_bounds__(256) reverse_in_kernel(const float* H0, float* const* Hs, int64_t K, int64_t ldh, Mat mt) {
  const float* H = Hs ? Hs[blockIdx.y] : H0;
  float* A = mt.A + blockIdx.y * mt.batch;
  const int64_t end = K + mt.pad;
  const bool quads = quads_ok(H, ldh, end);
  for (int64_t r = blockIdx.x; r < end; r += gridDim.x) {
    auto value = [&](int64_t c) { return c < mt.pad ? (c == r ? 1.0f : 0.0f) : H[(end - 1 - r) * ldh + (end - 1 - c)]; };
    if (quads && r >= mt.pad) {
      const int64_t first = (mt.pad + 3) & ~3;
      for (int64_t c = first + threadIdx.x * 4; c <= r; c += 4096) {
        float4 v[4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
          if (c + i * 1024 <= r) v[i] = *reinterpret_cast<const float4*>(H + (end - 1 - r) * ldh + (end - 4 - c - i * 1024));
#pragma unroll
        for (int i = 0; i < 4; ++i)
          if (c + i * 1024 <= r) *reinterpret_cast<float4*>(A + r * mt.lda + c + i * 1024) = reversed(v[i]);
      }
      for (int64_t c = threadIdx.x; c < first && c <= r; c += 256) A[r * mt.lda + c] = value(c);
      continue;
    }
    for (int64_t c = threadIdx.x; c <= r; c += 256) A[r * mt.lda + c] = value(c);
  }
}
// (`zeros`: the lower part of U; nothing reads it of the blocked form)
__global__ void __launch_bounds__(256) reverse_out_kernel(float* H0, float* const* Hs, int64_t K, int64_t ldh, Mat mt, bool zeros) {
  float* U = Hs ? Hs[blockIdx.y] : H0;
  const float* A = mt.A + blockIdx.y * mt.batch;
  const int64_t end = K + mt.pad;
  const bool quads = quads_ok(U, ldh, end) && (K & 3) == 0;
  for (int64_t r = blockIdx.x; r < K; r += gridDim.x) {
    const float* row = A + (end - 1 - r) * mt.lda;
    if (quads) {
      for (int64_t c = (zeros ? 0 : r & ~3LL) + threadIdx.x * 4; c < K; c += 4096) {
        float4 v[4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
          if (c + i * 1024 < K && c + i * 1024 + 3 >= r) v[i] = reversed(*reinterpret_cast<const float4*>(row + (end - 4 - c - i * 1024)));
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int64_t d = c + i * 1024 - r;   // of the first of the four from the diagonal
          if (c + i * 1024 >= K) break;
          if (d < -3) v[i] = make_float4(0.f, 0.f, 0.f, 0.f);
          else if (d < 0) { v[i].x = 0.0f; if (d < -1) v[i].y = 0.0f; if (d < -2) v[i].z = 0.0f; }
          *reinterpret_cast<float4*>(U + r * ldh + c + i * 1024) = v[i];
        }
      }
      continue;
    }
    for (int64_t c = (zeros ? 0 : r / 32 * 32) + threadIdx.x; c < K; c += 256)
      U[r * ldh + c] = (c >= r) ? row[end - 1 - c] : 0.0f;
  }
}

static int64_t round_up(int64_t v, int64_t m) { return (v + m - 1) / m * m; }

// floats of workspace per problem: the matrix, the scratch panel of the square, and (for more than one outer block) the
// operand forms: of the square, of the next block's rows of P (two copies), of the panel before its product with D; P; and
// two copies of the update's operand of halves with its scales, a row per matrix row
static int64_t problem_floats(int64_t K) {
  const int64_t rows = round_up(K, NB);
  return round_up(K, 32) * round_up(K, 32) + kScratchFloats + (K > OB ? 6 * OB * OB + 5 * rows * OB + 2 * rows : 0);
}

// SMs the bulk of an update leaves to the chain beside it: the square's kernels are small (24 to 120 CTAs of which
// several fit an SM), and while the matrix is narrow the chain is the longer of the two
static int chain_reserve(int64_t K) { return K <= 6144 ? 40 : 20; }

// `blocks`: the blocked form in place of U
static int factor(float* H, float* const* Hs, int batch, int64_t order, int64_t ldh, float* ws, int* status, bool lookahead,
                  bool blocks, cudaStream_t st) {
  using tgemm::Job;
  using tgemm::Operand;
  const int slice = Hs ? tgemm::kShortSlice : tgemm::kLongSlice;   // (measured where they are defined)
  const int slice16 = Hs ? tgemm::kShortestSlice16 : tgemm::kLongSlice16;
  int rc;
#define B200Q_RC(expr) do { rc = (expr); if (rc != B200Q_OK) return rc; } while (0)
  const int64_t lda = round_up(order, 32), K = blocks ? lda : order, rows = round_up(K, NB);
  Mat mt;
  mt.A = ws; mt.batch = K * lda; mt.lda = lda; mt.status = status; mt.pad = (int)(K - order);
  float* P = ws + (int64_t)batch * K * lda;
  float* d_hi = P + (int64_t)batch * kScratchFloats;
  float* d_lo = d_hi + (int64_t)batch * OB * OB;
  float* f_base = d_lo + (int64_t)batch * OB * OB;        // next block's rows of P, two copies used in turn
  float* a_hi = f_base + (int64_t)batch * 4 * OB * OB;    // panel before its product with D, and S[o,:o]^T
  const int64_t cap = (int64_t)batch * rows * OB, pb = rows * OB;
  float* a_lo = a_hi + cap;
  float* p_all = a_lo + cap;                              // the other rows of P
  __half* q_base = (__half*)(p_all + cap);                // the update's operand, two copies used in turn
  float* q_scales = (float*)(q_base + 4 * cap);
  const size_t chol_smem = kCholSmemFloats * sizeof(float), panel_smem = kPanelSmemFloats * sizeof(float);
  B200Q_TRY(cudaFuncSetAttribute(chol_diag_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)chol_smem));
  B200Q_TRY(cudaFuncSetAttribute(panel_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)panel_smem));
  auto grid = [&](int64_t x, int64_t cap_x) { return dim3((unsigned)(x < cap_x ? x : cap_x), (unsigned)batch, 1); };
  const int64_t row_ctas = batch > 8 ? 2 * kNumSMs / batch + 1 : 8 * kNumSMs;

  reverse_in_kernel<<<grid(K, row_ctas), 256, 0, st>>>(H, Hs, order, ldh, mt);
  B200Q_LAUNCH_CHECK();
  // Look-ahead: the chain (caller's stream) works on the next square while the products of this step that the next
  // square does not need run on a helper stream.  Arithmetic and its order do not depend on it.
  tgemm::SideStream* side = lookahead && K > 2 * OB ? tgemm::side_stream(st) : nullptr;
  cudaStream_t bulk = side ? side->stream : st;
  bool side_busy = false;
  const int64_t first = blocks && K % OB ? K % OB : OB;
  for (int64_t K0 = 0, K1 = 0, step = 0; K0 < K; K0 = K1, ++step) {
    const int whole = (int)(step == 0 ? first : OB), n = (int)(K - K0 < whole ? K - K0 : whole), inner = (n + NB - 1) / NB;
    K1 = K0 + n;
    const bool last = K1 >= K;
    for (int k = 0; k < inner; ++k) {
      const int bn = n - k * NB < NB ? n - k * NB : NB, below = n - k * NB - bn;
      B200Q_TRY(launch_chained(chol_diag_kernel, dim3(batch), kCholThreads, chol_smem, st, mt, (int)K0 + k * NB, bn));
      B200Q_LAUNCH_CHECK();
      const int units = (below + kVec - 1) / kVec + k * NB / kVec;
      if (units == 0) continue;
      B200Q_TRY(launch_chained(panel_kernel, dim3(2 * units, batch), kThreads, panel_smem, st, mt, P, (int)K0, n, k));
      B200Q_LAUNCH_CHECK();
      const int rt = (below + 31) / 32, base = (k + 1) * (NB / 32), tiles = rt * base + rt * (rt + 1) / 2;
      B200Q_TRY(launch_chained(square_update_kernel, dim3(tiles + k * 16, batch), kThreads, kUpdSmemFloats * sizeof(float), st,
                               mt, P, (int)K0, n, k, tiles));
      B200Q_LAUNCH_CHECK();
    }
    if (last && (K0 == 0 || blocks)) {
      if (side_busy) B200Q_TRY(cudaStreamWaitEvent(st, side->done, 0));
      break;
    }
    float* f_hi = f_base + (step & 1) * 2 * batch * (int64_t)OB * OB;
    float* f_lo = f_hi + batch * (int64_t)OB * OB;
    __half* q_hi = q_base + (step & 1) * 2 * cap;
    __half* q_lo = q_hi + cap;
    float* q_scale = q_scales + (step & 1) * (int64_t)batch * rows;
    const Operand D{d_hi, d_lo, OB, (int64_t)batch * OB, OB, 0}, Pan{a_hi, a_lo, OB, (int64_t)batch * rows, rows, 0},
        F{f_hi, f_lo, OB, (int64_t)batch * OB, OB, 0}, Q{q_hi, q_lo, OB, (int64_t)batch * rows, rows, 0, q_scale};
    const int n2 = last ? 0 : (int)(K - K1 < OB ? K - K1 : OB);
    if (side_busy) B200Q_TRY(cudaStreamWaitEvent(st, side->done, 0));   // products of the step before
    auto split_panel = [&](int64_t r0, int64_t r1, int64_t tcols, bool square, cudaStream_t on) -> int {
      const int64_t tiles = ((r1 - r0 + 31) / 32 + tcols / 32) * ((n + 31) / 32);
      if (tiles == 0 && !square) return B200Q_OK;
      const SquareForm form{d_hi, d_lo, square ? kSquareCtas : 0};
      dim3 g = tiles ? grid(tiles, row_ctas) : dim3(0, (unsigned)batch, 1);
      g.x += form.ctas;
      B200Q_TRY(launch_chained(split_panel_kernel, g, 256, 0, on, mt, (int)K0, n, (int)r0, (int)r1, (int)tcols, a_hi, a_lo, pb, form));
      B200Q_LAUNCH_CHECK();
      return B200Q_OK;
    };
    Job j;
    j.A = Pan; j.B = D; j.Kd = n; j.N = n; j.batch = batch; j.status = status + 2; j.status_stride = 4;
    j.out_ld = OB; j.out_batch = pb; j.slice = slice;
    if (!last) {
      // the next block's rows of P and its square: all the chain needs
      B200Q_RC(split_panel(K1, K1 + n2, 0, true, st));
      if (side) {
        B200Q_TRY(cudaEventRecord(side->ready, st));
        B200Q_TRY(cudaStreamWaitEvent(bulk, side->ready, 0));
      }
      Job f = j;
      f.A.row0 = (int)K1; f.M = n2; f.out_hi = f_hi; f.out_lo = f_lo; f.out_batch = (int64_t)OB * OB;
      B200Q_RC(tgemm::launch(f, st));
      if (side) B200Q_TRY(cudaEventRecord(side->next, st));
      Job d;
      d.A = d.B = F; d.M = d.N = n2; d.Kd = n; d.set = tgemm::kLower; d.batch = batch;
      d.alpha = -1.0f; d.beta = 1.0f; d.C = mt.A + K1 * (lda + 1); d.c_batch = mt.batch; d.ldc = lda;
      d.status = status + 2; d.status_stride = 4; d.slice = slice;
      B200Q_RC(tgemm::launch(d, st));
    } else {
      bulk = st;
    }
    // the other rows of P, and X[o,:o] with its transpose
    const int64_t left = blocks ? 0 : K0;   // columns before the square that take part
    B200Q_RC(split_panel(K1 + n2, K, left, last, bulk));
    Job r = j;
    r.set = tgemm::kPanel; r.skip0 = (int)left; r.skip1 = (int)(K1 + n2); r.M = (int)K;
    if (!last) r.out_hi = p_all;
    if (left) { r.X = mt.A + K0 * lda; r.x_batch = mt.batch; r.ldx = lda; r.xt_rows = (int)K0; }
    r.max_ctas = side && !last ? kNumSMs - chain_reserve(K) : 0;
    B200Q_RC(tgemm::launch(r, bulk));
    if (last) break;
    if (side) B200Q_TRY(cudaStreamWaitEvent(bulk, side->next, 0));
    // the update's operand: X[o,:o]^T and D^T, P (of the next block's rows from its operand form); everything from column c0 on
    const int64_t c0 = K0 - left;
    B200Q_RC(tgemm::split_update16(tgemm::UpdateOperand{mt.A + K0 * lda + c0, lda, mt.batch, n, K1 - c0, f_hi, f_lo,
                                                        (int64_t)OB * OB, n2, p_all + (K1 + n2) * OB, pb, K - K1 - n2,
                                                        q_hi + c0 * OB, q_lo + c0 * OB, q_scale + c0, rows}, batch, bulk));
    // S[below,o] = -P D, S[i,:o] -= P_i X[o,:o], A[i,j] -= P_i P_j^T, without the next square
    Job u;
    u.A = u.B = Q; u.A.row0 = u.B.row0 = (int)c0; u.M = u.N = (int)(K - c0); u.Kd = n; u.set = tgemm::kBulk; u.batch = batch;
    u.row_begin = u.skip0 = (int)(K1 - c0); u.skip1 = (int)(K1 + n2 - c0);
    u.alpha = -1.0f; u.beta = 1.0f; u.C = mt.A + c0 * (lda + 1); u.c_batch = mt.batch; u.ldc = lda;
    u.fresh0 = (int)(K0 - c0); u.fresh1 = (int)(K1 - c0);
    u.status = status + 2; u.status_stride = 4; u.max_ctas = r.max_ctas; u.slice = slice16;
    B200Q_RC(tgemm::launch(u, bulk));
    if (side) {
      B200Q_TRY(cudaEventRecord(side->done, bulk));
      side_busy = true;
    }
  }
#undef B200Q_RC
  reverse_out_kernel<<<grid(K, row_ctas), 256, 0, st>>>(H, Hs, order, ldh, mt, !blocks);
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
  return factor::factor(H, nullptr, 1, K, ldh, (float*)workspace, status, true, false, (cudaStream_t)stream);
}

int b200q_gptq_factor_blocks(float* H, int64_t K, int64_t ldh, void* workspace, int* status, void* stream) {
  if (!H || !workspace || !status || K <= 0 || ldh < K || K > (1 << 24)) return B200Q_ERR_ARG;
  return factor::factor(H, nullptr, 1, K, ldh, (float*)workspace, status, true, true, (cudaStream_t)stream);
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
  return factor::factor(nullptr, H, count, K, ldh, (float*)workspace, status, false, false, st);
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
