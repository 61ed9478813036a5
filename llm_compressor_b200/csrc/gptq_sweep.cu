// GPTQ solve, part 2: the column sweep, for one weight or a batch of weights of one shape.
//
// Rows of W are independent and the columns of a row form one dependent chain: quantise column i, divide the error
// by U[i,i], subtract its multiple of U[i, i+1:] from the rest of the row.  The columns are taken in superblocks of
// up to 512.  Inside one, a CTA carries 32 or 64 rows through all columns without touching device memory for them
// (sweep_block_kernel); between superblocks the rest of the matrix takes W[:, after] -= Err * U[block, after] as one
// fp32-accurate tensor-core product (tgemm).  What the reference calls its block size only orders float32 operations
// and does not change the result otherwise, so it does not decide the split here.
//
// With the factor's blocked form (V upper, H = V V^T, U = V^-1; b200q_gptq_factor_blocks) the products across superblocks
// use Err U = W - Q, that is Err = (W - Q) V: what the columns of superblock b get from those before it is
// (W - Q)[:, :b] V[:b, b] U_bb.  The same product with W - Q in place of the errors and -V U_bb in place of U, without the
// triangular inverse, half of the factor's work; W as it was is needed for it.  Error of the last column against float64, all
// codes zero, 4096 columns: 2.3e-7 of its root mean square.  Reading W again costs the sweep 2 to 5 % (4096 x 4096: 757 us with
// U, 787; 4096 x 14336: 4376, 4483), the factor saves more.
//
// Each correction is one fused multiply-add (the reference rounds the product first), true divisions decide a code
// wherever an ulp could matter.
#include <cstdlib>
#include <type_traits>

#include "common.cuh"
#include "tgemm_tf32.cuh"

namespace b200q {
namespace sweep {

constexpr int kMaxBlock = 128;               // largest block size callers may ask for
constexpr size_t kSweepHeaderBytes = 256;    // status word at the start of the workspace
constexpr int kMicro = 16;                   // columns whose errors make one operand of the MMAs
constexpr int kHalf = 8;                     // columns the chain takes at a time
constexpr int kSlots = 4;                    // micro-blocks whose parameters and band of U are in shared memory
constexpr int kBlockCols = 128;              // columns of W that one MMA corrects
constexpr int kRowBytes = 4 * kMicro;        // operand row of a micro-block: 16 hi and 16 lo halves
constexpr int kTileBytes = kBlockCols * kRowBytes;   // a block's columns of U for a micro-block's errors
constexpr int kLag = 3;                      // errors of micro-block m reach columns from m + kLag on by MMAs
constexpr int kBandCols = kLag * kMicro;     // columns of U that chain and feeder need of a micro-block's rows (8 rows at
                                             // most reach 5 half-blocks on)
constexpr int kGoAhead = 8;                  // half-blocks before the end at which the next kernel may be set up
constexpr int kErrSlots = 4;                 // micro-blocks whose errors are kept
constexpr int kBandFloats = kMicro * kBandCols + kMicro;   // and the reciprocals of the pivots

// One pointer per operand, or (table set) a device array with one per problem.
template <class T> struct Ptr {
  T* one; T* const* table;
  __device__ __forceinline__ T* at(int b) const { return table ? table[b] : one; }
};

struct Params {
  Ptr<float> W; Ptr<const float> U; Ptr<const void> scale; Ptr<const void> zp;
  Ptr<const int32_t> col_group; Ptr<const float> gscale; Ptr<float> losses;
  int64_t N, K, ldw, ldu;
  int strategy, group_size, block_h, zp_kind;
  int64_t groups_per_row;
  QRange qr;
  float* err; int64_t lde, err_batch;                     // the superblock's errors (null: nothing after it), or
  const void* W0; int64_t ld0; int w0dtype;               // (set) what its columns differ from these by
  int i1, sb;                                             // superblock: first column, width
  int sdtype;                                             // of the scales
  const unsigned char* tiles; int64_t tiles_batch;        // operand form of U[i1 : i1 + sb, i1 : i1 + sb], one a factor
  const int32_t* u_index;                                 // factor of problem b (null: one each)
  int* status;                                            // set if a bounded wait expires
};

// What a CTA of ROWS rows and SBLK columns holds, and where.
template <int ROWS, int SBLK> struct Shape {
  static constexpr int kChains = ROWS / 32;            // chain warps: a lane per row
  static constexpr int kBlocks = SBLK / kBlockCols;
  static constexpr int kHelpers = 4 * kBlocks;         // warps with 32 columns each
  // first warp of each role; two feeders per chain, one of each other kind of 32 rows, one for the MMAs and one for
  // the parameters
  static constexpr int kErrors = ROWS == 32 ? 3 : 2, kFeeder = ROWS == 32 ? 1 : 4, kMma = ROWS == 32 ? 4 : 8,
                       kOut = kMma + 1, kParams = kOut + kChains;
  static constexpr int kFirstHelper = ROWS == 32 ? 8 : 12;
  static constexpr int kThreads = 32 * (kFirstHelper + kHelpers);
  static constexpr int kStages = 3, kStageBytes = kBlocks * kTileBytes;   // ring of the tiles of a micro-block's errors
  static constexpr int kErrBytes = ROWS * kRowBytes;   // errors of a micro-block as operand
  static constexpr int kWld = ROWS + 4;                // stride of a column of W: float4 accesses conflict-free
  static constexpr int kRing = 0, kErr = kRing + kStages * kStageBytes, kW = kErr + 2 * kErrBytes,
                       kE = kW + SBLK * kWld * 4, kPar = kE + kErrSlots * kMicro * ROWS * 4,
                       kZ = kPar + kSlots * kMicro * ROWS * 8, kBand = kZ + kSlots * kMicro * ROWS * 4,
                       kSe = kBand + kSlots * kBandFloats * 4,
                       kNext = kSe + 4 * ROWS * 4, kPow = kNext + 2 * kHalf * ROWS * 4, kEnd = kPow + SBLK * 4;
  static constexpr size_t kSmem = kEnd + 1024;
  static constexpr int kMicros = SBLK / kMicro;
};
static_assert(Shape<32, 512>::kSmem <= 232448 - 2048 && Shape<64, 256>::kSmem <= 232448 - 2048, "shared memory");
// Registers a thread of the warpgroups, as many as at the launch: 32 rows 768 threads at 80 (160 + 64 + 4 * 64), 64 rows 640 at
// 96 (144 + 64 + 48 + 2 * 112).
template <int ROWS> struct Regs {
  static constexpr int kChain = ROWS == 32 ? 160 : 144, kFeeder = 64, kOther = ROWS == 32 ? 64 : 48, kHelper = ROWS == 32 ? 64 : 112;
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void bar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void bar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool bar_ready(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred P1;\n\tmbarrier.try_wait.parity.shared::cta.b64 P1, [%1], %2;\n\tselp.b32 %0, 1, 0, P1;\n\t}"
      : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
  return ok != 0;
}
// (try_wait above may suspend the thread for thousands of cycles, this one never does)
__device__ __forceinline__ bool bar_test(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred P1;\n\tmbarrier.test_wait.parity.shared::cta.b64 P1, [%1], %2;\n\tselp.b32 %0, 1, 0, P1;\n\t}"
      : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
  return ok != 0;
}
// After a wait has run out nothing waits any more: the CTA ends with garbage and the status says so.
__device__ __forceinline__ void bar_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
  if (bar_ready(bar, parity)) return;
  const long long t0 = clock64();
  while (!bar_ready(bar, parity)) {
    if (*abort_flag) return;
    if (clock64() - t0 > 4000000000LL) { *abort_flag = 1; return; }
  }
}
// the same for warps that nobody waits for soon: they leave the issue slots and the barrier unit to the others
__device__ __forceinline__ void bar_sleep(uint32_t bar, uint32_t parity, unsigned ns, volatile int* abort_flag) {
  if (bar_test(bar, parity)) return;
  const long long t0 = clock64();
  while (!bar_test(bar, parity)) {
    __nanosleep(ns);
    if (*abort_flag) return;
    if (clock64() - t0 > 4000000000LL) { *abort_flag = 1; return; }
  }
}
// the same without suspending: for the few warps whose reaction the chain waits for.  The limit is one of tries, a second
// at least and longer for a warp that is seldom scheduled: with the clock looked at every 1024 tries, sweeps of 1001 to 14336
// rows took 1 to 3 % longer (1001 x 4096 606 us, 620).
__device__ __forceinline__ void bar_spin(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
  for (uint32_t tries = 0; !bar_test(bar, parity);)
    if ((++tries & 1023u) == 0 && (*abort_flag || tries > (1u << 26))) { *abort_flag = 1; return; }
}
__device__ __forceinline__ void bulk_copy(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}
__device__ __forceinline__ void tc_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mma_f16(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                         uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate) : "memory");
}
// K-major operand in rows of 64 bytes, 64-byte swizzle: groups of eight rows are 512 bytes apart
__device__ __forceinline__ uint64_t make_desc(uint32_t saddr) {
  return (uint64_t)((saddr >> 4) & 0x3FFFu) | (uint64_t)1 << 16 | (uint64_t)(512 >> 4) << 32 | (uint64_t)1 << 46 |
         (uint64_t)4 << 61;
}
// D fp32, A / B f16, both K-major, M = 128
__host__ __device__ constexpr uint32_t instr_desc(int n) {
  return (1u << 4) | ((uint32_t)(n >> 3) << 17) | ((128u >> 4) << 24);
}
// ---- operands of the products inside a superblock
// Float32 values as two halves with a scale per operand row, as tgemm has them: a row is a column of the superblock (of
// U^T), or a row of a micro-block's errors.
using tgemm::row_scale;
using tgemm::split_pair;

// U[i1 : i1 + sb, i1 : i1 + sb] as the tiles that the sweep copies into shared memory: tile (micro-block m, block b) holds
// for each of the block's 128 columns 16 hi and 16 lo halves of the micro-block's rows of U, in 64-byte rows swizzled as
// the MMA reads them, rows taken times the power of their pivot (tgemm::pivot_power).  Behind the tiles the inverse scale of every column, the
// inverses of the pivots' powers (the errors are taken times these), and then for every micro-block its rows of U
// from the diagonal on (the identity beyond sb) and the reciprocals of its pivots.  A CTA takes 32 columns.
constexpr int kTileThreads = 256;
constexpr int64_t scales_offset(int sblk) { return (int64_t)(sblk / kMicro) * (sblk / kBlockCols) * kTileBytes; }
constexpr int64_t powers_offset(int sblk) { return scales_offset(sblk) + sblk * 4; }
constexpr int64_t band_offset(int sblk) { return powers_offset(sblk) + sblk * 4; }
constexpr int64_t tiles_bytes(int sblk) { return band_offset(sblk) + sblk / kMicro * kBandFloats * 4; }   // of one factor
// Further CTAs (from `squares` on) make the operand of the trailing product: the columns behind the square.
struct Slice { __half *hi, *lo; float* scale; int64_t cols, rows; bool inverse; };   // rows of the operand per factor
template <int SBLK>
__global__ void __launch_bounds__(kTileThreads) square_tiles_kernel(Ptr<const float> Us, int64_t ldu, int i1, int sb,
                                                                   unsigned char* tiles, int64_t batch_bytes, int squares,
                                                                   const Slice slice) {
  chain_wait();
  chain_go();
  extern __shared__ float stage[];   // [32][SBLK + 2]
  __shared__ float s_max[kTileThreads / 32][32];
  __shared__ float s_power[SBLK];   // of the rows' pivots
  constexpr int kWarps = kTileThreads / 32, kBlocks = SBLK / kBlockCols;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, c = blockIdx.x * 32 + lane;
  const float* U = Us.at(blockIdx.y) + (int64_t)i1 * ldu + i1;
  if ((int)blockIdx.x >= squares) {
    const int64_t at = blockIdx.y * slice.rows;
    tgemm::split_columns16<SBLK>(U + sb, ldu, sb, slice.cols, INT64_MAX / 2, slice.hi + at * SBLK, slice.lo + at * SBLK,
                                 slice.scale + at, slice.inverse ? tgemm::kInverses : tgemm::kPowers, blockIdx.x - squares, stage);
    return;
  }
  tiles += blockIdx.y * batch_bytes;
  float v[SBLK / kWarps], largest = 0.0f;
  // (no load depends on a condition: they go out together)
#pragma unroll
  for (int i = 0; i < SBLK / kWarps; ++i) v[i] = U[(int64_t)min(warp + i * kWarps, sb - 1) * ldu + min(c, sb - 1)];
  for (int p = threadIdx.x; p < SBLK; p += kTileThreads) {
    const float reciprocal = __frcp_rn(p < sb ? U[(int64_t)p * ldu + p] : 1.0f);
    s_power[p] = tgemm::pivot_power(reciprocal);
    if (blockIdx.x == 0) reinterpret_cast<float*>(tiles + powers_offset(SBLK))[p] = tgemm::pivot_inverse(reciprocal);
  }
#pragma unroll
  for (int i = 0; i < SBLK / kWarps; ++i)
    if (warp + i * kWarps > c || c >= sb) v[i] = 0.0f;
  __syncthreads();
  float* bands = reinterpret_cast<float*>(tiles + band_offset(SBLK));
#pragma unroll
  for (int i = 0; i < SBLK / kWarps; ++i) {
    const int p = warp + i * kWarps, c0 = p / kMicro * kMicro;
    const float x = (p == c && c >= sb) ? 1.0f : v[i];
    if (c >= c0 && c < c0 + kBandCols) bands[p / kMicro * kBandFloats + (p - c0) * kBandCols + c - c0] = x;
    if (c == p) bands[p / kMicro * kBandFloats + kMicro * kBandCols + p - c0] = __frcp_rn(x);
    v[i] *= s_power[p];
    largest = fmaxf(largest, fabsf(v[i]));
  }
  s_max[warp][lane] = largest;
  __syncthreads();
#pragma unroll
  for (int k = 0; k < kWarps; ++k) largest = fmaxf(largest, s_max[k][lane]);
  float scale, inverse;
  row_scale(largest, scale, inverse);
  if (warp == 0) reinterpret_cast<float*>(tiles + scales_offset(SBLK))[c] = inverse;
#pragma unroll
  for (int i = 0; i < SBLK / kWarps; ++i) stage[lane * (SBLK + 2) + warp + i * kWarps] = v[i] * scale;
  __syncthreads();
  const int b = c / kBlockCols, row = c % kBlockCols;
  for (int m = warp; (m + kLag) * kMicro <= c; m += kWarps) {
    const float* x = stage + lane * (SBLK + 2) + m * kMicro;
    unsigned char* d = tiles + (int64_t)(m * kBlocks + b) * kTileBytes + row * kRowBytes;
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      uint32_t hi[4], lo[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) split_pair(x[8 * j + 2 * k], x[8 * j + 2 * k + 1], hi[k], lo[k]);
      *reinterpret_cast<uint4*>(d + ((j ^ ((row >> 1) & 3)) << 4)) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
      *reinterpret_cast<uint4*>(d + (((j + 2) ^ ((row >> 1) & 3)) << 4)) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
    }
  }
}
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr) : "memory");
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ uint64_t pair(float lo, float hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void unpair(uint64_t v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}

// ---- quantisation of a column on the chain
// The code of x is settled by x * (1 / s) taken slightly low and slightly high: equal codes mean that the ulps between
// the product and the reference's division cannot matter.  Whether they are equal is not waited for column by column:
// a micro-block whose flags show a difference anywhere (some per mille of them) is swept again by the exact rules.
constexpr float kMargin = 0x1p-21f;   // > the 2^-22 by which reciprocal, product and division can differ in all
constexpr float kMagic = 12582912.0f; // 1.5 * 2^23: a float32 sum with it is rounded to the nearest integer, ties to even

// integer code of x * r + zz (the sign of a zero is put back later)
template <bool ZP>
__device__ __forceinline__ float code_of(float x, float r, float zz, float qmin, float qmax) {
  // product and rounding to an integer in one: beyond 2^22, where the sum's ulp grows, only the clamp matters
  if (!ZP) return fminf(fmaxf(fmaf(x, r, kMagic), kMagic + qmin), kMagic + qmax) - kMagic;
  return (fminf(fmaxf(fmaf(x, r, zz), qmin), qmax) + kMagic) - kMagic;
}
// FP8 or FP4 value of both ends through the hardware's pair and back: one conversion each way, which saturates (clamped and
// converted one by one FP8, 1001 x 1160, took 203 us, 192 now; 32 weights of 2048 x 768 1301, 1246).  A NaN, which the exact rules clamp, counts as a difference.
template <int KIND>
__device__ __forceinline__ float code_pair(float lo, float hi, bool& differ) {
  uint32_t h;
  if constexpr (KIND == kFp8)
    asm("{\n\t.reg .b16 c;\n\tcvt.rn.satfinite.e4m3x2.f32 c, %2, %1;\n\tcvt.rn.f16x2.e4m3x2 %0, c;\n\t}" : "=r"(h) : "f"(lo), "f"(hi));
  else
    asm("{\n\t.reg .b8 c;\n\tcvt.rn.satfinite.e2m1x2.f32 c, %2, %1;\n\tcvt.rn.f16x2.e2m1x2 %0, c;\n\t}" : "=r"(h) : "f"(lo), "f"(hi));
  differ |= __byte_perm(h, h, 0x1032) != h || lo != lo;
  return __half2float(__ushort_as_half((unsigned short)(h & 0xFFFFu)));
}
// bf16 rounding with the result already in place as a float
__device__ __forceinline__ float bf16_in_place(float v) {
  uint32_t d;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(v), "f"(0.0f));
  return __uint_as_float(d);
}
template <int KIND, bool SB, bool ZP>
__device__ __forceinline__ float dequant(float q, float s, float z) {
  if (ZP) {
    q = q - z;
    if (SB && KIND != kInt) q = bf16_in_place(q);   // (integer differences are exact in bf16)
  }
  q = q * s;
  return SB ? bf16_in_place(q) : q;
}

// What bounds it: the chain of columns, one warp of 32 rows.  Cycles of a CTA's launch, 4096 rows x 512 columns, clocks read
// in the chain's warp: 2100 setting up, 6000 until the first columns of W are there, 500 their parameters, 83000 the
// chain, 900 after it.  Eight columns of the chain take 1300, of which 210 are the hand-over from the feeder (180 where it has
// long been through: the chain hardly ever waits), 1060 at the end of the superblock where few other roles still run.
// What the roles cost one another is instruction fetch: from 35 KB of unrolled code, as they were at first, 3000 fetches a
// CTA went to the GPC's cache and the kernel took 140 us; with eight columns unrolled instead of sixteen and short loops
// everywhere else it takes 65 (81 when warp-level MMAs on 16-column tiles in shared memory did the corrections; ncu, warm
// caches).  The whole 4096 x 4096 sweep takes 0.82 ms, 0.88 with zero points (1.04).  So: nothing is unrolled further than the
// registers demand.
//
// Roles, all of them warps of one CTA that hand over by one-shot mbarriers, so that nobody waits for all:
//   chain    codes and errors of eight columns; applies them to these columns and sums what they are to the next eight
//   feeders  give the eight after these the errors of up to four half-blocks (even and odd ones a warp each)
//   errors   turn the errors of 16 columns into an MMA operand
//   MMA      U^T[128 columns, 16] E[16, rows] for everything from kLag micro-blocks on, accumulators in TMEM (two sets)
//   helpers  hold the columns of W in registers (a lane each, all rows), add the products to them, hand them over
//            when their turn comes and write the codes out when the chain is past, while it goes on
//   out      errors out for the trailing product, losses;  params  scales and zero points, copies of U
// U comes as tiles that one bulk copy brings in (as 64-byte rows of a tensor map it arrived at 18 bytes a clock and SM).
template <int ROWS, int SBLK, bool SB, int KIND, bool ZP>
__global__ void __launch_bounds__(Shape<ROWS, SBLK>::kThreads, 1)
sweep_block_kernel(const __grid_constant__ Params p) {
  using S = Shape<ROWS, SBLK>;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* sm = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  float* sW = reinterpret_cast<float*>(sm + S::kW);         // [SBLK][kWld]
  float* sE = reinterpret_cast<float*>(sm + S::kE);         // [kErrSlots][kMicro][ROWS] negated errors
  float2* sPar = reinterpret_cast<float2*>(sm + S::kPar);   // [kSlots][kMicro][ROWS] scale, 1 / scale
  float* sZ = reinterpret_cast<float*>(sm + S::kZ);         // [kSlots][kMicro][ROWS] zero point
  float* sBand = reinterpret_cast<float*>(sm + S::kBand);   // [kSlots][kMicro][kBandCols] U[c0 + t, c0 ...], [kMicro] 1 / U[i,i]
  float* sSe = reinterpret_cast<float*>(sm + S::kSe);       // [4][ROWS] inverse scales of a micro-block's errors
  float* sNext = reinterpret_cast<float*>(sm + S::kNext);   // [2][kHalf][ROWS] columns that the chain takes next
  // One-shot barriers.  Of a micro-block m: parameters and band are there; its columns have the errors up to m - kLag
  // (helpers); its errors are there as operand; its errors are out.  Of half a micro-block n: its columns have the errors up to n - 2 (feeder);
  // its errors and codes are there (chain).
  __shared__ __align__(8) uint64_t s_par[S::kMicros], s_raw[S::kMicros], s_opr[S::kMicros], s_out[S::kMicros], s_ready[2 * S::kMicros],
      s_done[2 * S::kMicros];
  __shared__ __align__(8) uint64_t s_full[S::kStages], s_empty[S::kStages];
  __shared__ __align__(8) uint64_t s_accf[2][S::kBlocks], s_acce[2][S::kBlocks];
  __shared__ int s_odd[S::kChains][kSlots];                        // some scale is outside the range the low / high test covers
  __shared__ uint32_t s_tmem;
  __shared__ volatile int s_abort;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

  if (tid == 0) {
    for (int m = 0; m < S::kMicros; ++m) {
      bar_init(smem_u32(&s_par[m]), 2); bar_init(smem_u32(&s_raw[m]), 1); bar_init(smem_u32(&s_opr[m]), S::kChains);
      bar_init(smem_u32(&s_out[m]), S::kChains);
    }
    for (int n = 0; n < 2 * S::kMicros; ++n) {
      bar_init(smem_u32(&s_ready[n]), S::kChains); bar_init(smem_u32(&s_done[n]), S::kChains);
    }
    for (int k = 0; k < S::kStages; ++k) { bar_init(smem_u32(&s_full[k]), 1); bar_init(smem_u32(&s_empty[k]), 1); }
    for (int k = 0; k < 2; ++k)
      for (int b = 0; b < S::kBlocks; ++b) { bar_init(smem_u32(&s_accf[k][b]), 1); bar_init(smem_u32(&s_acce[k][b]), 4); }
    s_abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == S::kMma) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem)), "r"(512) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = s_tmem;
  chain_wait();

  const int job = blockIdx.y, sb = p.sb, micros = (sb + kMicro - 1) / kMicro, blocks = (sb + kBlockCols - 1) / kBlockCols;
  const int64_t row0 = (int64_t)blockIdx.x * ROWS;
  const float* __restrict__ U = p.U.at(job);
  const bool has_u = U != nullptr;
  const unsigned char* tiles = p.tiles + (p.u_index ? p.u_index[job] : job) * p.tiles_batch;
  const float qmin = p.qr.qmin, qmax = p.qr.qmax;
  const int steps = micros - kLag;   // micro-blocks whose errors go anywhere by MMAs
  auto first_block = [](int m) { return (m + kLag) * kMicro / kBlockCols; };

  auto helper_role = [&] {
    // ---- helpers: warp (block b, quarter q) has columns 128 b + 32 q + lane in registers, all rows of them
    const int b = (warp - S::kFirstHelper) >> 2, q = warp & 3, own = 4 * b + q, col = own * 32 + lane;
    float* __restrict__ W = p.W.at(job) + p.i1 + col;
    float v[ROWS];
#pragma unroll
    for (int r = 0; r < ROWS; ++r) v[r] = (col < sb && row0 + r < p.N) ? W[(row0 + r) * p.ldw] : 0.0f;
    // columns of micro-block `m`, one of this warp's two, for the feeder
    auto hand_over = [&](int m) {
      if ((lane >> 4) == (m & 1)) {
        float4* d = reinterpret_cast<float4*>(sW + col * S::kWld);
#pragma unroll
        for (int r = 0; r < ROWS; r += 4) d[r / 4] = make_float4(v[r], v[r + 1], v[r + 2], v[r + 3]);
      }
      __syncwarp();
      if (lane == 0) bar_arrive(smem_u32(&s_raw[m]));
    };
    if (own == 0) { hand_over(0); hand_over(1); }
    if (own == 1) hand_over(2);
    const int last_step = min(2 * own + 1 - kLag, steps - 1);         // the last whose errors this warp's columns take
    const int last_mma = min(8 * b + 7 - kLag, steps - 1);            // the last that its block takes part in
    const float su = has_u && col < sb ? reinterpret_cast<const float*>(tiles + scales_offset(SBLK))[col] : 0.0f;
    if (b < blocks) {
#pragma unroll 1
      for (int m = 0; m <= last_mma; ++m) {
        const uint32_t acc = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)((m & 1) * 256 + b * 2 * ROWS);
        bar_sleep(smem_u32(&s_accf[m & 1][b]), (uint32_t)(m >> 1) & 1u, m + kLag + 2 >= 2 * own ? 20 : 100, &s_abort);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if (has_u && m <= last_step) {
#pragma unroll
          for (int r0 = 0; r0 < ROWS; r0 += 8) {
            uint32_t x[8], y[8];
            tmem_ld8(acc + r0, x);
            tmem_ld8(acc + ROWS + r0, y);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
            for (int r = 0; r < 8; r += 4) {
              const float4 se = *reinterpret_cast<const float4*>(sSe + (m & 3) * ROWS + r0 + r);
              const float f[4] = {se.x, se.y, se.z, se.w};
#pragma unroll
              for (int k = 0; k < 4; ++k)
                v[r0 + r + k] = fmaf((__uint_as_float(x[r + k]) + __uint_as_float(y[r + k])) * su, f[k], v[r0 + r + k]);
            }
          }
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) bar_arrive(smem_u32(&s_acce[m & 1][b]));
        if (m + kLag == 2 * own || m + kLag == 2 * own + 1) hand_over(m + kLag);
      }
      // the columns as the chain leaves them
      bar_sleep(smem_u32(&s_done[2 * min(2 * own + 1, micros - 1) + 1]), 0, 200, &s_abort);
      if (col < sb) {
        const float4* d = reinterpret_cast<const float4*>(sW + col * S::kWld);
#pragma unroll
        for (int r = 0; r < ROWS; r += 4) {
          const float4 x = d[r / 4];
          v[r] = x.x; v[r + 1] = x.y; v[r + 2] = x.z; v[r + 3] = x.w;
        }
#pragma unroll
        for (int r = 0; r < ROWS; ++r)
          if (row0 + r < p.N) W[(row0 + r) * p.ldw] = v[r];
      }
    }
  };
  auto chain_role = [&] {
    // ---- the chain, a lane per row: eight columns at a time
    const int r = warp * 32 + lane;
    uint64_t x[kHalf / 2];    // columns of half-block n, all corrections up to it done
    bar_wait(smem_u32(&s_raw[0]), 0, &s_abort);
    bar_wait(smem_u32(&s_par[0]), 0, &s_abort);
#pragma unroll
    for (int k = 0; k < kHalf / 2; ++k) x[k] = pair(sW[2 * k * S::kWld + r], sW[(2 * k + 1) * S::kWld + r]);
#pragma unroll 1
    for (int n = 0; n < 2 * micros; ++n) {
      // the next kernel's CTAs wait on the SMs that are free, where the helper stream makes the next slice of U meanwhile: not
      // before the end is near (from the start on, where warps without a role said so, they kept that slice, which the product
      // waits for, off the SMs until the sweep was over: 4096 x 4096 806 us, now 757; 4096 x 14336 4670, 4376)
      if (n == 2 * micros - kGoAhead) chain_go();
      const int slot = (n >> 1) & (kSlots - 1), t0 = (n & 1) * kHalf;
      float* wcol = sW + n * kHalf * S::kWld + r;
      float* eo = sE + (((n >> 1) & (kErrSlots - 1)) * kMicro + t0) * ROWS + r;
      const float* band = sBand + slot * kBandFloats + t0 * kBandCols + t0;
      const float2* par = sPar + (slot * kMicro + t0) * ROWS + r;
      const float* zero = sZ + (slot * kMicro + t0) * ROWS + r;
      uint64_t y[kHalf / 2] = {0, 0, 0, 0};   // what its errors are to the columns of n + 1
      const uint64_t x0[kHalf / 2] = {x[0], x[1], x[2], x[3]};
      uint64_t ne[kHalf];                     // negated errors, twice each
      bool differ = s_odd[warp][slot] != 0;
      float q[kHalf];
#pragma unroll
      for (int t = 0; t < kHalf; ++t) {
        float a, c;
        unpair(x[t / 2], a, c);
        const float2 sr = par[t * ROWS];
        const float wi = (t & 1) ? c : a, s = sr.x, z = ZP ? zero[t * ROWS] : 0.0f;
        const float mz = ZP ? fabsf(z) * (0.5f * kMargin) : 0.0f;
        const float rlo = sr.y * (1.0f - kMargin), rhi = sr.y * (1.0f + kMargin);
        float qc;
        if constexpr (KIND == kInt) {
          qc = code_of<ZP>(wi, rlo, z - mz, qmin, qmax);
          differ |= qc != code_of<ZP>(wi, rhi, z + mz, qmin, qmax);
        } else {
          qc = code_pair<KIND>(fmaf(wi, rlo, z - mz), fmaf(wi, rhi, z + mz), differ);
        }
        const float dq = dequant<KIND, SB, ZP>(qc, s, z);
        // loss and error use the reciprocal of the pivot (an ulp from the reference's divisions)
        const float e = __fmul_rn(__fsub_rn(dq, wi), sBand[slot * kBandFloats + kMicro * kBandCols + t0 + t]);
        ne[t] = pair(e, e);
        // a zero has the sign of the quotient: x / s + 0 is -0 for a small negative x, and stays it
        q[t] = (KIND == kInt && (!ZP || (dq == 0.0f && z == 0.0f))) ? copysignf(dq, fmaf(wi, rlo, z - mz)) : dq;
#pragma unroll
        for (int k = (t + 1) / 4; k < 4; ++k) {
          const ulonglong2 u = *reinterpret_cast<const ulonglong2*>(band + t * kBandCols + 4 * k);
          if (k < 2) {
            if (4 * k + 1 > t) x[2 * k] = fma2(ne[t], u.x, x[2 * k]);
            x[2 * k + 1] = fma2(ne[t], u.y, x[2 * k + 1]);
          } else {
            y[2 * k - 4] = fma2(ne[t], u.x, y[2 * k - 4]);
            y[2 * k - 3] = fma2(ne[t], u.y, y[2 * k - 3]);
          }
        }
      }
#pragma unroll
      for (int t = 0; t < kHalf; ++t) {
        float e, f;
        unpair(ne[t], e, f);
        eo[t * ROWS] = e;
        wcol[t * S::kWld] = q[t];
      }
      if (__any_sync(0xffffffffu, differ)) {
        // again by the exact rules, column by column in shared memory
#pragma unroll
        for (int k = 0; k < kHalf / 2; ++k) {
          float a, c;
          unpair(x0[k], a, c);
          wcol[2 * k * S::kWld] = a;
          wcol[(2 * k + 1) * S::kWld] = c;
          y[k] = 0;
        }
#pragma unroll 1
        for (int t = 0; t < kHalf; ++t) {
          const float wi = wcol[t * S::kWld], s = par[t * ROWS].x, z = ZP ? zero[t * ROWS] : 0.0f;
          const float v = dequant_code<SB>(round_code_k<KIND>(__fdiv_rn(wi, s) + z, qmin, qmax), s, z);
          const float e = __fmul_rn(__fsub_rn(v, wi), sBand[slot * kBandFloats + kMicro * kBandCols + t0 + t]);
          wcol[t * S::kWld] = v;
          eo[t * ROWS] = e;
#pragma unroll 1
          for (int k = t + 1; k < kHalf; ++k) wcol[k * S::kWld] = fmaf(e, band[t * kBandCols + k], wcol[k * S::kWld]);
          const uint64_t ee = pair(e, e);
#pragma unroll
          for (int k = 0; k < 2; ++k) {
            const ulonglong2 u = *reinterpret_cast<const ulonglong2*>(band + t * kBandCols + kHalf + 4 * k);
            y[2 * k] = fma2(ee, u.x, y[2 * k]);
            y[2 * k + 1] = fma2(ee, u.y, y[2 * k + 1]);
          }
        }
      }
      __syncwarp();
      if (lane == 0) bar_arrive(smem_u32(&s_done[n]));
      if (n + 1 == 2 * micros) break;
      if (n > 0) bar_spin(smem_u32(&s_ready[n + 1]), 0, &s_abort);
      const float* next = n > 0 ? sNext + ((n + 1) & 1) * kHalf * ROWS + r : wcol + kHalf * S::kWld;
      const int ld = n > 0 ? ROWS : S::kWld;
#pragma unroll
      for (int k = 0; k < kHalf / 2; ++k) x[k] = add2(pair(next[2 * k * ld], next[(2 * k + 1) * ld]), y[k]);
    }
  };
  auto feeder_role = [&] {
    // ---- feeders (of even and of odd half-blocks), a lane per row: half-block n takes the errors that no MMA gives it, up to those of n - 2
    const int r = ((warp - S::kFeeder) >> 1) * 32 + lane;
#pragma unroll 1
    for (int n = 2 + ((warp - S::kFeeder) & 1); n < 2 * micros; n += 2) {
      const int m = n >> 1;
      const float* wcol = sW + n * kHalf * S::kWld + r;
      uint64_t x[kHalf / 2] = {0, 0, 0, 0};   // summed apart: one rounding at the weight's magnitude
#pragma unroll 1
      for (int h = max(2 * (m - kLag + 1), 0); h <= n - 2; ++h) {
        bar_spin(smem_u32(&s_done[h]), 0, &s_abort);
        const int t0 = (h & 1) * kHalf;
        const float* e = sE + (((h >> 1) & (kErrSlots - 1)) * kMicro + t0) * ROWS + r;
        const float* band = sBand + ((h >> 1) & (kSlots - 1)) * kBandFloats + t0 * (kBandCols + 1) + (n - h) * kHalf;
#pragma unroll
        for (int t = 0; t < kHalf; ++t) {
          const float f = e[t * ROWS];
          const uint64_t ee = pair(f, f);
#pragma unroll
          for (int k = 0; k < 2; ++k) {
            const ulonglong2 u = *reinterpret_cast<const ulonglong2*>(band + t * kBandCols + 4 * k);
            x[2 * k] = fma2(ee, u.x, x[2 * k]);
            x[2 * k + 1] = fma2(ee, u.y, x[2 * k + 1]);
          }
        }
      }
      float* next = sNext + (n & 1) * kHalf * ROWS + r;
      bar_spin(smem_u32(&s_raw[m]), 0, &s_abort);
      // (the chain has taken n - 2 out of `next`)
#pragma unroll
      for (int k = 0; k < kHalf / 2; ++k) {
        float a, c;
        unpair(add2(x[k], pair(wcol[2 * k * S::kWld], wcol[(2 * k + 1) * S::kWld])), a, c);
        next[2 * k * ROWS] = a;
        next[(2 * k + 1) * ROWS] = c;
      }
      if ((n & 1) == 0) bar_spin(smem_u32(&s_par[m]), 0, &s_abort);
      __syncwarp();
      if (lane == 0) bar_arrive(smem_u32(&s_ready[n]));
    }
  };
  auto error_role = [&] {
    // ---- errors of 32 rows as operand of the MMAs
    const int r = (warp - S::kErrors) * 32 + lane;
    float* power = reinterpret_cast<float*>(sm + S::kPow);   // of the pivots, inverted (every one of these warps writes all)
    for (int i = lane; i < SBLK / 4; i += 32)
      reinterpret_cast<float4*>(power)[i] = has_u ? reinterpret_cast<const float4*>(tiles + powers_offset(SBLK))[i]
                                                  : make_float4(1.f, 1.f, 1.f, 1.f);
    __syncwarp();
#pragma unroll 1
    for (int m = 0; m < steps; ++m) {
      if (m >= 2)   // the operand buffer's last readers are done
        bar_spin(smem_u32(&s_accf[m & 1][blocks - 1]), (uint32_t)((m - 2) >> 1) & 1u, &s_abort);
      bar_spin(smem_u32(&s_done[2 * m + 1]), 0, &s_abort);
      const float* es = sE + (m & (kErrSlots - 1)) * kMicro * ROWS + r;
      const uint32_t eop = smem_u32(sm + S::kErr + (m & 1) * S::kErrBytes) + (uint32_t)(r * kRowBytes);
      float largest[4] = {0.0f, 0.0f, 0.0f, 0.0f}, to, back;
      const float* pw = power + m * kMicro;
#pragma unroll 8
      for (int t = 0; t < kMicro; ++t) largest[t & 3] = fmaxf(largest[t & 3], fabsf(es[t * ROWS] * pw[t]));
      row_scale(fmaxf(fmaxf(largest[0], largest[1]), fmaxf(largest[2], largest[3])), to, back);
      sSe[(m & 3) * ROWS + r] = back;
#pragma unroll 1
      for (int j = 0; j < 2; ++j) {   // 16 bytes of hi halves and of lo halves each; 64-byte swizzle
        uint32_t hi[4], lo[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const int t = 8 * j + 2 * k;
          split_pair(es[t * ROWS] * pw[t] * to, es[(t + 1) * ROWS] * pw[t + 1] * to, hi[k], lo[k]);
        }
        const uint32_t at = eop + ((uint32_t)(j ^ ((r >> 1) & 3)) << 4), at2 = eop + ((uint32_t)((j + 2) ^ ((r >> 1) & 3)) << 4);
        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(at), "r"(hi[0]), "r"(hi[1]), "r"(hi[2]), "r"(hi[3]) : "memory");
        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(at2), "r"(lo[0]), "r"(lo[1]), "r"(lo[2]), "r"(lo[3]) : "memory");
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) bar_arrive(smem_u32(&s_opr[m]));
    }
  };
  auto out_role = [&] {
    // ---- errors of 32 rows: out for the trailing product, into the losses
    const int r = (warp - S::kOut) * 32 + lane;
    const int64_t row = row0 + r;
    const bool live = row < p.N, out = p.err && live;   // (a superblock with columns after it is a whole one)
    float loss = 0.0f;
#pragma unroll 1
    for (int m = 0; m < micros; ++m) {
      const bool from = ROWS == 32 && p.W0 && out;   // (wider CTAs are never given the blocked form)
      uint4 w0[kMicro / 4];   // asked for before the wait
      if (from) {
        const bool half = p.w0dtype == B200Q_BF16;
        const int64_t col = row * p.ld0 + p.i1 + m * kMicro;
        const uint4* src = reinterpret_cast<const uint4*>((const char*)p.W0 + (half ? 2 : 4) * col);
        w0[0] = src[0]; w0[1] = src[1];
        if (!half) {
          w0[2] = src[2]; w0[3] = src[3];
        } else {
          auto wide = [](uint32_t a, uint32_t b) { return make_uint4(a << 16, a & 0xFFFF0000u, b << 16, b & 0xFFFF0000u); };
          const uint4 a = w0[0], b = w0[1];
          w0[0] = wide(a.x, a.y); w0[1] = wide(a.z, a.w); w0[2] = wide(b.x, b.y); w0[3] = wide(b.z, b.w);
        }
      }
      bar_wait(smem_u32(&s_done[2 * m + 1]), 0, &s_abort);
      const float* es = sE + (m & (kErrSlots - 1)) * kMicro * ROWS + r;
      const int64_t at = job * p.err_batch + row * p.lde + m * kMicro;
      float sum = 0.0f;
#pragma unroll 1
      for (int t = 0; t < kMicro; t += 4) {
        float x[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          x[k] = -es[(t + k) * ROWS];
          sum = fmaf(x[k], x[k], sum);
        }
        if (out && !from) *reinterpret_cast<float4*>(p.err + at + t) = make_float4(x[0], x[1], x[2], x[3]);
      }
      if (from) {
        const float* q = sW + m * kMicro * S::kWld + r;
#pragma unroll
        for (int k = 0; k < kMicro / 4; ++k)
          *reinterpret_cast<float4*>(p.err + at + 4 * k) =
              make_float4(__uint_as_float(w0[k].x) - q[4 * k * S::kWld], __uint_as_float(w0[k].y) - q[(4 * k + 1) * S::kWld],
                          __uint_as_float(w0[k].z) - q[(4 * k + 2) * S::kWld], __uint_as_float(w0[k].w) - q[(4 * k + 3) * S::kWld]);
      }
      __syncwarp();
      if (lane == 0) bar_arrive(smem_u32(&s_out[m]));
      loss += sum;   // (512 terms one after the other: 3.0e-7 off at K = 520, this way 0.9e-7)
    }
    if (live) {
      float* losses = p.losses.at(job);
      const float half = loss * 0.5f;
      losses[row] = p.i1 == 0 ? half : losses[row] + half;
    }
  };
  auto param_role = [&] {
    // ---- parameters of the rows, up to four micro-blocks ahead; copies of U: tiles (a stage per micro-block), bands
    const void* scale = p.scale.at(job);
    const void* zp = p.zp.at(job);
    const float* gs = p.gscale.at(job);
    const int32_t* col_group = p.col_group.at(job);
    const float g = gs ? *gs : 1.0f;
    const bool per_column = p.strategy != B200Q_TENSOR && p.strategy != B200Q_CHANNEL;
    int64_t pbase[S::kChains];
#pragma unroll
    for (int h = 0; h < S::kChains; ++h) {
      const int64_t row = min(row0 + h * 32 + lane, p.N - 1);
      pbase[h] = p.strategy == B200Q_CHANNEL ? row : p.strategy == B200Q_BLOCK ? (row / p.block_h) * p.groups_per_row
                 : p.strategy == B200Q_TENSOR ? 0 : row * p.groups_per_row;
    }
    auto load = [&](int64_t pi, float& s, float& z) {
      s = p.sdtype == B200Q_BF16 ? __bfloat162float(((const __nv_bfloat16*)scale)[pi]) : ((const float*)scale)[pi];
      z = ZP ? load_zp(zp, p.zp_kind, pi) : 0.0f;
    };
    auto groups = [&](int k) -> int {   // of column lane % 16 of micro-block k (columns beyond the superblock: of the last)
      if (!per_column) return 0;
      const int col = p.i1 + min(k * kMicro + (lane & 15), sb - 1);
      return col_group ? col_group[col] : col / p.group_size;
    };
    // asked for a micro-block ahead: the groups, and scale and zero point at the group of the first column
    int grp = groups(0), now = 0;
    float s1[S::kChains], z1[S::kChains];
    auto ask = [&](int k) {
      now = grp;
#pragma unroll
      for (int h = 0; h < S::kChains; ++h) load(pbase[h] + __shfl_sync(0xffffffffu, now, 0), s1[h], z1[h]);
      grp = groups(k + 1);
    };
    auto load_step = [&](int m) {
      if (!has_u || m >= steps) return;
      const int stage = m % S::kStages;
      if (m >= S::kStages) bar_wait(smem_u32(&s_empty[stage]), (uint32_t)(m / S::kStages - 1) & 1u, &s_abort);
      if (lane == 0 && !s_abort) {
        // (rows of columns that are past stay as they are: nobody takes their sums)
        const int first = first_block(m);
        const uint32_t bar = smem_u32(&s_full[stage]), skip = ((m + kLag) * kMicro - first * kBlockCols) * kRowBytes;
        const uint32_t dst = smem_u32(sm + S::kRing + stage * S::kStageBytes);
        const unsigned char* src = tiles + m * S::kStageBytes;
        const uint32_t begin = first * kTileBytes + skip, bytes = blocks * kTileBytes - begin;
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
        bulk_copy(dst + begin, src + begin, bytes, bar);
      }
      __syncwarp();
    };
    auto load_band = [&](int k) {
      if (k >= micros) return;
      if (k >= kSlots) {   // the feeders are through with the slot
        bar_wait(smem_u32(&s_ready[2 * k - 4]), 0, &s_abort);
        bar_wait(smem_u32(&s_ready[2 * k - 3]), 0, &s_abort);
      }
      if (lane == 0 && !s_abort) {
        const uint32_t bar = smem_u32(&s_par[k]);
        if (has_u) {
          asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(kBandFloats * 4) : "memory");
          bulk_copy(smem_u32(sBand + (k & (kSlots - 1)) * kBandFloats),
                    tiles + band_offset(SBLK) + (int64_t)k * kBandFloats * 4, kBandFloats * 4, bar);
        } else {
          bar_arrive(bar);
        }
      }
      __syncwarp();
    };
    if (!has_u)
      for (int i = lane; i < kSlots * kBandFloats; i += 32) {
        const int k = i % kBandFloats;
        sBand[i] = k >= kMicro * kBandCols || k / kBandCols == k % kBandCols ? 1.0f : 0.0f;
      }
    __syncwarp();
    for (int k = 0; k < kSlots - 1; ++k) load_band(k);
    for (int k = 0; k < S::kStages; ++k) load_step(k);
    ask(0);
#pragma unroll 1
    for (int k = 0; k < micros; ++k) {
      const int slot = k & (kSlots - 1);
      if (k >= kSlots) {   // the chain and the other readers of the slots are through with them
        bar_wait(smem_u32(&s_done[2 * (k - kSlots) + 1]), 0, &s_abort);
        bar_wait(smem_u32(&s_out[k - kSlots]), 0, &s_abort);
      }
      const bool same = __all_sync(0xffffffffu, now == __shfl_sync(0xffffffffu, now, 0));
#pragma unroll
      for (int h = 0; h < S::kChains; ++h) {
        const int r = h * 32 + lane;
        const bool live = row0 + r < p.N;
        bool odd = false;
        auto put = [&](int t, float s, float z) {   // the effective scale and its reciprocal
          if (!live) { s = 1.0f; z = 0.0f; }
          else if (gs) s = __fdiv_rn(s, g);
          odd |= !(s >= 0x1p-100f && s <= 0x1p100f);
          sPar[(slot * kMicro + t) * ROWS + r] = make_float2(s, __frcp_rn(s));
          if (ZP) sZ[(slot * kMicro + t) * ROWS + r] = z;
        };
        if (same) {
          put(0, s1[h], z1[h]);
          const float2 sr = sPar[slot * kMicro * ROWS + r];
          const float z = ZP ? sZ[slot * kMicro * ROWS + r] : 0.0f;
#pragma unroll 5
          for (int t = 1; t < kMicro; ++t) {
            sPar[(slot * kMicro + t) * ROWS + r] = sr;
            if (ZP) sZ[(slot * kMicro + t) * ROWS + r] = z;
          }
        } else {
#pragma unroll 1
          for (int t0 = 0; t0 < kMicro; t0 += 4) {
            float s[4], z[4];
#pragma unroll
            for (int t = 0; t < 4; ++t) load(pbase[h] + __shfl_sync(0xffffffffu, now, t0 + t), s[t], z[t]);
#pragma unroll 1
            for (int t = 0; t < 4; ++t) put(t0 + t, t == 0 ? s[0] : t == 1 ? s[1] : t == 2 ? s[2] : s[3],
                                            t == 0 ? z[0] : t == 1 ? z[1] : t == 2 ? z[2] : z[3]);
          }
        }
        odd = __any_sync(0xffffffffu, odd);
        if (lane == 0) s_odd[h][slot] = odd;
      }
      __syncwarp();
      if (lane == 0) bar_arrive(smem_u32(&s_par[k]));
      ask(k + 1);
      if (k - 1 >= S::kStages) load_step(k - 1);
      if (k - 1 >= kSlots - 1) load_band(k - 1);
    }
    if (micros - 1 >= kSlots - 1) load_band(micros - 1);
  };
  auto mma_role = [&] {
    // ---- MMAs
#pragma unroll 1
    for (int m = 0; m < steps; ++m) {
      {
        const int first = first_block(m);
        for (int b = first; b < blocks; ++b) bar_spin(smem_u32(&s_acce[m & 1][b]), ((uint32_t)(m >> 1) & 1u) ^ 1u, &s_abort);
        if (has_u) bar_spin(smem_u32(&s_full[m % S::kStages]), (uint32_t)(m / S::kStages) & 1u, &s_abort);
        bar_spin(smem_u32(&s_opr[m]), 0, &s_abort);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if (lane == 0) {
          constexpr uint32_t lo = kRowBytes / 2;
          const uint64_t e_hi = make_desc(smem_u32(sm + S::kErr + (m & 1) * S::kErrBytes)), e_lo = e_hi + (lo >> 4);
          uint64_t u_hi = make_desc(smem_u32(sm + S::kRing + (m % S::kStages) * S::kStageBytes + first * kTileBytes));
          uint32_t d = tmem + (uint32_t)((m & 1) * 256 + first * 2 * ROWS);
#pragma unroll 1
          for (int b = first; b < blocks; ++b, d += 2 * ROWS, u_hi += kTileBytes >> 4) {
            if (has_u) {   // hi * hi, and beside it hi * lo + lo * hi
              mma_f16(d, u_hi, e_hi, instr_desc(ROWS), 0u);
              mma_f16(d + ROWS, u_hi, e_lo, instr_desc(ROWS), 0u);
              mma_f16(d + ROWS, u_hi + (lo >> 4), e_hi, instr_desc(ROWS), 1u);
              tc_commit(smem_u32(&s_accf[m & 1][b]));
            } else {       // (nothing to add: the helpers still follow the steps)
              bar_arrive(smem_u32(&s_accf[m & 1][b]));
            }
          }
          if (has_u) tc_commit(smem_u32(&s_empty[m % S::kStages]));
        }
        __syncwarp();
      }
    }
  };
  if (warp >= S::kFirstHelper) {
    if constexpr (ROWS == 32) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(Regs<ROWS>::kHelper));
    else asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(Regs<ROWS>::kHelper));
    helper_role();
  } else if (warp < 4) {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(Regs<ROWS>::kChain));
    if (warp < S::kChains) chain_role();
    else if (warp >= S::kErrors && warp < S::kErrors + S::kChains) error_role();
    else if (ROWS == 32) feeder_role();
  } else if (ROWS == 64 && warp < 8) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(Regs<ROWS>::kFeeder));
    feeder_role();
  } else {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(Regs<ROWS>::kOther));
    if (warp == S::kMma) mma_role();
    else if (warp >= S::kOut && warp < S::kParams) out_role();
    else if (warp == S::kParams) param_role();
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (s_abort) {
    if (tid == 0 && p.status) atomicCAS(p.status, 0, B200Q_ERR_DEVICE);
    const long long t0 = clock64();
    while (clock64() - t0 < 2000000LL) __nanosleep(1000);   // copies in flight land
  }
  if (warp == S::kMma) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
  }
}

// Superblock width, rows of a CTA.  32 rows a CTA and 512 columns while that gives every CTA an SM of its own; more rows
// are carried 64 a CTA (two chains, the operand tiles of U read once for both), whose share of the superblock fits the
// helpers' registers up to 256 columns.
static bool wide(int64_t N, int batch) { return (N + 31) / 32 * batch <= kNumSMs; }
// The trailing product is split in the columns the next superblock needs and the rest on a helper stream only while
// a superblock's CTAs leave half of the GPU idle.
static bool look_ahead(int64_t ctas) { return ctas <= kNumSMs / 2; }

struct Layout {
  int rows, sb, sets;
  int64_t ctas, rows_n, rows_k, err, ub;   // CTAs, rows per problem of the operands; elements of the errors and of U's slice
  int64_t tiles;                           // bytes of the tiles of all factors
  size_t set;                              // bytes of a set: errors, their halves and scales, the slice's, the tiles
  size_t bytes;
};
static Layout layout_of(int64_t N, int64_t K, int batch, int distinct_u, bool may_overlap) {
  Layout l;
  l.rows = wide(N, batch) ? 32 : 64;
  l.sb = l.rows == 32 ? 512 : 256;
  l.ctas = (N + l.rows - 1) / l.rows;
  l.sets = may_overlap && K > l.sb ? 2 : 1;
  l.rows_n = (N + 127) / 128 * 128; l.rows_k = (K + 127) / 128 * 128;
  l.err = K > l.sb ? l.rows_n * l.sb * batch : 0; l.ub = K > l.sb ? l.rows_k * l.sb * distinct_u : 0;
  l.tiles = tiles_bytes(l.sb) * distinct_u;
  l.set = (size_t)(2 * l.err + l.ub + (l.err + l.ub) / l.sb) * sizeof(float) + (size_t)l.tiles;
  l.bytes = kSweepHeaderBytes + l.sets * l.set + 64;
  return l;
}

typedef void (*Kernel)(const Params);
template <int ROWS, int SBLK, bool SB, int KIND> static Kernel pick_zp(bool zp) {
  return zp ? sweep_block_kernel<ROWS, SBLK, SB, KIND, true> : sweep_block_kernel<ROWS, SBLK, SB, KIND, false>;
}
template <int ROWS, int SBLK, bool SB> static Kernel pick_kind(int kind, bool zp) {
  return kind == kInt ? pick_zp<ROWS, SBLK, SB, kInt>(zp)
                      : kind == kFp8 ? pick_zp<ROWS, SBLK, SB, kFp8>(zp) : pick_zp<ROWS, SBLK, SB, kFp4>(zp);
}
static Kernel pick_kernel(int rows, bool bf16_values, int kind, bool zp) {
  if (rows == 32) return bf16_values ? pick_kind<32, 512, true>(kind, zp) : pick_kind<32, 512, false>(kind, zp);
  return bf16_values ? pick_kind<64, 256, true>(kind, zp) : pick_kind<64, 256, false>(kind, zp);
}

// `Ud` / `u_index`: the distinct factors of a batch and the one each problem uses (null: the single U, or one each)
static int sweep(Params p, int sdtype, bool global, int batch, const float* const* Ud, int distinct_u,
                 const int32_t* u_index, bool may_overlap, void* workspace, cudaStream_t st) {
  const int64_t N = p.N, K = p.K;
  const bool has_u = p.U.one || p.U.table;
  const Layout l = layout_of(N, K, batch, distinct_u, may_overlap);
  const bool blocks = p.W0 != nullptr;
  // header of the workspace: a status word that a bounded wait expiring in a sweep or a trailing product sets to
  // B200Q_ERR_DEVICE (cleared here, read by the caller afterwards)
  int* status = (int*)workspace;
  struct Set { float* err; __half *e_hi, *e_lo, *u_hi, *u_lo; float *e_scale, *u_scale; unsigned char* tiles; };
  auto set = [&](int which) {
    Set t;
    t.err = (float*)((char*)workspace + kSweepHeaderBytes + which * l.set);
    t.e_hi = (__half*)(t.err + l.err); t.e_lo = t.e_hi + l.err;
    t.u_hi = t.e_lo + l.err; t.u_lo = t.u_hi + l.ub;
    t.e_scale = (float*)(t.u_lo + l.ub); t.u_scale = t.e_scale + l.err / l.sb;
    t.tiles = (unsigned char*)(t.u_scale + l.ub / l.sb);
    return t;
  };
  B200Q_TRY(cudaMemsetAsync(status, 0, sizeof(int), st));
  if (sdtype != B200Q_BF16 && sdtype != B200Q_F32) return B200Q_ERR_UNSUPPORTED;
  p.sdtype = sdtype; p.status = status; p.u_index = u_index; p.tiles_batch = tiles_bytes(l.sb);
  const bool with_zp = p.zp.one || p.zp.table, bf16_values = sdtype == B200Q_BF16 && !global;
  const Kernel kern = pick_kernel(l.rows, bf16_values, p.qr.kind, with_zp);
  const size_t smem = l.rows == 32 ? Shape<32, 512>::kSmem : Shape<64, 256>::kSmem;
  const int threads = l.rows == 32 ? Shape<32, 512>::kThreads : Shape<64, 256>::kThreads;
  B200Q_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  // A single weight makes the next superblock's slice of U beside the sweep, and with few rows the far columns'
  // product beside the sweep after it.
  tgemm::SideStream* side = l.sets == 2 && has_u ? tgemm::side_stream(st) : nullptr;
  const bool far_beside = side && look_ahead(l.ctas * batch);
  int rc;
  // the operand forms of U that superblock i1 needs: of its square, and of U[i1 : i1 + sb, i1 + sb :] for the trailing
  // product (row = column, contraction contiguous)
  Ptr<const float> factors = p.U;
  if (Ud) factors = {nullptr, Ud};
  auto square = l.sb == 512 ? square_tiles_kernel<512> : square_tiles_kernel<256>;
  const size_t square_smem = tgemm::split_columns16_smem(l.sb);
  B200Q_TRY(cudaFuncSetAttribute(square, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)square_smem));
  auto split_u = [&](int64_t i1, int which, bool tiles, bool rest, cudaStream_t on) -> int {
    const int w = (int)(K - i1 < l.sb ? K - i1 : l.sb), squares = tiles ? (w + 31) / 32 : 0;
    const int64_t cols = rest ? K - i1 - w : 0;
    const Set t = set(which);
    if (squares + cols == 0) return B200Q_OK;
    B200Q_TRY(launch_chained(square, dim3((unsigned)(squares + (cols + 31) / 32), distinct_u), kTileThreads, square_smem, on, factors,
                             p.ldu, (int)i1, w, t.tiles, p.tiles_batch, squares,
                             Slice{t.u_hi, t.u_lo, t.u_scale, cols, l.rows_k, blocks}));
    B200Q_LAUNCH_CHECK();
    return B200Q_OK;
  };
  if (has_u && side) {   // the first slice beside the first superblock, which needs its square only
    B200Q_TRY(cudaEventRecord(side->next, st));
    B200Q_TRY(cudaStreamWaitEvent(side->stream, side->next, 0));
    if ((rc = split_u(0, 0, true, false, st)) || (rc = split_u(0, 0, false, true, side->stream))) return rc;
  } else if (has_u && (rc = split_u(0, 0, true, true, st))) {
    return rc;
  }
  int blk = 0;
  for (int64_t i1 = 0; i1 < K; i1 += l.sb, ++blk) {
    const int w = (int)(K - i1 < l.sb ? K - i1 : l.sb), which = l.sets == 2 ? blk & 1 : 0;
    const int64_t i2 = i1 + w;
    const bool trailing = i2 < K && has_u;
    const Set t = set(which);
    p.i1 = (int)i1; p.sb = w;
    p.err = trailing ? t.err : nullptr;
    p.tiles = t.tiles; p.lde = l.sb; p.err_batch = l.rows_n * l.sb;
    if (trailing && side) {
      // the next superblock's slice of U: its buffer was last read by the products of the superblock before this one
      B200Q_TRY(cudaEventRecord(side->next, st));
      B200Q_TRY(cudaStreamWaitEvent(side->stream, side->next, 0));
      if ((rc = split_u(i2, which ^ 1, true, true, side->stream))) return rc;
      B200Q_TRY(cudaEventRecord(side->done, side->stream));
    }
    B200Q_TRY(launch_chained(kern, dim3((unsigned)l.ctas, batch), threads, smem, st, p));
    B200Q_LAUNCH_CHECK();
    if (!trailing) continue;
    // W[:, i2:] -= Err[N, w] * U[i1:i2, i2:].  What of this superblock's U the helper stream made, this stream may read
    // behind its wait for side->done only: the slice below.  The powers of the pivots come with the square's tiles, the
    // first of which are this stream's own; the others were waited for before the product of the superblock before.
    if ((rc = tgemm::split_rows16(t.err, l.sb, p.err_batch, N, w, t.e_hi, t.e_lo, t.e_scale, l.sb, l.rows_n, batch,
                                  (const float*)(t.tiles + powers_offset(l.sb)), blocks, p.tiles_batch / 4, u_index, st)))
      return rc;
    tgemm::Job j;
    j.A = tgemm::Operand{t.e_hi, t.e_lo, l.sb, l.rows_n * batch, l.rows_n, 0, t.e_scale};
    j.B = tgemm::Operand{t.u_hi, t.u_lo, l.sb, l.rows_k * distinct_u, l.rows_k, 0, t.u_scale};
    j.b_index = u_index;
    j.M = (int)N; j.N = (int)(K - i2); j.Kd = w; j.batch = batch; j.alpha = -1.0f; j.beta = 1.0f;
    if (p.W.one) j.C = p.W.one + i2;
    j.c_table = p.W.table; j.c_offset = i2; j.ldc = p.ldw; j.status = status;
    // (measured where they are defined)
    j.slice = p.W.table ? tgemm::kShortSlice16 : tgemm::kLongSlice16;
    if (!side) {
      if ((rc = tgemm::launch(j, st))) return rc;
      if ((rc = split_u(i2, l.sets == 2 ? which ^ 1 : 0, true, true, st))) return rc;
      continue;
    }
    tgemm::Job far = j;
    if (far_beside) {
      if (j.N > l.sb) j.N = l.sb;
      B200Q_TRY(cudaEventRecord(side->ready, st));
      B200Q_TRY(cudaStreamWaitEvent(side->stream, side->ready, 0));
    }
    // the far columns of the superblock before, and the next slice of U, made behind them
    B200Q_TRY(cudaStreamWaitEvent(st, side->done, 0));
    if ((rc = tgemm::launch(j, st))) return rc;
    if (far_beside && far.N > l.sb) {   // (waited for with the slice of U that the next round makes)
      far.B.row0 += l.sb; far.N -= l.sb; far.max_ctas = kNumSMs - (int)l.ctas * batch;
      if (p.W.one) far.C = p.W.one + i2 + l.sb;
      far.c_offset = i2 + l.sb;
      if ((rc = tgemm::launch(far, side->stream))) return rc;
    }
  }
  return B200Q_OK;
}

static int fill_scheme(Params* p, const b200q_qargs* qa, int64_t N, int64_t K, const int32_t* col_group) {
  int rc = make_qrange(qa, &p->qr); if (rc) return rc;
  ParamMap pm;
  rc = make_param_map(qa, N, K, col_group, &pm); if (rc) return rc;
  p->strategy = qa->strategy;
  p->group_size = (qa->strategy == B200Q_BLOCK) ? qa->block_w : qa->group_size;
  if (p->group_size <= 0) p->group_size = 1;
  p->block_h = qa->block_h > 0 ? qa->block_h : 1;
  p->zp_kind = qa->zp_kind;
  p->groups_per_row = pm.groups_per_row;
  return B200Q_OK;
}

}  // namespace sweep
}  // namespace b200q

using namespace b200q;

extern "C" {

size_t b200q_gptq_sweep_workspace_bytes(int64_t N, int64_t K, int blocksize) {
  if (N <= 0 || K <= 0 || blocksize <= 0) return 0;
  return sweep::layout_of(N, K, 1, 1, true).bytes;
}

int b200q_gptq_sweep_takes_blocks(int64_t N, int64_t K) { return N > 0 && sweep::wide(N, 1) && K > 512; }

static int sweep_one(float* Wf, int64_t N, int64_t K, int64_t ldf, const float* U, int64_t ldu, const void* scale,
                     int sdtype, const void* zp, const int32_t* col_group, const float* gscale,
                     const b200q_qargs* qa, int blocksize, float* losses, const void* W0, int w0dtype, int64_t ld0,
                     void* workspace, void* stream) {
  using namespace b200q::sweep;
  if (!Wf || !scale || !qa || !losses || !workspace || N <= 0 || K <= 0 || ldf < K) return B200Q_ERR_ARG;
  if (U && ldu < K) return B200Q_ERR_ARG;
  if (((uintptr_t)workspace) & 15) return B200Q_ERR_ARG;
  if (blocksize <= 0 || blocksize > kMaxBlock) return B200Q_ERR_UNSUPPORTED;
  Params p;
  int rc = fill_scheme(&p, qa, N, K, col_group); if (rc) return rc;
  p.W = {Wf, nullptr}; p.U = {U, nullptr}; p.scale = {scale, nullptr}; p.zp = {zp, nullptr};
  p.col_group = {col_group, nullptr}; p.gscale = {gscale, nullptr}; p.losses = {losses, nullptr};
  p.N = N; p.K = K; p.ldw = ldf; p.ldu = ldu; p.W0 = W0; p.w0dtype = w0dtype; p.ld0 = ld0;
  return sweep::sweep(p, sdtype, gscale != nullptr, 1, nullptr, 1, nullptr, true, workspace, (cudaStream_t)stream);
}

int b200q_gptq_sweep(float* Wf, int64_t N, int64_t K, int64_t ldf, const float* U, int64_t ldu, const void* scale,
                     int sdtype, const void* zp, const int32_t* col_group, const float* gscale,
                     const b200q_qargs* qa, int blocksize, float* losses, void* workspace, void* stream) {
  return sweep_one(Wf, N, K, ldf, U, ldu, scale, sdtype, zp, col_group, gscale, qa, blocksize, losses, nullptr, 0, 0, workspace, stream);
}

int b200q_gptq_sweep_blocks(float* Wf, int64_t N, int64_t K, int64_t ldf, const void* W0, int w0dtype, int64_t ld0,
                            const float* F, int64_t ldu, const void* scale, int sdtype, const void* zp, const int32_t* col_group, const float* gscale,
                            const b200q_qargs* qa, int blocksize, float* losses, void* workspace, void* stream) {
  if (!F || !W0 || !b200q_gptq_sweep_takes_blocks(N, K) || ld0 < K || (ld0 & 7) || ((uintptr_t)W0 & 15)) return B200Q_ERR_ARG;
  if (w0dtype != B200Q_BF16 && w0dtype != B200Q_F32) return B200Q_ERR_UNSUPPORTED;
  return sweep_one(Wf, N, K, ldf, F, ldu, scale, sdtype, zp, col_group, gscale, qa, blocksize, losses, W0, w0dtype, ld0,
                   workspace, stream);
}

size_t b200q_gptq_sweep_many_workspace_bytes(int64_t N, int64_t K, int count, int distinct) {
  if (N <= 0 || K <= 0 || count <= 0 || distinct <= 0) return 0;
  return sweep::layout_of(N, K, count, distinct, false).bytes;
}

int b200q_gptq_sweep_many(float* const* W, const float* const* U, const float* const* distinct_u, int distinct,
                          const int32_t* u_index, const void* const* scale, int sdtype, const void* const* zp,
                          const int32_t* const* col_group, const float* const* gscale, float* const* losses, int count,
                          int64_t N, int64_t K, int64_t ldw, int64_t ldu, const b200q_qargs* qa, void* workspace,
                          void* stream) {
  using namespace b200q::sweep;
  if (!W || !scale || !losses || !qa || !workspace || count <= 0 || N <= 0 || K <= 0 || ldw < K || (U && ldu < K)) return B200Q_ERR_ARG;
  if (count > 65535 || (U && (!distinct_u || distinct <= 0 || distinct > 65535)) || ((uintptr_t)workspace) & 15) return B200Q_ERR_ARG;
  Params p;
  int rc = fill_scheme(&p, qa, N, K, nullptr); if (rc) return rc;
  p.W0 = nullptr;
  p.W = {nullptr, W}; p.U = {nullptr, U}; p.scale = {nullptr, scale}; p.zp = {nullptr, zp};
  p.col_group = {nullptr, col_group}; p.gscale = {nullptr, gscale}; p.losses = {nullptr, losses};
  p.N = N; p.K = K; p.ldw = ldw; p.ldu = ldu;
  return sweep::sweep(p, sdtype, gscale != nullptr, count, distinct_u, U ? distinct : 1, u_index, false, workspace,
                      (cudaStream_t)stream);
}

int b200q_gptq_sweep_batched(float* const* W, const float* const* U, const void* const* scale, int sdtype,
                             const void* const* zp, const int32_t* const* col_group, const float* const* gscale,
                             float* const* losses, int count, int64_t N, int64_t K, int64_t ldw, int64_t ldu,
                             const b200q_qargs* qa, int blocksize, void* stream) {
  if (count <= 0 || N <= 0 || K <= 0) return B200Q_ERR_ARG;
  if (blocksize != 128) return B200Q_ERR_UNSUPPORTED;
  // no workspace in this entry point's arguments: taken from the stream's memory pool for the call
  void* ws = nullptr;
  cudaStream_t st = (cudaStream_t)stream;
  B200Q_TRY(cudaMallocAsync(&ws, b200q_gptq_sweep_many_workspace_bytes(N, K, count, count), st));
  int rc = b200q_gptq_sweep_many(W, U, U, count, nullptr, scale, sdtype, zp, col_group, gscale, losses, count, N, K,
                                 ldw, ldu, qa, ws, stream);
  // the status word goes with the workspace: whatever it says by then is kept for b200q_take_wait_status
  if (rc == B200Q_OK) rc = b200q_note_wait_status((const int*)ws, stream);
  B200Q_TRY(cudaFreeAsync(ws, st));
  return rc;
}

}  // extern "C"
