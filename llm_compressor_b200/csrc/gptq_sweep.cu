// GPTQ solve, part 2: the column sweep, for one weight or a batch of weights of one shape.
//
// Rows of W are independent and the columns of a row form one dependent chain: quantise column i, divide the error
// by U[i,i], subtract its multiple of U[i, i+1:] from the rest of the row.  The columns are taken in superblocks of
// up to 512.  Inside one, a CTA carries 32 rows through all columns with everything in shared memory
// (sweep_block_kernel); between superblocks the rest of the matrix takes W[:, after] -= Err * U[block, after] as one
// fp32-accurate tensor-core product (tgemm).  What the reference calls its block size only orders float32 operations
// and does not change the result otherwise, so it does not decide the split here.
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
constexpr int kRows = 32;                    // rows of a CTA: a lane each
constexpr int kMicro = 16;                   // columns a lane keeps in registers at a time
// 12 warps where a CTA has its SM to itself, 8 where two share one
constexpr int warps_of(int superblock) { return superblock == 512 ? 12 : 8; }
constexpr int WLD = kRows + 4, ELD = kRows + 8;   // columns of W and of the errors in shared memory: the strides
                                                  // make the MMA fragments' accesses conflict-free
__host__ __device__ constexpr int u_stride(int superblock) { return superblock + 8; }   // likewise

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
  float* err_hi; float* err_lo; int64_t lde, err_batch;   // operand form of the superblock's errors (null: nothing after it)
  int i1, sb;                                             // superblock: first column, width
  int sdtype;                                             // of the scales
  int* status;                                            // set if a bounded wait expires
};

__host__ __device__ constexpr size_t smem_bytes(int superblock) {
  return (size_t)(3 * kMicro * u_stride(superblock)   // rows of U of three micro-blocks
                  + 2 * 4 * kMicro * kRows            // parameters of two micro-blocks
                  + 2 * superblock                    // 1 / U[i,i], parameter column
                  + 32                                // one parameter column for all of a micro-block?
                  + 2 * kMicro * ELD                  // errors of two micro-blocks
                  + superblock * WLD) * sizeof(float);   // W, column-major
}

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void bulk_copy(float* dst, const float* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(smem_u32(dst)), "l"(src), "r"(bytes), "r"(bar) : "memory");
}
__device__ __forceinline__ bool bar_ready(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred P1;\n\tmbarrier.try_wait.parity.shared::cta.b64 P1, [%1], %2;\n\tselp.b32 %0, 1, 0, P1;\n\t}"
      : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
  return ok != 0;
}
__device__ __forceinline__ void fma2(uint64_t& d, uint64_t a, uint64_t b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
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

template <int KIND>
__device__ __forceinline__ float code_of(float v, float qmin, float qmax) {
  v = fminf(fmaxf(v, qmin), qmax);
  if constexpr (KIND == kInt) {
    return (v + 12582912.0f) - 12582912.0f;   // 1.5 * 2^23: rounds to nearest even (the sign of a zero is put back later)
  } else if constexpr (KIND == kFp8) {
    return e4m3_round(v);
  } else {
    uint32_t h;   // through the hardware's E2M1 pair and back
    asm("{\n\t.reg .b8 b;\n\tcvt.rn.satfinite.e2m1x2.f32 b, %1, %1;\n\tcvt.rn.f16x2.e2m1x2 %0, b;\n\t}" : "=r"(h) : "f"(v));
    return __half2float(__ushort_as_half((unsigned short)(h & 0xFFFFu)));
  }
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

// three tf32 MMAs per product of hi / lo splits, as in tgemm
__device__ __forceinline__ void split_tf32(float x, uint32_t& hi, uint32_t& lo) {
  hi = (__float_as_uint(x) + 0x1000u) & 0xFFFFE000u;
  lo = (__float_as_uint(x - __uint_as_float(hi)) + 0x1000u) & 0xFFFFE000u;
}
__device__ __forceinline__ void mma_tf32(float (&c)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
  asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

// A micro-block's errors as MMA operand: rows of the CTA x columns of the micro-block, [row tile][k step]
struct ErrFrag { uint32_t hi[2][2][4], lo[2][2][4]; };
// `upto12`: only the first twelve columns exist yet
__device__ __forceinline__ void load_errors(const float* e, int lane, bool upto12, ErrFrag& f) {
  const float* ei = e + (lane & 3) * ELD + (lane >> 2);
#pragma unroll
  for (int y = 0; y < 2; ++y)
#pragma unroll
    for (int ks = 0; ks < 2; ++ks)
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const bool out = upto12 && ks == 1 && k >= 2;
        split_tf32(out ? 0.0f : ei[(ks * 8 + (k >> 1) * 4) * ELD + y * 16 + (k & 1) * 8], f.hi[y][ks][k], f.lo[y][ks][k]);
      }
}
// W[32 rows, 16 columns] -= E[32, 16] U[16, 16 columns]; `w`, `u`: the first of the columns
template <int ULD>
__device__ __forceinline__ void apply_errors(const ErrFrag& f, const float* u, float* w, int lane) {
  float* o = w + 2 * (lane & 3) * WLD + (lane >> 2);
  const float* ub = u + (lane & 3) * ULD + (lane >> 2);
  float old[2][2][4], acc[2][2][4] = {}, part[2][2][4] = {};   // [row tile][column tile]
#pragma unroll
  for (int y = 0; y < 2; ++y)
#pragma unroll
    for (int x = 0; x < 2; ++x)
#pragma unroll
      for (int k = 0; k < 4; ++k) old[y][x][k] = o[(x * 8 + (k & 1)) * WLD + y * 16 + (k >> 1) * 8];
#pragma unroll
  for (int ks = 0; ks < 2; ++ks) {
    uint32_t bh[2][2], bl[2][2];
#pragma unroll
    for (int x = 0; x < 2; ++x)
#pragma unroll
      for (int k = 0; k < 2; ++k) split_tf32(ub[(ks * 8 + k * 4) * ULD + x * 8], bh[x][k], bl[x][k]);
#pragma unroll
    for (int y = 0; y < 2; ++y)
#pragma unroll
      for (int x = 0; x < 2; ++x) mma_tf32(acc[y][x], f.hi[y][ks], bh[x]);
#pragma unroll
    for (int y = 0; y < 2; ++y)
#pragma unroll
      for (int x = 0; x < 2; ++x) mma_tf32(part[y][x], f.hi[y][ks], bl[x]);
#pragma unroll
    for (int y = 0; y < 2; ++y)
#pragma unroll
      for (int x = 0; x < 2; ++x) mma_tf32(part[y][x], f.lo[y][ks], bh[x]);
  }
#pragma unroll
  for (int y = 0; y < 2; ++y)
#pragma unroll
    for (int x = 0; x < 2; ++x)
#pragma unroll
      for (int k = 0; k < 4; ++k)
        o[(x * 8 + (k & 1)) * WLD + y * 16 + (k >> 1) * 8] = old[y][x][k] - (acc[y][x][k] + part[y][x][k]);
}

// What bounds it: the chain of columns.  Its dependent instructions (product with 1 / s, clamp, round, dequantise,
// difference, product with the reciprocal pivot, correction of the next column) come to some 60 cycles a column by their
// latencies; measured it takes 308 (512 columns in 86.5 us at 1.82 GHz, 4096 rows), and where the rest goes has not been
// measured.  So one warp of the CTA does nothing but the chain: 16 columns at a time in registers, a lane per row.  Others apply a finished micro-block's
// 16 errors to the columns two micro-blocks on and later as warp-level tensor-core products (a float32 FMA formulation
// spends its time on the broadcast loads of U: 480 cycles a column against the chain's own), taking tasks of 16 columns
// from a counter.  The columns next in line take the first twelve errors from a warp that waits for them while the chain
// is on the last four, and those four from the chain warp.  Duties beside that: the warps that share the chain warp's
// scheduler ask for rows of U by bulk copies (as per-thread copies they block the warps that issue them: all CTAs want
// the same rows at the same time), and take tasks only while these, not the chain, decide; warp 5 fetches parameters,
// warp 6 writes the errors out as the operand of the trailing product.  One barrier per micro-block.  Every role is a
// latency-bound stream of instructions, a quarter of its stalls instruction fetch, hence short loops rather than
// unrolled code off the chain.
template <int SBLK, bool SB, int KIND, bool ZP>
__global__ void __launch_bounds__(32 * warps_of(SBLK), SBLK == 512 ? 1 : 2) sweep_block_kernel(const __grid_constant__ Params p) {
  const float qmin = p.qr.qmin, qmax = p.qr.qmax;
  chain_wait();
  extern __shared__ __align__(16) float sm[];
  constexpr int ULD = u_stride(SBLK);
  constexpr int NW = warps_of(SBLK), NT = 32 * NW;
  constexpr int kNextWarp = NW > 8 ? 9 : 1;            // brings the next micro-block's columns up to date
  constexpr int kHead = 12;                            // its share of a micro-block's errors
  float* sU = sm;                                      // [3][kMicro][ULD]
  float* sP = sU + 3 * kMicro * ULD;                   // [2][scale, low and high 1 / scale, zero point][kMicro][kRows]
  float* sRd = sP + 2 * 4 * kMicro * kRows;            // [SBLK]
  int* sGrp = reinterpret_cast<int*>(sRd + SBLK);      // [SBLK]
  int* sSame = sGrp + SBLK;                            // [32]
  float* sE = sRd + 2 * SBLK + 32;                     // [2][kMicro][ELD]
  float* sW = sE + 2 * kMicro * ELD;                   // [SBLK][WLD]
  __shared__ int s_odd;                                // some scale is outside the range the low / high test covers
  __shared__ int s_next[2];                            // next task of the helpers
  __shared__ __align__(8) uint64_t s_bar[3];           // rows of U of a micro-block have arrived
  const int job = blockIdx.y, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int sb = p.sb, micros = (sb + kMicro - 1) / kMicro;
  float* __restrict__ W = p.W.at(job) + p.i1;
  const float* __restrict__ U = p.U.at(job);
  if (U) U += (int64_t)p.i1 * p.ldu + p.i1;
  const int64_t row0 = (int64_t)blockIdx.x * kRows, row = row0 + lane;
  const bool live = row < p.N;
  const bool bulk = U && ((p.ldu & 3) == 0) && ((((uintptr_t)U) & 15) == 0) && (sb % kMicro) == 0;
  const bool vecw = ((p.ldw & 3) == 0) && ((((uintptr_t)W) & 15) == 0) && (sb & 3) == 0;
  // `ROWS` rows from t0 on of U's micro-block m, columns from its own first one on (columns beyond sb are zero).
  // Called by whole warps; with bulk copies one lane of each works, the one with t0 = 0 announces the bytes.
  auto fetch_u = [&](int m, int t0, auto ROWS) {
    float* dst = sU + (m % 3) * kMicro * ULD;
    const int c0 = m * kMicro, c_end = micros * kMicro;
    if (bulk) {
      if (lane == 0) {
        const uint32_t bytes = (uint32_t)(c_end - c0) * 4, bar = smem_u32(&s_bar[m % 3]);
        if (t0 == 0)
          asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes * kMicro) : "memory");
#pragma unroll
        for (int t = 0; t < ROWS; ++t)
          bulk_copy(dst + (t0 + t) * ULD + c0, U + (int64_t)(c0 + t0 + t) * p.ldu + c0, bytes, bar);
      }
      return;
    }
#pragma unroll 1
    for (int t = t0; t < t0 + ROWS; ++t) {
      const int i = c0 + t;
#pragma unroll 1
      for (int c = c0 + lane; c < c_end; c += 32) {
        float v = (i == c) ? 1.0f : 0.0f;
        if (U) v = (i < sb && c < sb) ? U[(int64_t)i * p.ldu + c] : 0.0f;
        dst[t * ULD + c] = v;
      }
    }
  };
  // a warp of twelve asks for half of a micro-block's rows, of eight for all
  constexpr std::integral_constant<int, NW == 12 ? kMicro / 2 : kMicro> kAskRows;
  auto wait_u = [&](int m) {
    if (!bulk) return;
    const uint32_t bar = smem_u32(&s_bar[m % 3]), parity = (uint32_t)(m / 3) & 1u;
    if (bar_ready(bar, parity)) return;
    const long long t0 = clock64();
    while (!bar_ready(bar, parity))
      if (clock64() - t0 > 4000000000LL) { atomicCAS(p.status, 0, B200Q_ERR_DEVICE); break; }
  };
  // parameters of micro-block m's columns for the CTA's rows, by one warp (columns beyond sb: unit scale)
  const void* scale = p.scale.at(job);
  const void* zp = p.zp.at(job);
  const float* gs = p.gscale.at(job);
  int64_t pbase;
  switch (p.strategy) {
    case B200Q_TENSOR: pbase = 0; break;
    case B200Q_CHANNEL: pbase = row; break;
    case B200Q_BLOCK: pbase = (row / p.block_h) * p.groups_per_row; break;
    default: pbase = row * p.groups_per_row; break;
  }
  auto fetch_params = [&](int m) {
    float* dst = sP + (m & 1) * 4 * kMicro * kRows + lane;
    const int c0 = m * kMicro;
    const bool same = sSame[m] != 0;
    const float g = gs ? *gs : 1.0f;
    auto put = [&](int t, float s) {
      if (gs) s = __fdiv_rn(s, g);
      const float rs = __frcp_rn(s);
      if (!(s >= 0x1p-100f && s <= 0x1p100f)) s_odd = 1;
      dst[t * kRows] = s;
      dst[(kMicro + t) * kRows] = rs * (1.0f - kMargin);
      dst[(2 * kMicro + t) * kRows] = rs * (1.0f + kMargin);
    };
    auto load = [&](int t, float& s, float& z) {
      s = 1.0f; z = 0.0f;
      if (c0 + t < sb && live) {
        const int64_t pi = pbase + sGrp[c0 + t];
        s = p.sdtype == B200Q_BF16 ? __bfloat162float(((const __nv_bfloat16*)scale)[pi]) : ((const float*)scale)[pi];
        if (ZP) z = load_zp(zp, p.zp_kind, pi);
      }
    };
    if (same) {
      float s, z;
      load(0, s, z);
      put(0, s);
      s = dst[0];
      const float lo = dst[kMicro * kRows], hi = dst[2 * kMicro * kRows];
#pragma unroll 4
      for (int t = 0; t < kMicro; ++t) {
        dst[t * kRows] = s;
        dst[(kMicro + t) * kRows] = lo;
        dst[(2 * kMicro + t) * kRows] = hi;
        if (ZP) dst[(3 * kMicro + t) * kRows] = z;
      }
    } else {
      float s[kMicro], z[kMicro];
#pragma unroll
      for (int t = 0; t < kMicro; ++t) load(t, s[t], z[t]);   // all of them on their way before the first is used
#pragma unroll
      for (int t = 0; t < kMicro; ++t) {
        dst[t * kRows] = s[t];
        if (ZP) dst[(3 * kMicro + t) * kRows] = z[t];
      }
#pragma unroll 1
      for (int t = 0; t < kMicro; ++t) put(t, dst[t * kRows]);
    }
  };
  if (tid == 32) {
    s_odd = 0; s_next[0] = s_next[1] = 0;
    for (int k = 0; k < 3; ++k) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&s_bar[k])) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    __syncwarp();
#pragma unroll 1
    for (int m = 0; m < micros && m < 2; ++m) fetch_u(m, 0, std::integral_constant<int, kMicro>());
  }
  const int32_t* col_group = p.col_group.at(job);
  for (int c = tid; c < micros * kMicro; c += NT) {
    float d = 1.0f;
    int grp = 0;
    if (c < sb) {
      if (U) d = U[(int64_t)c * p.ldu + c];
      const int col = p.i1 + c;
      grp = (p.strategy == B200Q_TENSOR || p.strategy == B200Q_CHANNEL) ? 0 : (col_group ? col_group[col] : col / p.group_size);
    }
    sRd[c] = __frcp_rn(d);
    sGrp[c] = grp;
  }
  // tile in: a lane per row, eight columns (a whole sector) at a time
  if (vecw) {
#pragma unroll 4
    for (int c = warp * 8; c < micros * kMicro; c += 8 * (NW)) {
      float4 v[2];
#pragma unroll
      for (int h = 0; h < 2; ++h)
        v[h] = (live && c + 4 * h < sb) ? *reinterpret_cast<const float4*>(W + row * p.ldw + c + 4 * h)
                                        : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        float* d = sW + (c + 4 * h) * WLD + lane;
        d[0] = v[h].x; d[WLD] = v[h].y; d[2 * WLD] = v[h].z; d[3 * WLD] = v[h].w;
      }
    }
  } else {
    for (int r = warp; r < kRows; r += NW) {
      const bool in = row0 + r < p.N;
      const float* src = W + (row0 + r) * p.ldw;
      for (int c = lane; c < micros * kMicro; c += 32) sW[c * WLD + r] = (in && c < sb) ? src[c] : 0.0f;
    }
  }
  __syncthreads();
  if (tid < micros) {
    bool same = true;
    for (int t = 1; t < kMicro; ++t) same = same && (tid * kMicro + t >= sb || sGrp[tid * kMicro + t] == sGrp[tid * kMicro]);
    sSame[tid] = same ? 1 : 0;
  }
  __syncthreads();
  if (warp == 5) fetch_params(0);
  wait_u(0);
  __syncthreads();

  float loss = 0.0f;   // of warp 6's rows, a lane each
  // the errors of micro-block `of`: their squares into the loss, and out as operand rows
  auto finish_errors = [&](int of) {
    const float* ei = sE + (of & 1) * kMicro * ELD + lane;
    float x[kMicro], sum = 0.0f;
#pragma unroll
    for (int t = 0; t < kMicro; ++t) { x[t] = ei[t * ELD]; sum = fmaf(x[t], x[t], sum); }
    loss += sum;   // (512 terms one after the other: 3.0e-7 off at K = 520, this way 0.9e-7)
    if (!p.err_hi || !live) return;
    const int64_t at = job * p.err_batch + row * p.lde + of * kMicro;
#pragma unroll
    for (int q = 0; q < kMicro; q += 4) {
      float h[4], l[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        h[k] = tgemm::tf32_rn(x[q + k]);
        l[k] = tgemm::tf32_rn(x[q + k] - h[k]);
      }
      *reinterpret_cast<float4*>(p.err_hi + at + q) = make_float4(h[0], h[1], h[2], h[3]);
      *reinterpret_cast<float4*>(p.err_lo + at + q) = make_float4(l[0], l[1], l[2], l[3]);
    }
  };
  float e[kMicro];
#pragma unroll
  for (int t = 0; t < kMicro; ++t) e[t] = 0.0f;
#pragma unroll 1
  for (int m = 0; m < micros; ++m) {
    const int c0 = m * kMicro;
    const float* u_prev = sU + ((m + 2) % 3) * kMicro * ULD;
    const float* u = sU + (m % 3) * kMicro * ULD + c0;
    if (warp == 0) {
      float* wcol = sW + c0 * WLD + lane;
      float* eo = sE + (m & 1) * kMicro * ELD + lane;
      const float* par = sP + (m & 1) * 4 * kMicro * kRows + lane;
      float w[kMicro];
      {
        // the last errors of the micro-block before this one
        uint64_t v[kMicro / 2];
#pragma unroll
        for (int k = 0; k < kMicro / 2; ++k) v[k] = pair(wcol[2 * k * WLD], wcol[(2 * k + 1) * WLD]);
        if (m > 0) {
#pragma unroll
          for (int t = kHead; t < kMicro; ++t) {
            const uint64_t ne = pair(-e[t], -e[t]);
#pragma unroll
            for (int k = 0; k < kMicro / 4; ++k) {
              const ulonglong2 uu = *reinterpret_cast<const ulonglong2*>(u_prev + t * ULD + c0 + 4 * k);
              fma2(v[2 * k], ne, uu.x);
              fma2(v[2 * k + 1], ne, uu.y);
            }
          }
        }
#pragma unroll
        for (int k = 0; k < kMicro / 2; ++k) unpair(v[k], w[2 * k], w[2 * k + 1]);
      }
      // columns [begin, end) in registers; true if the test of some code failed
      auto chain = [&](auto begin, auto end) -> bool {
        bool differ = false;
#pragma unroll
        for (int t = begin; t < end; ++t) {
          const float s = par[t * kRows], rlo = par[(kMicro + t) * kRows], rhi = par[(2 * kMicro + t) * kRows];
          const float z = ZP ? par[(3 * kMicro + t) * kRows] : 0.0f, mz = ZP ? fabsf(z) * (0.5f * kMargin) : 0.0f;
          const float wi = w[t], lo = fmaf(wi, rlo, z - mz);
          const float qc = code_of<KIND>(lo, qmin, qmax);
          differ |= qc != code_of<KIND>(fmaf(wi, rhi, z + mz), qmin, qmax);
          const float q = dequant<KIND, SB, ZP>(qc, s, z);
          // loss and error use the reciprocal of the pivot (an ulp from the reference's divisions)
          const float tt = __fmul_rn(__fsub_rn(wi, q), sRd[c0 + t]);
          e[t] = tt;
          // a zero has the sign of the quotient: x / s + 0 is -0 for a small negative x, and stays it
          w[t] = (KIND == kInt && (!ZP || (q == 0.0f && z == 0.0f))) ? copysignf(q, lo) : q;
#pragma unroll
          for (int k4 = (t + 1) / 4; k4 < kMicro / 4; ++k4) {
            const float4 uu = *reinterpret_cast<const float4*>(u + t * ULD + 4 * k4);
            if (4 * k4 + 0 > t) w[4 * k4 + 0] = fmaf(-tt, uu.x, w[4 * k4 + 0]);
            if (4 * k4 + 1 > t) w[4 * k4 + 1] = fmaf(-tt, uu.y, w[4 * k4 + 1]);
            if (4 * k4 + 2 > t) w[4 * k4 + 2] = fmaf(-tt, uu.z, w[4 * k4 + 2]);
            if (4 * k4 + 3 > t) w[4 * k4 + 3] = fmaf(-tt, uu.w, w[4 * k4 + 3]);
          }
        }
        return __any_sync(0xffffffffu, differ);
      };
      // columns from `begin` on by the exact rules, one by one in shared memory
      auto exact = [&](int begin) {
#pragma unroll 1
        for (int t = begin; t < kMicro; ++t) {
          const float wi = wcol[t * WLD], s = par[t * kRows], z = ZP ? par[(3 * kMicro + t) * kRows] : 0.0f;
          const float q = dequant_code<SB>(round_code_k<KIND>(__fdiv_rn(wi, s) + z, qmin, qmax), s, z);
          const float tt = __fmul_rn(__fsub_rn(wi, q), sRd[c0 + t]);
          wcol[t * WLD] = q;
          eo[t * ELD] = tt;
          for (int k = t + 1; k < kMicro; ++k) wcol[k * WLD] = fmaf(-tt, u[t * ULD + k], wcol[k * WLD]);
        }
#pragma unroll
        for (int t = kHead; t < kMicro; ++t) e[t] = eo[t * ELD];
      };
      auto announce = [&] {   // the first errors are there
        if (m + 1 < micros) asm volatile("bar.arrive 1, 64;" ::: "memory");
      };
      if (!chain(std::integral_constant<int, 0>(), std::integral_constant<int, kHead>()) && !s_odd) {
#pragma unroll
        for (int t = 0; t < kHead; ++t) eo[t * ELD] = e[t];
        announce();
#pragma unroll
        for (int t = 0; t < kMicro; ++t) wcol[t * WLD] = w[t];
        if (!chain(std::integral_constant<int, kHead>(), std::integral_constant<int, kMicro>())) {
#pragma unroll
          for (int t = kHead; t < kMicro; ++t) { wcol[t * WLD] = w[t]; eo[t * ELD] = e[t]; }
        } else {
          exact(kHead);
        }
      } else {
        // (the tile still is as the micro-block found it, without the last errors of the one before)
#pragma unroll 1
        for (int k = 0; k < kMicro && m > 0; ++k) {
          float v = wcol[k * WLD];
          for (int t = kHead; t < kMicro; ++t)
            v = fmaf(-sE[((m + 1) & 1) * kMicro * ELD + t * ELD + lane], u_prev[t * ULD + c0 + k], v);
          wcol[k * WLD] = v;
        }
        exact(0);
        announce();
      }
    } else if (m + 1 < micros) {
      const bool beside = (warp & 3) == 0;   // the chain warp's scheduler
      if (beside && m > 0) fetch_u(m + 1, (warp - 4) * (kAskRows / 4), kAskRows);   // into the buffer of micro-block m - 2
      if (tid == 32) s_next[(m + 1) & 1] = 0;   // (nobody takes from it before the barrier)
      if (warp == 5) fetch_params(m + 1);
      if (warp == 6 && m > 0) finish_errors(m - 1);
      ErrFrag f;
      if (m > 0 && (!beside || micros - m > 16)) {
        load_errors(sE + ((m - 1) & 1) * kMicro * ELD, lane, false, f);
        if (warp == kNextWarp) {
          apply_errors<ULD>(f, u_prev + c0 + kMicro, sW + (c0 + kMicro) * WLD, lane);
        } else {
#pragma unroll 1
          while (true) {
            int task = 0;
            if (lane == 0) task = atomicAdd(&s_next[m & 1], 1);
            const int c = c0 + (2 + __shfl_sync(0xffffffffu, task, 0)) * kMicro;
            if (c >= micros * kMicro) break;
            apply_errors<ULD>(f, u_prev + c, sW + c * WLD, lane);
          }
        }
      }
      if (warp == kNextWarp) {
        asm volatile("bar.sync 1, 64;" ::: "memory");
        load_errors(sE + (m & 1) * kMicro * ELD, lane, true, f);
        apply_errors<ULD>(f, u + kMicro, sW + (c0 + kMicro) * WLD, lane);
      }
    } else if (warp == 6 && m > 0) {
      finish_errors(m - 1);
    }
    if (m + 1 < micros) wait_u(m + 1);
    __syncthreads();
  }
  chain_go();
  if (warp == 6) finish_errors(micros - 1);   // (a superblock with columns after it is a whole one)
  // tile out
  if (vecw) {
#pragma unroll 2
    for (int c = warp * 8; c < sb; c += 8 * (NW)) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const float* d = sW + (c + 4 * h) * WLD + lane;
        if (live && c + 4 * h < sb)
          *reinterpret_cast<float4*>(W + row * p.ldw + c + 4 * h) = make_float4(d[0], d[WLD], d[2 * WLD], d[3 * WLD]);
      }
    }
  } else {
    for (int r = warp; r < kRows; r += NW) {
      if (row0 + r >= p.N) break;
      float* dst = W + (row0 + r) * p.ldw;
      for (int c = lane; c < sb; c += 32) dst[c] = sW[c * WLD + r];
    }
  }
  if (warp == 6 && live) {
    float* lo = p.losses.at(job);
    const float half = loss * 0.5f;
    lo[row] = p.i1 == 0 ? half : lo[row] + half;
  }
}

// Superblock width.  With at most one CTA per SM the chain decides and 512 columns halve the launches and the traffic
// of the trailing products; with more rows than that the CTA's own updates (width / 2 multiply-adds per element) do,
// and 256 columns leave room for two CTAs per SM.
static int superblock_of(int64_t ctas) { return ctas <= kNumSMs ? 512 : 256; }
// The trailing product is split in the columns the next superblock needs and the rest on a helper stream only while
// a superblock's CTAs leave half of the GPU idle.
static bool look_ahead(int64_t ctas) { return ctas <= kNumSMs / 2; }

struct Layout {
  int sb, sets;
  int64_t rows_n, rows_k, err, ub;   // rows per problem of the operands; floats of one hi or lo array
  size_t bytes;
};
static Layout layout_of(int64_t N, int64_t K, int batch, int distinct_u, bool may_overlap) {
  const int64_t ctas = (N + kRows - 1) / kRows * batch;
  Layout l;
  l.sb = superblock_of(ctas);
  l.sets = may_overlap && look_ahead(ctas) ? 2 : 1;
  l.rows_n = (N + 127) / 128 * 128; l.rows_k = (K + 127) / 128 * 128;
  l.err = l.rows_n * l.sb * batch; l.ub = l.rows_k * l.sb * distinct_u;
  l.bytes = kSweepHeaderBytes + (K > l.sb ? (size_t)(2 * l.sets * (l.err + l.ub)) * sizeof(float) : 0) + 64;
  return l;
}

// `Ud` / `u_index`: the distinct factors of a batch and the one each problem uses (null: the single U, or one each)
static int sweep(Params p, int sdtype, bool global, int batch, const float* const* Ud, int distinct_u,
                 const int32_t* u_index, bool may_overlap, void* workspace, cudaStream_t st) {
  const int64_t N = p.N, K = p.K;
  const bool has_u = p.U.one || p.U.table;
  const Layout l = layout_of(N, K, batch, distinct_u, may_overlap);
  // header of the workspace: a status word that a bounded wait expiring inside one of the trailing products sets to
  // B200Q_ERR_DEVICE (cleared here, read by the caller afterwards)
  int* status = (int*)workspace;
  float* err = (float*)((char*)workspace + kSweepHeaderBytes);   // [sets][hi, lo]
  float* ub = err + 2 * l.sets * l.err;                          // [sets][hi, lo]
  B200Q_TRY(cudaMemsetAsync(status, 0, sizeof(int), st));
  if (sdtype != B200Q_BF16 && sdtype != B200Q_F32) return B200Q_ERR_UNSUPPORTED;
  p.sdtype = sdtype; p.status = status;
  const bool with_zp = p.zp.one || p.zp.table, bf16_values = sdtype == B200Q_BF16 && !global;
  void (*kern)(const Params) = nullptr;
#define B200Q_SWEEP_ZP(S, B, K) kern = with_zp ? sweep_block_kernel<S, B, K, true> : sweep_block_kernel<S, B, K, false>
#define B200Q_SWEEP_SB(S, K) do { if (bf16_values) B200Q_SWEEP_ZP(S, true, K); else B200Q_SWEEP_ZP(S, false, K); } while (0)
#define B200Q_SWEEP_PICK(S)                            \
  do {                                                 \
    if (p.qr.kind == kInt) B200Q_SWEEP_SB(S, kInt);      \
    else if (p.qr.kind == kFp8) B200Q_SWEEP_SB(S, kFp8); \
    else B200Q_SWEEP_SB(S, kFp4);                        \
  } while (0)
  if (l.sb == 512) B200Q_SWEEP_PICK(512); else B200Q_SWEEP_PICK(256);
#undef B200Q_SWEEP_PICK
#undef B200Q_SWEEP_SB
#undef B200Q_SWEEP_ZP
  B200Q_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_bytes(l.sb)));
  const int ctas = (int)((N + kRows - 1) / kRows);
  tgemm::SideStream* side = l.sets == 2 && has_u && K > 2 * l.sb ? tgemm::side_stream(st) : nullptr;
  bool side_busy = false;
  int rc;
  auto split_u = [&](int64_t i1, int which, cudaStream_t on) -> int {
    // operand form of U[i1 : i1 + sb, i1 + sb :] (independent of the sweep: kept off its chain)
    const int64_t i2 = i1 + l.sb;
    if (i2 >= K) return B200Q_OK;
    float* hi = ub + (int64_t)which * 2 * l.ub;
    return tgemm::split_transposed(p.U.one ? p.U.one + i1 * p.ldu + i2 : nullptr, Ud, i1 * p.ldu + i2, p.ldu, l.sb,
                                   (int)(K - i2), hi, hi + l.ub, l.sb, l.rows_k * l.sb, distinct_u, on);
  };
  if (has_u && (rc = split_u(0, 0, st))) return rc;
  int blk = 0;
  for (int64_t i1 = 0; i1 < K; i1 += l.sb, ++blk) {
    const int w = (int)(K - i1 < l.sb ? K - i1 : l.sb), which = l.sets == 2 ? blk & 1 : 0;
    const int64_t i2 = i1 + w;
    const bool trailing = i2 < K && has_u;
    p.i1 = (int)i1; p.sb = w;
    p.err_hi = trailing ? err + (int64_t)which * 2 * l.err : nullptr;
    p.err_lo = trailing ? p.err_hi + l.err : nullptr;
    p.lde = l.sb; p.err_batch = l.rows_n * l.sb;
    B200Q_TRY(launch_chained(kern, dim3(ctas, batch), 32 * warps_of(l.sb), smem_bytes(l.sb), st, p));
    B200Q_LAUNCH_CHECK();
    if (!trailing) continue;
    // W[:, i2:] -= Err[N, w] * U[i1:i2, i2:]
    float* bhi = ub + (int64_t)which * 2 * l.ub;
    tgemm::Job j;
    j.A = tgemm::Operand{p.err_hi, p.err_lo, l.sb, l.rows_n * batch, l.rows_n, 0};
    j.B = tgemm::Operand{bhi, bhi + l.ub, l.sb, l.rows_k * distinct_u, l.rows_k, 0};
    j.b_index = u_index;
    j.M = (int)N; j.N = (int)(K - i2); j.Kd = w; j.batch = batch; j.alpha = -1.0f; j.beta = 1.0f;
    if (p.W.one) j.C = p.W.one + i2;
    j.c_table = p.W.table; j.c_offset = i2; j.ldc = p.ldw; j.status = status;
    // a batch: error of the last of 2048 columns 2.6e-7 of its root mean square, with long slices 7.5e-7, by float32
    // multiply-adds 4.1e-7; 64 weights of 768 x 2048: 4.0 ms, 3.8 with long slices.  The single weight keeps the long
    // ones (6.4e-7; 8.8e-7 when its products had rank 128).
    j.slice = p.W.table ? tgemm::kShortSlice : tgemm::kLongSlice;
    if (!side) {
      if ((rc = tgemm::launch(j, st))) return rc;
      if ((rc = split_u(i2, l.sets == 2 ? which ^ 1 : 0, st))) return rc;
      continue;
    }
    tgemm::Job far = j;
    if (j.N > l.sb) j.N = l.sb;
    B200Q_TRY(cudaEventRecord(side->ready, st));
    B200Q_TRY(cudaStreamWaitEvent(side->stream, side->ready, 0));
    // the far columns of the superblock before, and this one's operand form of U made behind them
    if (side_busy) B200Q_TRY(cudaStreamWaitEvent(st, side->done, 0));
    if ((rc = tgemm::launch(j, st))) return rc;
    if (far.N > l.sb) {
      far.B.row0 = l.sb; far.N -= l.sb; far.max_ctas = kNumSMs - ctas * batch;
      if (p.W.one) far.C = p.W.one + i2 + l.sb;
      far.c_offset = i2 + l.sb;
      if ((rc = tgemm::launch(far, side->stream))) return rc;
    }
    // the next superblock's slice of U: its buffer was last read by the superblock before this one
    if ((rc = split_u(i2, which ^ 1, side->stream))) return rc;
    B200Q_TRY(cudaEventRecord(side->done, side->stream));
    side_busy = true;
  }
  if (side_busy) B200Q_TRY(cudaStreamWaitEvent(st, side->done, 0));
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

int b200q_gptq_sweep(float* Wf, int64_t N, int64_t K, int64_t ldf, const float* U, int64_t ldu, const void* scale,
                     int sdtype, const void* zp, const int32_t* col_group, const float* gscale,
                     const b200q_qargs* qa, int blocksize, float* losses, void* workspace, void* stream) {
  using namespace b200q::sweep;
  if (!Wf || !scale || !qa || !losses || !workspace || N <= 0 || K <= 0 || ldf < K) return B200Q_ERR_ARG;
  if (U && ldu < K) return B200Q_ERR_ARG;
  if (((uintptr_t)workspace) & 15) return B200Q_ERR_ARG;
  if (blocksize <= 0 || blocksize > kMaxBlock) return B200Q_ERR_UNSUPPORTED;
  Params p;
  int rc = fill_scheme(&p, qa, N, K, col_group); if (rc) return rc;
  p.W = {Wf, nullptr}; p.U = {U, nullptr}; p.scale = {scale, nullptr}; p.zp = {zp, nullptr};
  p.col_group = {col_group, nullptr}; p.gscale = {gscale, nullptr}; p.losses = {losses, nullptr};
  p.N = N; p.K = K; p.ldw = ldf; p.ldu = ldu;
  return sweep::sweep(p, sdtype, gscale != nullptr, 1, nullptr, 1, nullptr, true, workspace, (cudaStream_t)stream);
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
