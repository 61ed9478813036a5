// MSE shrink-grid observer: all shrink candidates evaluated in one pass over the weight.
//
// For each group the elements stay in registers (GROUP strategies) or shared memory
// (CHANNEL) while every candidate p = 1 - i/grid is tried: qparams from (p*min, p*max),
// fake-quantise, sum |q - x|^norm, keep the strictly smallest.  Arithmetic is done in the
// weight's dtype step by step (bf16 weights: every elementwise result is rounded to bf16,
// sums are accumulated in float32 and rounded once), like the element-wise torch ops of the
// reference.  The reference stops the whole search once `patience` consecutive candidates
// improved no group anywhere; pass 1 records per candidate whether any group improved, a
// one-thread kernel derives the stopping step, and pass 2 (a no-op unless the search stops
// early) repeats the search up to that step.
#include "common.cuh"

#include <string.h>

#include <mutex>

namespace b200q {
namespace mse {

struct Cfg {
  int symmetric, scale_kind, zp_kind, mx_offset;
  float qmin, qmax, half_range, range, eps, inv_half_range;
  int kind;
  int steps, patience;
  double grid;
  float norm, expand;
};

// qparams of calculate_qparams without a global scale, in dtype T (TB: bf16).
template <bool TB>
__device__ __forceinline__ void qparams_local(float mn, float mx, const Cfg& c, float& s, float& zp) {
  mn = fminf(mn, 0.0f);
  mx = fmaxf(mx, 0.0f);
  if (c.symmetric) {
    float amax = fmaxf(fabsf(mn), fabsf(mx));
    if (c.scale_kind == B200Q_SCALE_E8M0) {
      int biased;
      if (TB) { uint32_t b = __float_as_uint(amax) >> 16; b = (b + 32u) & 0xFF80u; biased = (int)((b >> 7) & 0xFFu); }
      else { uint32_t b = __float_as_uint(amax); b = (b + (1u << 21)) & 0xFF800000u; biased = (int)((b >> 23) & 0xFFu); }
      float e = (biased == 0) ? 0.0f : fminf(fmaxf((float)(biased - c.mx_offset), 0.0f), 255.0f);
      s = __uint_as_float(e >= 1.0f ? ((uint32_t)e << 23) : 0x00400000u);
    } else {
      // (bf16 statistics: the product with the reciprocal rounds to the same bf16 value, see qparams_one)
      s = TB ? bf16r(amax * c.inv_half_range) : __fdiv_rn(amax, c.half_range);
      if (c.scale_kind == B200Q_SCALE_FP8) s = e4m3_round(fminf(fmaxf(s, -448.0f), 448.0f));
    }
    zp = 0.0f;
  } else {
    float d = rnd_if<TB>(mx - mn);
    s = rnd_if<TB>(__fdiv_rn(d, c.range));
    float z = rnd_if<TB>(__fdiv_rn(mn, s));
    z = rnd_if<TB>(c.qmin - z);
    // 0/0 for an all-zero group: torch's clamp keeps the NaN and the integer cast makes it 0
    zp = (z != z) ? 0.0f : fminf(fmaxf(z, c.qmin), c.qmax);
  }
  if (s == 0.0f) s = c.eps;
  if (c.zp_kind == B200Q_ZP_INT8) zp = rintf(fminf(fmaxf(zp, -128.0f), 127.0f));
  else if (c.zp_kind == B200Q_ZP_UINT8) zp = rintf(fminf(fmaxf(zp, 0.0f), 255.0f));
  else zp = e4m3_round(fminf(fmaxf(zp, -448.0f), 448.0f));
}

template <bool TB>
__device__ __forceinline__ float elem_error(float x, float s, float z, const Cfg& c) {
  QRange qr{c.qmin, c.qmax, c.kind};
  float q = quant_code<TB>(x, s, z, qr);
  float fq = dequant_code<TB>(q, s, z);
  float d = rnd_if<TB>(fabsf(rnd_if<TB>(fq - x)));
  float e = (d == 0.0f) ? 0.0f : powf(d, c.norm);
  return rnd_if<TB>(e);
}

__device__ __forceinline__ float shrink_factor(int i, double grid) {
  return (float)(1.0 - (double)i / grid);
}

// ctl[0] = number of steps to run, ctl[1..] = per-step "some group improved" flags
template <int DT>
__global__ void __launch_bounds__(256) mse_group_kernel(const void* __restrict__ W, int64_t N, int64_t K,
                                                        int64_t ldw, int g, Cfg c, int* __restrict__ ctl,
                                                        int pass, void* __restrict__ mn_out,
                                                        void* __restrict__ mx_out) {
  using E = Elem<DT>;
  using T = typename E::type;
  constexpr bool TB = E::is_bf16;
  const int limit = (pass == 0) ? c.steps : ctl[0];
  if (pass == 1 && limit >= c.steps) return;  // the search never stopped early
  const int lanes = g >> 3;
  const int64_t cpr = K >> 3, total = N * cpr, gpr = K / g;
  for (int64_t ch = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; ch < ((total + 31) & ~31LL);
       ch += (int64_t)gridDim.x * blockDim.x) {
    const bool live = ch < total;
    float v[8];
    float lo = INFINITY, hi = -INFINITY;
    int64_t row = 0, cc = 0;
    if (live) {
      row = ch / cpr; cc = ch - row * cpr;
      const T* src = (const T*)W + row * ldw + cc * 8;
#pragma unroll
      for (int i = 0; i < 8; ++i) { v[i] = E::load(src + i); lo = fminf(lo, v[i]); hi = fmaxf(hi, v[i]); }
    } else {
#pragma unroll
      for (int i = 0; i < 8; ++i) v[i] = 0.0f;
    }
    for (int o = lanes >> 1; o > 0; o >>= 1) {
      lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, o));
      hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, o));
    }
    const float mn = rnd_if<TB>(lo * c.expand), mx = rnd_if<TB>(hi * c.expand);
    float best_err = TB ? 3.3895313892515355e38f : 3.402823466e38f;  // finfo(dtype).max
    float best_mn = mn, best_mx = mx;
    for (int i = 0; i < limit; ++i) {
      const float p = shrink_factor(i, c.grid);
      const float smn = rnd_if<TB>(mn * p), smx = rnd_if<TB>(mx * p);
      float s, z;
      qparams_local<TB>(smn, smx, c, s, z);
      float err = 0.0f;
#pragma unroll
      for (int e = 0; e < 8; ++e) err += elem_error<TB>(v[e], s, z, c);
      for (int o = lanes >> 1; o > 0; o >>= 1) err += __shfl_xor_sync(0xffffffffu, err, o);
      err = rnd_if<TB>(err);
      if (live && err < best_err) {
        best_err = err; best_mn = smn; best_mx = smx;
        if (pass == 0 && (cc % lanes) == 0 && ((volatile int*)ctl)[1 + i] == 0) atomicOr(&ctl[1 + i], 1);
      }
    }
    if (live && (cc % lanes) == 0) {
      int64_t gi = row * gpr + (cc * 8) / g;
      E::store((T*)mn_out + gi, best_mn);
      E::store((T*)mx_out + gi, best_mx);
    }
  }
}

// ---------------------------------------------------------------------------------------
// bf16 weights: the same search in packed bf16x2 arithmetic with the power read from a table.
//
// torch evaluates a candidate with element-wise bf16 ops.  For bf16 operands a packed HADD2 / HMUL2 / HFMA2 gives
// exactly the rounded result of the float32 operation followed by a rounding to bf16 (the _rn forms of the intrinsics:
// the plain ones let the compiler fuse a product and a subtraction into one rounding).  The quotient bf16(x / s) is
// fma(x, r_hi, fma(x, r_lo, +0)) with 1 / s split into two bf16 parts, exact for every pair of bf16 significands (see
// stream_kernels.cuh); scales outside 2^-100 .. 2^100 take element-wise divisions.  The error |q - x| is a bf16 value,
// so its rounded power is one of 32768: a table in shared memory, made once per call with powf.
//
// What bounds it: the table look-ups (about three cycles a warp, bank conflicts of 32 random entries) and about ten
// instructions an element (4096 x 4096, groups of 128, 20 candidates: 186 us).  Evaluating exp2(norm * log2 d) instead costs two special-function results, checks against
// rounding midpoints and a fallback: 685 us for 20 candidates on 4096 x 4096.
constexpr int kTable = 32768;
constexpr size_t kTableBytes = kTable * 2;

// Where entry i stands.  An error is a difference of two close numbers with few significant bits left, so the low bits of
// its pattern are mostly zero: in plain order the look-ups of a warp meet in a few banks (FP8 errors use 16 of 128
// patterns of an exponent).  Both halves of a pair at once.
__device__ __forceinline__ uint32_t table_place(uint32_t i) { return i ^ ((i >> 4) & 0x07FF07FFu); }

__global__ void __launch_bounds__(256) make_table_kernel(__nv_bfloat16* __restrict__ table, float norm, int* __restrict__ ctl,
                                                         int n) {
  const int i = blockIdx.x * 256 + threadIdx.x;
  const float d = __uint_as_float((uint32_t)i << 16);
  if (i < kTable) table[table_place((uint32_t)i)] = __float2bfloat16_rn(d == 0.0f ? 0.0f : powf(d, norm));
  if (blockIdx.x == 0)
    for (int k = threadIdx.x; k < n; k += 256) ctl[k] = 0;
}

__device__ __forceinline__ uint32_t bf2_of(float v) {
  __nv_bfloat162 r = __float2bfloat162_rn(v);
  return *reinterpret_cast<uint32_t*>(&r);
}
__device__ __forceinline__ uint32_t bf2_pack(float hi, float lo) {
  uint32_t d;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(hi), "f"(lo));
  return d;
}
#define B200Q_BF2(op, ...) ([&] { __nv_bfloat162 r_ = op(__VA_ARGS__); return *reinterpret_cast<uint32_t*>(&r_); }())
#define B200Q_B(v) *reinterpret_cast<const __nv_bfloat162*>(&(v))

enum MseKind { kMseInt4 = 0, kMseInt8 = 1, kMseFp8 = 2, kMseFp4 = 3 };

// what the elements need from one candidate
struct Cand {
  float s, z;
  uint32_t rhi2, rlo2, s2, z2;
  bool slow;
};
__device__ __forceinline__ Cand make_cand(float smn, float smx, const Cfg& c) {
  Cand q;
  qparams_local<true>(smn, smx, c, q.s, q.z);
  const float rs = __frcp_rn(q.s), rhi = bf16r(rs);
  q.rhi2 = bf2_of(rhi); q.rlo2 = bf2_of(rs - rhi); q.s2 = bf2_of(q.s); q.z2 = bf2_of(q.z);
  q.slow = !(q.s >= 0x1p-100f && q.s <= 0x1p100f);
  return q;
}
// fake_quantize(x) - x of a pair
template <int KIND, bool SYM>
__device__ __forceinline__ uint32_t pair_error(uint32_t w, const Cand& q, uint32_t qmin2, uint32_t qmax2) {
  const uint32_t zero = 0u, magic = 0x43404340u;   // {192, 192}: integers are 1 apart in [128, 256)
  uint32_t v = B200Q_BF2(__hfma2, B200Q_B(w), B200Q_B(q.rlo2), B200Q_B(zero));
  v = B200Q_BF2(__hfma2, B200Q_B(w), B200Q_B(q.rhi2), B200Q_B(v));
  if (!SYM) v = B200Q_BF2(__hadd2_rn, B200Q_B(v), B200Q_B(q.z2));
  if (KIND == kMseInt4 || KIND == kMseInt8) {
    v = B200Q_BF2(__hmax2, B200Q_B(v), B200Q_B(qmin2));
    v = B200Q_BF2(__hmin2, B200Q_B(v), B200Q_B(qmax2));
    if (KIND == kMseInt4) {
      v = B200Q_BF2(__hadd2_rn, B200Q_B(v), B200Q_B(magic));
      v = B200Q_BF2(__hsub2_rn, B200Q_B(v), B200Q_B(magic));
    } else {
      v = B200Q_BF2(h2rint, B200Q_B(v));
    }
  } else {
    // through the hardware's code (round to nearest even, saturating) and back
    const float lo = __uint_as_float(v << 16), hi = __uint_as_float(v & 0xFFFF0000u);
    uint32_t h;
    if (KIND == kMseFp8)
      asm("{\n\t.reg .b16 b;\n\tcvt.rn.satfinite.e4m3x2.f32 b, %2, %1;\n\tcvt.rn.f16x2.e4m3x2 %0, b;\n\t}" : "=r"(h) : "f"(lo), "f"(hi));
    else
      asm("{\n\t.reg .b8 b;\n\tcvt.rn.satfinite.e2m1x2.f32 b, %2, %1;\n\tcvt.rn.f16x2.e2m1x2 %0, b;\n\t}" : "=r"(h) : "f"(lo), "f"(hi));
    const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&h));
    v = bf2_pack(f.y, f.x);
  }
  if (!SYM) v = B200Q_BF2(__hsub2_rn, B200Q_B(v), B200Q_B(q.z2));
  v = B200Q_BF2(__hmul2_rn, B200Q_B(v), B200Q_B(q.s2));
  return B200Q_BF2(__hsub2_rn, B200Q_B(v), B200Q_B(w));
}
// Twice the places of a pair's magnitudes, which are byte offsets: the signs leave at the top of either half.
__device__ __forceinline__ uint32_t table_offsets(uint32_t d) {
  const uint32_t i = (d << 1) & 0xFFFEFFFEu;
  return i ^ ((i >> 4) & 0x0FFE0FFEu);
}
__device__ __forceinline__ float add_power(float sum, const unsigned char* tab, uint32_t offset) {
  unsigned short p = *reinterpret_cast<const unsigned short*>(tab + offset);
  float r;
  asm("add.rn.f32.bf16 %0, %1, %2;" : "=f"(r) : "h"(p), "f"(sum));
  return r;
}
// error sum of a chunk of 8 elements, in element order
template <int KIND, bool SYM>
__device__ __forceinline__ float chunk_error(const uint32_t (&w)[4], const Cand& q, uint32_t qmin2, uint32_t qmax2,
                                             const Cfg& c, const unsigned short* __restrict__ tab) {
  float err = 0.0f;
  if (q.slow) {
    for (int k = 0; k < 4; ++k) {
      err += elem_error<true>(__uint_as_float(w[k] << 16), q.s, q.z, c);
      err += elem_error<true>(__uint_as_float(w[k] & 0xFFFF0000u), q.s, q.z, c);
    }
    return err;
  }
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const uint32_t d = table_offsets(pair_error<KIND, SYM>(w[k], q, qmin2, qmax2));
    err = add_power(err, reinterpret_cast<const unsigned char*>(tab), d & 0xFFFFu);
    err = add_power(err, reinterpret_cast<const unsigned char*>(tab), d >> 16);
  }
  return err;
}
__device__ __forceinline__ void load_table(uint4* dst, const __nv_bfloat16* __restrict__ table) {
#pragma unroll 4
  for (int i = threadIdx.x; i < (int)(kTableBytes / 16); i += blockDim.x) dst[i] = reinterpret_cast<const uint4*>(table)[i];
}
__device__ __forceinline__ void chunk_range(const uint4& raw, float& lo, float& hi) {
  const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const float a = __uint_as_float(w[k] << 16), b = __uint_as_float(w[k] & 0xFFFF0000u);
    lo = fminf(lo, fminf(a, b)); hi = fmaxf(hi, fmaxf(a, b));
  }
}

// GROUP strategies.  The chunks of a group are shared by L lanes, R each (L apart), so that a candidate's parameters
// are derived once per R * 8 elements.  The chunk sums are added in the order of a butterfly over all chunks of the
// group, whatever R is.
template <int KIND, bool SYM, int R>
__global__ void __launch_bounds__(256, 3) mse_group_bf16_kernel(const void* __restrict__ W, int64_t N, int64_t K, int64_t ldw,
                                                             int g, Cfg c, const __nv_bfloat16* __restrict__ table,
                                                             int* __restrict__ ctl, int pass, void* __restrict__ mn_out,
                                                             void* __restrict__ mx_out, uint32_t* __restrict__ better) {
  using T = __nv_bfloat16;
  extern __shared__ __align__(16) unsigned short s_table[];
  __shared__ float s_shrink[1024];
  const int limit = (pass == 0) ? c.steps : ctl[0];
  if (pass == 1 && limit >= c.steps) return;  // the search never stopped early
  load_table(reinterpret_cast<uint4*>(s_table), table);
  for (int i = threadIdx.x; i < limit && i < 1024; i += blockDim.x) s_shrink[i] = shrink_factor(i, c.grid);
  __syncthreads();
  const int L = (g >> 3) / R;
  const int64_t gpr = K / g, total = N * gpr * L;
  const uint32_t qmin2 = bf2_of(c.qmin), qmax2 = bf2_of(c.qmax);
  for (int64_t slot = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; slot < ((total + 31) & ~31LL);
       slot += (int64_t)gridDim.x * blockDim.x) {
    const bool live = slot < total;
    const int64_t gi = live ? slot / L : 0, row = gi / gpr;
    const int j = (int)(slot - gi * L);
    uint32_t w[R][4];
    float lo = INFINITY, hi = -INFINITY;
    const T* src = (const T*)W + row * ldw + (gi - row * gpr) * g + j * 8;
#pragma unroll
    for (int k = 0; k < R; ++k) {
      uint4 raw = make_uint4(0u, 0u, 0u, 0u);
      if (live) {
        raw = __ldg(reinterpret_cast<const uint4*>(src + (int64_t)k * L * 8));
        chunk_range(raw, lo, hi);
      }
      w[k][0] = raw.x; w[k][1] = raw.y; w[k][2] = raw.z; w[k][3] = raw.w;
    }
    for (int o = L >> 1; o > 0; o >>= 1) {
      lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, o));
      hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, o));
    }
    const float mn = bf16r(lo * c.expand), mx = bf16r(hi * c.expand);
    float best_err = 3.3895313892515355e38f;  // finfo(bfloat16).max
    float best_mn = mn, best_mx = mx;
    uint32_t mask = 0;
#pragma unroll 1   // (unrolled, the candidates outgrow the instruction cache: 188 us instead of 136 for int4, 3000 x 3840)
    for (int i = 0; i < limit; ++i) {
      const float p = i < 1024 ? s_shrink[i] : shrink_factor(i, c.grid);
      const float smn = bf16r(mn * p), smx = bf16r(mx * p);
      const Cand q = make_cand(smn, smx, c);
      float part[R];
#pragma unroll
      for (int k = 0; k < R; ++k) part[k] = chunk_error<KIND, SYM>(w[k], q, qmin2, qmax2, c, s_table);
      float err = R == 4 ? (part[0] + part[R / 2]) + (part[R / 4] + part[R - 1]) : R == 2 ? part[0] + part[R - 1] : part[0];
      for (int o = L >> 1; o > 0; o >>= 1) err += __shfl_xor_sync(0xffffffffu, err, o);
      err = bf16r(err);
      if (live && err < best_err) {
        best_err = err; best_mn = smn; best_mx = smx; mask |= 1u << (i & 31);
        if (pass == 0 && j == 0 && ((volatile int*)ctl)[1 + i] == 0) atomicOr(&ctl[1 + i], 1);
      }
    }
    if (live && j == 0) {
      if (better) better[gi] = mask;
      ((T*)mn_out)[gi] = __float2bfloat16_rn(better ? mn : best_mn);
      ((T*)mx_out)[gi] = __float2bfloat16_rn(better ? mx : best_mx);
    }
  }
}

// CHANNEL and BLOCK strategies: a CTA per row or bh x bw block, kept packed in shared memory (blocks that stick out of
// the matrix are completed with zeros, as in mse_tile_kernel).  Candidates are evaluated four at a time, so that the
// CTA-wide sum costs a barrier for four.
template <int KIND, bool SYM>
__global__ void __launch_bounds__(256) mse_tile_bf16_kernel(const void* __restrict__ W, int64_t N, int64_t K, int64_t ldw,
                                                            int bh, int bw, Cfg c, const __nv_bfloat16* __restrict__ table,
                                                            int* __restrict__ ctl, int pass, void* __restrict__ mn_out,
                                                            void* __restrict__ mx_out, uint32_t* __restrict__ better) {
  using T = __nv_bfloat16;
  extern __shared__ __align__(16) unsigned short s_table[];
  uint4* data = reinterpret_cast<uint4*>(s_table + kTable);
  __shared__ float s_part[2][8][4], s_lo[8], s_hi[8];
  const int limit = (pass == 0) ? c.steps : ctl[0];
  if (pass == 1 && limit >= c.steps) return;
  load_table(reinterpret_cast<uint4*>(s_table), table);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int cw = bw >> 3, chunks = bh * cw;
  const int64_t gpr = (K + bw - 1) / bw, groups = ((N + bh - 1) / bh) * gpr;
  const uint32_t qmin2 = bf2_of(c.qmin), qmax2 = bf2_of(c.qmax);
  for (int64_t grp = blockIdx.x; grp < groups; grp += gridDim.x) {
    const int64_t r0 = (grp / gpr) * bh, c0 = (grp % gpr) * bw;
    float lo = INFINITY, hi = -INFINITY;
    for (int x = threadIdx.x; x < chunks; x += 256) {
      const int y = x / cw;
      const int64_t r = r0 + y, cc = c0 + (x - y * cw) * 8;
      uint4 raw = make_uint4(0u, 0u, 0u, 0u);
      if (r < N && cc < K) raw = __ldg(reinterpret_cast<const uint4*>((const T*)W + r * ldw + cc));
      data[x] = raw;
      chunk_range(raw, lo, hi);
    }
    lo = warp_min(lo); hi = warp_max(hi);
    if (lane == 0) { s_lo[warp] = lo; s_hi[warp] = hi; }
    __syncthreads();
    for (int w = 0; w < 8; ++w) { lo = fminf(lo, s_lo[w]); hi = fmaxf(hi, s_hi[w]); }
    const float mn = bf16r(lo * c.expand), mx = bf16r(hi * c.expand);
    float best_err = 3.3895313892515355e38f, best_mn = mn, best_mx = mx;
    uint32_t mask = 0;
    for (int i0 = 0, turn = 0; i0 < limit; i0 += 4, turn ^= 1) {
      Cand q[4];
      float smn[4], smx[4], err[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const float p = shrink_factor(i0 + k, c.grid);
        smn[k] = bf16r(mn * p); smx[k] = bf16r(mx * p);
        q[k] = make_cand(smn[k], smx[k], c);
      }
      for (int x = threadIdx.x; x < chunks; x += 256) {
        const uint4 raw = data[x];
        const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
        for (int k = 0; k < 4; ++k) err[k] += chunk_error<KIND, SYM>(w, q[k], qmin2, qmax2, c, s_table);
      }
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        err[k] = warp_sum(err[k]);
        if (lane == 0) s_part[turn][warp][k] = err[k];
      }
      __syncthreads();
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        float tot = 0.0f;
        for (int w = 0; w < 8; ++w) tot += s_part[turn][w][k];
        tot = bf16r(tot);
        if (i0 + k < limit && tot < best_err) {
          best_err = tot; best_mn = smn[k]; best_mx = smx[k]; mask |= 1u << ((i0 + k) & 31);
          if (pass == 0 && threadIdx.x == 0 && ((volatile int*)ctl)[1 + i0 + k] == 0) atomicOr(&ctl[1 + i0 + k], 1);
        }
      }
    }
    if (threadIdx.x == 0) {
      if (better) better[grp] = mask;
      ((T*)mn_out)[grp] = __float2bfloat16_rn(better ? mn : best_mn);
      ((T*)mx_out)[grp] = __float2bfloat16_rn(better ? mx : best_mx);
    }
    __syncthreads();
  }
}
#undef B200Q_BF2
#undef B200Q_B

// One CTA per group held in shared memory: a row (CHANNEL, bh = 1, bw = K) or a bh x bw block
// (BLOCK; blocks that stick out of the matrix are completed with zeros, which take part in the
// statistics like the reference's padding).  The per-candidate error is summed in a fixed order
// (thread-strided partial sums, warp tree, warps in order), so results do not depend on timing.
template <int DT>
__global__ void __launch_bounds__(256) mse_tile_kernel(const void* __restrict__ W, int64_t N, int64_t K,
                                                       int64_t ldw, int bh, int bw, Cfg c, int* __restrict__ ctl,
                                                       int pass, void* __restrict__ mn_out, void* __restrict__ mx_out) {
  using E = Elem<DT>;
  using T = typename E::type;
  constexpr bool TB = E::is_bf16;
  extern __shared__ float srow[];
  __shared__ float s_a[8], s_b[8];
  __shared__ float s_bc[2];
  const int limit = (pass == 0) ? c.steps : ctl[0];
  if (pass == 1 && limit >= c.steps) return;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  const int64_t gpr = (K + bw - 1) / bw, groups = ((N + bh - 1) / bh) * gpr;
  const int elems = bh * bw;
  for (int64_t grp = blockIdx.x; grp < groups; grp += gridDim.x) {
    const int64_t r0 = (grp / gpr) * bh, c0 = (grp % gpr) * bw;
    float lo = INFINITY, hi = -INFINITY;
    for (int x = threadIdx.x; x < elems; x += blockDim.x) {
      const int64_t r = r0 + x / bw, cc = c0 + x % bw;
      const float v = (r < N && cc < K) ? E::load((const T*)W + r * ldw + cc) : 0.0f;
      srow[x] = v; lo = fminf(lo, v); hi = fmaxf(hi, v);
    }
    lo = warp_min(lo); hi = warp_max(hi);
    if (lane == 0) { s_a[warp] = lo; s_b[warp] = hi; }
    __syncthreads();
    if (threadIdx.x == 0) {
      for (int w = 1; w < nw; ++w) { lo = fminf(lo, s_a[w]); hi = fmaxf(hi, s_b[w]); }
      s_bc[0] = lo; s_bc[1] = hi;
    }
    __syncthreads();
    const float mn = rnd_if<TB>(s_bc[0] * c.expand), mx = rnd_if<TB>(s_bc[1] * c.expand);
    float best_err = TB ? 3.3895313892515355e38f : 3.402823466e38f;
    float best_mn = mn, best_mx = mx;
    for (int i = 0; i < limit; ++i) {
      const float p = shrink_factor(i, c.grid);
      const float smn = rnd_if<TB>(mn * p), smx = rnd_if<TB>(mx * p);
      float s, z;
      qparams_local<TB>(smn, smx, c, s, z);
      float err = 0.0f;
      for (int x = threadIdx.x; x < elems; x += blockDim.x) err += elem_error<TB>(srow[x], s, z, c);
      err = warp_sum(err);
      __syncthreads();
      if (lane == 0) s_a[warp] = err;
      __syncthreads();
      float tot = 0.0f;
      for (int w = 0; w < nw; ++w) tot += s_a[w];
      tot = rnd_if<TB>(tot);
      if (tot < best_err) {
        best_err = tot; best_mn = smn; best_mx = smx;
        if (pass == 0 && threadIdx.x == 0 && ((volatile int*)ctl)[1 + i] == 0) atomicOr(&ctl[1 + i], 1);
      }
    }
    if (threadIdx.x == 0) {
      E::store((T*)mn_out + grp, best_mn);
      E::store((T*)mx_out + grp, best_mx);
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------------------
// TENSOR strategy: the whole matrix is one group.  One launch per shrink candidate sums the
// element errors into per-CTA partials (grid-stride, fixed order inside a CTA); a one-warp kernel
// folds the partials in index order, compares with the best so far and keeps the reference's
// patience counter, all on the device.  After the search has stopped the remaining launches return
// at once.  state: [0] min, [1] max (expanded), [2] best error, [3] best min, [4] best max,
// [5] stale count, [6] stopped flag (both as int bit patterns), then the partials.
constexpr int kSpanState = 8;

template <int DT>
__global__ void __launch_bounds__(256) mse_span_range_kernel(const void* __restrict__ W, int64_t N, int64_t K,
                                                             int64_t ldw, float* __restrict__ partial) {
  using E = Elem<DT>;
  using T = typename E::type;
  __shared__ float s_a[8], s_b[8];
  float lo = INFINITY, hi = -INFINITY;
  const int64_t total = N * K;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t r = i / K, cc = i - r * K;
    const float v = E::load((const T*)W + r * ldw + cc);
    lo = fminf(lo, v); hi = fmaxf(hi, v);
  }
  lo = warp_min(lo); hi = warp_max(hi);
  if ((threadIdx.x & 31) == 0) { s_a[threadIdx.x >> 5] = lo; s_b[threadIdx.x >> 5] = hi; }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < (int)(blockDim.x >> 5); ++w) { lo = fminf(lo, s_a[w]); hi = fmaxf(hi, s_b[w]); }
    partial[2 * blockIdx.x] = lo; partial[2 * blockIdx.x + 1] = hi;
  }
}
template <bool TB>
__global__ void mse_span_init_kernel(float* __restrict__ state, const float* __restrict__ partial, int nblocks, Cfg c) {
  float lo = INFINITY, hi = -INFINITY;
  for (int i = 0; i < nblocks; ++i) { lo = fminf(lo, partial[2 * i]); hi = fmaxf(hi, partial[2 * i + 1]); }
  const float mn = rnd_if<TB>(lo * c.expand), mx = rnd_if<TB>(hi * c.expand);
  state[0] = mn; state[1] = mx;
  state[2] = TB ? 3.3895313892515355e38f : 3.402823466e38f;
  state[3] = mn; state[4] = mx;
  ((int*)state)[5] = 0; ((int*)state)[6] = 0;
}
template <int DT>
__global__ void __launch_bounds__(256) mse_span_error_kernel(const void* __restrict__ W, int64_t N, int64_t K,
                                                             int64_t ldw, Cfg c, int step,
                                                             const float* __restrict__ state,
                                                             float* __restrict__ partial) {
  using E = Elem<DT>;
  using T = typename E::type;
  constexpr bool TB = E::is_bf16;
  __shared__ float s_a[8];
  if (((const int*)state)[6]) return;
  const float p = shrink_factor(step, c.grid);
  const float smn = rnd_if<TB>(state[0] * p), smx = rnd_if<TB>(state[1] * p);
  float s, z;
  qparams_local<TB>(smn, smx, c, s, z);
  float err = 0.0f;
  const int64_t total = N * K;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t r = i / K, cc = i - r * K;
    err += elem_error<TB>(E::load((const T*)W + r * ldw + cc), s, z, c);
  }
  err = warp_sum(err);
  if ((threadIdx.x & 31) == 0) s_a[threadIdx.x >> 5] = err;
  __syncthreads();
  if (threadIdx.x == 0) {
    float tot = 0.0f;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) tot += s_a[w];
    partial[blockIdx.x] = tot;
  }
}
template <bool TB>
__global__ void mse_span_fold_kernel(float* __restrict__ state, const float* __restrict__ partial, int nblocks, Cfg c,
                                     int step) {
  int* istate = (int*)state;
  if (istate[6]) return;
  float tot = 0.0f;
  for (int i = 0; i < nblocks; ++i) tot += partial[i];
  tot = rnd_if<TB>(tot);
  if (tot < state[2]) {
    const float p = shrink_factor(step, c.grid);
    state[2] = tot; state[3] = rnd_if<TB>(state[0] * p); state[4] = rnd_if<TB>(state[1] * p);
    istate[5] = 0;
  } else if (++istate[5] >= c.patience) {
    istate[6] = 1;
  }
}
template <int DT>
__global__ void mse_span_store_kernel(const float* __restrict__ state, void* __restrict__ mn_out,
                                      void* __restrict__ mx_out) {
  using E = Elem<DT>;
  using T = typename E::type;
  E::store((T*)mn_out, state[3]);
  E::store((T*)mx_out, state[4]);
}

// Which candidate counts is known once every group has been through all of them: the search ends for all groups at once,
// when no group has found a better one for `patience` candidates.  Groups with up to 32 candidates note which ones were
// better than all before (`better`, bit i), and the last of these before the end is taken here; with more, the search is
// run a second time up to the end (half as long again where it ends early: FP8 per channel 365 us, 205 without).
__global__ void __launch_bounds__(256) pick_kernel(const int* __restrict__ ctl, const uint32_t* __restrict__ better,
                                                   int64_t groups, Cfg c, __nv_bfloat16* __restrict__ mn,
                                                   __nv_bfloat16* __restrict__ mx) {
  int stale = 0, run = c.steps;
  for (int i = 0; i < c.steps; ++i) {
    if (ctl[1 + i]) stale = 0;
    else if (++stale >= c.patience) { run = i + 1; break; }
  }
  const uint32_t before = run >= 32 ? 0xFFFFFFFFu : (1u << run) - 1u;
  for (int64_t g = (int64_t)blockIdx.x * 256 + threadIdx.x; g < groups; g += (int64_t)gridDim.x * 256) {
    const uint32_t m = better[g] & before;
    if (m == 0) continue;   // none: the range as it is
    const float p = shrink_factor(31 - __clz(m), c.grid);
    mn[g] = __float2bfloat16_rn(__bfloat162float(mn[g]) * p);
    mx[g] = __float2bfloat16_rn(__bfloat162float(mx[g]) * p);
  }
}

// ctl[0] <- number of candidates the reference's loop evaluates before it breaks
__global__ void stop_step_kernel(int* ctl, int steps, int patience) {
  int stale = 0, run = steps;
  for (int i = 0; i < steps; ++i) {
    if (ctl[1 + i]) stale = 0;
    else if (++stale >= patience) { run = i + 1; break; }
  }
  ctl[0] = run;
}
__global__ void clear_ctl_kernel(int* ctl, int n) {
  for (int i = threadIdx.x; i < n; i += blockDim.x) ctl[i] = 0;
}

// Blocks per SM of the table-driven kernels (the table takes 64 KiB of shared memory a block)
constexpr int kTableBlocksPerSM = 3;

template <int KIND, bool SYM>
static int launch_group(const void* W, int64_t N, int64_t K, int64_t ldw, int g, const Cfg& c, const __nv_bfloat16* table,
                        int* ctl, int pass, void* mn, void* mx, uint32_t* better, cudaStream_t st) {
  const int chunks = g >> 3, r = chunks >= 4 ? 4 : chunks;
  const int64_t slots = N * (K / g) * (chunks / r);
  const int grid = grid_for((slots + 255) / 256, kTableBlocksPerSM);
  auto kern = r == 4 ? mse_group_bf16_kernel<KIND, SYM, 4> : r == 2 ? mse_group_bf16_kernel<KIND, SYM, 2> : mse_group_bf16_kernel<KIND, SYM, 1>;
  B200Q_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTableBytes));
  kern<<<grid, 256, kTableBytes, st>>>(W, N, K, ldw, g, c, table, ctl, pass, mn, mx, better);
  return B200Q_OK;
}
template <int KIND, bool SYM>
static int launch_tile(const void* W, int64_t N, int64_t K, int64_t ldw, int bh, int bw, const Cfg& c,
                       const __nv_bfloat16* table, int* ctl, int pass, void* mn, void* mx, uint32_t* better,
                       cudaStream_t st) {
  const size_t smem = kTableBytes + (size_t)bh * bw * 2;
  const int64_t groups = ((N + bh - 1) / bh) * ((K + bw - 1) / bw);
  const int per_sm = (int)(220 * 1024 / (smem + 1024));
  auto kern = mse_tile_bf16_kernel<KIND, SYM>;
  B200Q_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  kern<<<grid_for(groups, per_sm < 1 ? 1 : per_sm), 256, smem, st>>>(W, N, K, ldw, bh, bw, c, table, ctl, pass, mn, mx, better);
  return B200Q_OK;
}

}  // namespace mse
}  // namespace b200q

using namespace b200q;

extern "C" {

// int(maxshrink * grid) in double precision, as the reference's Python evaluates it
int b200q_observe_mse_steps(double maxshrink, double grid) {
  const double v = maxshrink * grid;
  if (!(v >= 0.0)) return -1;
  return v > 2147483647.0 ? 2147483647 : (int)v;
}

static size_t mse_flag_bytes(int steps) {
  return (sizeof(int) * (size_t)(steps + 1 > 1 ? steps + 1 : 1) + 255) / 256 * 256;
}

// groups that a packed search notes its better candidates for
static int64_t mse_groups(int64_t N, int64_t K, const b200q_qargs* qa) {
  if (N <= 0 || K <= 0 || !qa) return 0;
  switch (qa->strategy) {
    case B200Q_GROUP: case B200Q_TENSOR_GROUP: return qa->group_size > 0 ? N * ((K + qa->group_size - 1) / qa->group_size) : 0;
    case B200Q_CHANNEL: return N;
    case B200Q_BLOCK:
      return qa->block_h > 0 && qa->block_w > 0 ? ((N + qa->block_h - 1) / qa->block_h) * ((K + qa->block_w - 1) / qa->block_w) : 0;
    default: return 0;
  }
}

size_t b200q_observe_mse_workspace_bytes(int64_t N, int64_t K, const b200q_qargs* qa, int steps) {
  const size_t flags = mse_flag_bytes(steps);
  if (qa && qa->strategy == B200Q_TENSOR)   // search state and per-CTA partials
    return flags + sizeof(float) * (size_t)(b200q::mse::kSpanState + 2 * 4 * b200q::kNumSMs);
  return flags + b200q::mse::kTableBytes + 256 + (steps <= 32 ? sizeof(uint32_t) * (size_t)mse_groups(N, K, qa) : 0);   // (the table starts on a 16-byte boundary of whatever it is given)
}

}  // extern "C"

// `table`: 64 KiB for the powers of bf16 errors, 16-byte aligned; `notes`: 4 bytes a group (null: the search runs twice)
static int observe_mse(const void* W, int wdtype, int64_t N, int64_t K, int64_t ldw, const b200q_qargs* qa,
                       double maxshrink, int patience, double grid, float norm, float expand, void* mn_out,
                       void* mx_out, void* scratch, void* table_mem, void* notes, void* stream) {
  using namespace b200q::mse;
  if (!W || !qa || !mn_out || !mx_out || !scratch || N <= 0 || K <= 0 || ldw < K) return B200Q_ERR_ARG;
  if (wdtype != B200Q_BF16 && wdtype != B200Q_F32) return B200Q_ERR_UNSUPPORTED;
  QRange qr;
  int rc = make_qrange(qa, &qr); if (rc) return rc;
  Cfg c;
  c.symmetric = qa->symmetric; c.scale_kind = qa->scale_kind; c.zp_kind = qa->zp_kind;
  c.mx_offset = (qa->num_bits == 4) ? 2 : 8;
  c.qmin = qr.qmin; c.qmax = qr.qmax; c.range = qr.qmax - qr.qmin; c.half_range = c.range / 2.0f; c.kind = qr.kind;
  c.inv_half_range = 1.0f / c.half_range;
  if (!qa->symmetric && qr.kind == kFp4) return B200Q_ERR_UNSUPPORTED;
  if (qa->scale_kind == B200Q_SCALE_FP8) c.eps = 0.125f;
  else if (qa->scale_kind == B200Q_SCALE_E8M0) c.eps = 1.0f;
  else c.eps = (wdtype == B200Q_BF16) ? 0.0078125f : 1.1920928955078125e-07f;
  c.steps = b200q_observe_mse_steps(maxshrink, grid);
  c.patience = patience; c.grid = grid; c.norm = norm; c.expand = expand;
  if (wdtype == B200Q_BF16) {
    // torch casts the python exponent to the tensor's dtype: |e|.pow(2.4) on bf16 uses 2.40625
    uint32_t b;
    memcpy(&b, &norm, 4);
    b = (b + 0x7FFFu + ((b >> 16) & 1u)) & 0xFFFF0000u;
    memcpy(&c.norm, &b, 4);
  }
  if (c.steps < 0) return B200Q_ERR_ARG;
  cudaStream_t st = (cudaStream_t)stream;
  int* ctl = (int*)scratch;
  const bool grp = qa->strategy == B200Q_GROUP || qa->strategy == B200Q_TENSOR_GROUP;
  // bf16 weights in whole 16-byte pieces: the table-driven kernels
  const bool blk = qa->strategy == B200Q_BLOCK;
  const bool packed = wdtype == B200Q_BF16 && qa->strategy != B200Q_TENSOR && (K & 7) == 0 && (ldw & 7) == 0 &&
                      (((uintptr_t)W) & 15) == 0 && (!blk || (qa->block_w > 0 && qa->block_w % 8 == 0)) &&
                      (qr.kind != kInt || qa->num_bits == 4 || qa->num_bits == 8);
  __nv_bfloat16* table = (__nv_bfloat16*)table_mem;
  uint32_t* better = packed && (qa->symmetric || qr.kind == kInt) && c.steps <= 32 ? (uint32_t*)notes : nullptr;
  if (packed) make_table_kernel<<<kTable / 256, 256, 0, st>>>(table, c.norm, ctl, c.steps + 1);
  else clear_ctl_kernel<<<1, 128, 0, st>>>(ctl, c.steps + 1);
  B200Q_LAUNCH_CHECK();
#define B200Q_MSE_PICK(fn, ...)                                                                                     \
  do {                                                                                                              \
    if (qr.kind == kFp8) rc = fn<kMseFp8, true>(__VA_ARGS__);                                                       \
    else if (qr.kind == kFp4) rc = fn<kMseFp4, true>(__VA_ARGS__);                                                  \
    else if (qa->num_bits == 4) rc = qa->symmetric ? fn<kMseInt4, true>(__VA_ARGS__) : fn<kMseInt4, false>(__VA_ARGS__); \
    else rc = qa->symmetric ? fn<kMseInt8, true>(__VA_ARGS__) : fn<kMseInt8, false>(__VA_ARGS__);                    \
    if (rc) return rc;                                                                                              \
  } while (0)
  for (int pass = 0; pass < 2; ++pass) {
    if (grp) {
      int g = qa->group_size;
      if (!(g >= 8 && g <= 256 && (g & (g - 1)) == 0 && K % g == 0)) return B200Q_ERR_UNSUPPORTED;
      int grid_sz = grid_for((N * (K >> 3) + 255) / 256, 4);
      if (packed && (qa->symmetric || qr.kind == kInt)) B200Q_MSE_PICK(launch_group, W, N, K, ldw, g, c, table, ctl, pass, mn_out, mx_out, better, st);
      else if (wdtype == B200Q_BF16) mse_group_kernel<B200Q_BF16><<<grid_sz, 256, 0, st>>>(W, N, K, ldw, g, c, ctl, pass, mn_out, mx_out);
      else mse_group_kernel<B200Q_F32><<<grid_sz, 256, 0, st>>>(W, N, K, ldw, g, c, ctl, pass, mn_out, mx_out);
    } else if (qa->strategy == B200Q_CHANNEL || qa->strategy == B200Q_BLOCK) {
      if (blk && (qa->block_h <= 0 || qa->block_w <= 0)) return B200Q_ERR_ARG;
      const int64_t bh = blk ? qa->block_h : 1, bw = blk ? qa->block_w : K;
      const size_t smem = (size_t)(bh * bw) * sizeof(float);
      if (bh * bw > (int64_t)50 * 1024) return B200Q_ERR_UNSUPPORTED;   // group does not fit in shared memory
      const int64_t groups = ((N + bh - 1) / bh) * ((K + bw - 1) / bw);
      int grid_sz = grid_for(groups, smem > 100 * 1024 ? 1 : 2);
      if (packed && (qa->symmetric || qr.kind == kInt)) B200Q_MSE_PICK(launch_tile, W, N, K, ldw, (int)bh, (int)bw, c, table, ctl, pass, mn_out, mx_out, better, st);
      else if (wdtype == B200Q_BF16) {
        B200Q_TRY(cudaFuncSetAttribute(mse_tile_kernel<B200Q_BF16>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        mse_tile_kernel<B200Q_BF16><<<grid_sz, 256, smem, st>>>(W, N, K, ldw, (int)bh, (int)bw, c, ctl, pass, mn_out, mx_out);
      } else {
        B200Q_TRY(cudaFuncSetAttribute(mse_tile_kernel<B200Q_F32>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        mse_tile_kernel<B200Q_F32><<<grid_sz, 256, smem, st>>>(W, N, K, ldw, (int)bh, (int)bw, c, ctl, pass, mn_out, mx_out);
      }
    } else if (qa->strategy == B200Q_TENSOR) {
      // one group: the search runs candidate by candidate, with its state on the device
      if (pass == 1) break;
      float* state = (float*)(ctl + c.steps + 1);
      float* partial = state + kSpanState;
      const int nblk = grid_for((N * K + 255) / 256, 4);
      const bool tb = wdtype == B200Q_BF16;
      if (tb) mse_span_range_kernel<B200Q_BF16><<<nblk, 256, 0, st>>>(W, N, K, ldw, partial);
      else mse_span_range_kernel<B200Q_F32><<<nblk, 256, 0, st>>>(W, N, K, ldw, partial);
      B200Q_LAUNCH_CHECK();
      if (tb) mse_span_init_kernel<true><<<1, 1, 0, st>>>(state, partial, nblk, c);
      else mse_span_init_kernel<false><<<1, 1, 0, st>>>(state, partial, nblk, c);
      B200Q_LAUNCH_CHECK();
      for (int i = 0; i < c.steps; ++i) {
        if (tb) mse_span_error_kernel<B200Q_BF16><<<nblk, 256, 0, st>>>(W, N, K, ldw, c, i, state, partial);
        else mse_span_error_kernel<B200Q_F32><<<nblk, 256, 0, st>>>(W, N, K, ldw, c, i, state, partial);
        B200Q_LAUNCH_CHECK();
        if (tb) mse_span_fold_kernel<true><<<1, 1, 0, st>>>(state, partial, nblk, c, i);
        else mse_span_fold_kernel<false><<<1, 1, 0, st>>>(state, partial, nblk, c, i);
        B200Q_LAUNCH_CHECK();
      }
      if (tb) mse_span_store_kernel<B200Q_BF16><<<1, 1, 0, st>>>(state, mn_out, mx_out);
      else mse_span_store_kernel<B200Q_F32><<<1, 1, 0, st>>>(state, mn_out, mx_out);
      B200Q_LAUNCH_CHECK();
      return B200Q_OK;
    } else {
      return B200Q_ERR_UNSUPPORTED;
    }
    B200Q_LAUNCH_CHECK();
    if (better) {
      const int64_t groups = mse_groups(N, K, qa);
      pick_kernel<<<grid_for((groups + 255) / 256, 4), 256, 0, st>>>(ctl, better, groups, c, (__nv_bfloat16*)mn_out,
                                                                     (__nv_bfloat16*)mx_out);
      B200Q_LAUNCH_CHECK();
      break;
    }
    if (pass == 0) {
      stop_step_kernel<<<1, 1, 0, st>>>(ctl, c.steps, c.patience);
      B200Q_LAUNCH_CHECK();
    }
  }
#undef B200Q_MSE_PICK
  return B200Q_OK;
}

extern "C" int b200q_observe_mse(const void* W, int wdtype, int64_t N, int64_t K, int64_t ldw, const b200q_qargs* qa,
                                 double maxshrink, int patience, double grid, float norm, float expand, void* mn_out,
                                 void* mx_out, void* scratch, void* stream) {
  if (!scratch) return B200Q_ERR_ARG;
  const int steps = b200q_observe_mse_steps(maxshrink, grid);
  if (steps < 0) return B200Q_ERR_ARG;
  const uintptr_t table = ((uintptr_t)scratch + mse_flag_bytes(steps) + 15) & ~(uintptr_t)15;
  return observe_mse(W, wdtype, N, K, ldw, qa, maxshrink, patience, grid, norm, expand, mn_out, mx_out, scratch,
                     (void*)table, (void*)(table + b200q::mse::kTableBytes), stream);
}

// ---------------------------------------------------------------------------------------
// Allocation-free variant of b200q_observe_mse.
//
// Some callers cannot obtain device memory at the moment they need an MSE observation: a
// serving process that has handed its whole memory budget to a KV-cache pool and re-calibrates
// a layer in place, code running inside a framework callback where the caching allocator must
// not be re-entered, or a C program that links this library without any allocator of its own.
// For them the search's scratch (one flag per shrink candidate plus the stop step, 4 KiB, and the 64 KiB
// table of powers of bf16 errors) lives in fixed arrays inside the library image instead of a
// caller-supplied buffer.  Calls that overlap on the GPU would share both: the caller keeps them on one stream.
namespace b200q {
namespace mse {

constexpr int kStaticMaxSteps = 1023;  // candidates; the array holds kStaticMaxSteps + 1 ints (4 KiB)
static __device__ __align__(256) int g_static_ctl[kStaticMaxSteps + 1];
static __device__ __align__(256) __nv_bfloat16 g_static_table[kTable];   // powers of bf16 errors

constexpr int kMaxDevices = 64;
static int* g_static_ctl_ptr[kMaxDevices] = {nullptr};
static void* g_static_table_ptr[kMaxDevices] = {nullptr};
static std::mutex g_static_mutex;

// Device addresses of the arrays on the current device.  In host code the symbols' names are only
// handles, not addresses, so they are resolved once per device with cudaGetSymbolAddress.
static int static_addresses(int** out, void** table) {
  int dev = -1;
  B200Q_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kMaxDevices) return B200Q_ERR_UNSUPPORTED;
  std::lock_guard<std::mutex> lock(g_static_mutex);
  if (g_static_ctl_ptr[dev] == nullptr) {
    void* p = nullptr;
    B200Q_TRY(cudaGetSymbolAddress(&p, g_static_ctl));
    if (p == nullptr) return B200Q_ERR_CUDA;
    void* t = nullptr;
    B200Q_TRY(cudaGetSymbolAddress(&t, g_static_table));
    if (t == nullptr) return B200Q_ERR_CUDA;
    g_static_table_ptr[dev] = t;
    g_static_ctl_ptr[dev] = static_cast<int*>(p);
  }
  *out = g_static_ctl_ptr[dev];
  *table = g_static_table_ptr[dev];
  return B200Q_OK;
}

}  // namespace mse
}  // namespace b200q

extern "C" int b200q_observe_mse_noalloc(const void* W, int wdtype, int64_t N, int64_t K, int64_t ldw,
                                         const b200q_qargs* qa, double maxshrink, int patience, double grid,
                                         float norm, float expand, void* mn_out, void* mx_out, void* stream) {
  using namespace b200q::mse;
  const int steps = b200q_observe_mse_steps(maxshrink, grid);
  if (steps < 0 || steps > kStaticMaxSteps) {
    b200q::set_last_error("b200q_observe_mse_noalloc: int(maxshrink*grid) exceeds the built-in scratch (1023 candidates)",
                          cudaErrorInvalidValue);
    return B200Q_ERR_ARG;
  }
  if (qa && qa->strategy == B200Q_TENSOR) {
    // the whole-tensor search keeps per-CTA partial sums in its scratch, more than the array holds
    b200q::set_last_error("b200q_observe_mse_noalloc: the TENSOR strategy needs more scratch than the built-in array",
                          cudaErrorInvalidValue);
    return B200Q_ERR_UNSUPPORTED;
  }
  int* ctl = nullptr;
  void* table = nullptr;
  int rc = static_addresses(&ctl, &table);
  if (rc != B200Q_OK) return rc;
  // the search clears the flags it uses before its first pass, so the contents left by the
  // previous call do not matter
  return observe_mse(W, wdtype, N, K, ldw, qa, maxshrink, patience, grid, norm, expand, mn_out, mx_out, ctl, table, nullptr,
                     stream);
}
