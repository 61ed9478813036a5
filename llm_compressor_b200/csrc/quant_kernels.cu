// HBM-bound kernels of the observer / qparams / quantize / pack path (sm_100a).
//
// All kernels stream the weight matrix once with 16-byte loads, keep the group
// statistics in registers (warp shuffles between the lanes that share a group) and
// write packed codes with 4..16-byte stores.  Grids are whole multiples of the SM count.
#include "common.cuh"

#include <algorithm>
#include <atomic>
#include <cstdlib>
#include <mutex>
#include <string>

namespace b200q {

static thread_local std::string g_last_error;
static std::atomic<long long> g_launches{0};
void count_launch() { g_launches.fetch_add(1, std::memory_order_relaxed); }
void set_last_error(const char* what, cudaError_t e) {
  g_last_error = std::string(what) + ": " + cudaGetErrorString(e);
}

// ----------------------------------------------------------------------------------------
// qparams of one group, in the statistics' dtype (TB: bf16), following calculate_qparams.
struct QParamCfg {
  int symmetric, scale_kind, zp_kind, mx_offset, has_global;
  float qmin, qmax, half_range, range, eps;
  float inv_half_range, inv_range;   // float32 reciprocals, used for bf16 statistics (see qparams_one)
};

static int make_qparam_cfg(const b200q_qargs* qa, bool stat_bf16, bool has_global, QParamCfg* c) {
  QRange r;
  int st = make_qrange(qa, &r);
  if (st) return st;
  c->symmetric = qa->symmetric; c->scale_kind = qa->scale_kind; c->zp_kind = qa->zp_kind;
  c->has_global = has_global ? 1 : 0;
  c->qmin = r.qmin; c->qmax = r.qmax; c->range = r.qmax - r.qmin; c->half_range = c->range / 2.0f;
  c->inv_half_range = 1.0f / c->half_range; c->inv_range = 1.0f / c->range;
  c->mx_offset = (qa->num_bits == 4) ? 2 : 8;
  if (qa->scale_kind == B200Q_SCALE_E8M0 &&
      !(qa->qtype == B200Q_QFLOAT && qa->group_size == 32 && qa->symmetric))
    return B200Q_ERR_UNSUPPORTED;
  if (!qa->symmetric && r.kind == kFp4) return B200Q_ERR_UNSUPPORTED;
  if (qa->scale_kind == B200Q_SCALE_FP8) c->eps = 0.125f;
  else if (qa->scale_kind == B200Q_SCALE_E8M0) c->eps = 1.0f;
  else c->eps = (stat_bf16 && !has_global) ? 0.0078125f : 1.1920928955078125e-07f;
  return B200Q_OK;
}

template <bool TB>
__device__ __forceinline__ void qparams_one(float mn, float mx, const QParamCfg& c, float g,
                                            float& scale, float& zp) {
  mn = fminf(mn, 0.0f);
  mx = fmaxf(mx, 0.0f);
  float s;
  if (c.symmetric) {
    float amax = fmaxf(fabsf(mn), fabsf(mx));
    if (c.scale_kind == B200Q_SCALE_E8M0) {
      // keep sign+exponent after adding a quarter exponent step to the mantissa
      int biased;
      if (TB) {
        uint32_t b = __float_as_uint(amax) >> 16;
        b = (b + 32u) & 0xFF80u;
        biased = (int)((b >> 7) & 0xFFu);
      } else {
        uint32_t b = __float_as_uint(amax);
        b = (b + (1u << 21)) & 0xFF800000u;
        biased = (int)((b >> 23) & 0xFFu);
      }
      s = (biased == 0) ? -INFINITY : (float)(biased - c.mx_offset);
    } else {
      // bf16 statistics: the quotient of an 8-bit significand by 7.5, 127.5, 448 or 6 stays at least
      // 129 float32 ulps away from every bf16 rounding midpoint (checked over all significands), so
      // the product with the float32 reciprocal rounds to the same bf16 value as the division
      s = TB ? bf16r(amax * c.inv_half_range) : __fdiv_rn(amax, c.half_range);
    }
    zp = 0.0f;
  } else {
    float d = rnd_if<TB>(mx - mn);
    s = TB ? bf16r(d * c.inv_range) : __fdiv_rn(d, c.range);
    float z = rnd_if<TB>(__fdiv_rn(mn, s));
    z = rnd_if<TB>(c.qmin - z);
    // 0/0 for an all-zero group: torch's clamp keeps the NaN and the integer cast makes it 0
    zp = (z != z) ? 0.0f : fminf(fmaxf(z, c.qmin), c.qmax);
  }
  if (c.has_global) s = g * s;
  if (c.scale_kind == B200Q_SCALE_FP8) {
    s = e4m3_round(fminf(fmaxf(s, -448.0f), 448.0f));
  } else if (c.scale_kind == B200Q_SCALE_E8M0) {
    float e = rintf(fminf(fmaxf(s, 0.0f), 255.0f));
    s = __uint_as_float(e >= 1.0f ? ((uint32_t)e << 23) : 0x00400000u);  // 2^(e-127)
  }
  if (s == 0.0f) s = c.eps;
  if (!c.symmetric) {   // a symmetric zero point is exactly 0 in every storage type
    if (c.zp_kind == B200Q_ZP_INT8) zp = rintf(fminf(fmaxf(zp, -128.0f), 127.0f));
    else if (c.zp_kind == B200Q_ZP_UINT8) zp = rintf(fminf(fmaxf(zp, 0.0f), 255.0f));
    else zp = e4m3_round(fminf(fmaxf(zp, -448.0f), 448.0f));
  }
  scale = s;
}

__device__ __forceinline__ void store_zp(void* out, int zp_kind, int64_t i, float zp) {
  if (zp_kind == B200Q_ZP_INT8) ((int8_t*)out)[i] = (int8_t)zp;
  else if (zp_kind == B200Q_ZP_UINT8) ((uint8_t*)out)[i] = (uint8_t)zp;
  else ((uint8_t*)out)[i] = e4m3_bits(zp);
}

// 127 + floor(log2 s) of a positive power-of-two scale (also right for any positive float).
__device__ __forceinline__ uint8_t e8m0_of(float s) {
  uint32_t b = __float_as_uint(s);
  uint32_t e = (b >> 23) & 0xFFu;
  if (e == 0) {  // subnormal float: 2^-127 has mantissa 0x400000
    uint32_t m = b & 0x7FFFFFu;
    if (m == 0) return 0;
    int lz = __clz(m) - 9;  // leading zeros inside the 23-bit mantissa
    int v = 127 + (-127 - lz);
    return (uint8_t)(v < 0 ? 0 : v);
  }
  return (uint8_t)e;
}

// ----------------------------------------------------------------------------------------
// 8 consecutive elements of a row as floats
template <int DT>
__device__ __forceinline__ void load8(const void* base, int64_t off, float (&v)[8]) {
  if constexpr (DT == B200Q_BF16) {
    uint4 u = __ldg(reinterpret_cast<const uint4*>((const __nv_bfloat16*)base + off));
    const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      v[2 * i] = __uint_as_float(w[i] << 16);
      v[2 * i + 1] = __uint_as_float(w[i] & 0xFFFF0000u);
    }
  } else {
    const float4* p = reinterpret_cast<const float4*>((const float*)base + off);
    float4 a = __ldg(p), b = __ldg(p + 1);
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
    v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
  }
}
template <int DT>
__device__ __forceinline__ void store8(void* base, int64_t off, const float (&v)[8]) {
  if constexpr (DT == B200Q_BF16) {
    uint32_t w[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      __nv_bfloat162 h = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
      w[i] = *reinterpret_cast<uint32_t*>(&h);
    }
    *reinterpret_cast<uint4*>((__nv_bfloat16*)base + off) = make_uint4(w[0], w[1], w[2], w[3]);
  } else {
    float4* p = reinterpret_cast<float4*>((float*)base + off);
    p[0] = make_float4(v[0], v[1], v[2], v[3]);
    p[1] = make_float4(v[4], v[5], v[6], v[7]);
  }
}

}  // namespace b200q
#include "stream_kernels.cuh"
#include "stream_tma.cuh"
namespace b200q {

// ---- tensor map of a bf16 weight for the TMA-fed kernels: rows cut into 128-byte pieces -------
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
static EncodeTiledFn tensor_map_encoder() {
  static const EncodeTiledFn fn = [] {
    void* sym = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &qres) == cudaSuccess &&
        qres == cudaDriverEntryPointSuccess)
      return (EncodeTiledFn)sym;
    return (EncodeTiledFn) nullptr;
  }();
  return fn;
}
// dims (64 elements, K/64 pieces, N rows), box (64, 32, 1) = one 4 KiB tile, 128-byte swizzle
static bool make_weight_tile_map(CUtensorMap* m, const void* W, int64_t N, int64_t K, int64_t ldw) {
  EncodeTiledFn enc = tensor_map_encoder();
  if (!enc) return false;
  cuuint64_t dims[3] = {64u, (cuuint64_t)(K / 64), (cuuint64_t)N};
  cuuint64_t strides[2] = {128u, (cuuint64_t)ldw * 2u};
  cuuint32_t box[3] = {64u, 32u, 1u};
  cuuint32_t estr[3] = {1, 1, 1};
  return enc(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(W), dims, strides, box, estr,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}
static bool tma_path_enabled() {
  static const bool on = [] { const char* e = getenv("B200Q_STREAM_TMA"); return !(e && e[0] == '0'); }();
  return on;
}

static bool vec_ok(const void* p, int64_t K, int64_t ld, int elem_bytes) {
  return (K % 8 == 0) && (ld % 8 == 0) && (((uintptr_t)p) % 16 == 0) && elem_bytes > 0;
}
static bool pow2(int v) { return v > 0 && (v & (v - 1)) == 0; }

// ========================================================================================
// observe_minmax (the streaming group kernels are in stream_kernels.cuh)
// ========================================================================================
// generic: one thread per group, any sizes
template <int DT>
__global__ void minmax_generic_kernel(const void* __restrict__ W, int64_t N, int64_t K, int64_t ldw, int g,
                                      void* __restrict__ mn_out, void* __restrict__ mx_out) {
  using E = Elem<DT>;
  using T = typename E::type;
  const int64_t gpr = (K + g - 1) / g, total = N * gpr;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total;
       i += (int64_t)gridDim.x * blockDim.x) {
    int64_t r = i / gpr, c = i - r * gpr;
    float lo = INFINITY, hi = -INFINITY;
    for (int64_t x = c * g; x < min((int64_t)(c * g + g), K); ++x) {
      float v = E::load((const T*)W + r * ldw + x);
      lo = fminf(lo, v); hi = fmaxf(hi, v);
    }
    E::store((T*)mn_out + i, lo);
    E::store((T*)mx_out + i, hi);
  }
}

// BLOCK: a CTA per block (rows of the block over warps, 8 elements a lane, or an element a lane where the layout does
// not allow more).  HBM-bound from a few hundred blocks on; a thread per block, which the generic kernel gives it, took
// 1114 us for 128 x 128 blocks of 4096 x 4096.
template <int DT, bool VEC>
__global__ void __launch_bounds__(256) minmax_block_kernel(const void* __restrict__ W, int64_t N, int64_t K, int64_t ldw,
                                                           int bh, int bw, int64_t blocks_per_row, int64_t blocks,
                                                           void* __restrict__ mn_out, void* __restrict__ mx_out) {
  using E = Elem<DT>;
  using T = typename E::type;
  __shared__ float s_lo[8], s_hi[8];
  constexpr int PER = VEC ? 8 : 1;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int cw = bw / PER;
  for (int64_t b = blockIdx.x; b < blocks; b += gridDim.x) {
    const int64_t r0 = (b / blocks_per_row) * bh, c0 = (b % blocks_per_row) * bw;
    const int rows = (int)min((int64_t)bh, N - r0), cols = (int)min((int64_t)bw, K - c0);
    // zero padding of ragged blocks takes part in the statistics
    const bool ragged = rows < bh || cols < bw;
    float lo = ragged ? 0.0f : INFINITY, hi = ragged ? 0.0f : -INFINITY;
    const T* base = (const T*)W + r0 * ldw + c0;
#pragma unroll 4
    for (int i = threadIdx.x; i < rows * cw; i += 256) {
      const int y = i / cw, x = (i - y * cw) * PER;
      if (x >= cols) continue;
      if constexpr (VEC) {
        float v[8];
        load8<DT>(base, (int64_t)y * ldw + x, v);
#pragma unroll
        for (int k = 0; k < 8; ++k) { lo = fminf(lo, v[k]); hi = fmaxf(hi, v[k]); }
      } else {
        const float v = E::load(base + (int64_t)y * ldw + x);
        lo = fminf(lo, v); hi = fmaxf(hi, v);
      }
    }
    lo = warp_min(lo); hi = warp_max(hi);
    if (lane == 0) { s_lo[warp] = lo; s_hi[warp] = hi; }
    __syncthreads();
    if (threadIdx.x == 0) {
      for (int w = 1; w < 8; ++w) { lo = fminf(lo, s_lo[w]); hi = fmaxf(hi, s_hi[w]); }
      E::store((T*)mn_out + b, lo);
      E::store((T*)mx_out + b, hi);
    }
    __syncthreads();
  }
}

// CHANNEL: one CTA per row
template <int DT>
__global__ void __launch_bounds__(256) minmax_channel_kernel(const void* __restrict__ W, int64_t N,
                                                             int64_t K, int64_t ldw, bool vec,
                                                             void* __restrict__ mn_out,
                                                             void* __restrict__ mx_out) {
  using E = Elem<DT>;
  using T = typename E::type;
  __shared__ float s_lo[8], s_hi[8];
  for (int64_t row = blockIdx.x; row < N; row += gridDim.x) {
    float lo = INFINITY, hi = -INFINITY;
    if (vec) {
      for (int64_t c = threadIdx.x; c < (K >> 3); c += blockDim.x) {
        float v[8];
        load8<DT>(W, row * ldw + c * 8, v);
#pragma unroll
        for (int i = 0; i < 8; ++i) { lo = fminf(lo, v[i]); hi = fmaxf(hi, v[i]); }
      }
    } else {
      for (int64_t x = threadIdx.x; x < K; x += blockDim.x) {
        float v = E::load((const T*)W + row * ldw + x);
        lo = fminf(lo, v); hi = fmaxf(hi, v);
      }
    }
    lo = warp_min(lo); hi = warp_max(hi);
    if ((threadIdx.x & 31) == 0) { s_lo[threadIdx.x >> 5] = lo; s_hi[threadIdx.x >> 5] = hi; }
    __syncthreads();
    if (threadIdx.x == 0) {
      for (int w = 1; w < (blockDim.x >> 5); ++w) { lo = fminf(lo, s_lo[w]); hi = fmaxf(hi, s_hi[w]); }
      E::store((T*)mn_out + row, lo);
      E::store((T*)mx_out + row, hi);
    }
    __syncthreads();
  }
}

// TENSOR: per-CTA partials, then one CTA folds them
template <int DT>
__global__ void __launch_bounds__(256) minmax_tensor_partial_kernel(const void* __restrict__ W,
                                                                    int64_t N, int64_t K,
                                                                    int64_t ldw, bool vec,
                                                                    float* __restrict__ partial) {
  using E = Elem<DT>;
  using T = typename E::type;
  __shared__ float s_lo[8], s_hi[8];
  float lo = INFINITY, hi = -INFINITY;
  if (vec) {
    int64_t cpr = K >> 3, total = N * cpr;
    for (int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; c < total;
         c += (int64_t)gridDim.x * blockDim.x) {
      int64_t row = c / cpr, cc = c - row * cpr;
      float v[8];
      load8<DT>(W, row * ldw + cc * 8, v);
#pragma unroll
      for (int i = 0; i < 8; ++i) { lo = fminf(lo, v[i]); hi = fmaxf(hi, v[i]); }
    }
  } else {
    int64_t total = N * K;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total;
         i += (int64_t)gridDim.x * blockDim.x) {
      int64_t row = i / K, x = i - row * K;
      float v = E::load((const T*)W + row * ldw + x);
      lo = fminf(lo, v); hi = fmaxf(hi, v);
    }
  }
  lo = warp_min(lo); hi = warp_max(hi);
  if ((threadIdx.x & 31) == 0) { s_lo[threadIdx.x >> 5] = lo; s_hi[threadIdx.x >> 5] = hi; }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < (blockDim.x >> 5); ++w) { lo = fminf(lo, s_lo[w]); hi = fmaxf(hi, s_hi[w]); }
    partial[2 * blockIdx.x] = lo;
    partial[2 * blockIdx.x + 1] = hi;
  }
}
template <int DT>
__global__ void minmax_tensor_final_kernel(const float* __restrict__ partial, int n,
                                           void* __restrict__ mn_out, void* __restrict__ mx_out) {
  using E = Elem<DT>;
  using T = typename E::type;
  float lo = INFINITY, hi = -INFINITY;
  for (int i = threadIdx.x; i < n; i += 32) { lo = fminf(lo, partial[2 * i]); hi = fmaxf(hi, partial[2 * i + 1]); }
  lo = warp_min(lo); hi = warp_max(hi);
  if (threadIdx.x == 0) { E::store((T*)mn_out, lo); E::store((T*)mx_out, hi); }
}

constexpr int kTensorPartialBlocks = kNumSMs * 4;

template <int DT>
static int observe_minmax_impl(const void* W, int64_t N, int64_t K, int64_t ldw,
                               const b200q_qargs* qa, void* mn, void* mx, void* scratch, float* absmax,
                               cudaStream_t st) {
  const bool vec = vec_ok(W, K, ldw, 2);
  if (absmax && qa->strategy != B200Q_GROUP && qa->strategy != B200Q_TENSOR_GROUP) return B200Q_ERR_UNSUPPORTED;
  switch (qa->strategy) {
    case B200Q_GROUP:
    case B200Q_TENSOR_GROUP: {
      int g = qa->group_size;
      if (g <= 0) return B200Q_ERR_ARG;
      if (vec && pow2(g) && g >= 8 && g <= 256 && K % g == 0) {
        if constexpr (DT == B200Q_BF16) {
          const stream::GroupSplit gsp = stream::make_group_split(g);
          const int64_t slots = (K / g) * gsp.L;
          int tx2 = 32;
          while (tx2 < 256 && tx2 < slots) tx2 <<= 1;
          const int rows2 = stream::kThreads / tx2;
          const int grid2 = grid_for((N + rows2 - 1) / rows2, 8);
          const int txl2 = __builtin_ctz(tx2), ll2 = __builtin_ctz(gsp.L);
          if (gsp.R == 8) stream::minmax_group_bf16_kernel<8><<<grid2, stream::kThreads, 0, st>>>(W, (int)N, (int)K, ldw, g, ll2, txl2, mn, mx, absmax);
          else if (gsp.R == 4) stream::minmax_group_bf16_kernel<4><<<grid2, stream::kThreads, 0, st>>>(W, (int)N, (int)K, ldw, g, ll2, txl2, mn, mx, absmax);
          else if (gsp.R == 2) stream::minmax_group_bf16_kernel<2><<<grid2, stream::kThreads, 0, st>>>(W, (int)N, (int)K, ldw, g, ll2, txl2, mn, mx, absmax);
          else stream::minmax_group_bf16_kernel<1><<<grid2, stream::kThreads, 0, st>>>(W, (int)N, (int)K, ldw, g, ll2, txl2, mn, mx, absmax);
        } else {
          if (absmax) return B200Q_ERR_UNSUPPORTED;
          stream::RowTiling t = stream::make_tiling(N, K, 8);
          stream::minmax_group_kernel<DT><<<t.grid, stream::kThreads, 0, st>>>(W, (int)N, (int)K, ldw, g, __builtin_ctz(t.tx), mn, mx);
        }
      } else {
        if (absmax) return B200Q_ERR_UNSUPPORTED;
        int64_t total = N * ((K + g - 1) / g);
        minmax_generic_kernel<DT><<<grid_for((total + 127) / 128, 8), 128, 0, st>>>(W, N, K, ldw, g, mn, mx);
      }
      break;
    }
    case B200Q_BLOCK: {
      if (qa->block_h <= 0 || qa->block_w <= 0) return B200Q_ERR_ARG;
      const int64_t per_row = (K + qa->block_w - 1) / qa->block_w;
      const int64_t total = ((N + qa->block_h - 1) / qa->block_h) * per_row;
      // (K % 8 == 0: a chunk of 8 is inside the matrix as a whole)
      if (vec && qa->block_w % 8 == 0)
        minmax_block_kernel<DT, true><<<grid_for(total, 8), 256, 0, st>>>(W, N, K, ldw, qa->block_h, qa->block_w, per_row, total, mn, mx);
      else
        minmax_block_kernel<DT, false><<<grid_for(total, 8), 256, 0, st>>>(W, N, K, ldw, qa->block_h, qa->block_w, per_row, total, mn, mx);
      break;
    }
    case B200Q_CHANNEL:
      minmax_channel_kernel<DT><<<grid_for(N, 8), 256, 0, st>>>(W, N, K, ldw, vec, mn, mx);
      break;
    case B200Q_TENSOR: {
      if (!scratch) return B200Q_ERR_ARG;
      int blocks = grid_for((N * K / 8 + 255) / 256, 4);
      minmax_tensor_partial_kernel<DT><<<blocks, 256, 0, st>>>(W, N, K, ldw, vec, (float*)scratch);
      minmax_tensor_final_kernel<DT><<<1, 32, 0, st>>>((const float*)scratch, blocks, mn, mx);
      break;
    }
    default: return B200Q_ERR_ARG;
  }
  B200Q_LAUNCH_CHECK();
  return B200Q_OK;
}

// ========================================================================================
// global scale
// ========================================================================================
template <int DT>
__global__ void absmax_kernel(const void* __restrict__ mn, const void* __restrict__ mx, int64_t n,
                              float* __restrict__ absmax) {
  using E = Elem<DT>;
  using T = typename E::type;
  float a = 0.0f;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    a = fmaxf(a, fmaxf(fabsf(E::load((const T*)mn + i)), fabsf(E::load((const T*)mx + i))));
  }
  a = warp_max(a);
  // non-negative floats order like their bit patterns
  if ((threadIdx.x & 31) == 0) atomicMax(reinterpret_cast<int*>(absmax), __float_as_int(a));
}
// largest magnitude of a whole bf16 matrix, folded into *absmax: 16-byte loads, four in flight,
// sign bits cleared and a packed unsigned 16-bit maximum (bf16 magnitudes order like integers)
__global__ void __launch_bounds__(256) absmax_weight_bf16_kernel(const void* __restrict__ W, int64_t N, int64_t K,
                                                                 int64_t ldw, float* __restrict__ absmax) {
  const int64_t cpr = K >> 3, total = N * cpr;
  const int64_t step = (int64_t)gridDim.x * blockDim.x;
  uint32_t m = 0;
  int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  auto chunk = [&](int64_t i) {
    const int64_t row = i / cpr, cc = i - row * cpr;
    return stream::ldg_stream((const __nv_bfloat16*)W + row * ldw + cc * 8);
  };
  for (; c + 3 * step < total; c += 4 * step) {
    const uint4 a = chunk(c), b = chunk(c + step), d = chunk(c + 2 * step), e = chunk(c + 3 * step);
    const uint4 v[4] = {a, b, d, e};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      m = __vimax3_u16x2(m, v[k].x & 0x7FFF7FFFu, v[k].y & 0x7FFF7FFFu);
      m = __vimax3_u16x2(m, v[k].z & 0x7FFF7FFFu, v[k].w & 0x7FFF7FFFu);
    }
  }
  for (; c < total; c += step) {
    const uint4 a = chunk(c);
    m = __vimax3_u16x2(m, a.x & 0x7FFF7FFFu, a.y & 0x7FFF7FFFu);
    m = __vimax3_u16x2(m, a.z & 0x7FFF7FFFu, a.w & 0x7FFF7FFFu);
  }
  uint32_t h = max(m & 0xFFFFu, m >> 16);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) h = max(h, __shfl_xor_sync(0xffffffffu, h, o));
  __shared__ uint32_t s_m[8];
  if ((threadIdx.x & 31) == 0) s_m[threadIdx.x >> 5] = h;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < (int)(blockDim.x >> 5); ++w) h = max(h, s_m[w]);
    // non-negative floats order like their bit patterns
    atomicMax(reinterpret_cast<int*>(absmax), (int)(h << 16));
  }
}

__device__ __forceinline__ float global_scale_of(float a, bool stat_bf16) {
  float tiny = 1.17549435e-38f;  // smallest normal of both bf16 and float32
  a = fmaxf(a, tiny);
  // "scalar / tensor" in torch is tensor.reciprocal() * scalar: two roundings in the statistics' dtype
  float r = __frcp_rn(a);
  if (stat_bf16) r = bf16r(r);
  float g = __fmul_rn(r, 448.0f * 6.0f);
  if (stat_bf16) g = bf16r(g);
  if (!(fabsf(g) <= 3.402823466e38f)) g = 1.0f;  // NaN / Inf -> 1
  return g;
}
__global__ void global_scale_kernel(const float* __restrict__ absmax, int stat_bf16,
                                    float* __restrict__ out) {
  *out = global_scale_of(*absmax, stat_bf16 != 0);
}

// ========================================================================================
// qparams
// ========================================================================================
template <int DT, bool GLOBAL>
__global__ void qparams_kernel(const void* __restrict__ mn, const void* __restrict__ mx, int64_t n,
                               QParamCfg c, const float* __restrict__ gscale,
                               void* __restrict__ scale_out, void* __restrict__ zp_out) {
  using E = Elem<DT>;
  using T = typename E::type;
  float g = GLOBAL ? *gscale : 1.0f;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    float s, z;
    qparams_one<E::is_bf16>(E::load((const T*)mn + i), E::load((const T*)mx + i), c, g, s, z);
    if (GLOBAL) ((float*)scale_out)[i] = s;
    else E::store((T*)scale_out + i, s);
    if (zp_out) store_zp(zp_out, c.zp_kind, i, z);
  }
}

// ========================================================================================
// statistics -> qparams in one pass, for one weight or a batch of weights of one shape
// ========================================================================================
// What min / max and qparams kernels do one after the other for a memoryless min-max observer, without the statistics
// in between: bf16 weights in 16-byte pieces, the scale in the weight's dtype.  blockIdx.y = weight.  (By MinMax2, which
// leaves a NaN out as the separate kernels do; RangeQ loses the chunk's other values with it.)
struct StatJob {
  const void* one; const void* const* table;   // the weight, or a device array of them
  void* scale; void* zp;                       // [count][entries], contiguous
  int64_t entries;
  __device__ __forceinline__ const __nv_bfloat16* weight() const { return (const __nv_bfloat16*)(table ? table[blockIdx.y] : one); }
  __device__ __forceinline__ void put(int64_t i, float lo, float hi, const QParamCfg& c) const {
    float s, z;
    qparams_one<true>(lo, hi, c, 1.0f, s, z);
    const int64_t at = blockIdx.y * entries + i;
    ((__nv_bfloat16*)scale)[at] = __float2bfloat16_rn(s);
    if (zp) store_zp(zp, c.zp_kind, at, z);
  }
};
// groups of R * L chunks: the lane / chunk split of the fused round-to-nearest kernel
template <int R>
__global__ void __launch_bounds__(256) group_qparams_kernel(StatJob j, int N, int K, int64_t ldw, int l_log2, int tx_log2,
                                                            QParamCfg qc) {
  const int TX = 1 << tx_log2, rows = 256 >> tx_log2, L = 1 << l_log2;
  const int tx = threadIdx.x & (TX - 1), ty = threadIdx.x >> tx_log2;
  const int cpg = R << l_log2, gpr = (K >> 3) / cpg, slots = gpr << l_log2, send = (slots + 31) & ~31;
  const __nv_bfloat16* W = j.weight();
  for (int row = blockIdx.x * rows + ty; row < N; row += gridDim.x * rows) {
    const __nv_bfloat16* wrow = W + (int64_t)row * ldw;
    for (int t = tx; t < send; t += TX) {
      const bool live = t < slots;
      const int grp = t >> l_log2, ln = t & (L - 1);
      const int c0 = grp * cpg + ln;
      uint4 raw[R];
#pragma unroll
      for (int k = 0; k < R; ++k)
        raw[k] = live ? stream::ldg_stream(wrow + (int64_t)(c0 + k * L) * 8) : make_uint4(0, 0, 0, 0);
      stream::MinMax2 r;
      r.first(raw[0]);
#pragma unroll
      for (int k = 1; k < R; ++k) r.add(raw[k]);
      float lo, hi;
      r.finish(lo, hi);
      for (int o = L >> 1; o > 0; o >>= 1) {
        lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, o));
        hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, o));
      }
      if (live && ln == 0) j.put((int64_t)row * gpr + grp, lo, hi, qc);
    }
  }
}
// rows, a warp each: no barrier between the rows of a CTA, whose loads follow one another (25 us for 6001 x 7168 with a
// CTA per row).  For fewer rows than a few warps per SM scheduler the CTA per row below.
__global__ void __launch_bounds__(256) row_qparams_kernel(StatJob j, int64_t N, int64_t K, int64_t ldw, QParamCfg qc) {
  const int lane = threadIdx.x & 31;
  const __nv_bfloat16* W = j.weight();
  const int64_t warps = (int64_t)gridDim.x * 8;
  for (int64_t r = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5); r < N; r += warps) {
    const __nv_bfloat16* row = W + r * ldw;
    stream::MinMax2 q;
    q.mn = q.mx = __nv_bfloat162(0.0f, 0.0f);   // (zeros change nothing: the range is made to contain zero anyway)
    int64_t c = lane * 8;
    for (; c + 7 * 256 < K; c += 8 * 256) {
      uint4 raw[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) raw[k] = stream::ldg_stream(row + c + k * 256);
#pragma unroll
      for (int k = 0; k < 8; ++k) q.add(raw[k]);
    }
#pragma unroll 4
    for (; c < K; c += 256) q.add(stream::ldg_stream(row + c));
    float lo, hi;
    q.finish(lo, hi);
    lo = warp_min(lo); hi = warp_max(hi);
    if (lane == 0) j.put(r, lo, hi, qc);
  }
}
// rows (bh = 1, bw = K) or bh x bw blocks: a CTA each
__global__ void __launch_bounds__(256) span_qparams_kernel(StatJob j, int64_t N, int64_t K, int64_t ldw, int bh, int bw,
                                                           int64_t per_row, int64_t spans, int cw_log2, QParamCfg qc) {
  __shared__ float s_lo[2][8], s_hi[2][8];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, cw = bw >> 3;
  const __nv_bfloat16* W = j.weight();
  int par = 0;
  for (int64_t b = blockIdx.x; b < spans; b += gridDim.x, par ^= 1) {
    const int64_t br = b / per_row, r0 = br * bh, c0 = (b - br * per_row) * bw;
    const int rows = (int)min((int64_t)bh, N - r0), cols = (int)min((int64_t)bw, K - c0);
    const __nv_bfloat16* base = W + r0 * ldw + c0;
    // (the zero padding of ragged blocks changes nothing: the range is made to contain zero anyway)
    float lo = 0.0f, hi = 0.0f;
#pragma unroll 4
    for (int i = threadIdx.x; i < rows * cw; i += 256) {
      const int y = cw_log2 >= 0 ? i >> cw_log2 : i / cw, x = (i - y * cw) * 8;
      if (x >= cols) continue;
      stream::MinMax2 r;
      r.first(stream::ldg_stream(base + (int64_t)y * ldw + x));
      float l, h;
      r.finish(l, h);
      lo = fminf(lo, l); hi = fmaxf(hi, h);
    }
    lo = warp_min(lo); hi = warp_max(hi);
    if (lane == 0) { s_lo[par][warp] = lo; s_hi[par][warp] = hi; }
    __syncthreads();   // one barrier per span: the buffers alternate
    if (threadIdx.x == 0) {
      for (int w = 1; w < 8; ++w) { lo = fminf(lo, s_lo[par][w]); hi = fmaxf(hi, s_hi[par][w]); }
      j.put(b, lo, hi, qc);
    }
  }
}

// The same for symmetric schemes with a global scale that up to eight contiguous weights share: a symmetric scale needs only
// the largest magnitude of its group, so that is what pass one leaves in the place of the scale (while it finds the
// largest of all), and pass two turns it into the scale.  W is read once; the statistics of the separate kernels
// (min, max, float32 scale, copy) moved another 66 bytes a group.  blockIdx.y = weight.
constexpr int kMaxShared = 8;
struct SharedJob {
  const __nv_bfloat16* w[kMaxShared];
  __nv_bfloat16* scale[kMaxShared];
  void* zp[kMaxShared];
  float* global_scale[kMaxShared];
  int64_t groups[kMaxShared];
  float* absmax;
};
template <int R>
__global__ void __launch_bounds__(256) shared_absmax_kernel(const __grid_constant__ SharedJob j) {
  const int64_t n = j.groups[blockIdx.y], step = (int64_t)gridDim.x * 256;
  const uint4* w = reinterpret_cast<const uint4*>(j.w[blockIdx.y]);
  __nv_bfloat16* out = j.scale[blockIdx.y];
  constexpr int U = 8 / R;      // groups of a thread whose loads are in flight together
  float top = 0.0f;
  for (int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x; i < n; i += U * step) {
    uint4 raw[U][R];
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int r = 0; r < R; ++r)
        raw[u][r] = i + u * step < n ? stream::ldg_stream(w + (i + u * step) * R + r) : make_uint4(0, 0, 0, 0);
#pragma unroll
    for (int u = 0; u < U; ++u) {
      __nv_bfloat162 m = __float2bfloat162_rn(0.0f);
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const __nv_bfloat162* e = reinterpret_cast<const __nv_bfloat162*>(&raw[u][r]);
#pragma unroll
        for (int q = 0; q < 4; ++q) m = __hmax2(m, __habs2(e[q]));
      }
      const __nv_bfloat16 a = __hmax(m.x, m.y);
      if (i + u * step < n) out[i + u * step] = a;
      top = fmaxf(top, __bfloat162float(a));
    }
  }
  top = warp_max(top);
  if ((threadIdx.x & 31) == 0) atomicMax(reinterpret_cast<int*>(j.absmax), __float_as_int(top));
}
__global__ void __launch_bounds__(256) shared_qparams_kernel(const __grid_constant__ SharedJob j, QParamCfg qc) {
  const float g = global_scale_of(*j.absmax, true);
  const int64_t n = j.groups[blockIdx.y];
  __nv_bfloat16* scale = j.scale[blockIdx.y];
  void* zp = j.zp[blockIdx.y];
  if (blockIdx.x == 0 && threadIdx.x == 0) *j.global_scale[blockIdx.y] = g;
  for (int64_t i = ((int64_t)blockIdx.x * 256 + threadIdx.x) * 8; i < n; i += (int64_t)gridDim.x * 2048) {
    const int m = (int)(n - i < 8 ? n - i : 8);
    alignas(16) __nv_bfloat16 v[8];
    if (m == 8) *reinterpret_cast<uint4*>(v) = *reinterpret_cast<const uint4*>(scale + i);
    else for (int e = 0; e < m; ++e) v[e] = scale[i + e];
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      if (e >= m) break;
      float s, z;
      const float a = __bfloat162float(v[e]);
      qparams_one<true>(-a, a, qc, g, s, z);
      v[e] = __float2bfloat16_rn(s);
    }
    if (m == 8) {
      *reinterpret_cast<uint4*>(scale + i) = *reinterpret_cast<const uint4*>(v);
      *reinterpret_cast<uint2*>((uint8_t*)zp + i) = make_uint2(0u, 0u);   // (zero in every storage type)
    } else {
      for (int e = 0; e < m; ++e) { scale[i + e] = v[e]; ((uint8_t*)zp)[i + e] = 0; }
    }
  }
}

// ========================================================================================
// fake_quantize / quantize_pack with given parameters
// ========================================================================================
enum PackMode { kPackFake = 0, kPackInt4 = 1, kPackByte = 2, kPackFp4 = 3, kPackInt8Word = 4 };

template <int SDT>
__device__ __forceinline__ float load_scale(const void* scale, int64_t i) {
  return Elem<SDT>::load((const typename Elem<SDT>::type*)scale + i);
}

// Scalar path for ragged shapes: one thread per output unit (word / byte / element).
template <int XDT, int SDT, bool GLOBAL, int MODE>
__global__ void quant_scalar_kernel(const void* __restrict__ W, int64_t N, int64_t K, int64_t ldw,
                                    const void* __restrict__ scale, const void* __restrict__ zp,
                                    int zp_kind, ParamMap pm, const float* __restrict__ gscale,
                                    QRange qr, void* __restrict__ out, int64_t ldo) {
  using EX = Elem<XDT>;
  constexpr bool XB = EX::is_bf16;
  constexpr bool SB = Elem<SDT>::is_bf16 && !GLOBAL;
  constexpr bool CB = XB && SB;
  constexpr int per = (MODE == kPackInt4) ? 8 : (MODE == kPackInt8Word) ? 4 : (MODE == kPackFp4) ? 2 : 1;
  const float g = GLOBAL ? *gscale : 1.0f;
  const int64_t upr = (K + per - 1) / per, total = N * upr;
  for (int64_t u = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; u < total;
       u += (int64_t)gridDim.x * blockDim.x) {
    int64_t row = u / upr, uc = u - row * upr;
    uint32_t word = 0;
    for (int i = 0; i < per; ++i) {
      int64_t col = uc * per + i;
      if (col >= K) break;  // zero padding of the last word
      int64_t pi = pm.index(row, col);
      float s = load_scale<SDT>(scale, pi);
      if (GLOBAL) s = __fdiv_rn(s, g);
      float z = zp ? load_zp(zp, zp_kind, pi) : 0.0f;
      float x = EX::load((const typename EX::type*)W + row * ldw + col);
      float q = quant_code<CB>(x, s, z, qr);
      if constexpr (MODE == kPackFake) {
        EX::store((typename EX::type*)out + row * ldo + col, dequant_code<SB>(q, s, z));
      } else if constexpr (MODE == kPackInt4) {
        word |= ((uint32_t)((int)q + 8) & 0xFu) << (4 * i);
      } else if constexpr (MODE == kPackInt8Word) {
        word |= ((uint32_t)((int)q + 128) & 0xFFu) << (8 * i);
      } else if constexpr (MODE == kPackFp4) {
        word |= e2m1_nibble(q) << (4 * i);
      } else {
        word = (qr.kind == kFp8) ? e4m3_bits(q) : ((uint32_t)(int)q & 0xFFu);
      }
    }
    if constexpr (MODE == kPackInt4 || MODE == kPackInt8Word) ((uint32_t*)out)[u] = word;
    else if constexpr (MODE == kPackFp4 || MODE == kPackByte) ((uint8_t*)out)[u] = (uint8_t)word;
  }
}

template <int XDT, int SDT, bool GLOBAL, int MODE>
static int quant_launch(const void* W, int64_t N, int64_t K, int64_t ldw, const void* scale,
                        const void* zp, int zp_kind, const ParamMap& pm, const float* gscale,
                        const QRange& qr, void* out, int64_t ldo, cudaStream_t st) {
  bool vec = vec_ok(W, K, ldw, 2) && (((uintptr_t)out) % 16 == 0) &&
             (MODE != kPackFake || ldo % 8 == 0);
  if (vec && N < (1LL << 31) && K < (1LL << 31)) {
    const bool uniform = (pm.strategy == B200Q_TENSOR) || (pm.strategy == B200Q_CHANNEL) ||
                         ((pm.strategy == B200Q_GROUP || pm.strategy == B200Q_TENSOR_GROUP) &&
                          pm.g_idx == nullptr && (pm.group_size & 7) == 0) ||
                         (pm.strategy == B200Q_BLOCK && (pm.block_w & 7) == 0);
    // bf16 weights with per-group parameters in column order: lane / chunk split kernels.  The
    // combinations that occur: a bf16 scale without a global scale, or a scale with one (FP4 only: the
    // observer's float32 scale, or the module's bf16 copy, with which the row kernel took 116 us for
    // 14336 x 4096); everything else takes the row kernel below.
    if constexpr (XDT == B200Q_BF16 && MODE != kPackFake && ((SDT == B200Q_BF16 && !GLOBAL) || (GLOBAL && MODE == kPackFp4))) {
      const int g = pm.group_size;
      if ((pm.strategy == B200Q_GROUP || pm.strategy == B200Q_TENSOR_GROUP) && pm.g_idx == nullptr && g >= 8 &&
          g <= 256 && (g & (g - 1)) == 0 && K % g == 0) {
        const stream::GroupSplit gsp = stream::make_group_split(g, 4);
        const int64_t slots = (K / g) * gsp.L;
        int tx2 = 32;
        while (tx2 < 256 && tx2 < slots) tx2 <<= 1;
        const int rows2 = stream::kThreads / tx2;
        const int txl2 = __builtin_ctz(tx2);
#define B200Q_QG(RR, LL) const int grid2 = resident_grid<stream::quant_group_bf16_kernel<SDT, GLOBAL, MODE, RR, LL>>(stream::kThreads, 0, (N + rows2 - 1) / rows2); stream::quant_group_bf16_kernel<SDT, GLOBAL, MODE, RR, LL><<<grid2, stream::kThreads, 0, st>>>(W, (int)N, (int)K, ldw, txl2, scale, zp, zp_kind, gscale, qr, out)
        switch (g) {
          case 8: { B200Q_QG(1, 1); break; }
          case 16: { B200Q_QG(2, 1); break; }
          case 32: { B200Q_QG(4, 1); break; }
          case 64: { B200Q_QG(4, 2); break; }
          case 128: { B200Q_QG(4, 4); break; }
          default: { B200Q_QG(4, 8); break; }
        }
#undef B200Q_QG
        B200Q_LAUNCH_CHECK();
        return B200Q_OK;
      }
    }
    const stream::RowTiling t = stream::make_tiling(N, K, 6);
    const int grid = resident_grid<stream::quant_rows_kernel<XDT, SDT, GLOBAL, MODE>>(stream::kThreads, 0, (N + t.rows - 1) / t.rows);
    const int width = pm.strategy == B200Q_BLOCK ? pm.block_w : pm.group_size;
    const int width_log2 = width > 0 && (width & (width - 1)) == 0 ? __builtin_ctz((unsigned)width) : -1;
    stream::quant_rows_kernel<XDT, SDT, GLOBAL, MODE><<<grid, stream::kThreads, 0, st>>>(
        W, (int)N, (int)K, ldw, __builtin_ctz(t.tx), scale, zp, zp_kind, pm, uniform, width_log2, gscale, qr, out, ldo);
  } else {
    int64_t blocks = (N * K + 255) / 256;
    quant_scalar_kernel<XDT, SDT, GLOBAL, MODE><<<grid_for(blocks, 8), 256, 0, st>>>(
        W, N, K, ldw, scale, zp, zp_kind, pm, gscale, qr, out, ldo);
  }
  B200Q_LAUNCH_CHECK();
  return B200Q_OK;
}

template <int MODE>
static int quant_dispatch(const void* W, int wdtype, int64_t N, int64_t K, int64_t ldw,
                          const void* scale, int sdtype, const void* zp, const int32_t* g_idx,
                          const float* gscale, const b200q_qargs* qa, void* out, int64_t ldo,
                          cudaStream_t st) {
  if (!W || !scale || !out || !qa || N <= 0 || K <= 0) return B200Q_ERR_ARG;
  QRange qr; ParamMap pm;
  int rc = make_qrange(qa, &qr); if (rc) return rc;
  rc = make_param_map(qa, N, K, g_idx, &pm); if (rc) return rc;
  int zk = qa->zp_kind;
#define B200Q_Q(X, S, G) return quant_launch<X, S, G, MODE>(W, N, K, ldw, scale, zp, zk, pm, gscale, qr, out, ldo, st)
  if (wdtype == B200Q_BF16 && sdtype == B200Q_BF16) { if (gscale) B200Q_Q(B200Q_BF16, B200Q_BF16, true); else B200Q_Q(B200Q_BF16, B200Q_BF16, false); }
  if (wdtype == B200Q_BF16 && sdtype == B200Q_F32)  { if (gscale) B200Q_Q(B200Q_BF16, B200Q_F32, true);  else B200Q_Q(B200Q_BF16, B200Q_F32, false); }
  if (wdtype == B200Q_F32 && sdtype == B200Q_BF16)  { if (gscale) B200Q_Q(B200Q_F32, B200Q_BF16, true);  else B200Q_Q(B200Q_F32, B200Q_BF16, false); }
  if (wdtype == B200Q_F32 && sdtype == B200Q_F32)   { if (gscale) B200Q_Q(B200Q_F32, B200Q_F32, true);   else B200Q_Q(B200Q_F32, B200Q_F32, false); }
#undef B200Q_Q
  return B200Q_ERR_UNSUPPORTED;
}

// ========================================================================================
// zero-point packing along dim 0 and scale compression
// ========================================================================================
__global__ void pack_zp_kernel(const int8_t* __restrict__ zp, int64_t N, int64_t G, int bits,
                               int32_t* __restrict__ out) {
  const int pf = 32 / bits;
  const int64_t rows_out = (N + pf - 1) / pf, total = rows_out * G;
  const int off = 1 << (bits - 1);
  const uint32_t mask = (bits == 32) ? 0xFFFFFFFFu : ((1u << bits) - 1u);
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total;
       i += (int64_t)gridDim.x * blockDim.x) {
    int64_t ro = i / G, c = i - ro * G;
    uint32_t w = 0;
    for (int j = 0; j < pf; ++j) {
      int64_t r = ro * pf + j;
      if (r >= N) break;
      w |= (((uint32_t)((int)zp[r * G + c] + off)) & mask) << (bits * j);
    }
    out[i] = (int32_t)w;
  }
}

template <int DT>
__global__ void compress_scale_kernel(const void* __restrict__ scale, int64_t n, int kind,
                                      uint8_t* __restrict__ out) {
  using E = Elem<DT>;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    float s = E::load((const typename E::type*)scale + i);
    out[i] = (kind == B200Q_SCALE_FP8) ? e4m3_bits(s) : e8m0_of(s);
  }
}

// ========================================================================================
// fused round-to-nearest: statistics -> qparams -> codes -> packed, one read of W
// ========================================================================================
// GROUP strategies (g power of two, 8..256): thread = 8 elements, lanes of a group shuffle.
template <int DT, int MODE, bool GLOBAL>
__global__ void __launch_bounds__(256) rtn_group_kernel(
    const void* __restrict__ W, int64_t N, int64_t K, int64_t ldw, int g, QParamCfg qc, QRange qr,
    const float* __restrict__ gscale, void* __restrict__ scale_out, void* __restrict__ zp_out,
    uint8_t* __restrict__ scale_store, void* __restrict__ out) {
  using E = Elem<DT>;
  using T = typename E::type;
  constexpr bool XB = E::is_bf16;
  constexpr bool SB = XB && !GLOBAL;  // scale dtype: stats dtype unless a global scale promotes it
  constexpr bool CB = XB && SB;
  const float gs = GLOBAL ? *gscale : 1.0f;
  const int lanes = g >> 3;
  const int64_t cpr = K >> 3, total = N * cpr, gpr = K / g;
  for (int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; c < ((total + 31) & ~31LL);
       c += (int64_t)gridDim.x * blockDim.x) {
    const bool live = c < total;
    float v[8];
    float lo = INFINITY, hi = -INFINITY;
    int64_t row = 0, cc = 0;
    if (live) {
      row = c / cpr; cc = c - row * cpr;
      load8<DT>(W, row * ldw + cc * 8, v);
#pragma unroll
      for (int i = 0; i < 8; ++i) { lo = fminf(lo, v[i]); hi = fmaxf(hi, v[i]); }
    }
    for (int o = lanes >> 1; o > 0; o >>= 1) {
      lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, o));
      hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, o));
    }
    if (!live) continue;
    float s, z;
    qparams_one<XB>(lo, hi, qc, gs, s, z);
    if ((cc % lanes) == 0) {
      int64_t gi = row * gpr + (cc * 8) / g;
      // the module keeps the scale in the weight dtype (exact: FP8-grid and power-of-two
      // scales are bf16 values; plain scales already are bf16 when the statistics are)
      E::store((T*)scale_out + gi, s);
      if (zp_out) store_zp(zp_out, qc.zp_kind, gi, z);
      if (scale_store) scale_store[gi] = (qc.scale_kind == B200Q_SCALE_FP8) ? e4m3_bits(s) : e8m0_of(s);
    }
    float se = GLOBAL ? __fdiv_rn(s, gs) : s;
    uint32_t w0 = 0, w1 = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      float q = quant_code<CB>(v[i], se, z, qr);
      if (MODE == kPackInt4) w0 |= ((uint32_t)((int)q + 8) & 0xFu) << (4 * i);
      else if (MODE == kPackFp4) w0 |= e2m1_nibble(q) << (4 * i);
      else {
        uint32_t b = (qr.kind == kFp8) ? e4m3_bits(q)
                   : (MODE == kPackInt8Word) ? ((uint32_t)((int)q + 128) & 0xFFu)
                                             : ((uint32_t)(int)q & 0xFFu);
        if (i < 4) w0 |= b << (8 * i); else w1 |= b << (8 * (i - 4));
      }
    }
    if (MODE == kPackInt4 || MODE == kPackFp4) ((uint32_t*)out)[row * cpr + cc] = w0;
    else reinterpret_cast<uint2*>(out)[row * cpr + cc] = make_uint2(w0, w1);
  }
}

// CHANNEL strategy: one CTA per row, the row staged in shared memory between the two passes.
template <int DT, int MODE>
__global__ void __launch_bounds__(256) rtn_channel_kernel(
    const void* __restrict__ W, int64_t N, int64_t K, int64_t ldw, QParamCfg qc, QRange qr,
    void* __restrict__ scale_out, void* __restrict__ zp_out, void* __restrict__ out) {
  using E = Elem<DT>;
  using T = typename E::type;
  constexpr bool XB = E::is_bf16;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* srow = reinterpret_cast<T*>(smem_raw);
  __shared__ float s_lo[8], s_hi[8], s_par[2];
  const int64_t cpr = K >> 3;
  for (int64_t row = blockIdx.x; row < N; row += gridDim.x) {
    float lo = INFINITY, hi = -INFINITY;
    for (int64_t c = threadIdx.x; c < cpr; c += blockDim.x) {
      float v[8];
      load8<DT>(W, row * ldw + c * 8, v);
      store8<DT>(srow, c * 8, v);
#pragma unroll
      for (int i = 0; i < 8; ++i) { lo = fminf(lo, v[i]); hi = fmaxf(hi, v[i]); }
    }
    lo = warp_min(lo); hi = warp_max(hi);
    if ((threadIdx.x & 31) == 0) { s_lo[threadIdx.x >> 5] = lo; s_hi[threadIdx.x >> 5] = hi; }
    __syncthreads();
    if (threadIdx.x == 0) {
      for (int w = 1; w < (blockDim.x >> 5); ++w) { lo = fminf(lo, s_lo[w]); hi = fmaxf(hi, s_hi[w]); }
      float s, z;
      qparams_one<XB>(lo, hi, qc, 1.0f, s, z);
      s_par[0] = s; s_par[1] = z;
      E::store((T*)scale_out + row, s);
      if (zp_out) store_zp(zp_out, qc.zp_kind, row, z);
    }
    __syncthreads();
    const float s = s_par[0], z = s_par[1];
    for (int64_t c = threadIdx.x; c < cpr; c += blockDim.x) {
      float v[8];
      if constexpr (XB) {
        uint4 u = *reinterpret_cast<const uint4*>(srow + c * 8);
        const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) { v[2 * i] = __uint_as_float(w[i] << 16); v[2 * i + 1] = __uint_as_float(w[i] & 0xFFFF0000u); }
      } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] = ((const float*)srow)[c * 8 + i];
      }
      uint32_t w0 = 0, w1 = 0;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        float q = quant_code<XB>(v[i], s, z, qr);
        if (MODE == kPackInt4) w0 |= ((uint32_t)((int)q + 8) & 0xFu) << (4 * i);
        else {
          uint32_t b = (qr.kind == kFp8) ? e4m3_bits(q)
                     : (MODE == kPackInt8Word) ? ((uint32_t)((int)q + 128) & 0xFFu)
                                               : ((uint32_t)(int)q & 0xFFu);
          if (i < 4) w0 |= b << (8 * i); else w1 |= b << (8 * (i - 4));
        }
      }
      if (MODE == kPackInt4) ((uint32_t*)out)[row * cpr + c] = w0;
      else reinterpret_cast<uint2*>(out)[row * cpr + c] = make_uint2(w0, w1);
    }
    __syncthreads();
  }
}

// ========================================================================================
// Q(W * s) / s, one grid point of the AWQ search, for bf16 weights and integer codes
// ========================================================================================
// The chain of the element-wise formulation - scale and round to bf16, min / max of the group or row, qparams,
// fake-quantise, divide by the scale in float32 and round - in one pass over the weight: 4 B of traffic an element
// where the separate passes moved 30 (231 us for 4096 x 4096).
struct ColScale { float s[8], rs[8]; bool plain; };   // plain: all of them within 2^-24 .. 2^24
__device__ __forceinline__ void load_col_scale(const float* __restrict__ col, int64_t c, ColScale& k) {
  const float4 a = __ldg(reinterpret_cast<const float4*>(col + c)), b = __ldg(reinterpret_cast<const float4*>(col + c) + 1);
  k.s[0] = a.x; k.s[1] = a.y; k.s[2] = a.z; k.s[3] = a.w; k.s[4] = b.x; k.s[5] = b.y; k.s[6] = b.z; k.s[7] = b.w;
  k.plain = true;
#pragma unroll
  for (int i = 0; i < 8; ++i) { k.rs[i] = __frcp_rn(k.s[i]); k.plain = k.plain && k.s[i] >= 0x1p-24f && k.s[i] <= 0x1p24f; }
}
__device__ __forceinline__ uint4 scale_chunk(const uint4& raw, const ColScale& k) {
  const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
  uint32_t o[4];
#pragma unroll
  for (int p = 0; p < 4; ++p)
    o[p] = stream::cvt_bf16x2(__uint_as_float(w[p] & 0xFFFF0000u) * k.s[2 * p + 1], __uint_as_float(w[p] << 16) * k.s[2 * p]);
  return make_uint4(o[0], o[1], o[2], o[3]);
}
// bf16(fq / s) of a chunk by the division itself (arguments by value and out of line: rarely needed)
__device__ __noinline__ uint4 unscale_exact(uint4 fq, float4 s0, float4 s1) {
  auto one = [](uint32_t w, float lo, float hi) {
    return stream::cvt_bf16x2(__fdiv_rn(__uint_as_float(w & 0xFFFF0000u), hi), __fdiv_rn(__uint_as_float(w << 16), lo));
  };
  return make_uint4(one(fq.x, s0.x, s0.y), one(fq.y, s0.z, s0.w), one(fq.z, s1.x, s1.y), one(fq.w, s1.z, s1.w));
}
__device__ __forceinline__ uint32_t rint_bf16x2(uint32_t v, bool four_bit) {
  if (four_bit) {   // integers are 1 apart in [128, 256)
    const uint32_t magic = 0x43404340u;
    const __nv_bfloat162 m = *reinterpret_cast<const __nv_bfloat162*>(&magic);
    __nv_bfloat162 r = __hsub2_rn(__hadd2_rn(*reinterpret_cast<__nv_bfloat162*>(&v), m), m);
    return *reinterpret_cast<uint32_t*>(&r);
  }
  __nv_bfloat162 r = h2rint(*reinterpret_cast<__nv_bfloat162*>(&v));
  return *reinterpret_cast<uint32_t*>(&r);
}
__device__ __forceinline__ uint4 fake_quant_unscale(const uint4& ws, const stream::GroupQ& g, const QRange& qr, bool sym,
                                                    bool four_bit, const ColScale& k) {
  uint32_t fq[4];
  if (g.slow) {
    const uint32_t w[4] = {ws.x, ws.y, ws.z, ws.w};
#pragma unroll
    for (int p = 0; p < 4; ++p) {
      float f[2];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const float x = h ? __uint_as_float(w[p] & 0xFFFF0000u) : __uint_as_float(w[p] << 16);
        f[h] = dequant_code<true>(quant_code<true>(x, g.se, g.z, qr), g.se, g.z);
      }
      fq[p] = stream::cvt_bf16x2(f[1], f[0]);
    }
  } else {
    uint32_t v[4];
    stream::quot8_bf16<false>(ws, g, v);
    const uint32_t lo2 = stream::bf2_splat(qr.qmin), hi2 = stream::bf2_splat(qr.qmax), s2 = stream::bf2_splat(g.se);
#pragma unroll
    for (int p = 0; p < 4; ++p) {
      if (!sym) v[p] = stream::bf2_add(v[p], g.z2);
      const uint32_t sign = v[p] & 0x80008000u;     // rounding to zero keeps the sign
      uint32_t q = rint_bf16x2(stream::bf2_min(stream::bf2_max(v[p], lo2), hi2), four_bit);
      q = (q & 0x7FFF7FFFu) | sign;
      __nv_bfloat162 d = *reinterpret_cast<__nv_bfloat162*>(&q);
      if (!sym) d = __hsub2_rn(d, *reinterpret_cast<const __nv_bfloat162*>(&g.z2));
      d = __hmul2_rn(d, *reinterpret_cast<const __nv_bfloat162*>(&s2));
      fq[p] = *reinterpret_cast<uint32_t*>(&d);
    }
  }
  // The product with 1 / s is a few float32 ulps off the quotient, so it rounds to the same bf16 value unless it lies
  // within 16 ulps of a midpoint, which one test settles for the chunk.  The scales' ranges keep every product that is
  // not zero a normal number.
  uint32_t o[4], near = 0xFFFFFFFFu;
#pragma unroll
  for (int p = 0; p < 4; ++p) {
    const float lo = __uint_as_float(fq[p] << 16) * k.rs[2 * p], hi = __uint_as_float(fq[p] & 0xFFFF0000u) * k.rs[2 * p + 1];
    near = min(near, min((__float_as_uint(lo) & 0xFFFFu) - 0x7FF0u, (__float_as_uint(hi) & 0xFFFFu) - 0x7FF0u));
    o[p] = stream::cvt_bf16x2(hi, lo);
  }
  if (near > 0x20u && k.plain && g.se >= 0x1p-60f && g.se <= 0x1p60f) return make_uint4(o[0], o[1], o[2], o[3]);
  return unscale_exact(make_uint4(fq[0], fq[1], fq[2], fq[3]), make_float4(k.s[0], k.s[1], k.s[2], k.s[3]),
                       make_float4(k.s[4], k.s[5], k.s[6], k.s[7]));
}

// Weights of one width behind the same column scales, as one matrix of all their rows.
constexpr int kScaledMax = 8;
struct ScaledRows {
  const void* W[kScaledMax]; void* out[kScaledMax];
  int64_t ldw[kScaledMax], end[kScaledMax];   // row stride, rows of this and the weights before it
};
// GROUP: a thread owns R chunks of 8 columns of a group and walks down the rows, so that its column scales and their
// reciprocals stay in registers; the g / 8 / R lanes of a group shuffle, and derive its parameters once for R chunks.
// Bound by issue.  Three weights of 4096 x 4096, groups of 128: 60.6 us, 79 with a chunk a lane and a launch a weight.
template <int R>
__global__ void __launch_bounds__(256) scaled_group_kernel(const __grid_constant__ ScaledRows m, int64_t N, int64_t K,
                                                           int lanes, const float* __restrict__ col, QParamCfg qc, QRange qr,
                                                           bool four_bit) {
  using T = __nv_bfloat16;
  const int64_t slot = (int64_t)blockIdx.x * 32 + (threadIdx.x & 31), cpr = K >> 3;
  const bool live = slot * R < cpr;
  const int64_t first = (slot / lanes * lanes * R + slot % lanes) * 8;   // column of the first chunk; the others `lanes` chunks apart
  ColScale k[R];
  if (live) {
#pragma unroll
    for (int i = 0; i < R; ++i) load_col_scale(col, first + (int64_t)i * lanes * 8, k[i]);
  }
  const int64_t step = (int64_t)gridDim.y * 8;
  int64_t row = (int64_t)blockIdx.y * 8 + (threadIdx.x >> 5);
  int at = 0, at_next = 0;   // the weight that a row is of
  uint4 next[R];
  auto fetch = [&](int64_t r) {
    while (r >= m.end[at_next]) ++at_next;
    if (!live) return;
    const T* src = (const T*)m.W[at_next] + (r - (at_next ? m.end[at_next - 1] : 0)) * m.ldw[at_next] + first;
#pragma unroll
    for (int i = 0; i < R; ++i) next[i] = stream::ldg_stream(src + i * lanes * 8);
  };
#pragma unroll
  for (int i = 0; i < R; ++i) next[i] = make_uint4(0, 0, 0, 0);
  if (row < N) fetch(row);
  for (; row < N; row += step) {
    at = at_next;
    uint4 ws[R];
#pragma unroll
    for (int i = 0; i < R; ++i) ws[i] = live ? scale_chunk(next[i], k[i]) : make_uint4(0, 0, 0, 0);
    if (row + step < N) fetch(row + step);
    stream::RangeQ r;
    r.first(ws[0]);
#pragma unroll
    for (int i = 1; i < R; ++i) r.add(ws[i]);
    float lo, hi;
    r.finish(lo, hi);
    for (int o = lanes >> 1; o > 0; o >>= 1) {
      lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, o));
      hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, o));
    }
    float s, z;
    qparams_one<true>(lo, hi, qc, 1.0f, s, z);
    const stream::GroupQ gq = stream::make_group_q<true>(s, z + 0.0f);   // (a stored zero point has no -0)
    if (live) {
      T* dst = (T*)m.out[at] + (row - (at ? m.end[at - 1] : 0)) * K + first;
#pragma unroll
      for (int i = 0; i < R; ++i)
        *reinterpret_cast<uint4*>(dst + i * lanes * 8) = fake_quant_unscale(ws[i], gq, qr, qc.symmetric != 0, four_bit, k[i]);
    }
  }
}
// CHANNEL: a CTA per row, the scaled row in registers between the two halves (R chunks of 8 per thread)
template <int R>
__global__ void __launch_bounds__(256) scaled_channel_kernel(const void* __restrict__ W, int64_t N, int64_t K, int64_t ldw,
                                                             const float* __restrict__ col, QParamCfg qc, QRange qr,
                                                             bool four_bit, void* __restrict__ out) {
  using T = __nv_bfloat16;
  __shared__ float s_lo[2][8], s_hi[2][8];
  const int cpr = (int)(K >> 3), warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int par = 0;
  for (int64_t row = blockIdx.x; row < N; row += gridDim.x, par ^= 1) {
    uint4 ws[R];
    stream::RangeQ r;
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const int c = threadIdx.x + i * 256;
      ws[i] = c < cpr ? stream::ldg_stream((const T*)W + row * ldw + (int64_t)c * 8) : make_uint4(0, 0, 0, 0);
    }
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const int c = threadIdx.x + i * 256;
      if (c < cpr) {
        ColScale k;
        load_col_scale(col, (int64_t)c * 8, k);
        ws[i] = scale_chunk(ws[i], k);
      }
      if (i == 0) r.first(ws[0]); else r.add(ws[i]);
    }
    float lo, hi;
    r.finish(lo, hi);
    lo = warp_min(lo); hi = warp_max(hi);
    if (lane == 0) { s_lo[par][warp] = lo; s_hi[par][warp] = hi; }
    __syncthreads();   // one barrier per row: the buffers alternate
#pragma unroll
    for (int w = 0; w < 8; ++w) { lo = fminf(lo, s_lo[par][w]); hi = fmaxf(hi, s_hi[par][w]); }
    float s, z;
    qparams_one<true>(lo, hi, qc, 1.0f, s, z);
    const stream::GroupQ gq = stream::make_group_q<true>(s, z + 0.0f);
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const int c = threadIdx.x + i * 256;
      if (c < cpr) {
        ColScale k;
        load_col_scale(col, (int64_t)c * 8, k);
        *reinterpret_cast<uint4*>((T*)out + row * K + (int64_t)c * 8) = fake_quant_unscale(ws[i], gq, qr, qc.symmetric != 0, four_bit, k);
      }
    }
  }
}

__global__ void note_wait_kernel(const int* status) {
  if (*status != 0) atomicExch(&tma::g_wait_expired, 1);
}

}  // namespace b200q

using namespace b200q;

// ========================================================================================
// C ABI
// ========================================================================================
extern "C" {

const char* b200q_version(void) { return "b200q 0.1 (sm_100a)"; }
const char* b200q_last_error(void) { return g_last_error.c_str(); }
long long b200q_launch_count(void) { return g_launches.load(std::memory_order_relaxed); }

int b200q_take_wait_status(void) {
  int v = 0;
  B200Q_TRY(cudaDeviceSynchronize());   // (the copy alone does not wait for non-blocking streams)
  B200Q_TRY(cudaMemcpyFromSymbol(&v, tma::g_wait_expired, sizeof(int)));
  if (v == 0) return B200Q_OK;
  v = 0;
  B200Q_TRY(cudaMemcpyToSymbol(tma::g_wait_expired, &v, sizeof(int)));
  return B200Q_ERR_DEVICE;
}

int b200q_note_wait_status(const int* status, void* stream) {
  if (!status) return B200Q_ERR_ARG;
  note_wait_kernel<<<1, 1, 0, (cudaStream_t)stream>>>(status);
  B200Q_LAUNCH_CHECK();
  return B200Q_OK;
}

size_t b200q_observe_minmax_workspace_bytes(int64_t, int64_t, const b200q_qargs* qa) {
  return (qa && qa->strategy == B200Q_TENSOR) ? sizeof(float) * 2 * kTensorPartialBlocks : 0;
}

int b200q_observe_minmax_absmax(const void* W, int wdtype, int64_t N, int64_t K, int64_t ldw, const b200q_qargs* qa, void* mn,
                                void* mx, void* scratch, float* absmax, void* stream) {
  if (!W || !qa || !mn || !mx || N <= 0 || K <= 0 || ldw < K) return B200Q_ERR_ARG;
  cudaStream_t st = (cudaStream_t)stream;
  if (wdtype == B200Q_BF16) return observe_minmax_impl<B200Q_BF16>(W, N, K, ldw, qa, mn, mx, scratch, absmax, st);
  if (wdtype == B200Q_F32) return observe_minmax_impl<B200Q_F32>(W, N, K, ldw, qa, mn, mx, scratch, absmax, st);
  return B200Q_ERR_UNSUPPORTED;
}

int b200q_observe_minmax(const void* W, int wdtype, int64_t N, int64_t K, int64_t ldw,
                         const b200q_qargs* qa, void* mn, void* mx, void* scratch, void* stream) {
  return b200q_observe_minmax_absmax(W, wdtype, N, K, ldw, qa, mn, mx, scratch, nullptr, stream);
}

int b200q_absmax_accumulate(const void* mn, const void* mx, int dtype, int64_t count, float* absmax,
                            void* stream) {
  if (!mn || !mx || !absmax || count <= 0) return B200Q_ERR_ARG;
  cudaStream_t st = (cudaStream_t)stream;
  int grid = grid_for((count + 255) / 256, 2);
  if (dtype == B200Q_BF16) absmax_kernel<B200Q_BF16><<<grid, 256, 0, st>>>(mn, mx, count, absmax);
  else if (dtype == B200Q_F32) absmax_kernel<B200Q_F32><<<grid, 256, 0, st>>>(mn, mx, count, absmax);
  else return B200Q_ERR_UNSUPPORTED;
  B200Q_LAUNCH_CHECK();
  return B200Q_OK;
}

int b200q_absmax_accumulate_weight(const void* W, int wdtype, int64_t N, int64_t K, int64_t ldw, float* absmax,
                                   void* stream) {
  if (!W || !absmax || N <= 0 || K <= 0 || ldw < K) return B200Q_ERR_ARG;
  if (wdtype != B200Q_BF16 || !vec_ok(W, K, ldw, 2)) return B200Q_ERR_UNSUPPORTED;
  const int grid = grid_for((N * (K >> 3) + 1023) / 1024, 8);
  absmax_weight_bf16_kernel<<<grid, 256, 0, (cudaStream_t)stream>>>(W, N, K, ldw, absmax);
  B200Q_LAUNCH_CHECK();
  return B200Q_OK;
}

int b200q_global_scale_finalize(const float* absmax, int stat_dtype, float* global_scale, void* stream) {
  if (!absmax || !global_scale) return B200Q_ERR_ARG;
  global_scale_kernel<<<1, 1, 0, (cudaStream_t)stream>>>(absmax, stat_dtype == B200Q_BF16, global_scale);
  B200Q_LAUNCH_CHECK();
  return B200Q_OK;
}

int b200q_qparams(const void* mn, const void* mx, int stat_dtype, int64_t count, const b200q_qargs* qa,
                  const float* gscale, void* scale_out, void* zp_out, void* stream) {
  if (!mn || !mx || !qa || !scale_out || count <= 0) return B200Q_ERR_ARG;
  QParamCfg c;
  int rc = make_qparam_cfg(qa, stat_dtype == B200Q_BF16, gscale != nullptr, &c);
  if (rc) return rc;
  cudaStream_t st = (cudaStream_t)stream;
  int grid = grid_for((count + 255) / 256, 8);
  if (stat_dtype == B200Q_BF16) {
    if (gscale) qparams_kernel<B200Q_BF16, true><<<grid, 256, 0, st>>>(mn, mx, count, c, gscale, scale_out, zp_out);
    else qparams_kernel<B200Q_BF16, false><<<grid, 256, 0, st>>>(mn, mx, count, c, gscale, scale_out, zp_out);
  } else if (stat_dtype == B200Q_F32) {
    if (gscale) qparams_kernel<B200Q_F32, true><<<grid, 256, 0, st>>>(mn, mx, count, c, gscale, scale_out, zp_out);
    else qparams_kernel<B200Q_F32, false><<<grid, 256, 0, st>>>(mn, mx, count, c, gscale, scale_out, zp_out);
  } else return B200Q_ERR_UNSUPPORTED;
  B200Q_LAUNCH_CHECK();
  return B200Q_OK;
}

int b200q_minmax_qparams(const void* W, const void* const* table, int count, int wdtype, int64_t N, int64_t K, int64_t ldw,
                         const b200q_qargs* qa, void* scale_out, void* zp_out, void* stream) {
  if ((!W && !table) || !qa || !scale_out || count <= 0 || count > 65535 || N <= 0 || K <= 0 || ldw < K) return B200Q_ERR_ARG;
  if (wdtype != B200Q_BF16 || !vec_ok(W, K, ldw, 2) || N >= (1 << 30) || K >= (1 << 30)) return B200Q_ERR_UNSUPPORTED;
  QParamCfg qc;
  int rc = make_qparam_cfg(qa, true, false, &qc); if (rc) return rc;
  cudaStream_t st = (cudaStream_t)stream;
  StatJob j;
  j.one = W; j.table = table; j.scale = scale_out; j.zp = zp_out;
  const int cap = count > 1 ? 8 * kNumSMs / count + 1 : 8 * kNumSMs;
  auto grid = [&](int64_t need) { return dim3((unsigned)(need < cap ? need : cap), (unsigned)count, 1); };
  if (qa->strategy == B200Q_GROUP) {
    const int g = qa->group_size;
    if (!(pow2(g) && g >= 8 && g <= 256 && K % g == 0)) return B200Q_ERR_UNSUPPORTED;
    j.entries = N * (K / g);
    const stream::GroupSplit gsp = stream::make_group_split(g);
    const int64_t slots = (K / g) * gsp.L;
    int tx = 32;
    while (tx < 256 && tx < slots) tx <<= 1;
    const dim3 gd = grid((N + 256 / tx - 1) / (256 / tx));
    const int ll = __builtin_ctz(gsp.L), txl = __builtin_ctz(tx);
    if (gsp.R == 8) group_qparams_kernel<8><<<gd, 256, 0, st>>>(j, (int)N, (int)K, ldw, ll, txl, qc);
    else if (gsp.R == 4) group_qparams_kernel<4><<<gd, 256, 0, st>>>(j, (int)N, (int)K, ldw, ll, txl, qc);
    else if (gsp.R == 2) group_qparams_kernel<2><<<gd, 256, 0, st>>>(j, (int)N, (int)K, ldw, ll, txl, qc);
    else group_qparams_kernel<1><<<gd, 256, 0, st>>>(j, (int)N, (int)K, ldw, ll, txl, qc);
  } else if (qa->strategy == B200Q_CHANNEL || qa->strategy == B200Q_BLOCK) {
    const bool blk = qa->strategy == B200Q_BLOCK;
    if (blk && (qa->block_h <= 0 || qa->block_w <= 0 || qa->block_w % 8)) return B200Q_ERR_UNSUPPORTED;
    const int bh = blk ? qa->block_h : 1, bw = blk ? qa->block_w : (int)K;
    if ((int64_t)bh * bw >= (1LL << 31)) return B200Q_ERR_UNSUPPORTED;
    const int64_t per_row = (K + bw - 1) / bw;
    j.entries = ((N + bh - 1) / bh) * per_row;
    const int cw = bw / 8;
    if (!blk && N * count >= 16 * kNumSMs)
      row_qparams_kernel<<<grid((N + 7) / 8), 256, 0, st>>>(j, N, K, ldw, qc);
    else
      span_qparams_kernel<<<grid(j.entries), 256, 0, st>>>(j, N, K, ldw, bh, bw, per_row, j.entries,
                                                           (cw & (cw - 1)) == 0 ? __builtin_ctz((unsigned)cw) : -1, qc);
  } else {
    return B200Q_ERR_UNSUPPORTED;
  }
  B200Q_LAUNCH_CHECK();
  return B200Q_OK;
}

int b200q_shared_qparams(const void* const* W, void* const* scale, void* const* zp, float* const* global_scale,
                         const int64_t* N, int count, int64_t K, const b200q_qargs* qa, float* absmax, void* stream) {
  if (!W || !scale || !zp || !global_scale || !N || count <= 0 || K <= 0 || !qa || !absmax) return B200Q_ERR_ARG;
  const int g = qa->group_size;
  if (count > kMaxShared || qa->strategy != B200Q_TENSOR_GROUP || !qa->symmetric || (g != 16 && g != 32) || K % g)
    return B200Q_ERR_UNSUPPORTED;
  QParamCfg qc;
  int rc = make_qparam_cfg(qa, true, true, &qc); if (rc) return rc;
  SharedJob j = {};
  int64_t most = 0;
  for (int i = 0; i < count; ++i) {
    if (!W[i] || !scale[i] || !zp[i] || !global_scale[i] || N[i] <= 0) return B200Q_ERR_ARG;
    if ((((uintptr_t)W[i]) | ((uintptr_t)scale[i]) | ((uintptr_t)zp[i])) & 15) return B200Q_ERR_UNSUPPORTED;
    j.w[i] = (const __nv_bfloat16*)W[i]; j.scale[i] = (__nv_bfloat16*)scale[i]; j.zp[i] = zp[i];
    j.global_scale[i] = global_scale[i];
    j.groups[i] = N[i] * (K / g);
    most = most > j.groups[i] ? most : j.groups[i];
  }
  j.absmax = absmax;
  cudaStream_t st = (cudaStream_t)stream;
  B200Q_TRY(cudaMemsetAsync(absmax, 0, sizeof(float), st));
  const int cap = (8 * kNumSMs + count - 1) / count;
  auto grid = [&](int64_t need) { return dim3((unsigned)(need < cap ? need : cap), (unsigned)count, 1); };
  if (g == 16) shared_absmax_kernel<2><<<grid((most + 255) / 256), 256, 0, st>>>(j);
  else shared_absmax_kernel<4><<<grid((most + 255) / 256), 256, 0, st>>>(j);
  B200Q_LAUNCH_CHECK();
  shared_qparams_kernel<<<grid((most + 2047) / 2048), 256, 0, st>>>(j, qc);
  B200Q_LAUNCH_CHECK();
  return B200Q_OK;
}

int b200q_fake_quantize(const void* W, int wdtype, int64_t N, int64_t K, int64_t ldw, const void* scale,
                        int sdtype, const void* zp, const int32_t* g_idx, const float* gscale,
                        const b200q_qargs* qa, void* out, int64_t ldo, void* stream) {
  if (ldw < K || ldo < K) return B200Q_ERR_ARG;
  return quant_dispatch<kPackFake>(W, wdtype, N, K, ldw, scale, sdtype, zp, g_idx, gscale, qa, out, ldo,
                                   (cudaStream_t)stream);
}

int b200q_quantize_pack(const void* W, int wdtype, int64_t N, int64_t K, int64_t ldw, const void* scale,
                        int sdtype, const void* zp, const int32_t* g_idx, const float* gscale,
                        const b200q_qargs* qa, int pack_int8, void* out, void* stream) {
  if (!qa || ldw < K) return B200Q_ERR_ARG;
  cudaStream_t st = (cudaStream_t)stream;
  if (qa->qtype == B200Q_QINT && qa->num_bits == 4)
    return quant_dispatch<kPackInt4>(W, wdtype, N, K, ldw, scale, sdtype, zp, g_idx, gscale, qa, out, 0, st);
  if (qa->qtype == B200Q_QINT && qa->num_bits == 8) {
    if (pack_int8)
      return quant_dispatch<kPackInt8Word>(W, wdtype, N, K, ldw, scale, sdtype, zp, g_idx, gscale, qa, out, 0, st);
    return quant_dispatch<kPackByte>(W, wdtype, N, K, ldw, scale, sdtype, zp, g_idx, gscale, qa, out, 0, st);
  }
  if (qa->qtype == B200Q_QFLOAT && qa->num_bits == 8)
    return quant_dispatch<kPackByte>(W, wdtype, N, K, ldw, scale, sdtype, zp, g_idx, gscale, qa, out, 0, st);
  if (qa->qtype == B200Q_QFLOAT && qa->num_bits == 4) {
    if (K % 2) return B200Q_ERR_ARG;
    return quant_dispatch<kPackFp4>(W, wdtype, N, K, ldw, scale, sdtype, zp, g_idx, gscale, qa, out, 0, st);
  }
  return B200Q_ERR_UNSUPPORTED;
}

int b200q_scaled_fake_quantize_many(const void* const* W, int wdtype, int count, const int64_t* N, int64_t K, const int64_t* ldw,
                                    const float* col_scale, const b200q_qargs* qa, void* const* out, void* stream) {
  if (!W || !N || !ldw || !col_scale || !qa || !out || count <= 0 || K <= 0) return B200Q_ERR_ARG;
  if (wdtype != B200Q_BF16 || qa->qtype != B200Q_QINT || (qa->num_bits != 4 && qa->num_bits != 8) ||
      qa->scale_kind != B200Q_SCALE_PLAIN || (((uintptr_t)col_scale) % 16))
    return B200Q_ERR_UNSUPPORTED;
  for (int i = 0; i < count; ++i) {
    if (!W[i] || !out[i] || N[i] <= 0 || ldw[i] < K) return B200Q_ERR_ARG;
    if (!vec_ok(W[i], K, ldw[i], 2) || (((uintptr_t)out[i]) % 16)) return B200Q_ERR_UNSUPPORTED;
  }
  QParamCfg qc; QRange qr;
  int rc = make_qparam_cfg(qa, true, false, &qc); if (rc) return rc;
  rc = make_qrange(qa, &qr); if (rc) return rc;
  cudaStream_t st = (cudaStream_t)stream;
  const bool four = qa->num_bits == 4;
  const int64_t cpr = K >> 3;
  if (qa->strategy == B200Q_GROUP) {
    const int g = qa->group_size;
    if (!(pow2(g) && g >= 8 && g <= 256 && K % g == 0)) return B200Q_ERR_UNSUPPORTED;
    const int R = g >= 16 ? 2 : 1, lanes = g / 8 / R;
    const int64_t gx = (cpr / R + 31) / 32;
    if (gx > 2147483647LL) return B200Q_ERR_UNSUPPORTED;
    for (int at = 0; at < count; at += kScaledMax) {
      ScaledRows m;
      int64_t rows = 0;
      for (int i = 0; i < kScaledMax; ++i) {
        const int w = at + i < count ? at + i : count - 1;
        rows += at + i < count ? N[w] : 0;
        m.W[i] = W[w]; m.out[i] = out[w]; m.ldw[i] = ldw[w]; m.end[i] = rows;
      }
      // as many CTAs as are resident at once: each walks down its share of the rows, which earns the column scales'
      // reciprocals (six per SM where four fit: 33 us for 4096 x 4096)
      int64_t gy = (R == 2 ? resident_grid<scaled_group_kernel<2>>(256, 0, (int64_t)1 << 40)
                           : resident_grid<scaled_group_kernel<1>>(256, 0, (int64_t)1 << 40)) / gx;
      if (gy < 1) gy = 1;
      if (gy > (rows + 7) / 8) gy = (rows + 7) / 8;
      if (gy > 65535) gy = 65535;
      auto kernel = R == 2 ? scaled_group_kernel<2> : scaled_group_kernel<1>;
      kernel<<<dim3((unsigned)gx, (unsigned)gy), 256, 0, st>>>(m, rows, K, lanes, col_scale, qc, qr, four);
      B200Q_LAUNCH_CHECK();
    }
  } else if (qa->strategy == B200Q_CHANNEL) {
    if (cpr > 8 * 256) return B200Q_ERR_UNSUPPORTED;
    for (int i = 0; i < count; ++i) {
#define B200Q_SC(R) scaled_channel_kernel<R><<<resident_grid<scaled_channel_kernel<R>>(256, 0, N[i]), 256, 0, st>>>(W[i], N[i], K, ldw[i], col_scale, qc, qr, four, out[i])
      if (cpr <= 256) B200Q_SC(1);
      else if (cpr <= 512) B200Q_SC(2);
      else if (cpr <= 1024) B200Q_SC(4);
      else B200Q_SC(8);
#undef B200Q_SC
      B200Q_LAUNCH_CHECK();
    }
  } else {
    return B200Q_ERR_UNSUPPORTED;
  }
  return B200Q_OK;
}

int b200q_scaled_fake_quantize(const void* W, int wdtype, int64_t N, int64_t K, int64_t ldw, const float* col_scale,
                               const b200q_qargs* qa, void* out, void* stream) {
  return b200q_scaled_fake_quantize_many(&W, wdtype, 1, &N, K, &ldw, col_scale, qa, &out, stream);
}

int b200q_pack_zero_points(const int8_t* zp, int64_t N, int64_t G, int num_bits, int32_t* out, void* stream) {
  if (!zp || !out || N <= 0 || G <= 0 || num_bits < 1 || num_bits > 8) return B200Q_ERR_ARG;
  int64_t total = ((N + 32 / num_bits - 1) / (32 / num_bits)) * G;
  pack_zp_kernel<<<grid_for((total + 255) / 256, 4), 256, 0, (cudaStream_t)stream>>>(zp, N, G, num_bits, out);
  B200Q_LAUNCH_CHECK();
  return B200Q_OK;
}

int b200q_compress_scale(const void* scale, int sdtype, int64_t count, int scale_kind, uint8_t* out, void* stream) {
  if (!scale || !out || count <= 0) return B200Q_ERR_ARG;
  if (scale_kind != B200Q_SCALE_FP8 && scale_kind != B200Q_SCALE_E8M0) return B200Q_ERR_ARG;
  cudaStream_t st = (cudaStream_t)stream;
  int grid = grid_for((count + 255) / 256, 8);
  if (sdtype == B200Q_BF16) compress_scale_kernel<B200Q_BF16><<<grid, 256, 0, st>>>(scale, count, scale_kind, out);
  else if (sdtype == B200Q_F32) compress_scale_kernel<B200Q_F32><<<grid, 256, 0, st>>>(scale, count, scale_kind, out);
  else return B200Q_ERR_UNSUPPORTED;
  B200Q_LAUNCH_CHECK();
  return B200Q_OK;
}

}  // extern "C"

template <int DT>
static int rtn_impl(const void* W, int64_t N, int64_t K, int64_t ldw, const b200q_qargs* qa,
                    const float* gscale, void* scale_out, void* zp_out, uint8_t* scale_store, void* out,
                    cudaStream_t st) {
  QParamCfg qc; QRange qr;
  int rc = make_qparam_cfg(qa, DT == B200Q_BF16, gscale != nullptr, &qc); if (rc) return rc;
  rc = make_qrange(qa, &qr); if (rc) return rc;
  if (!vec_ok(W, K, ldw, 2) || (((uintptr_t)out) % 16)) return B200Q_ERR_UNSUPPORTED;
  if (!qa->symmetric && !zp_out) return B200Q_ERR_ARG;
  const bool grp = qa->strategy == B200Q_GROUP || qa->strategy == B200Q_TENSOR_GROUP;
  if (grp) {
    int g = qa->group_size;
    if (!(pow2(g) && g >= 8 && g <= 256 && K % g == 0)) return B200Q_ERR_UNSUPPORTED;
    stream::RowTiling t = stream::make_tiling(N, K, 6);
    const int txl = __builtin_ctz(t.tx);
    // bf16 weights whose rows are whole 2048-element tiles: the TMA-fed kernel
    if constexpr (DT == B200Q_BF16) {
      const bool aligned = (((uintptr_t)scale_out) % 16 == 0) && (!zp_out || ((uintptr_t)zp_out) % 4 == 0) &&
                           (!scale_store || ((uintptr_t)scale_store) % 4 == 0) && (((uintptr_t)out) % 16 == 0);
      if (tma_path_enabled() && aligned && K % tma::kTileElems == 0 && (g == 16 || g == 32 || g == 128) &&
          N < (1 << 30) && (!gscale || (g == 16 && qr.kind == kFp4))) {
        CUtensorMap wm;
        if (make_weight_tile_map(&wm, W, N, K, ldw)) {
          const int64_t tiles = N * (K / tma::kTileElems);
          const int gridt = (int)std::min<int64_t>((tiles + tma::kWarps - 1) / tma::kWarps, 2 * kNumSMs);
          // test hook: B200Q_TEST_DROP_TILE=n makes one warp skip its n-th tile request (see the kernel)
          const char* drop_env = getenv("B200Q_TEST_DROP_TILE");
          const int drop_request = drop_env ? atoi(drop_env) : -1;
#define B200Q_T3(MODE, GL, GG)                                                                                   \
  do {                                                                                                           \
    B200Q_TRY(cudaFuncSetAttribute(tma::rtn_group_tma_kernel<stream::MODE, GL, GG>,                              \
                                   cudaFuncAttributeMaxDynamicSharedMemorySize, tma::kSmemBytes));               \
    tma::rtn_group_tma_kernel<stream::MODE, GL, GG><<<gridt, tma::kWarps * 32, tma::kSmemBytes, st>>>(           \
        wm, (int)N, (int)K, qc, qr, gscale, scale_out, zp_out, scale_store, out, drop_request);                  \
  } while (0)
#define B200Q_T2(MODE)                                     \
  do {                                                     \
    if (g == 16) B200Q_T3(MODE, false, 16);                \
    else if (g == 32) B200Q_T3(MODE, false, 32);           \
    else B200Q_T3(MODE, false, 128);                       \
  } while (0)
          if (gscale) B200Q_T3(kFp4, true, 16);
          else if (qr.kind == kInt && qa->num_bits == 4) B200Q_T2(kInt4);
          else if (qr.kind == kInt && qa->num_bits == 8) B200Q_T2(kInt8Word);
          else if (qr.kind == kFp8) B200Q_T2(kByte);
          else if (qr.kind == kFp4) B200Q_T2(kFp4);
          else return B200Q_ERR_UNSUPPORTED;
#undef B200Q_T2
#undef B200Q_T3
          B200Q_LAUNCH_CHECK();
          return B200Q_OK;
        }
      }
    }
    // bf16 weights: R chunks per lane, L lanes per group (both compile-time)
    const stream::GroupSplit gsp = stream::make_group_split(g, 4);
    const int64_t slots = (K / g) * gsp.L;
    int tx2 = 32;
    while (tx2 < 256 && tx2 < slots) tx2 <<= 1;
    const int rows2 = stream::kThreads / tx2;
    const int grid2 = grid_for((N + rows2 - 1) / rows2, 6);
    const int txl2 = __builtin_ctz(tx2);
#define B200Q_RB3(MODE, GL, RR, LL) stream::rtn_group_bf16_kernel<stream::MODE, GL, RR, LL><<<grid2, stream::kThreads, 0, st>>>(W, (int)N, (int)K, ldw, txl2, qc, qr, gscale, scale_out, zp_out, scale_store, out)
#define B200Q_RB2(MODE, GL)                          \
  do {                                               \
    switch (g) {                                     \
      case 8: B200Q_RB3(MODE, GL, 1, 1); break;      \
      case 16: B200Q_RB3(MODE, GL, 2, 1); break;     \
      case 32: B200Q_RB3(MODE, GL, 4, 1); break;     \
      case 64: B200Q_RB3(MODE, GL, 4, 2); break;     \
      case 128: B200Q_RB3(MODE, GL, 4, 4); break;    \
      default: B200Q_RB3(MODE, GL, 4, 8); break;     \
    }                                                \
  } while (0)
#define B200Q_RB(MODE)                                                            \
  do {                                                                            \
    if (gscale) {                                                                 \
      if constexpr (stream::MODE == stream::kFp4) {                               \
        if (g != 16) return B200Q_ERR_UNSUPPORTED;                                \
        B200Q_RB3(MODE, true, 2, 1);                                              \
      } else {                                                                    \
        return B200Q_ERR_UNSUPPORTED;                                             \
      }                                                                           \
    } else {                                                                      \
      B200Q_RB2(MODE, false);                                                     \
    }                                                                             \
  } while (0)
#define B200Q_R(MODE)                                                                              \
  do {                                                                                             \
    if constexpr (DT == B200Q_BF16) {                                                              \
      B200Q_RB(MODE);                                                                               \
    } else if (gscale) stream::rtn_group_kernel<DT, stream::MODE, true><<<t.grid, stream::kThreads, 0, st>>>(W, (int)N, (int)K, ldw, g, txl, qc, qr, gscale, scale_out, zp_out, scale_store, out); \
    else stream::rtn_group_kernel<DT, stream::MODE, false><<<t.grid, stream::kThreads, 0, st>>>(W, (int)N, (int)K, ldw, g, txl, qc, qr, gscale, scale_out, zp_out, scale_store, out);      \
  } while (0)
    if (qr.kind == kInt && qa->num_bits == 4) B200Q_R(kInt4);
    else if (qr.kind == kInt && qa->num_bits == 8) B200Q_R(kInt8Word);
    else if (qr.kind == kFp8) B200Q_R(kByte);
    else if (qr.kind == kFp4) B200Q_R(kFp4);
    else return B200Q_ERR_UNSUPPORTED;
#undef B200Q_R
#undef B200Q_RB
#undef B200Q_RB2
#undef B200Q_RB3
  } else if (qa->strategy == B200Q_CHANNEL) {
    if (gscale) return B200Q_ERR_UNSUPPORTED;
    if constexpr (DT == B200Q_BF16) {
      const int64_t cpr = K >> 3;
      if ((K & 7) == 0 && cpr <= 16 * stream::kThreads && N < (1 << 30)) {
        const int r = cpr <= 2 * stream::kThreads ? 2 : cpr <= 4 * stream::kThreads ? 4
                    : cpr <= 8 * stream::kThreads ? 8 : 16;
        const int gridc = grid_for(N, r <= 4 ? 4 : 2);
#define B200Q_CB2(MODE, RR) stream::rtn_channel_bf16_kernel<stream::MODE, RR><<<gridc, stream::kThreads, 0, st>>>(W, (int)N, (int)K, ldw, qc, qr, scale_out, zp_out, out)
#define B200Q_CB(MODE)                       \
  do {                                       \
    if (r == 2) B200Q_CB2(MODE, 2);          \
    else if (r == 4) B200Q_CB2(MODE, 4);     \
    else if (r == 8) B200Q_CB2(MODE, 8);     \
    else B200Q_CB2(MODE, 16);                \
  } while (0)
        if (qr.kind == kInt && qa->num_bits == 4) B200Q_CB(kInt4);
        else if (qr.kind == kInt && qa->num_bits == 8) B200Q_CB(kInt8Word);
        else if (qr.kind == kFp8) B200Q_CB(kByte);
        else return B200Q_ERR_UNSUPPORTED;
#undef B200Q_CB
#undef B200Q_CB2
        B200Q_LAUNCH_CHECK();
        return B200Q_OK;
      }
    }
    size_t smem = (size_t)K * (DT == B200Q_BF16 ? 2 : 4);
    if (smem > 200 * 1024) return B200Q_ERR_UNSUPPORTED;
    int grid = grid_for(N, smem > 100 * 1024 ? 1 : 2);
#define B200Q_C(MODE)                                                                               \
  do {                                                                                              \
    B200Q_TRY(cudaFuncSetAttribute(rtn_channel_kernel<DT, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)); \
    rtn_channel_kernel<DT, MODE><<<grid, 256, smem, st>>>(W, N, K, ldw, qc, qr, scale_out, zp_out, out); \
  } while (0)
    if (qr.kind == kInt && qa->num_bits == 4) B200Q_C(kPackInt4);
    else if (qr.kind == kInt && qa->num_bits == 8) B200Q_C(kPackInt8Word);
    else if (qr.kind == kFp8) B200Q_C(kPackByte);
    else return B200Q_ERR_UNSUPPORTED;
#undef B200Q_C
  } else {
    return B200Q_ERR_UNSUPPORTED;
  }
  B200Q_LAUNCH_CHECK();
  return B200Q_OK;
}

extern "C" {

int b200q_rtn_quantize_pack(const void* W, int wdtype, int64_t N, int64_t K, int64_t ldw,
                            const b200q_qargs* qa, void* scale_out, void* zp_out, uint8_t* scale_store,
                            void* out, void* stream) {
  if (!W || !qa || !scale_out || !out || N <= 0 || K <= 0 || ldw < K) return B200Q_ERR_ARG;
  if (qa->strategy == B200Q_TENSOR_GROUP) return B200Q_ERR_UNSUPPORTED;  // needs the global scale
  cudaStream_t st = (cudaStream_t)stream;
  if (wdtype == B200Q_BF16) return rtn_impl<B200Q_BF16>(W, N, K, ldw, qa, nullptr, scale_out, zp_out, scale_store, out, st);
  if (wdtype == B200Q_F32) return rtn_impl<B200Q_F32>(W, N, K, ldw, qa, nullptr, scale_out, zp_out, scale_store, out, st);
  return B200Q_ERR_UNSUPPORTED;
}

int b200q_nvfp4_quantize_pack(const void* W, int wdtype, int64_t N, int64_t K, int64_t ldw,
                              const float* global_scale, void* scale_out, uint8_t* scale_store, void* out,
                              void* stream) {
  if (!W || !global_scale || !scale_out || !out || N <= 0 || K <= 0 || ldw < K) return B200Q_ERR_ARG;
  b200q_qargs qa = {4, B200Q_QFLOAT, 1, B200Q_TENSOR_GROUP, 16, 0, 0, B200Q_SCALE_FP8, B200Q_ZP_FP8};
  cudaStream_t st = (cudaStream_t)stream;
  if (wdtype == B200Q_BF16) return rtn_impl<B200Q_BF16>(W, N, K, ldw, &qa, global_scale, scale_out, nullptr, scale_store, out, st);
  if (wdtype == B200Q_F32) return rtn_impl<B200Q_F32>(W, N, K, ldw, &qa, global_scale, scale_out, nullptr, scale_store, out, st);
  return B200Q_ERR_UNSUPPORTED;
}

}  // extern "C"
