// GPTQ solve, part 1: act-order permutation, gathers and scatters, dead columns and dampening, on device in fp32.
// The factorisation is in gptq_factor.cu, the column sweep in gptq_sweep.cu.
#include "common.cuh"
#include "tgemm_tf32.cuh"

#include <cstring>

namespace b200q {
namespace solve {

// ---------------------------------------------------------------------------------------
// act-order: stable descending rank by counting.  The comparison runs on an integer key that
// orders every float the way torch.sort does (NaN above +inf, -0 equal to +0), so the ranks are
// a permutation of 0..K-1 whatever the diagonal holds.
__device__ __forceinline__ uint32_t order_key(float d) {
  if (d != d) return 0xFFFFFFFFu;
  const uint32_t b = __float_as_uint(d + 0.0f);   // -0 + 0 = +0
  return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
// A CTA ranks 32 columns, its eight warps counting an eighth of the others each (one thread per column counted all
// of them: 26 us at K = 1160).  blockIdx.y = problem.
__global__ void __launch_bounds__(256) perm_kernel(const float* H0, const float* const* Hs, int64_t K, int64_t ldh,
                                                   int32_t* __restrict__ perm) {
  __shared__ uint32_t sd[1024];
  __shared__ int s_rank[8][32];
  const float* __restrict__ H = Hs ? Hs[blockIdx.y] : H0;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t i = (int64_t)blockIdx.x * 32 + lane;
  const uint32_t ki = (i < K) ? order_key(H[i * ldh + i]) : 0u;
  int rank = 0;
  for (int64_t j0 = 0; j0 < K; j0 += 1024) {
    for (int t = threadIdx.x; t < 1024; t += 256) {
      const int64_t j = j0 + t;
      sd[t] = (j < K) ? order_key(H[j * ldh + j]) : 0u;
    }
    __syncthreads();
    const int lim = (int)min((int64_t)1024, K - j0);
#pragma unroll 8
    for (int t = warp; t < lim; t += 8) {
      const uint32_t kj = sd[t];
      rank += (kj > ki) || (kj == ki && (j0 + t) < i);
    }
    __syncthreads();
  }
  s_rank[warp][lane] = rank;
  __syncthreads();
  if (warp == 0 && i < K) {
#pragma unroll
    for (int w = 1; w < 8; ++w) rank += s_rank[w][lane];
    perm[blockIdx.y * K + rank] = (int32_t)i;
  }
}

// column index taken from a caller-supplied permutation, kept inside the matrix
__device__ __forceinline__ int64_t perm_at(const int32_t* __restrict__ perm, int64_t c, int64_t K) {
  const int64_t v = (int64_t)perm[c];
  return v < 0 ? 0 : (v >= K ? K - 1 : v);
}

// ---------------------------------------------------------------------------------------
// columns in another order, to and from float32
// Both kernels are bound by HBM (the weight once in, once out).  One problem (src, dst), or a batch (tables of pointers,
// blockIdx.y = problem; dst without a table: every dst_batch elements).
struct Columns {
  const void* src; const void* const* src_table;
  void* dst; void* const* dst_table; int64_t dst_batch;
  const int32_t* perm; const int32_t* const* perm_table; int64_t perm_batch;
  const float* const* diag_table;     // gather: columns with a zero entry come out as zeros
  const float* diag;                  // the same of a single problem
  void* keep; int64_t ldk;            // gather: the values in the source's type as well, columns with a zero entry of
  const float* keep_diag;             // this as zeros
  const float* damp;                  // gather of a square matrix with `rows`: diagonal 0 -> 1, + damp[problem]
  int64_t N, K, lds, ldd;
  bool rows;                          // gather: rows in the order of perm too
  bool vec;                           // sizes allow 16-byte pieces (whether the addresses do is seen per problem)
  __device__ __forceinline__ const void* in() const { return src_table ? src_table[blockIdx.y] : src; }
  template <typename T> __device__ __forceinline__ T* out() const {
    return dst_table ? (T*)dst_table[blockIdx.y] : (T*)dst + blockIdx.y * dst_batch;
  }
  __device__ __forceinline__ const int32_t* order() const {
    return perm_table ? perm_table[blockIdx.y] : (perm ? perm + blockIdx.y * perm_batch : nullptr);
  }
};
// four rows of a column, next to each other in shared memory
template <typename T> struct alignas(4 * sizeof(T)) Quad { T v[4]; };

__device__ __forceinline__ bool aligned16(const void* p) { return ((uintptr_t)p & 15) == 0; }

// Columns as they are: a thread moves 8 (a 64-bit division per element took 48 us for 4096 x 4096 where HBM needs 16).
// Also any order, element by element, where four rows do not fit in shared memory.
template <int DT, bool GATHER>
__global__ void __launch_bounds__(256) plain_columns_kernel(Columns j, int tx_log2) {
  using E = Elem<DT>;
  using T = typename E::type;
  const int TX = 1 << tx_log2, tx = threadIdx.x & (TX - 1), ty = threadIdx.x >> tx_log2, rows = 256 >> tx_log2;
  const int32_t* perm = j.order();
  const float* dg = GATHER ? (j.diag_table ? j.diag_table[blockIdx.y] : j.diag) : nullptr;
  T* keep = GATHER ? (T*)j.keep : nullptr;
  const void* in = j.in();
  const bool vec = j.vec && !perm && aligned16(in) && aligned16(GATHER ? (void*)j.template out<float>() : (void*)j.template out<T>());
  for (int64_t r = (int64_t)blockIdx.x * rows + ty; r < j.N; r += (int64_t)gridDim.x * rows) {
    const int64_t from = GATHER && j.rows && perm ? perm_at(perm, r, j.K) : r;
    if (vec) {
      for (int64_t c = tx * 8; c < j.K; c += TX * 8) {
        alignas(16) float v[8];
        if constexpr (GATHER) {
          const T* w = (const T*)in + from * j.lds + c;
          alignas(16) T t[8];
#pragma unroll
          for (int e = 0; e < (int)sizeof(T) / 2; ++e) reinterpret_cast<uint4*>(t)[e] = reinterpret_cast<const uint4*>(w)[e];
#pragma unroll
          for (int e = 0; e < 8; ++e) v[e] = E::load(t + e);
          if (dg) {
#pragma unroll
            for (int e = 0; e < 8; ++e) v[e] = dg[c + e] == 0.0f ? 0.0f : v[e];
          }
          float4* o = reinterpret_cast<float4*>(j.template out<float>() + r * j.ldd + c);
          o[0] = make_float4(v[0], v[1], v[2], v[3]);
          o[1] = make_float4(v[4], v[5], v[6], v[7]);
          if (keep) {
#pragma unroll
            for (int e = 0; e < 8; ++e)
              if (j.keep_diag[c + e] == 0.0f) E::store(t + e, 0.0f);
            T* k = keep + r * j.ldk + c;
#pragma unroll
            for (int e = 0; e < (int)sizeof(T) / 2; ++e) reinterpret_cast<uint4*>(k)[e] = reinterpret_cast<const uint4*>(t)[e];
          }
        } else {
          const float4* w = reinterpret_cast<const float4*>((const float*)in + r * j.lds + c);
          *reinterpret_cast<float4*>(v) = w[0];
          *reinterpret_cast<float4*>(v + 4) = w[1];
          alignas(16) T t[8];
#pragma unroll
          for (int e = 0; e < 8; ++e) E::store(t + e, v[e]);
          T* o = j.template out<T>() + r * j.ldd + c;
#pragma unroll
          for (int e = 0; e < (int)sizeof(T) / 2; ++e) reinterpret_cast<uint4*>(o)[e] = reinterpret_cast<const uint4*>(t)[e];
        }
      }
    } else {
      for (int64_t c = tx; c < j.K; c += TX) {
        const int64_t at = perm ? perm_at(perm, c, j.K) : c;
        if constexpr (GATHER) {
          float v = (dg && dg[c] == 0.0f) ? 0.0f : E::load((const T*)in + from * j.lds + at);
          if (keep) keep[r * j.ldk + c] = j.keep_diag[c] == 0.0f ? T(0.0f) : ((const T*)in)[from * j.lds + at];
          if (j.damp && c == r) v = (v == 0.0f ? 1.0f : v) + j.damp[blockIdx.y];
          j.template out<float>()[r * j.ldd + c] = v;
        } else {
          E::store(j.template out<T>() + r * j.ldd + at, ((const float*)in)[r * j.lds + c]);
        }
      }
    }
  }
}

// Another order: four rows at a time go through shared memory, column by column, so that the scattered side is one
// shared-memory access for four rows and both sides of device memory stay in order (32 to 64 experts of 768 x 2048:
// gather 348 -> 103 us, scatter 552 -> 128 us a launch).
template <int DT>
__global__ void __launch_bounds__(256) gather_columns_kernel(Columns j) {
  using E = Elem<DT>;
  using T = typename E::type;
  constexpr int V = 16 / sizeof(T);
  extern __shared__ __align__(16) unsigned char smem[];
  Quad<T>* s = reinterpret_cast<Quad<T>*>(smem);
  const int32_t* perm = j.order();
  const float* dg = j.diag_table ? j.diag_table[blockIdx.y] : j.diag;
  const T* in = (const T*)j.in();
  T* keep = (T*)j.keep;
  float* out = j.template out<float>();
  const bool vec = j.vec && aligned16(in);
  for (int64_t r0 = (int64_t)blockIdx.x * 4; r0 < j.N; r0 += (int64_t)gridDim.x * 4) {
    const int nr = (int)min((int64_t)4, j.N - r0);
    const T* row[4];
#pragma unroll
    for (int y = 0; y < 4; ++y) {
      const int64_t r = r0 + (y < nr ? y : 0);
      row[y] = in + (j.rows ? perm_at(perm, r, j.K) : r) * j.lds;
    }
    if (vec) {
      for (int c = threadIdx.x * V; c < j.K; c += 256 * V) {
        alignas(16) T v[4][V];
#pragma unroll
        for (int y = 0; y < 4; ++y) *reinterpret_cast<uint4*>(v[y]) = *reinterpret_cast<const uint4*>(row[y] + c);
#pragma unroll
        for (int e = 0; e < V; ++e) s[c + e] = Quad<T>{{v[0][e], v[1][e], v[2][e], v[3][e]}};
      }
    } else {
      for (int c = threadIdx.x; c < j.K; c += 256) s[c] = Quad<T>{{row[0][c], row[1][c], row[2][c], row[3][c]}};
    }
    __syncthreads();
#pragma unroll 4
    for (int c = threadIdx.x; c < j.K; c += 256) {
      const Quad<T> q = s[perm_at(perm, c, j.K)];
      const bool dead = dg && dg[c] == 0.0f, none = keep && j.keep_diag[c] == 0.0f;
#pragma unroll
      for (int y = 0; y < 4; ++y) {
        if (y >= nr) break;
        float v = dead ? 0.0f : E::load(&q.v[y]);
        if (keep) keep[(r0 + y) * j.ldk + c] = none ? T(0.0f) : q.v[y];
        if (j.damp && c == r0 + y) v = (v == 0.0f ? 1.0f : v) + j.damp[blockIdx.y];
        out[(r0 + y) * j.ldd + c] = v;
      }
    }
    __syncthreads();
  }
}
template <int DT>
__global__ void __launch_bounds__(256) scatter_columns_kernel(Columns j) {
  using E = Elem<DT>;
  using T = typename E::type;
  constexpr int V = 16 / sizeof(T);
  extern __shared__ __align__(16) unsigned char smem[];
  Quad<T>* s = reinterpret_cast<Quad<T>*>(smem);
  const int32_t* perm = j.order();
  const float* in = (const float*)j.in();
  T* out = j.template out<T>();
  const bool vec = j.vec && aligned16(out);
  for (int64_t r0 = (int64_t)blockIdx.x * 4; r0 < j.N; r0 += (int64_t)gridDim.x * 4) {
    const int nr = (int)min((int64_t)4, j.N - r0);
    const float* row[4];
#pragma unroll
    for (int y = 0; y < 4; ++y) row[y] = in + (r0 + (y < nr ? y : 0)) * j.lds;
#pragma unroll 4
    for (int c = threadIdx.x; c < j.K; c += 256) {
      Quad<T> q;
#pragma unroll
      for (int y = 0; y < 4; ++y) E::store(&q.v[y], row[y][c]);
      s[perm_at(perm, c, j.K)] = q;
    }
    __syncthreads();
    if (vec) {
      for (int c = threadIdx.x * V; c < j.K; c += 256 * V) {
        alignas(16) T v[4][V];
#pragma unroll
        for (int e = 0; e < V; ++e) {
          const Quad<T> q = s[c + e];
#pragma unroll
          for (int y = 0; y < 4; ++y) v[y][e] = q.v[y];
        }
#pragma unroll
        for (int y = 0; y < 4; ++y)
          if (y < nr) *reinterpret_cast<uint4*>(out + (r0 + y) * j.ldd + c) = *reinterpret_cast<const uint4*>(v[y]);
      }
    } else {
      for (int c = threadIdx.x; c < j.K; c += 256) {
        const Quad<T> q = s[c];
#pragma unroll
        for (int y = 0; y < 4; ++y)
          if (y < nr) out[(r0 + y) * j.ldd + c] = q.v[y];
      }
    }
    __syncthreads();
  }
}

static bool pieces_ok(const void* p, int64_t ld, int64_t K) { return K % 8 == 0 && ld % 8 == 0 && ((uintptr_t)p & 15) == 0; }

template <int DT, bool GATHER>
static int launch_columns(const Columns& j, int count, cudaStream_t st) {
  using T = typename Elem<DT>::type;
  const int cap = count > 1 ? 8 * kNumSMs / count + 1 : 8 * kNumSMs;
  auto grid = [&](int64_t need) { return dim3((unsigned)(need < cap ? need : cap), (unsigned)count, 1); };
  const bool ordered = j.perm || j.perm_table;
  const int64_t bytes = j.K * 4 * (int64_t)sizeof(T);
  if (ordered && bytes <= 227 * 1024) {
    auto kernel = GATHER ? gather_columns_kernel<DT> : scatter_columns_kernel<DT>;
    static thread_local int attr_device = -1;
    int dev = 0;
    B200Q_TRY(cudaGetDevice(&dev));
    if (attr_device != dev) {
      B200Q_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024));
      attr_device = dev;
    }
    kernel<<<grid((j.N + 3) / 4), 256, (size_t)bytes, st>>>(j);
  } else {
    int tx = 5;
    while (tx < 8 && (1 << tx) * 8 < j.K) ++tx;
    plain_columns_kernel<DT, GATHER><<<grid((j.N + (256 >> tx) - 1) / (256 >> tx)), 256, 0, st>>>(j, tx);
  }
  B200Q_LAUNCH_CHECK();
  return B200Q_OK;
}

// A few words of host data (pointer tables, shapes) as kernel arguments: ordered in the stream like any launch.  A copy
// from pageable memory waited for everything queued before it (0.5 ms each in an epoch of 96 expert modules).
constexpr int kUploadWords = 448;
struct UploadWords { unsigned long long v[kUploadWords]; };
__global__ void __launch_bounds__(kUploadWords) upload_kernel(const __grid_constant__ UploadWords w, int n,
                                                              unsigned long long* __restrict__ dst) {
  if ((int)threadIdx.x < n) dst[threadIdx.x] = w.v[threadIdx.x];
}

// The prologue of many factorisations of one size: per problem (blockIdx.y) the diagonal in the new order, the damping
// (summed in that order, as damp_kernel does on the permuted matrix) ...
__global__ void __launch_bounds__(1024) diag_damp_kernel(const float* const* __restrict__ Hs, int64_t K, int64_t ldh,
                                                         const int32_t* __restrict__ perm, float percdamp,
                                                         float* __restrict__ diag, float* __restrict__ damp) {
  __shared__ float s_part[32];
  const float* H = Hs[blockIdx.y];
  const int32_t* pm = perm ? perm + blockIdx.y * K : nullptr;
  float sum = 0.0f;
  for (int64_t i = threadIdx.x; i < K; i += 1024) {
    const int64_t r = pm ? pm[i] : i;
    const float d = H[r * ldh + r];
    diag[blockIdx.y * K + i] = d;
    sum += d == 0.0f ? 1.0f : d;
  }
  sum = warp_sum(sum);
  if ((threadIdx.x & 31) == 0) s_part[threadIdx.x >> 5] = sum;
  __syncthreads();
  if (threadIdx.x < 32) {
    const float v = warp_sum(s_part[threadIdx.x]);
    if (threadIdx.x == 0) damp[blockIdx.y] = percdamp * (v / (float)K);
  }
}
// ... and, without a permutation, dead diagonal entries set to 1 and the damping added, in place.
__global__ void __launch_bounds__(256) damp_many_kernel(float* const* __restrict__ Hs, int64_t K, int64_t ldh,
                                                        const float* __restrict__ damp) {
  float* H = Hs[blockIdx.y];
  const int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x;
  if (i >= K) return;
  const float d = H[i * ldh + i];
  H[i * ldh + i] = (d == 0.0f ? 1.0f : d) + damp[blockIdx.y];
}

// ---------------------------------------------------------------------------------------
// dead columns and dampening
__global__ void zero_dead_columns_kernel(const float* __restrict__ H, int64_t K, int64_t diag_stride,
                                         float* __restrict__ W, int64_t N, int64_t ldf) {
  // one warp per column; only dead columns touch W
  const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t c = warp; c < K; c += nwarps) {
    if (H[c * diag_stride] == 0.0f)
      for (int64_t r = lane; r < N; r += 32) W[r * ldf + c] = 0.0f;
  }
}
__global__ void __launch_bounds__(1024) damp_kernel(float* __restrict__ H, int64_t K, int64_t ldh,
                                                    float percdamp) {
  __shared__ float s_part[32];
  __shared__ float s_damp;
  float sum = 0.0f;
  for (int64_t i = threadIdx.x; i < K; i += blockDim.x) {
    float d = H[i * ldh + i];
    if (d == 0.0f) { d = 1.0f; H[i * ldh + i] = 1.0f; }
    sum += d;
  }
  sum = warp_sum(sum);
  if ((threadIdx.x & 31) == 0) s_part[threadIdx.x >> 5] = sum;
  __syncthreads();
  if (threadIdx.x < 32) {
    float v = (threadIdx.x < (blockDim.x >> 5)) ? s_part[threadIdx.x] : 0.0f;
    v = warp_sum(v);
    if (threadIdx.x == 0) s_damp = percdamp * (v / (float)K);
  }
  __syncthreads();
  const float damp = s_damp;
  for (int64_t i = threadIdx.x; i < K; i += blockDim.x) H[i * ldh + i] += damp;
}

}  // namespace solve
}  // namespace b200q

using namespace b200q;
using namespace b200q::solve;

extern "C" {

int b200q_actorder_perm(const float* H, int64_t K, int64_t ldh, int32_t* perm, void* stream) {
  if (!H || !perm || K <= 0 || ldh < K) return B200Q_ERR_ARG;
  perm_kernel<<<(int)((K + 31) / 32), 256, 0, (cudaStream_t)stream>>>(H, nullptr, K, ldh, perm);
  B200Q_LAUNCH_CHECK();
  return B200Q_OK;
}

int b200q_upload(const void* host, int64_t nbytes, void* dst, void* stream) {
  if (!host || !dst || nbytes < 0 || nbytes % 8 || ((uintptr_t)dst) % 8) return B200Q_ERR_ARG;
  for (int64_t at = 0; at < nbytes; at += (int64_t)sizeof(UploadWords)) {
    UploadWords w;
    const int64_t n = nbytes - at < (int64_t)sizeof(w) ? nbytes - at : (int64_t)sizeof(w);
    memcpy(w.v, (const char*)host + at, (size_t)n);
    upload_kernel<<<1, kUploadWords, 0, (cudaStream_t)stream>>>(w, (int)(n / 8), (unsigned long long*)((char*)dst + at));
    B200Q_LAUNCH_CHECK();
  }
  return B200Q_OK;
}

int b200q_gptq_prologue_many(float* const* H, int count, int64_t K, int64_t ldh, float percdamp, int32_t* perm, float* diag,
                             float* damp, float* out, void* stream) {
  if (!H || !diag || !damp || count <= 0 || count > 65535 || K <= 0 || ldh < K || (perm && !out)) return B200Q_ERR_ARG;
  cudaStream_t st = (cudaStream_t)stream;
  if (perm) {
    perm_kernel<<<dim3((unsigned)((K + 31) / 32), (unsigned)count), 256, 0, st>>>(nullptr, H, K, ldh, perm);
    B200Q_LAUNCH_CHECK();
  }
  diag_damp_kernel<<<dim3(1, (unsigned)count), 1024, 0, st>>>(H, K, ldh, perm, percdamp, diag, damp);
  B200Q_LAUNCH_CHECK();
  if (!perm) {
    damp_many_kernel<<<dim3((unsigned)((K + 255) / 256), (unsigned)count), 256, 0, st>>>(H, K, ldh, damp);
    B200Q_LAUNCH_CHECK();
    return B200Q_OK;
  }
  Columns j = {};
  j.src_table = (const void* const*)H;
  j.dst = out; j.dst_batch = (K * K + 3) & ~(int64_t)3;
  j.perm = perm; j.perm_batch = K;
  j.damp = damp;
  j.N = j.K = j.ldd = K; j.lds = ldh;
  j.rows = true;
  j.vec = pieces_ok(nullptr, ldh, K);
  return launch_columns<B200Q_F32, true>(j, count, st);
}

int b200q_gather_columns_f32(const void* W, int wdtype, int64_t N, int64_t K, int64_t ldw, const int32_t* perm,
                             float* Wf, int64_t ldf, void* stream) {
  if (!W || !Wf || N <= 0 || K <= 0 || ldw < K || ldf < K) return B200Q_ERR_ARG;
  Columns j = {};
  j.src = W; j.dst = Wf; j.perm = perm;
  j.N = N; j.K = K; j.lds = ldw; j.ldd = ldf;
  j.vec = pieces_ok(W, ldw, K) && (perm || pieces_ok(Wf, ldf, K));
  if (wdtype == B200Q_BF16) return launch_columns<B200Q_BF16, true>(j, 1, (cudaStream_t)stream);
  if (wdtype == B200Q_F32) return launch_columns<B200Q_F32, true>(j, 1, (cudaStream_t)stream);
  return B200Q_ERR_UNSUPPORTED;
}

int b200q_gather_columns_keep(const void* W, int wdtype, int64_t N, int64_t K, int64_t ldw, const int32_t* perm,
                              const float* diag, int zero, float* Wf, int64_t ldf, void* keep, int64_t ldk, void* stream) {
  if (!W || !Wf || N <= 0 || K <= 0 || ldw < K || ldf < K || (keep && ldk < K) || ((zero || keep) && !diag)) return B200Q_ERR_ARG;
  Columns j = {};
  j.src = W; j.dst = Wf; j.perm = perm; j.diag = zero ? diag : nullptr;
  j.keep = keep; j.ldk = ldk; j.keep_diag = diag;
  j.N = N; j.K = K; j.lds = ldw; j.ldd = ldf;
  j.vec = pieces_ok(W, ldw, K) && (perm || (pieces_ok(Wf, ldf, K) && (!keep || pieces_ok(keep, ldk, K))));
  if (wdtype == B200Q_BF16) return launch_columns<B200Q_BF16, true>(j, 1, (cudaStream_t)stream);
  if (wdtype == B200Q_F32) return launch_columns<B200Q_F32, true>(j, 1, (cudaStream_t)stream);
  return B200Q_ERR_UNSUPPORTED;
}

int b200q_permute_hessian(const float* H, int64_t K, int64_t ldh, const int32_t* perm, float* Hp, int64_t ldp,
                          void* stream) {
  if (!H || !perm || !Hp || K <= 0 || ldh < K || ldp < K || H == Hp) return B200Q_ERR_ARG;
  Columns j = {};
  j.src = H; j.dst = Hp; j.perm = perm;
  j.N = j.K = K; j.lds = ldh; j.ldd = ldp;
  j.rows = true;
  j.vec = pieces_ok(H, ldh, K);
  return launch_columns<B200Q_F32, true>(j, 1, (cudaStream_t)stream);
}

int b200q_scatter_columns_cast(const float* Wf, int64_t N, int64_t K, int64_t ldf, const int32_t* perm, void* out,
                               int odtype, int64_t ldo, void* stream) {
  if (!Wf || !out || N <= 0 || K <= 0 || ldf < K || ldo < K) return B200Q_ERR_ARG;
  Columns j = {};
  j.src = Wf; j.dst = out; j.perm = perm;
  j.N = N; j.K = K; j.lds = ldf; j.ldd = ldo;
  j.vec = pieces_ok(out, ldo, K) && (perm || pieces_ok(Wf, ldf, K));
  if (odtype == B200Q_BF16) return launch_columns<B200Q_BF16, false>(j, 1, (cudaStream_t)stream);
  if (odtype == B200Q_F32) return launch_columns<B200Q_F32, false>(j, 1, (cudaStream_t)stream);
  return B200Q_ERR_UNSUPPORTED;
}

int b200q_gather_columns_f32_batched(const void* const* W, int wdtype, const int32_t* const* perm,
                                     const float* const* dead_diag, float* const* Wf, int count, int64_t N,
                                     int64_t K, int64_t ldw, int64_t ldf, void* stream) {
  if (!W || !Wf || count <= 0 || count > 65535 || N <= 0 || K <= 0 || ldw < K || ldf < K) return B200Q_ERR_ARG;
  Columns j = {};
  j.src_table = W; j.dst_table = (void* const*)Wf; j.perm_table = perm; j.diag_table = dead_diag;
  j.N = N; j.K = K; j.lds = ldw; j.ldd = ldf;
  j.vec = pieces_ok(nullptr, ldw, K) && (perm || pieces_ok(nullptr, ldf, K));
  if (wdtype == B200Q_BF16) return launch_columns<B200Q_BF16, true>(j, count, (cudaStream_t)stream);
  if (wdtype == B200Q_F32) return launch_columns<B200Q_F32, true>(j, count, (cudaStream_t)stream);
  return B200Q_ERR_UNSUPPORTED;
}

int b200q_scatter_columns_cast_batched(const float* const* Wf, const int32_t* const* perm, void* const* out,
                                       int odtype, int count, int64_t N, int64_t K, int64_t ldf, int64_t ldo,
                                       void* stream) {
  if (!Wf || !out || count <= 0 || count > 65535 || N <= 0 || K <= 0 || ldf < K || ldo < K) return B200Q_ERR_ARG;
  Columns j = {};
  j.src_table = (const void* const*)Wf; j.dst_table = out; j.perm_table = perm;
  j.N = N; j.K = K; j.lds = ldf; j.ldd = ldo;
  j.vec = pieces_ok(nullptr, ldo, K) && (perm || pieces_ok(nullptr, ldf, K));
  if (odtype == B200Q_BF16) return launch_columns<B200Q_BF16, false>(j, count, (cudaStream_t)stream);
  if (odtype == B200Q_F32) return launch_columns<B200Q_F32, false>(j, count, (cudaStream_t)stream);
  return B200Q_ERR_UNSUPPORTED;
}

int b200q_gptq_prepare(float* H, int64_t K, int64_t ldh, float* Wf, int64_t N, int64_t ldf, float percdamp,
                       void* stream) {
  if (!H || K <= 0 || ldh < K) return B200Q_ERR_ARG;
  cudaStream_t st = (cudaStream_t)stream;
  if (Wf && N > 0) {
    zero_dead_columns_kernel<<<grid_for((K * 32 + 255) / 256, 4), 256, 0, st>>>(H, K, ldh + 1, Wf, N, ldf);
    B200Q_LAUNCH_CHECK();
  }
  damp_kernel<<<1, 1024, 0, st>>>(H, K, ldh, percdamp);
  B200Q_LAUNCH_CHECK();
  return B200Q_OK;
}

int b200q_gptq_zero_dead_columns(const float* diag, int64_t diag_stride, int64_t K, float* Wf, int64_t N,
                                 int64_t ldf, void* stream) {
  if (!diag || !Wf || K <= 0 || N <= 0 || ldf < K || diag_stride <= 0) return B200Q_ERR_ARG;
  zero_dead_columns_kernel<<<grid_for((K * 32 + 255) / 256, 4), 256, 0, (cudaStream_t)stream>>>(diag, K, diag_stride,
                                                                                                Wf, N, ldf);
  B200Q_LAUNCH_CHECK();
  return B200Q_OK;
}

}  // extern "C"

// fp32-accurate tile GEMM of the solve, exposed for testing and reuse:
//   C[M,N] = beta*C + alpha * A[M,Kd] * (trans_b ? B[N,Kd]^T : B[Kd,N]),  Kd <= 128.
extern "C" size_t b200q_gemm_tf32x3_workspace_bytes(int64_t M, int64_t N, int64_t Kd) {
  if (M <= 0 || N <= 0 || Kd <= 0) return 0;
  const int64_t kp = tgemm::split_ld(Kd);
  const int64_t a = (M + 127) / 128 * 128 * kp, b = (N + 127) / 128 * 128 * kp;
  return (size_t)(2 * a + 2 * b) * sizeof(float);
}
extern "C" int b200q_gemm_tf32x3(int trans_b, const float* A, int64_t lda, const float* B, int64_t ldb, float* C,
                                 int64_t ldc, int64_t M, int64_t N, int64_t Kd, float alpha, float beta,
                                 int lower_tiles, void* workspace, int* status, void* stream) {
  if (!A || !B || !C || !workspace || M <= 0 || N <= 0 || Kd <= 0 || Kd > 128) return B200Q_ERR_ARG;
  cudaStream_t st = (cudaStream_t)stream;
  const int64_t kp = tgemm::split_ld(Kd);
  const int64_t asz = (M + 127) / 128 * 128 * kp, bsz = (N + 127) / 128 * 128 * kp;
  float* a_hi = (float*)workspace;
  float* a_lo = a_hi + asz;
  float* b_hi = a_lo + asz;
  float* b_lo = b_hi + bsz;
  int rc = tgemm::split(A, lda, (int)M, (int)Kd, a_hi, a_lo, st);
  if (rc) return rc;
  if (trans_b) rc = tgemm::split(B, ldb, (int)N, (int)Kd, b_hi, b_lo, st);
  else rc = tgemm::split_transposed(B, ldb, (int)Kd, (int)N, b_hi, b_lo, kp, st);
  if (rc) return rc;
  tgemm::Job j;
  j.A = tgemm::Operand{a_hi, a_lo, kp, (M + 127) / 128 * 128, 0, 0};
  j.B = tgemm::Operand{b_hi, b_lo, kp, (N + 127) / 128 * 128, 0, 0};
  j.M = (int)M; j.N = (int)N; j.Kd = (int)Kd; j.alpha = alpha; j.beta = beta; j.C = C; j.ldc = ldc; j.status = status;
  j.set = lower_tiles ? tgemm::kLowerBlocks : tgemm::kAll;
  return tgemm::launch(j, st);
}
