// GPTQ solve, part 1: act-order permutation, gathers and scatters, dead columns and dampening, on device in fp32.
// The factorisation is in gptq_factor.cu, the column sweep in gptq_sweep.cu.
#include "common.cuh"
#include "tgemm_tf32.cuh"

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

template <int DT>
__global__ void gather_cols_kernel(const void* __restrict__ W, int64_t N, int64_t K, int64_t ldw,
                                   const int32_t* __restrict__ perm, float* __restrict__ out, int64_t ldo) {
  using E = Elem<DT>;
  const int64_t total = N * K;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total;
       i += (int64_t)gridDim.x * blockDim.x) {
    int64_t r = i / K, c = i - r * K;
    int64_t src = perm ? perm_at(perm, c, K) : c;
    out[r * ldo + c] = E::load((const typename E::type*)W + r * ldw + src);
  }
}

// Batched forms for many weights of one shape (device arrays of pointers, blockIdx.y = problem):
// the gather also zeroes the columns whose Hessian diagonal entry (after the permutation) is zero.
template <int DT>
__global__ void gather_cols_batched_kernel(const void* const* __restrict__ W, int64_t N, int64_t K, int64_t ldw,
                                           const int32_t* const* __restrict__ perm,
                                           const float* const* __restrict__ diag, float* const* __restrict__ out,
                                           int64_t ldo) {
  using E = Elem<DT>;
  const int j = blockIdx.y;
  const typename E::type* w = (const typename E::type*)W[j];
  const int32_t* pm = perm ? perm[j] : nullptr;
  const float* dg = diag ? diag[j] : nullptr;
  float* o = out[j];
  const int64_t total = N * K;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t r = i / K, c = i - r * K;
    const int64_t src = pm ? perm_at(pm, c, K) : c;
    const bool dead = dg && dg[c] == 0.0f;
    o[r * ldo + c] = dead ? 0.0f : E::load(w + r * ldw + src);
  }
}

template <int DT>
__global__ void scatter_cols_batched_kernel(const float* const* __restrict__ Wf, int64_t N, int64_t K, int64_t ldf,
                                            const int32_t* const* __restrict__ perm, void* const* __restrict__ out,
                                            int64_t ldo) {
  using E = Elem<DT>;
  const int j = blockIdx.y;
  const float* wf = Wf[j];
  const int32_t* pm = perm ? perm[j] : nullptr;
  typename E::type* o = (typename E::type*)out[j];
  const int64_t total = N * K;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t r = i / K, c = i - r * K;
    const int64_t dst = pm ? perm_at(pm, c, K) : c;
    E::store(o + r * ldo + dst, wf[r * ldf + c]);
  }
}

__global__ void permute_hessian_kernel(const float* __restrict__ H, int64_t K, int64_t ldh,
                                       const int32_t* __restrict__ perm, float* __restrict__ out,
                                       int64_t ldo) {
  const int64_t total = K * K;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total;
       i += (int64_t)gridDim.x * blockDim.x) {
    int64_t r = i / K, c = i - r * K;
    out[r * ldo + c] = H[perm_at(perm, r, K) * ldh + perm_at(perm, c, K)];
  }
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
// ... and the matrix: out[r][c] = H[perm r][perm c], dead diagonal entries 1, damping added.  In place without a
// permutation, where only the diagonal changes.
__global__ void __launch_bounds__(256) permute_damp_kernel(float* const* __restrict__ Hs, int64_t K, int64_t ldh,
                                                           const int32_t* __restrict__ perm, const float* __restrict__ damp,
                                                           float* __restrict__ out) {
  const float* H = Hs[blockIdx.y];
  const float dm = damp[blockIdx.y];
  if (!perm) {
    for (int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x; i < K; i += (int64_t)gridDim.x * 256) {
      const float d = H[i * ldh + i];
      Hs[blockIdx.y][i * ldh + i] = (d == 0.0f ? 1.0f : d) + dm;
    }
    return;
  }
  const int32_t* pm = perm + blockIdx.y * K;
  float* o = out + blockIdx.y * ((K * K + 3) & ~(int64_t)3);
  for (int64_t r = blockIdx.x; r < K; r += gridDim.x) {
    const float* row = H + (int64_t)pm[r] * ldh;
    for (int64_t c = threadIdx.x; c < K; c += 256) {
      float v = row[pm[c]];
      if (c == r) v = (v == 0.0f ? 1.0f : v) + dm;
      o[r * K + c] = v;
    }
  }
}

template <int DT>
__global__ void scatter_cols_kernel(const float* __restrict__ Wf, int64_t N, int64_t K, int64_t ldf,
                                    const int32_t* __restrict__ perm, void* __restrict__ out, int64_t ldo) {
  using E = Elem<DT>;
  const int64_t total = N * K;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total;
       i += (int64_t)gridDim.x * blockDim.x) {
    int64_t r = i / K, c = i - r * K;
    int64_t dst = perm ? perm_at(perm, c, K) : c;
    E::store((typename E::type*)out + r * ldo + dst, Wf[r * ldf + c]);
  }
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
  const int64_t need = perm ? K : (K + 255) / 256, cap = 8 * kNumSMs / count + 1;
  permute_damp_kernel<<<dim3((unsigned)(need < cap ? need : cap), (unsigned)count), 256, 0, st>>>(H, K, ldh, perm, damp, out);
  B200Q_LAUNCH_CHECK();
  return B200Q_OK;
}

int b200q_gather_columns_f32(const void* W, int wdtype, int64_t N, int64_t K, int64_t ldw, const int32_t* perm,
                             float* Wf, int64_t ldf, void* stream) {
  if (!W || !Wf || N <= 0 || K <= 0 || ldw < K || ldf < K) return B200Q_ERR_ARG;
  int grid = grid_for((N * K + 255) / 256, 8);
  cudaStream_t st = (cudaStream_t)stream;
  if (wdtype == B200Q_BF16) gather_cols_kernel<B200Q_BF16><<<grid, 256, 0, st>>>(W, N, K, ldw, perm, Wf, ldf);
  else if (wdtype == B200Q_F32) gather_cols_kernel<B200Q_F32><<<grid, 256, 0, st>>>(W, N, K, ldw, perm, Wf, ldf);
  else return B200Q_ERR_UNSUPPORTED;
  B200Q_LAUNCH_CHECK();
  return B200Q_OK;
}

int b200q_permute_hessian(const float* H, int64_t K, int64_t ldh, const int32_t* perm, float* Hp, int64_t ldp,
                          void* stream) {
  if (!H || !perm || !Hp || K <= 0 || ldh < K || ldp < K || H == Hp) return B200Q_ERR_ARG;
  permute_hessian_kernel<<<grid_for((K * K + 255) / 256, 8), 256, 0, (cudaStream_t)stream>>>(H, K, ldh, perm, Hp, ldp);
  B200Q_LAUNCH_CHECK();
  return B200Q_OK;
}

int b200q_scatter_columns_cast(const float* Wf, int64_t N, int64_t K, int64_t ldf, const int32_t* perm, void* out,
                               int odtype, int64_t ldo, void* stream) {
  if (!Wf || !out || N <= 0 || K <= 0 || ldf < K || ldo < K) return B200Q_ERR_ARG;
  int grid = grid_for((N * K + 255) / 256, 8);
  cudaStream_t st = (cudaStream_t)stream;
  if (odtype == B200Q_BF16) scatter_cols_kernel<B200Q_BF16><<<grid, 256, 0, st>>>(Wf, N, K, ldf, perm, out, ldo);
  else if (odtype == B200Q_F32) scatter_cols_kernel<B200Q_F32><<<grid, 256, 0, st>>>(Wf, N, K, ldf, perm, out, ldo);
  else return B200Q_ERR_UNSUPPORTED;
  B200Q_LAUNCH_CHECK();
  return B200Q_OK;
}

int b200q_gather_columns_f32_batched(const void* const* W, int wdtype, const int32_t* const* perm,
                                     const float* const* dead_diag, float* const* Wf, int count, int64_t N,
                                     int64_t K, int64_t ldw, int64_t ldf, void* stream) {
  if (!W || !Wf || count <= 0 || count > 65535 || N <= 0 || K <= 0 || ldw < K || ldf < K) return B200Q_ERR_ARG;
  int gx = grid_for((N * K + 255) / 256, 8);
  const int cap = 8 * kNumSMs / count + 1;          // enough blocks over all problems to fill the machine
  if (gx > cap) gx = cap;
  dim3 grid((unsigned)gx, (unsigned)count, 1);
  cudaStream_t st = (cudaStream_t)stream;
  if (wdtype == B200Q_BF16) gather_cols_batched_kernel<B200Q_BF16><<<grid, 256, 0, st>>>(W, N, K, ldw, perm, dead_diag, Wf, ldf);
  else if (wdtype == B200Q_F32) gather_cols_batched_kernel<B200Q_F32><<<grid, 256, 0, st>>>(W, N, K, ldw, perm, dead_diag, Wf, ldf);
  else return B200Q_ERR_UNSUPPORTED;
  B200Q_LAUNCH_CHECK();
  return B200Q_OK;
}

int b200q_scatter_columns_cast_batched(const float* const* Wf, const int32_t* const* perm, void* const* out,
                                       int odtype, int count, int64_t N, int64_t K, int64_t ldf, int64_t ldo,
                                       void* stream) {
  if (!Wf || !out || count <= 0 || count > 65535 || N <= 0 || K <= 0 || ldf < K || ldo < K) return B200Q_ERR_ARG;
  int gx = grid_for((N * K + 255) / 256, 8);
  const int cap = 8 * kNumSMs / count + 1;
  if (gx > cap) gx = cap;
  dim3 grid((unsigned)gx, (unsigned)count, 1);
  cudaStream_t st = (cudaStream_t)stream;
  if (odtype == B200Q_BF16) scatter_cols_batched_kernel<B200Q_BF16><<<grid, 256, 0, st>>>(Wf, N, K, ldf, perm, out, ldo);
  else if (odtype == B200Q_F32) scatter_cols_batched_kernel<B200Q_F32><<<grid, 256, 0, st>>>(Wf, N, K, ldf, perm, out, ldo);
  else return B200Q_ERR_UNSUPPORTED;
  B200Q_LAUNCH_CHECK();
  return B200Q_OK;
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
  else rc = tgemm::split_transposed(B, nullptr, 0, ldb, (int)Kd, (int)N, b_hi, b_lo, kp, 0, 1, st);
  if (rc) return rc;
  tgemm::Job j;
  j.A = tgemm::Operand{a_hi, a_lo, kp, (M + 127) / 128 * 128, 0, 0};
  j.B = tgemm::Operand{b_hi, b_lo, kp, (N + 127) / 128 * 128, 0, 0};
  j.M = (int)M; j.N = (int)N; j.Kd = (int)Kd; j.alpha = alpha; j.beta = beta; j.C = C; j.ldc = ldc; j.status = status;
  j.set = lower_tiles ? tgemm::kLower : tgemm::kAll;
  return tgemm::launch(j, st);
}
