// fp32-accurate tile GEMM on the tensor cores (tcgen05, kind::tf32, "3xTF32").
//
//   C[M,N] = beta * C + alpha * A[M,Kd] * B[N,Kd]^T,   Kd <= 512
//
// Each float32 operand x is given as two tf32-exact arrays hi = tf32(x), lo = tf32(x - hi); every
// k-step issues three MMAs into one TMEM accumulator, hi*hi + hi*lo + lo*hi, which keeps ~22
// significant bits per product.  What limits the accuracy is the accumulation, which cuts off
// instead of rounding: see Job::slice.
//
// Structure: persistent CTAs, each with a contiguous range of the tile list (128 x TN tiles).  Warp 0
// streams 32-deep chunks of both operands (A_hi, A_lo, B_hi, B_lo) through a shared-memory ring by
// TMA.  Warp 1 issues the MMAs and owns TMEM.  A contraction is cut into slices of 32 to 128 terms:
// each slice accumulates in its own TMEM buffer (two, used in turn) and the epilogue (warps 4-11) adds
// the slices in registers, so no tensor-core accumulation chain is longer than that whatever Kd is, and
// C is read and written once per launch.
//
// Why Kd up to 512: a rank-128 update of a 128 x 128 tile moves 128 KB of C for 1.7 us of MMA work,
// which made the factorisation HBM-bound (222 us for 6105 tiles, 43 % of DRAM, tensor pipe 40 %).
// At rank 512 the C traffic per flop is a quarter and the launch count drops with it.
// Why three tile widths: the operands of a chunk come from L2 at 64 B/clk and SM for TN = 256, 85 for
// 128 and 128 for 64, so wide tiles run closer to the tensor pipe, narrow ones spread a small update
// over more SMs; pick_tiles() takes whatever finishes its waves first, CTA pairs of 256 x 256 among them.
//
// Operands of halves (kind::f16, "3xFP16" with a power-of-two scale per operand row) run the same way with chunks of 64
// terms: half the bytes and half the MMAs for as many bits.  The scales go onto the finished sums.
//
// All mbarrier waits are bounded.  CTA pairs are clusters of two; no load is multicast.
#include <cuda.h>

#include <cstdlib>
#include <mutex>
#include <type_traits>

#include "common.cuh"
#include "tgemm_tf32.cuh"

namespace b200q {
namespace tgemm {

constexpr int kChunkBytes = 128;                     // of an operand row: 32 floats or 64 halves
constexpr int kChunkK = kChunkBytes / 4, kChunkK16 = kChunkBytes / 2;
constexpr int kAPart = kTile * kChunkBytes;          // A_hi or A_lo of a chunk: 16 KiB
constexpr int kRingBytes = 196608;                   // 2, 3 or 4 stages for TN = 256, 128, 64
constexpr int kEpiWarps = 8;                         // two per TMEM lane quarter, each half of the columns
constexpr int kEpiBytes = kEpiWarps * 32 * 33 * 4;   // per-warp staging tiles of the epilogue
constexpr int kSmemBytes = kRingBytes + 1024 + 256 + kEpiBytes;
constexpr int kFirstEpiWarp = 4;                    // warpgroup 0: producer, MMA issuer, two idle warps
constexpr int kThreads = 32 * (kFirstEpiWarp + kEpiWarps);
// 384 threads at 168 registers; warpgroup 0 gives up 96 a thread and the epilogue's two take 48 each
// (72 + 216 + 216 = 3 * 168), so that a thread can hold 128 sums
constexpr int kIssueRegs = 72, kEpiRegs = 216;
constexpr long long kWaitCycles = 4000000000LL;

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred P1;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 P1, [%1], %2;\n\t"
      "selp.b32 %0, 1, 0, P1;\n\t}"
      : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
  return ok != 0;
}
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
  if (mbar_try_wait(bar, parity)) return true;
  const long long t0 = clock64();
  while (true) {
    if (mbar_try_wait(bar, parity)) return true;
    if (*abort_flag) return false;
    if (clock64() - t0 > kWaitCycles) { *abort_flag = 1; return false; }
  }
}
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int c1) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1) : "memory");
}
// CTA pairs (cta_group::2): the same location in CTA `rank` of the cluster, a load whose bytes count on a barrier of the
// even CTA, an arrival there, and the commit that arrives in both CTAs
__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t map_to_cta(uint32_t addr, uint32_t rank) {
  uint32_t out;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(out) : "r"(addr), "r"(rank));
  return out;
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const CUtensorMap* map, uint32_t bar_cluster_addr,
                                                 int c0, int c1) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4}], [%2];"
      ::"r"(dst), "l"(map), "r"(bar_cluster_addr), "r"(c0), "r"(c1) : "memory");
}
__device__ __forceinline__ void tc_commit_pair(uint32_t bar) {
  const uint16_t both = 3;
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
      ::"r"(bar), "h"(both) : "memory");
}
template <bool F16>
__device__ __forceinline__ void mma_pair(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                              uint32_t accumulate) {
  const uint32_t z = 0;
  if constexpr (F16)
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, {%5, %5, %5, %5, %5, %5, %5, %5}, p;\n\t}"
        ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate), "r"(z) : "memory");
  else
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::tf32 [%0], %1, %2, %3, {%5, %5, %5, %5, %5, %5, %5, %5}, p;\n\t}"
        ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate), "r"(z) : "memory");
}
__device__ __forceinline__ void tc_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
template <bool F16>
__device__ __forceinline__ void mma_one(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                        uint32_t accumulate) {
  if constexpr (F16)
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate) : "memory");
  else
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr) : "memory");
}
// x += v in L2: an update neither waits for C nor holds registers for it.  With loads and stores the epilogue (two waits
// on C per 32 columns) was slower than the MMAs of its tile, and the tensor pipe stood at 53 %.
__device__ __forceinline__ void red_add_v4(float* p, float a, float b, float c, float d) {
  asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(a), "f"(b), "f"(c), "f"(d) : "memory");
}
// shared-memory matrix descriptor, 128-byte swizzle, descriptor version 1
__device__ __forceinline__ uint64_t make_desc(uint32_t saddr, uint32_t lbo_bytes, uint32_t sbo_bytes) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr >> 4) & 0x3FFFu);
  d |= (uint64_t)((lbo_bytes >> 4) & 0x3FFFu) << 16;
  d |= (uint64_t)((sbo_bytes >> 4) & 0x3FFFu) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;
  return d;
}
// D fp32, A/B tf32 or f16, both K-major, M = tm, N = tn
__host__ __device__ constexpr uint32_t instr_desc(int tm, int tn, bool f16) {
  return (1u << 4) | (f16 ? 0u : (2u << 7) | (2u << 10)) | ((uint32_t)(tn >> 3) << 17) | ((uint32_t)(tm >> 4) << 24);
}

struct Params {
  Job j;
  int row_tiles, tm_rows, tn_log2;      // rows of a tile: 128, or 256 for a CTA pair
  int64_t num_tiles;                    // over all problems
  uint16_t start[kNumSMs][3];           // (problem, row tile, column tile) each CTA or pair starts at
};

__host__ __device__ __forceinline__ int tile_row(const Job& j, int tm, int rows) {
  int r = j.row_begin + tm * rows;
  if (j.set == kPanel && r >= j.skip0) r += j.skip1 - j.skip0;
  return r;
}
// column tiles of row tile tm (they are contiguous from column 0)
__host__ __device__ __forceinline__ int col_tiles(const Job& j, int tm, int rows, int tn_log2) {
  int lim = j.N;
  if (j.set == kLower || j.set == kBulk || j.set == kLowerBlocks) {
    const int r = tile_row(j, tm, rows);
    const int diag = (j.set == kBulk && r < j.skip1) ? j.skip0 : r + rows;
    lim = diag < lim ? diag : lim;
  }
  return (lim + (1 << tn_log2) - 1) >> tn_log2;
}
__device__ __forceinline__ void next_tile(const Params& p, int& b, int& tm, int& tn) {
  ++tn;
  while (tn >= col_tiles(p.j, tm, p.tm_rows, p.tn_log2)) {   // a row tile may have no column at all
    tn = 0;
    if (++tm == p.row_tiles) { tm = 0; ++b; return; }
  }
}

// PAIR: two CTAs on neighbouring SMs (a cluster of 2) share a 256 x 256 tile.  One MMA issued by the even CTA runs on both
// SMs; each stages its own 128 rows of A and its own 128 of B, 64 KiB a chunk instead of 96, and has its own half of the
// accumulator and its own epilogue.  full[] and acc_empty[] live in the even CTA, empty[] and acc_full[] in both.
template <int TN, bool SPLIT_OUT, bool PAIR, bool F16>
__global__ void __launch_bounds__(kThreads, 1)
tgemm_kernel(const __grid_constant__ CUtensorMap a_hi, const __grid_constant__ CUtensorMap a_lo,
             const __grid_constant__ CUtensorMap b_hi, const __grid_constant__ CUtensorMap b_lo,
             const __grid_constant__ Params p) {
  constexpr int kRows = PAIR ? 2 * kTile : kTile;      // rows of a tile
  constexpr int kBRows = PAIR ? TN / 2 : TN;           // rows of B that this CTA stages
  constexpr int kBPart = kBRows * kChunkBytes, kChunk = F16 ? kChunkK16 : kChunkK;
  static_assert(!(F16 && SPLIT_OUT), "");
  constexpr int kStageBytes = 2 * kAPart + 2 * kBPart;
  constexpr int kStages = kRingBytes / kStageBytes;
  constexpr uint32_t kTmemCols = 2 * TN;
  extern __shared__ unsigned char smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  unsigned char* aligned = smem_raw + (base - raw);
  uint64_t* bars = reinterpret_cast<uint64_t*>(aligned + kRingBytes);
  const uint32_t bar0 = smem_u32(bars);
  auto full_bar = [&](int s) { return bar0 + 8u * s; };
  auto empty_bar = [&](int s) { return bar0 + 8u * (kStages + s); };
  auto accf_bar = [&](int b) { return bar0 + 8u * (2 * kStages + b); };
  auto acce_bar = [&](int b) { return bar0 + 8u * (2 * kStages + 2 + b); };
  __shared__ uint32_t s_tmem_base;
  __shared__ volatile int s_abort;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = PAIR ? (int)cluster_ctarank() : 0;
  const int unit = PAIR ? blockIdx.x >> 1 : blockIdx.x, units = PAIR ? gridDim.x >> 1 : gridDim.x;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) { mbar_init(full_bar(s), 1); mbar_init(empty_bar(s), 1); }
    for (int b = 0; b < 2; ++b) { mbar_init(accf_bar(b), 1); mbar_init(acce_bar(b), PAIR ? 2 * kEpiWarps : kEpiWarps); }
    s_abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    if constexpr (PAIR) {
      asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem_base)),
                   "r"(kTmemCols) : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    } else {
      asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem_base)),
                   "r"(kTmemCols) : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (PAIR) cluster_sync_all();   // the peer's barriers are initialised before anything signals them
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_base = s_tmem_base;
  chain_wait();
  const Job& j = p.j;
  constexpr int kSteps = kChunkBytes / 32;   // k-steps of a chunk
  const int chunks = (j.Kd + kChunk - 1) / kChunk;
  const int64_t count = p.num_tiles * (unit + 1) / units - p.num_tiles * unit / units;
  int b = p.start[unit][0], tm = p.start[unit][1], tn = p.start[unit][2];

  if (warp < kFirstEpiWarp) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kIssueRegs));
    if (warp == 0 && lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int64_t i = 0; i < count && ok; ++i, next_tile(p, b, tm, tn)) {
        const int ra = (int)(b * j.A.batch_rows) + j.A.row0 + tile_row(j, tm, kRows) + rank * kTile;
        const int rb = (int)((j.b_index ? j.b_index[b] : b) * j.B.batch_rows) + j.B.row0 + tn * TN + rank * kBRows;
        for (int c = 0; c < chunks; ++c) {
          if (!mbar_wait(empty_bar(stage), phase ^ 1u, &s_abort)) { ok = false; break; }
          const uint32_t s = base + stage * kStageBytes;
          if constexpr (PAIR) {
            if (rank == 0) mbar_expect_tx(full_bar(stage), 2 * kStageBytes);
            const uint32_t full = map_to_cta(full_bar(stage), 0);
            tma_load_2d_pair(s, &a_hi, full, c * kChunk, ra);
            tma_load_2d_pair(s + 2 * kAPart, &b_hi, full, c * kChunk, rb);
            tma_load_2d_pair(s + 2 * kAPart + kBPart, &b_lo, full, c * kChunk, rb);
            tma_load_2d_pair(s + kAPart, &a_lo, full, c * kChunk, ra);
          } else {
          mbar_expect_tx(full_bar(stage), kStageBytes);
          tma_load_2d(s, &a_hi, full_bar(stage), c * kChunk, ra);
          tma_load_2d(s + 2 * kAPart, &b_hi, full_bar(stage), c * kChunk, rb);
          tma_load_2d(s + 2 * kAPart + kBPart, &b_lo, full_bar(stage), c * kChunk, rb);
          tma_load_2d(s + kAPart, &a_lo, full_bar(stage), c * kChunk, ra);
          }
          if (++stage == kStages) { stage = 0; phase ^= 1u; }
        }
      }
    }
    if (warp == 1 && rank == 0) {
    int stage = 0, slice = 0;
    uint32_t phase = 0;
    bool ok = true;
    constexpr uint32_t idesc = instr_desc(kRows, TN, F16);
    for (int64_t i = 0; i < count && ok; ++i) {
      for (int c = 0; c < chunks; ++c) {
        if (!mbar_wait(full_bar(stage), phase, &s_abort)) { ok = false; break; }
        const uint32_t sa = base + stage * kStageBytes, sb = sa + 2 * kAPart;
        // k-steps k0 .. k0 + N of the chunk, to the slice under way (unrolled: descriptors made in a loop cost 5 us a launch)
        auto issue = [&](int k0, auto N, bool first, bool last) {
          const int buf = slice & 1;
          if (first && !mbar_wait(acce_bar(buf), (uint32_t)(((slice >> 1) & 1) ^ 1), &s_abort)) { ok = false; return; }
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          if (lane == 0) {
            const uint32_t d_tmem = tmem_base + (uint32_t)(buf * TN), a = sa + k0 * 32, b = sb + k0 * 32;
            // K-major, 128-byte rows: 8-row groups 1024 bytes apart; a k-step of 8 tf32 or 16 halves is 32 bytes
            auto mma = [&](uint32_t x, uint32_t y, uint32_t accumulate) {
              if constexpr (PAIR) mma_pair<F16>(d_tmem, make_desc(x, 16, 1024), make_desc(y, 16, 1024), idesc, accumulate);
              else mma_one<F16>(d_tmem, make_desc(x, 16, 1024), make_desc(y, 16, 1024), idesc, accumulate);
            };
            // the small products first: in a short slice they lose next to nothing, the sum being as small as they are
#pragma unroll
            for (int kk = 0; kk < N; ++kk) {
              mma(a + kk * 32, b + kBPart + kk * 32, (first && kk == 0) ? 0u : 1u);
              mma(a + kAPart + kk * 32, b + kk * 32, 1u);
            }
#pragma unroll
            for (int kk = 0; kk < N; ++kk) mma(a + kk * 32, b + kk * 32, 1u);
            if (k0 + N == kSteps) {
              if constexpr (PAIR) tc_commit_pair(empty_bar(stage));
              else tc_commit(empty_bar(stage));
            }
            if (last) {
              if constexpr (PAIR) tc_commit_pair(accf_bar(buf));
              else tc_commit(accf_bar(buf));
            }
          }
          __syncwarp();
          if (last) ++slice;
        };
        if (!F16 || j.slice >= kSteps) {
          const int whole = j.slice / kSteps;
          issue(0, std::integral_constant<int, kSteps>(), c % whole == 0, c % whole == whole - 1 || c == chunks - 1);
        } else {
          issue(0, std::integral_constant<int, kSteps / 2>(), true, true);
          if (ok) issue(kSteps / 2, std::integral_constant<int, kSteps / 2>(), true, true);
        }
        if (!ok) break;
        if (++stage == kStages) { stage = 0; phase ^= 1u; }
      }
    }
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kEpiRegs));
    constexpr int kHalf = TN / 2;          // columns of this warp
    const int q = warp & 3, half = (warp - kFirstEpiWarp) >> 2;
    // per-warp staging tile [32 rows][33]: accumulator rows come out of TMEM one row per lane; going
    // through shared memory lets every global access cover whole 128-byte row segments
    float* stage = reinterpret_cast<float*>(aligned + kRingBytes + 256) + (warp - kFirstEpiWarp) * (32 * 33);
    const int sub_row = lane >> 3, sub_col = (lane & 7) * 4;  // 4 rows x 8 float4 per instruction
    int slice = 0;
    bool ok = true;
    for (int64_t i = 0; i < count && ok; ++i, next_tile(p, b, tm, tn)) {
      const int row0 = tile_row(j, tm, kRows) + rank * kTile + q * 32, colw = tn * TN + half * kHalf;
      float sum[kHalf];
      // scales of halves: the lane's row, a column of every 32 (asked for now, they are needed when the sums are there)
      float row_factor = j.alpha, col_factor[kHalf / 32];
      if constexpr (F16) {
        row_factor *= row0 + lane < j.M ? j.A.scale[(int64_t)b * j.A.batch_rows + j.A.row0 + row0 + lane] : 0.0f;
        const float* cf = j.B.scale + (j.b_index ? j.b_index[b] : b) * j.B.batch_rows + j.B.row0;
#pragma unroll
        for (int k = 0; k < kHalf / 32; ++k) col_factor[k] = colw + k * 32 + lane < j.N ? cf[colw + k * 32 + lane] : 0.0f;
      }
      for (int c = 0; c < chunks * kSteps; c += j.slice, ++slice) {
        const int buf = slice & 1;
        if (!mbar_wait(accf_bar(buf), (uint32_t)((slice >> 1) & 1), &s_abort)) { ok = false; break; }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
        for (int k = 0; k < kHalf / 16; ++k) {
          uint32_t r[16];
          tmem_ld16(tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(buf * TN + half * kHalf + k * 16), r);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
          for (int e = 0; e < 16; ++e)
            sum[k * 16 + e] = (c == 0) ? __uint_as_float(r[e]) : sum[k * 16 + e] + __uint_as_float(r[e]);
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) {
          if (rank == 0) mbar_arrive(acce_bar(buf));
          else mbar_arrive_cluster(map_to_cta(acce_bar(buf), 0));
        }
      }
      if (!ok) break;
      float* C = nullptr;
      bool vec = true;
      if (!SPLIT_OUT) {
        C = j.c_table ? j.c_table[b] + j.c_offset : j.C + (int64_t)b * j.c_batch;
        vec = ((j.ldc & 3) == 0) && ((((uintptr_t)C) & 15) == 0);
      }
      const int cols = j.set == kBulk && row0 < j.skip1 ? j.skip0 : j.N;   // (a tile may reach beyond skip0)
#pragma unroll
      for (int k = 0; k < kHalf / 32; ++k) {
        const int col0 = colw + k * 32;
        if (col0 >= cols) break;   // warp-uniform
        const int cc = col0 + sub_col;
        if constexpr (SPLIT_OUT) {
          if (j.X && row0 < j.xt_rows && row0 + lane < j.M) {
            // lanes hold consecutive rows: the transposed store is contiguous as it stands
            float* x = j.X + (int64_t)b * j.x_batch + row0 + lane;
#pragma unroll
            for (int e = 0; e < 32; ++e)
              if (col0 + e < j.N) x[(int64_t)(col0 + e) * j.ldx] = j.alpha * sum[k * 32 + e];
          }
          if (j.out_hi) {
#pragma unroll
            for (int e = 0; e < 32; ++e) stage[lane * 33 + e] = sum[k * 32 + e] * j.alpha;
            __syncwarp();
#pragma unroll
            for (int s = 0; s < 8; ++s) {
              const int lr = s * 4 + sub_row, row = row0 + lr;
              if (row < j.M && (j.out_lo || row >= j.xt_rows)) {
                const float* sp = stage + lr * 33 + sub_col;
                const int64_t at = (int64_t)b * j.out_batch + (int64_t)(row + j.out_row0) * j.out_ld + cc;
                if (!j.out_lo) {
                  *reinterpret_cast<float4*>(j.out_hi + at) = make_float4(sp[0], sp[1], sp[2], sp[3]);
                  continue;
                }
                float4 h, l;
                h.x = tf32_rn(sp[0]); h.y = tf32_rn(sp[1]); h.z = tf32_rn(sp[2]); h.w = tf32_rn(sp[3]);
                l.x = tf32_rn(sp[0] - h.x); l.y = tf32_rn(sp[1] - h.y);
                l.z = tf32_rn(sp[2] - h.z); l.w = tf32_rn(sp[3] - h.w);
                *reinterpret_cast<float4*>(j.out_hi + at) = h;
                *reinterpret_cast<float4*>(j.out_lo + at) = l;
              }
            }
            __syncwarp();
          }
        } else {
          const float beta = (col0 >= j.fresh0 && col0 < j.fresh1) ? 0.0f : j.beta;
          const bool fast = vec && col0 + 31 < j.N;
          float4 f = make_float4(1.f, 1.f, 1.f, 1.f);   // of the four columns that this lane writes
          if constexpr (F16) {
            f.x = __shfl_sync(0xffffffffu, col_factor[k], sub_col); f.y = __shfl_sync(0xffffffffu, col_factor[k], sub_col + 1);
            f.z = __shfl_sync(0xffffffffu, col_factor[k], sub_col + 2); f.w = __shfl_sync(0xffffffffu, col_factor[k], sub_col + 3);
          }
          const float fs[4] = {f.x, f.y, f.z, f.w};
#pragma unroll
          for (int e = 0; e < 32; ++e) stage[lane * 33 + e] = sum[k * 32 + e] * row_factor;
          __syncwarp();
          if (fast) {
            float* c = C + (int64_t)(row0 + sub_row) * j.ldc + cc;
            if (beta == 1.0f) {
#pragma unroll
              for (int s = 0; s < 8; ++s) {
                const int lr = s * 4 + sub_row;
                if (row0 + lr < j.M) {
                  const float* sp = stage + lr * 33 + sub_col;
                  red_add_v4(c + (int64_t)(s * 4) * j.ldc, sp[0] * f.x, sp[1] * f.y, sp[2] * f.z, sp[3] * f.w);
                }
              }
            } else {
#pragma unroll
            for (int s0 = 0; s0 < 8; s0 += 4) {
              float4 h[4];
#pragma unroll
              for (int s = 0; s < 4; ++s) {
                h[s] = make_float4(0.f, 0.f, 0.f, 0.f);
                if (beta != 0.0f && row0 + (s0 + s) * 4 + sub_row < j.M)
                  h[s] = *reinterpret_cast<const float4*>(c + (int64_t)((s0 + s) * 4) * j.ldc);
              }
#pragma unroll
              for (int s = 0; s < 4; ++s) {
                const int lr = (s0 + s) * 4 + sub_row;
                if (row0 + lr < j.M) {
                  const float* sp = stage + lr * 33 + sub_col;
                  float4 o;
                  o.x = beta * h[s].x + sp[0] * f.x; o.y = beta * h[s].y + sp[1] * f.y;
                  o.z = beta * h[s].z + sp[2] * f.z; o.w = beta * h[s].w + sp[3] * f.w;
                  *reinterpret_cast<float4*>(c + (int64_t)((s0 + s) * 4) * j.ldc) = o;
                }
              }
            }
            }
          } else {
            for (int s = 0; s < 8; ++s) {
              const int lr = s * 4 + sub_row, row = row0 + lr;
              if (row >= j.M) continue;
              for (int e = 0; e < 4; ++e)
                if (cc + e < j.N) {
                  float* d = C + (int64_t)row * j.ldc + cc + e;
                  const float old = (beta != 0.0f) ? *d : 0.0f;
                  *d = beta * old + stage[lr * 33 + sub_col + e] * fs[e];
                }
            }
          }
          __syncwarp();
        }
      }
    }
  }

  chain_go();
  if (s_abort) {
    if (threadIdx.x == 0 && j.status)
      for (int k = 0; k < j.batch; ++k) atomicCAS(j.status + k * j.status_stride, 0, B200Q_ERR_DEVICE);
    const long long t0 = clock64();
    while (clock64() - t0 < 2000000LL) __nanosleep(1000);
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (PAIR) cluster_sync_all();   // nothing of the peer's is still on its way here
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if constexpr (PAIR)
      asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(kTmemCols) : "memory");
    else
      asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(kTmemCols) : "memory");
  }
}

// hi = tf32(x) (round to nearest even on 10 mantissa bits), lo = tf32(x - hi); both stored as
// float32 words whose low 13 mantissa bits are zero.  dst rows are zero-padded to ld_dst.
__global__ void split_kernel(const float* __restrict__ src, int64_t ld_src, int rows, int cols,
                             float* __restrict__ hi, float* __restrict__ lo, int64_t ld_dst) {
  const int64_t total = (int64_t)rows * ld_dst;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t r = i / ld_dst, c = i - r * ld_dst;
    float h = 0.0f, l = 0.0f;
    if (c < cols) {
      const float x = src[r * ld_src + c];
      h = tf32_rn(x);
      l = tf32_rn(x - h);
    }
    hi[i] = h;
    lo[i] = l;
  }
}

// Transposing variant: row c of hi/lo (ld_dst floats) holds column c of src, zero-padded.  Turns a
// [Kd][N] operand into the K-major [N][Kd] form the MMA reads.
__global__ void __launch_bounds__(256) split_transposed_kernel(const float* __restrict__ src,
                                                               int64_t ld_src, int rows, int cols,
                                                               float* __restrict__ hi, float* __restrict__ lo,
                                                               int64_t ld_dst) {
  __shared__ float tile[32][33];
  chain_wait();
  chain_go();
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;  // 32 x 8
  const int tiles_c = (cols + 31) / 32, tiles_r = (int)(ld_dst / 32);
  for (int t = blockIdx.x; t < tiles_c * tiles_r; t += gridDim.x) {
    const int tc = t % tiles_c, tr = t / tiles_c;
    float v[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int gr = tr * 32 + ty + 8 * k, gc = tc * 32 + tx;
      v[k] = (gr < rows && gc < cols) ? src[(int64_t)gr * ld_src + gc] : 0.0f;
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) tile[ty + 8 * k][tx] = v[k];
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int c = ty + 8 * k, gc = tc * 32 + c, gr = tr * 32 + tx;  // output row = source column
      if (gc < cols) {
        const float x = tile[tx][c];
        const float h = tf32_rn(x);
        hi[(int64_t)gc * ld_dst + gr] = h;
        lo[(int64_t)gc * ld_dst + gr] = tf32_rn(x - h);
      }
    }
    __syncthreads();
  }
}

template <int LD>
__global__ void __launch_bounds__(256) split_rows16_kernel(const float* __restrict__ src, int64_t ld_src, int64_t src_batch,
                                                           int64_t rows, int cols, __half* hi, __half* lo, float* scale,
                                                           int64_t dst_rows, const float* __restrict__ columns,
                                                           bool inverse, int64_t columns_batch, const int32_t* __restrict__ index) {
  chain_wait();
  chain_go();
  const int64_t at = blockIdx.y * dst_rows;
  split_rows16<LD>(src + blockIdx.y * src_batch, nullptr, ld_src, rows, cols, hi + at * LD, lo + at * LD, scale + at,
                   columns ? columns + (index ? index[blockIdx.y] : blockIdx.y) * columns_batch : nullptr, inverse, blockIdx.x, gridDim.x);
}
// The operand of an update of the factor in one launch: `transposed` CTAs take the columns of the block row, the others rows
// from its end on, `first` of them from a tf32 operand form.
__global__ void __launch_bounds__(256) split_update16_kernel(const UpdateOperand u, int transposed) {
  chain_wait();
  chain_go();
  extern __shared__ float stage16[];
  const int64_t at = blockIdx.y * u.dst_rows;
  __half *hi = u.hi + at * kMaxDepth, *lo = u.lo + at * kMaxDepth;
  float* scale = u.scale + at;
  if ((int)blockIdx.x < transposed) {
    split_columns16<kMaxDepth>(u.row + blockIdx.y * u.row_batch, u.row_ld, u.n, u.end, u.end - u.n, hi, lo, scale, kNoPivots, blockIdx.x,
                               stage16);
    return;
  }
  const int64_t cta = blockIdx.x - transposed, ctas = gridDim.x - transposed;
  hi += u.end * kMaxDepth; lo += u.end * kMaxDepth; scale += u.end;
  split_rows16<kMaxDepth>(u.f_hi + blockIdx.y * u.f_batch, u.f_lo + blockIdx.y * u.f_batch, kMaxDepth, u.first, u.n, hi, lo, scale,
                          nullptr, false, cta, ctas);
  hi += u.first * kMaxDepth; lo += u.first * kMaxDepth; scale += u.first;
  split_rows16<kMaxDepth>(u.p + blockIdx.y * u.p_batch, nullptr, kMaxDepth, u.rows, u.n, hi, lo, scale, nullptr, false, cta, ctas);
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
inline EncodeTiledFn encode_fn() {
  // function-local static: initialised once, thread-safely (several host threads start solving at
  // the same moment)
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
// matrix [rows][ld] of floats or halves, boxes of box_rows rows of 128 bytes
inline bool make_map(CUtensorMap* m, const void* base, int64_t rows, int64_t ld, int box_rows, bool f16) {
  EncodeTiledFn enc = encode_fn();
  if (!enc) return false;
  cuuint64_t dims[2] = {(cuuint64_t)ld, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)ld * (f16 ? 2 : 4)};
  cuuint32_t box[2] = {f16 ? (cuuint32_t)kChunkK16 : (cuuint32_t)kChunkK, (cuuint32_t)box_rows};
  cuuint32_t estr[2] = {1, 1};
  return enc(m, f16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<void*>(base), dims, strides, box, estr,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// src [rows][cols] -> hi/lo [rows][split_ld(cols)]
int split(const float* src, int64_t ld_src, int rows, int cols, float* hi, float* lo, cudaStream_t st) {
  if (rows <= 0 || cols <= 0) return B200Q_OK;
  const int64_t ld = split_ld(cols);
  split_kernel<<<grid_for(((int64_t)rows * ld + 255) / 256, 8), 256, 0, st>>>(src, ld_src, rows, cols, hi, lo, ld);
  B200Q_LAUNCH_CHECK();
  return B200Q_OK;
}

int split_transposed(const float* src, int64_t ld_src, int rows, int cols, float* hi, float* lo, int64_t ld_dst, cudaStream_t st) {
  if (rows <= 0 || cols <= 0) return B200Q_OK;
  const int64_t tiles = (int64_t)((cols + 31) / 32) * (ld_dst / 32);
  const int64_t cap = 8 * kNumSMs;
  B200Q_TRY(launch_chained(split_transposed_kernel, dim3((unsigned)(tiles < cap ? tiles : cap)), 256, 0, st, src, ld_src, rows, cols,
                           hi, lo, ld_dst));
  B200Q_LAUNCH_CHECK();
  return B200Q_OK;
}

int split_rows16(const float* src, int64_t ld_src, int64_t src_batch, int64_t rows, int cols, __half* hi, __half* lo, float* scale,
                 int ld, int64_t dst_rows, int batch, const float* columns, bool inverse, int64_t columns_batch, const int32_t* index,
                 cudaStream_t st) {
  if (rows <= 0 || cols <= 0) return B200Q_OK;
  auto kernel = ld == 512 ? split_rows16_kernel<512> : split_rows16_kernel<256>;
  const int64_t blocks = (rows + 7) / 8, cap = 8 * kNumSMs / batch + 1;
  B200Q_TRY(launch_chained(kernel, dim3((unsigned)(blocks < cap ? blocks : cap), (unsigned)batch), 256, 0, st, src, ld_src,
                           src_batch, rows, cols, hi, lo, scale, dst_rows, columns, inverse, columns_batch, index));
  B200Q_LAUNCH_CHECK();
  return B200Q_OK;
}
int split_update16(const UpdateOperand& u, int batch, cudaStream_t st) {
  const size_t smem = split_columns16_smem(kMaxDepth);
  static thread_local int attr_device = -1;
  int dev = 0;
  B200Q_TRY(cudaGetDevice(&dev));
  if (attr_device != dev) {
    B200Q_TRY(cudaFuncSetAttribute(split_update16_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    attr_device = dev;
  }
  const int transposed = (int)((u.end + 31) / 32);
  const int64_t blocks = (u.first + u.rows + 7) / 8, cap = 3 * kNumSMs / batch + 1;
  B200Q_TRY(launch_chained(split_update16_kernel, dim3((unsigned)(transposed + (blocks < cap ? blocks : cap)), (unsigned)batch), 256,
                           smem, st, u, transposed));
  B200Q_LAUNCH_CHECK();
  return B200Q_OK;
}

// Tensor maps are cached per (array, shape, box): one encode serves every launch that reads an operand
// buffer.  Rows beyond an operand's extent inside its buffer may hold anything; they only reach
// output rows / columns that the epilogue masks.  Columns beyond Kd are zero (the splits pad them).
struct MapKey { const void* base; int64_t ld, rows; int box; bool f16; };
struct MapCache {
  // one place per key: a solve has some 25 operand buffers, and one host thread queues several solves at a time
  static constexpr uint32_t kSlots = 512;
  MapKey key[kSlots] = {};
  CUtensorMap map[kSlots];
  bool get(const void* base, int64_t ld, int64_t rows, int box, bool f16, CUtensorMap* out) {
    const uint64_t mixed = ((uint64_t)(uintptr_t)base / 128 * 64 + (uint64_t)box + (f16 ? 1 : 0)) * 0x9E3779B97F4A7C15ull;
    const uint32_t slot = (uint32_t)(mixed >> 40) % kSlots;
    MapKey& k = key[slot];
    if (!(k.base == base && k.ld == ld && k.rows == rows && k.box == box && k.f16 == f16)) {
      k = MapKey{nullptr, 0, 0, 0, false};
      if (!make_map(&map[slot], base, rows, ld, box, f16)) return false;
      k = MapKey{base, ld, rows, box, f16};
    }
    *out = map[slot];
    return true;
  }
};
inline MapCache& map_cache() {
  static thread_local MapCache c;
  return c;
}

// Row tiles of `rows` rows: kPanel leaves out [skip0, skip1), which tiles of 256 rows can only do at multiples of 256.
static int count_rows(const Job& j, int rows) {
  if (j.set != kPanel) return j.M > j.row_begin ? (j.M - j.row_begin + rows - 1) / rows : 0;
  return j.skip0 / rows + (j.M > j.skip1 ? (j.M - j.skip1 + rows - 1) / rows : 0);
}
static bool rows_fit(const Job& j, int rows) {
  if (j.set == kLowerBlocks) return rows <= kTile;
  if (j.set == kPanel) return j.skip0 % rows == 0;
  return j.set != kBulk || j.skip1 <= j.row_begin || (j.skip1 - j.row_begin) % rows == 0;
}
static int64_t count_tiles(const Job& j, int rows, int tn_log2) {
  const int row_tiles = count_rows(j, rows);
  if (j.set == kAll || j.set == kPanel) return row_tiles ? (int64_t)row_tiles * col_tiles(j, 0, rows, tn_log2) : 0;
  int64_t n = 0;
  for (int tm = 0; tm < row_tiles; ++tm) n += col_tiles(j, tm, rows, tn_log2);
  return n;
}

// CTA pairs that can be resident at once on the current device; 0 if a cluster of two cannot be launched
static int pair_capacity() {
  static std::mutex mu;
  static int cached[64];
  static bool have[64] = {false};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
  std::lock_guard<std::mutex> lock(mu);
  if (have[dev]) return cached[dev];
  auto kernel = tgemm_kernel<256, false, true, false>;
  int n = 0;
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes) == cudaSuccess) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2 * (kNumSMs / 2), 1, 1);
    cfg.blockDim = dim3(kThreads, 1, 1);
    cfg.dynamicSmemBytes = kSmemBytes;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess) n = 0;
  }
  (void)cudaGetLastError();
  cached[dev] = n < 0 ? 0 : (n < kNumSMs / 2 ? n : kNumSMs / 2);
  have[dev] = true;
  return cached[dev];
}

// Tile width, and whether CTA pairs take 256 x 256: SM cycles of the busiest CTA.  A chunk of 128 bytes takes the longer of its
// MMAs (12 of 32 / 64 / 128 cycles) and the arrival of its operands from L2 (about 64 B/clk and SM); the last tile's
// epilogue, about 20 cycles per column, is not hidden.
static void pick_tiles(Params& p, int ctas, int pairs) {
  const double chunk[3] = {800.0, 1150.0, 1700.0};
  // Above 1700 pairs are never taken.  A chunk of halves holds twice the terms at the same bytes and MMA cycles, so the
  // same line serves both, but with halves it decides next to nothing.  Without / with pairs, us:
  // factor (halves) K = 4096 1215 / 1212, 8192 2903 / 2911, 14336 9830 to 10380 / 9670 to 10330; sweep (halves) 4096 x 4096
  // 821 / 809, 14336 x 4096 2417 / 2430, 4096 x 14336 4627 / 4606, 32 weights of 768 x 2048 1820 / 1834; from 1000 to 2200, and
  // with an epilogue of 10 to 40 cycles a column, within 2 % of these.  With products of tf32 14336 columns took 13353 / 11398.
  const double pair_chunk = 1600.0;
  const Job& j = p.j;
  const int depth = j.A.scale ? kChunkK16 : kChunkK, chunks = (j.Kd + depth - 1) / depth;
  double best_cost = 0.0;
  for (int w = 6; w <= (j.set == kLowerBlocks ? 7 : 8); ++w) {
    const int64_t tiles = count_tiles(j, kTile, w) * j.batch;
    const double cost = (double)((tiles + ctas - 1) / ctas) * chunks * chunk[w - 6] + 20.0 * (1 << w);
    if (w == 6 || cost < best_cost) { p.tn_log2 = w; p.tm_rows = kTile; best_cost = cost; }
  }
  if (pairs > 0 && rows_fit(j, 2 * kTile)) {
    const int64_t tiles = count_tiles(j, 2 * kTile, 8) * j.batch;
    const double cost = (double)((tiles + pairs - 1) / pairs) * chunks * pair_chunk + 20.0 * 256;
    if (cost < best_cost) { p.tn_log2 = 8; p.tm_rows = 2 * kTile; }
  }
}

template <int TN, bool SPLIT_OUT, bool PAIR, bool F16>
static int launch_tiles(const Params& p, int units, cudaStream_t st) {
  const Job& j = p.j;
  constexpr int kBRows = PAIR ? TN / 2 : TN;
  MapCache& mc = map_cache();
  CUtensorMap mah, mal, mbh, mbl;
  if (!mc.get(j.A.hi, j.A.ld, j.A.rows, kTile, F16, &mah) || !mc.get(j.A.lo, j.A.ld, j.A.rows, kTile, F16, &mal) ||
      !mc.get(j.B.hi, j.B.ld, j.B.rows, kBRows, F16, &mbh) || !mc.get(j.B.lo, j.B.ld, j.B.rows, kBRows, F16, &mbl)) {
    set_last_error("cuTensorMapEncodeTiled (tgemm)", cudaErrorInvalidValue);
    return B200Q_ERR_CUDA;
  }
  auto kernel = tgemm_kernel<TN, SPLIT_OUT, PAIR, F16>;
  static thread_local int attr_device = -1;
  int dev = 0;
  B200Q_TRY(cudaGetDevice(&dev));
  if (attr_device != dev) {
    B200Q_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes));
    attr_device = dev;
  }
  if constexpr (PAIR) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(2 * units), 1, 1);
    cfg.blockDim = dim3(kThreads, 1, 1);
    cfg.dynamicSmemBytes = kSmemBytes;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    B200Q_TRY(cudaLaunchKernelEx(&cfg, kernel, mah, mal, mbh, mbl, p));
  } else {
    B200Q_TRY(launch_chained(kernel, dim3((unsigned)units), kThreads, kSmemBytes, st, mah, mal, mbh, mbl, p));
  }
  B200Q_LAUNCH_CHECK();
  return B200Q_OK;
}

int launch(const Job& j, cudaStream_t st) {
  if (j.Kd <= 0 || j.batch <= 0) return B200Q_OK;
  const bool f16 = j.A.scale != nullptr;
  if (f16 != (j.B.scale != nullptr) || (f16 && ((j.A.ld | j.B.ld) & 63 || j.out_hi || j.X))) return B200Q_ERR_ARG;
  if (j.Kd > kMaxDepth || j.batch > 65535 || (j.A.ld & 31) || (j.B.ld & 31) || j.A.ld < j.Kd || j.B.ld < j.Kd)
    return B200Q_ERR_ARG;
  if (count_rows(j, kTile) <= 0 || j.N <= 0) return B200Q_OK;
  Params p;
  p.j = j;
  const int ctas = j.max_ctas > 0 && j.max_ctas < kNumSMs ? j.max_ctas : kNumSMs;
  const int resident = pair_capacity(), pairs = ctas / 2 < resident ? ctas / 2 : resident;
  pick_tiles(p, ctas, pairs);
  p.row_tiles = count_rows(j, p.tm_rows);
  const bool pair = p.tm_rows == 2 * kTile;
  const int64_t per_problem = count_tiles(j, p.tm_rows, p.tn_log2);
  p.num_tiles = per_problem * j.batch;
  if (p.num_tiles <= 0) return B200Q_OK;
  const int most = pair ? pairs : ctas;
  const int units = (int)(p.num_tiles < most ? p.num_tiles : most);
  // where each CTA's (pair's) range starts: problem, row tile, column tile
  // (without divisions: two of 64 bits for each of 148 took longer than the launch itself)
  const int64_t share = p.num_tiles / units, rest = p.num_tiles % units;
  int tm = 0, n = col_tiles(j, 0, p.tm_rows, p.tn_log2);
  int64_t in = 0, before = 0, part = 0, b = 0;   // tile i * num_tiles / units of problem b, tiles before row tile tm
  for (int i = 0; i < units; ++i) {
    while (in >= per_problem) { in -= per_problem; ++b; tm = 0; before = 0; n = col_tiles(j, 0, p.tm_rows, p.tn_log2); }
    while (in >= before + n) { before += n; n = col_tiles(j, ++tm, p.tm_rows, p.tn_log2); }
    p.start[i][0] = (uint16_t)b; p.start[i][1] = (uint16_t)tm; p.start[i][2] = (uint16_t)(in - before);
    in += share;
    if ((part += rest) >= units) { part -= units; ++in; }
  }
  const bool split_out = j.out_hi || j.X;
#define B200Q_TILES(TN, PAIR)                                                                             \
  (f16 ? launch_tiles<TN, false, PAIR, true>(p, units, st)                                                \
       : split_out ? launch_tiles<TN, true, PAIR, false>(p, units, st) : launch_tiles<TN, false, PAIR, false>(p, units, st))
  if (pair) return B200Q_TILES(256, true);
  if (p.tn_log2 == 8) return B200Q_TILES(256, false);
  if (p.tn_log2 == 7) return B200Q_TILES(128, false);
  return B200Q_TILES(64, false);
#undef B200Q_TILES
}

SideStream* side_stream(cudaStream_t like) {
  // one helper per (device, caller stream), kept for the life of the process: host threads come
  // and go, the streams they launch on do not
  struct Entry { int device; cudaStream_t like; SideStream s; };
  constexpr int kMax = 64;
  static Entry entries[kMax];
  static int used = 0;
  static std::mutex mu;
  int dev = 0, prio = 0;
  static const bool enabled = [] { const char* e = getenv("B200Q_LOOKAHEAD"); return !(e && e[0] == '0'); }();
  if (!enabled) return nullptr;
  if (cudaGetDevice(&dev) != cudaSuccess) return nullptr;
  std::lock_guard<std::mutex> lock(mu);
  for (int i = 0; i < used; ++i)
    if (entries[i].device == dev && entries[i].like == like) return &entries[i].s;
  if (used == kMax) return nullptr;
  if (cudaStreamGetPriority(like, &prio) != cudaSuccess) { (void)cudaGetLastError(); prio = 0; }
  Entry& e = entries[used];
  e.device = dev; e.like = like;
  if (cudaStreamCreateWithPriority(&e.s.stream, cudaStreamNonBlocking, prio) != cudaSuccess ||
      cudaEventCreateWithFlags(&e.s.ready, cudaEventDisableTiming) != cudaSuccess ||
      cudaEventCreateWithFlags(&e.s.next, cudaEventDisableTiming) != cudaSuccess ||
      cudaEventCreateWithFlags(&e.s.done, cudaEventDisableTiming) != cudaSuccess) {
    (void)cudaGetLastError();
    return nullptr;
  }
  ++used;
  return &e.s;
}

}  // namespace tgemm
}  // namespace b200q
