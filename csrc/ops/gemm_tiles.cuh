// The bf16 GEMM of the model operators: D[M, N] = A[M, K] * B[N, K]^T on tcgen05, one persistent kernel template.
//
// Two shapes of tile:
//   one CTA    128 x BN (BN 64, 128 or 192): cta_group::1; every SM works alone, no cluster launch, no cluster barriers
//   CTA pair   256 x 256: cta_group::2; each CTA loads its 128 rows of A and half of the B tile and the even CTA issues
//              the MMAs for both, so a 128 x 256 block costs 32 KB of operands per 64 of K instead of 48
//
// What bounds it, from probes that ran loads and MMAs apart and together (148 SMs, operands in L2):
//   * L2 to shared memory is not the limit: 90 B / clk / SM for every SM at once (over 20 TB/s).
//   * Issue is.  Under `lane == 0` a k-block (two loads, four MMAs, a commit, two waits) took 608 clocks whatever the
//     tile; under elect.sync 430-515.  Hence elect_one() around the two role loops, and stage and phase counters
//     instead of divisions.
//   * Then the TMA unit: about 105 B / clk / SM and 50 clocks per load, so the 32 KB of a 128 x 128 k-block take 342
//     clocks (measured, at its bound) where its MMAs need 256.  Six stages of 64 of K do better than three of 128
//     (4096 x 512 x 2048: 11.8 -> 11.2 us): a stage is refilled sooner.
//   * A tile's epilogue was 1.8 us for 64 columns per warp, 3.6 us with a residual: instruction fetch and exposed
//     global loads.  Extra inputs with the layout of the output (residual, multiplier) are therefore fetched by TMA into
//     the staging buffer the result will leave from, before the accumulator is awaited; bias is fetched then too, four
//     values per lane, and spread by shuffles (read where it is used, even from L1, it cost 0.9 us); and a trip of the
//     epilogue loop is 32 columns.
//
//   warp 0        producer: one elected thread issues the TMA loads
//   warp 1        MMA issuer (even CTA of a pair), tensor-memory allocation
//   warps 2..     epilogue, one per tensor-memory lane quarter and 64 columns; the accumulator is double buffered
//
// No load uses cluster multicast.  Every wait is bounded (two seconds); a wait that runs out sets the error word the
// host checks, the roles leave their loops, and the CTAs of a pair still meet before tensor memory is freed.
#pragma once

#include "gemm_common.cuh"

#include "../core/launch.hpp"

#include <atomic>
#include <type_traits>

namespace mccl {
namespace ops {
namespace tiles {

// OUT_BF16_SCALED, OUT_F32_SCALED: times the scalar at GemmDev::alpha (the upstream gradient of a loss).  Instantiations of their own: the
// multiplications in the other epilogues, even where they were skipped, cost 2 us of a 134 us training step (instruction
// fetch, and fewer loads in flight).
// OUT_F32_SLABS: every part of K into a slab of its own (GemmDev::slab_rows rows further down in D), for a reader that adds the slabs in
// order.  Partial sums that are added in memory arrive in any order, and a forward pass or an input gradient that went that way
// no longer repeated bit for bit.
// OUT_BF16_SUM: the bf16 output and, added into GemmDev::colsum, its column sums (a bias gradient).
// OUT_BF16_PARTS: the sums of every 32 rows are written to a row of their own instead, for finish_sums or sum_parts.
// OUT_SWIGLU (pair tile only): B is [gate | up], 2 n rows; the even CTA brings 128 rows of gate and the odd one the same 128 of up,
// so that a tile's accumulator holds both factors of 128 outputs and silu(gate) * up is the epilogue.  The [m, 2 n] product
// itself, which backward reads, is written too where `aux` is given.  As a kernel of its own the activation read it back:
// 1537 x 16384 x 2048 (no aux) 86 + 17.6 us against 86, 4096 x 8192 x 1024 53 + 22 us against 54.
// OUT_SWIGLU_GRAD (pair tile only): the input gradient of the product behind the activation, turned into the gradient of
// [gate | up] (D, [m, 2 n]) with the saved [gate | up] (`aux`) on its way out; the [m, n] tensor between the two is neither
// written nor read.
enum Out : int { OUT_BF16 = 0, OUT_GELU = 1, OUT_F32 = 2, OUT_BF16_SUM = 3, OUT_SWIGLU = 4, OUT_SWIGLU_GRAD = 5, OUT_BF16_SCALED = 6, OUT_F32_SCALED = 7, OUT_F32_SLABS = 8, OUT_BF16_PARTS = 9 };
constexpr bool fp32_out(int out) { return out == OUT_F32 || out == OUT_F32_SCALED || out == OUT_F32_SLABS; }
constexpr bool half_boxes(int out) { return out == OUT_GELU || out == OUT_SWIGLU || out == OUT_SWIGLU_GRAD; }   // 32-column output boxes

// One product, or several with the same K whose tiles one launch works through (the weight gradients of one or more layers:
// alone, a 512 x 2048 gradient is 64 tiles and leaves half the SMs without one).
constexpr int kMaxGroup = 16;
struct NoSums {};
struct WithSums {
  PartSums sums;   // finished by the epilogue warps while the first tile's main loop runs
};
template <int kMax>
struct Problems : std::conditional_t<(kMax > 1), WithSums, NoSums> {
  CUtensorMap a[kMax], b[kMax], d[kMax];
  CUtensorMap x;              // the second output of the GELU instantiation, or the extra input of the bf16 ones
  int m[kMax], n[kMax];
  int first[kMax + 1];        // first tile of each product
  int n_tiles[kMax];
  int atoms[kMax];            // bit 0 / 1: the MN-major A / B has whole groups of 64 columns and is fetched by one load
  int count;
};

template <int BN, bool kPair, bool kGelu = false>
struct Shape {
  static constexpr int kStages = kPair ? 5 : (BN == 64 ? 8 : (BN == 192 ? 4 : (kGelu ? 5 : 6)));
  static constexpr int kRowsB = kPair ? BN / 2 : BN;   // rows of the B tile this CTA loads
  static constexpr int kABytes = BM * BK * 2;
  static constexpr int kBBytes = kRowsB * BK * 2;
  static constexpr int kStageBytes = kABytes + kBBytes;
  // GELU: 11 instructions per value and two of them long; twice the warps, half the columns each, so that more chains are in
  // flight per scheduler, and a staging buffer per output
  static constexpr int kEpiWarps = BN / 16 * (kGelu ? 2 : 1);   // 64 (GELU: 32) accumulator columns each
  static constexpr int kThreads = 64 + 32 * kEpiWarps;
  static constexpr int kCols = BN / (kEpiWarps / 4);
  static constexpr int kTiles = kStages * kStageBytes;
  static constexpr int kStagingOff = kTiles;
  static constexpr int kBarOff = kStagingOff + kEpiWarps * 4096;
  static constexpr int kTmem = BN > 128 ? 512 : 4 * BN / 2;       // two accumulators; allocations are powers of two
  static constexpr int kBarriers = 2 * kStages + 4 + kEpiWarps;
  static constexpr int kTotal = kBarOff + kBarriers * 8 + 16 + 1024;
  static_assert(kTotal <= 227 * 1024, "shared memory of one CTA");
};

__device__ __forceinline__ unsigned long long now_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
static __device__ __noinline__ bool wait_slow(uint64_t* bar, uint32_t parity, volatile int* abort_flag) {
  const unsigned long long t0 = now_ns();
  for (uint32_t i = 0;; ++i) {
    if (tc::mbar_try_wait(bar, parity)) return true;
    if ((i & 255u) == 255u) {
      if (*abort_flag) return false;
      if (now_ns() - t0 > 2000000000ull) return false;
    }
  }
}
__device__ __forceinline__ bool wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag) {
  if (tc::mbar_try_wait(bar, parity)) return true;
  return wait_slow(bar, parity, abort_flag);
}

__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
// Address, in the cluster's shared window, of the even CTA's copy of a shared-memory object of this CTA.
__device__ __forceinline__ uint32_t leader_addr(const void* p) {
  uint32_t a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(tc::smem_u32(p)), "r"(0));
  return a;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// The bytes land in this CTA's shared memory and complete on a barrier of the cluster window (the even CTA's).
__device__ __forceinline__ void load_2d_pair(void* dst, const CUtensorMap* map, uint32_t bar_cluster_addr, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(tc::smem_u32(dst)), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar_cluster_addr), "r"(x), "r"(y)
      : "memory");
}
// All 64-column groups of an MN-major tile at once: the matrix [K, MN] seen as [MN / 64][K][64].
__device__ __forceinline__ void load_groups(void* dst, const CUtensorMap* map, uint64_t* bar, int group, int k) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
      ::"r"(tc::smem_u32(dst)), "l"(reinterpret_cast<uint64_t>(map)), "r"(tc::smem_u32(bar)), "r"(0), "r"(k), "r"(group)
      : "memory");
}
__device__ __forceinline__ void load_groups_pair(void* dst, const CUtensorMap* map, uint32_t bar_cluster_addr, int group, int k) {
  asm volatile(
      "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
      ::"r"(tc::smem_u32(dst)), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar_cluster_addr), "r"(0), "r"(k), "r"(group)
      : "memory");
}
__device__ __forceinline__ void mma_pair(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc, bool accumulate) {
  uint32_t acc = accumulate ? 1u : 0u;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(acc)
      : "memory");
}
// Arrives on the barrier at this offset in BOTH CTAs once every MMA issued so far has finished (an mbarrier arrive, not a load).
__device__ __forceinline__ void commit_pair(uint64_t* bar) {
  const uint16_t mask = 3;
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
               ::"r"(tc::smem_u32(bar)), "h"(mask)
               : "memory");
}
__device__ __forceinline__ void arrive_cluster(uint32_t bar_cluster_addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar_cluster_addr) : "memory");
}
__device__ __forceinline__ void store_2d(const CUtensorMap* map, const void* src, int x, int y) {
  asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];"
               ::"l"(reinterpret_cast<uint64_t>(map)), "r"(tc::smem_u32(src)), "r"(x), "r"(y)
               : "memory");
}
__device__ __forceinline__ void reduce_add_2d(const CUtensorMap* map, const void* src, int x, int y) {
  asm volatile("cp.reduce.async.bulk.tensor.2d.global.shared::cta.add.tile.bulk_group [%0, {%2, %3}], [%1];"
               ::"l"(reinterpret_cast<uint64_t>(map)), "r"(tc::smem_u32(src)), "r"(x), "r"(y)
               : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
// All but the last N groups committed by this thread have read their shared-memory source.
template <int N>
__device__ __forceinline__ void bulk_wait_read() {
  asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(N) : "memory");
}
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
// Sums that kernels before this one left in parts (bias and norm gradients), by the W epilogue warps of each CTA: 32 columns at a time,
// rows dealt out to the warps with eight in flight, the warps' shares added in order.  A launch of its own for them is 4 us per layer
// (70M training loop 3870 -> 3941 us); here nobody waits for it (3868).
template <int W>
__device__ __forceinline__ void finish_sums(const PartSums& p, float* red, int warp, int lane) {
  const int groups = p.first[p.count];
  for (int q = blockIdx.x; q < groups; q += gridDim.x) {
    int i = 0;
    while (i + 1 < p.count && q >= p.first[i + 1]) ++i;
    const float* in = p.s[i].in;
    const int rows = p.s[i].rows, cols = p.s[i].cols, c = (q - p.first[i]) * 32 + lane;
    float t = 0.f;
    if (c < cols)
      for (int r0 = warp; r0 < rows; r0 += 8 * W) {
        float v[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) v[k] = r0 + W * k < rows ? __ldcg(in + static_cast<size_t>(r0 + W * k) * cols + c) : 0.f;
#pragma unroll
        for (int k = 0; k < 8; ++k) t += v[k];
      }
    red[warp * 32 + lane] = t;
    asm volatile("bar.sync 1, %0;" ::"n"(W * 32) : "memory");
    if (warp == 0 && c < cols) {
      for (int w = 1; w < W; ++w) t += red[w * 32 + lane];
      p.s[i].out[c] = t;
    }
    asm volatile("bar.sync 1, %0;" ::"n"(W * 32) : "memory");
  }
}

template <int BN, bool kPair, bool kAMn, bool kBMn, int kOut, int kMax>
__global__ void __launch_bounds__(Shape<BN, kPair, kOut == OUT_GELU>::kThreads, 1)
gemm_tile_kernel(const __grid_constant__ Problems<kMax> P, GemmDev g, int splits) {
  constexpr bool kSum = kOut == OUT_BF16_SUM || kOut == OUT_BF16_PARTS, kBf16 = kOut == OUT_BF16 || kSum, kF32 = fp32_out(kOut), kScaled = kOut == OUT_BF16_SCALED || kOut == OUT_F32_SCALED;
  using S = Shape<BN, kPair, kOut == OUT_GELU>;
  constexpr int kStages = S::kStages, kTileM = kPair ? 2 * BM : BM;
  constexpr bool kGated = kOut == OUT_SWIGLU;
  static_assert(!kGated || (kPair && !kBMn && kMax == 1), "gate and up come by one CTA each");
  constexpr int kTileN = kGated ? BN / 2 : BN, kCols = kGated ? S::kCols / 2 : S::kCols;   // output columns of a tile, of an epilogue warp
  extern __shared__ uint8_t smem_raw[];
  // the same offset in both CTAs of a pair: the MMA addresses the peer's operands by this CTA's offsets
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + S::kBarOff);
  uint64_t* empty = full + kStages;
  uint64_t* acc_full = empty + kStages;   // [2]
  uint64_t* acc_empty = acc_full + 2;     // [2]
  uint64_t* extra_full = acc_empty + 2;   // [epilogue warp][buffer]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(extra_full + S::kEpiWarps);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const unsigned long long tl_t0 = tl_begin(g.tl);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = kPair ? cluster_ctarank() : 0u;
  const int worker = static_cast<int>(kPair ? blockIdx.x >> 1 : blockIdx.x), workers = static_cast<int>(kPair ? gridDim.x >> 1 : gridDim.x);
  const int all_kb = (g.k + BK - 1) / BK;
  // splits >= 1: work items are (tile, part of K), taken in turn.  splits == 0: every worker gets an equal run of k-blocks,
  // across tile borders, and adds what it has of each tile into D.
  const int tiles = P.first[P.count];
  const bool runs = kF32 && kOut != OUT_F32_SLABS && splits == 0;
  const int work_begin = runs ? static_cast<int>(static_cast<long long>(tiles) * all_kb * worker / workers) : worker;
  const int work_end = runs ? static_cast<int>(static_cast<long long>(tiles) * all_kb * (worker + 1) / workers) : tiles * splits;

  if (warp == 0 && tc::elect_one()) {
    for (int s = 0; s < kStages; ++s) {
      tc::mbar_init(&full[s], 1);     // the (even CTA's) producer arrives once and expects the bytes of every load
      tc::mbar_init(&empty[s], 1);    // one commit per use
    }
    for (int b = 0; b < 2; ++b) {
      tc::mbar_init(&acc_full[b], 1);
      tc::mbar_init(&acc_empty[b], (kPair ? 2 : 1) * S::kEpiWarps);
    }
    for (int b = 0; b < S::kEpiWarps; ++b) tc::mbar_init(&extra_full[b], 1);
    *abort_flag = 0;
    tc::mbar_init_fence();
    for (int p = 0; p < P.count; ++p) {
      tc::tma_prefetch_desc(&P.a[p]);
      tc::tma_prefetch_desc(&P.b[p]);
      tc::tma_prefetch_desc(&P.d[p]);
    }
    if (kMax == 1) tc::tma_prefetch_desc(&P.x);
  }
  if (warp == 1) {
    if constexpr (kPair) {
      asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tc::smem_u32(tmem_slot)), "r"(S::kTmem) : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    } else {
      tc::tmem_alloc(tmem_slot, S::kTmem);
    }
  }
  tc::fence_before_sync();
  __syncthreads();
  // the peer's barriers exist and its tensor memory is allocated before anything is sent its way
  if constexpr (kPair) cluster_sync_all();
  tc::fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  pdl_wait();   // set-up done: from here on operands are read and outputs written
  if (tl_t0 != 0ull && tl_detail(g.tl)) tl_mark(g.tl, tl_t0, tl_now(), TL_GEMM_PHASE, 0u);

  // product, tile row, tile column and range of k-blocks of the work item at w, and where the next one is
  struct Item {
    int p, m_blk, n_blk, kb0, kb1, next, piece;
  };
  auto item = [&](int w) {
    Item it;
    int t;
    if (runs) {
      t = w / all_kb;
      it.kb0 = w - t * all_kb;
      it.kb1 = work_end - w < all_kb - it.kb0 ? it.kb0 + work_end - w : all_kb;
      it.next = w + it.kb1 - it.kb0;
      it.piece = 0;
    } else {
      t = splits > 1 ? w / splits : w;
      const int s = w - t * splits;
      it.kb0 = splits > 1 ? all_kb * s / splits : 0;
      it.kb1 = splits > 1 ? all_kb * (s + 1) / splits : all_kb;
      it.next = w + workers;
      it.piece = s;
    }
    it.p = 0;
    if constexpr (kMax > 1) {
      while (it.p + 1 < P.count && t >= P.first[it.p + 1]) ++it.p;
      t -= P.first[it.p];
    }
    it.m_blk = t / P.n_tiles[it.p];
    it.n_blk = t - it.m_blk * P.n_tiles[it.p];
    return it;
  };

  if (warp == 0) {
    // ------------------------------------------------------ TMA producer --
    if (tc::elect_one()) {
      bool ok = true;
      int s = 0;
      uint32_t parity = 1;   // a fresh barrier counts as the phase before the first: the first round does not wait
      for (int w = work_begin; w < work_end && ok;) {
        const Item it = item(w);
        w = it.next;
        const CUtensorMap* map_a = &P.a[it.p];
        const CUtensorMap* map_b = &P.b[it.p];
        const int a_row = it.m_blk * kTileM + static_cast<int>(rank) * BM;
        const int b_row = it.n_blk * kTileN + static_cast<int>(rank) * (kGated ? P.n[it.p] : S::kRowsB);
        for (int kb = it.kb0; kb < it.kb1; ++kb) {
          ok = wait(&empty[s], parity, abort_flag);
          if (!ok) break;
          uint8_t* a_dst = smem + s * S::kStageBytes;
          uint8_t* b_dst = a_dst + S::kABytes;
          const int k0 = kb * BK;
          if constexpr (kPair) {
            if (rank == 0) tc::mbar_expect_tx(&full[s], 2 * S::kStageBytes);
            const uint32_t bar = leader_addr(&full[s]);
            if (kAMn && (P.atoms[it.p] & 1)) {
              load_groups_pair(a_dst, map_a, bar, a_row / 64, k0);
            } else if (kAMn) {
#pragma unroll
              for (int q = 0; q < BM / 64; ++q) load_2d_pair(a_dst + q * (BK * 128), map_a, bar, a_row + q * 64, k0);
            } else {
              load_2d_pair(a_dst, map_a, bar, k0, a_row);
            }
            if (kBMn && (P.atoms[it.p] & 2)) {
              load_groups_pair(b_dst, map_b, bar, b_row / 64, k0);
            } else if (kBMn) {
#pragma unroll
              for (int q = 0; q < S::kRowsB / 64; ++q) load_2d_pair(b_dst + q * (BK * 128), map_b, bar, b_row + q * 64, k0);
            } else {
              load_2d_pair(b_dst, map_b, bar, k0, b_row);
            }
          } else {
            tc::mbar_expect_tx(&full[s], S::kStageBytes);
            if (kAMn && (P.atoms[it.p] & 1)) {
              load_groups(a_dst, map_a, &full[s], a_row / 64, k0);
            } else if (kAMn) {
#pragma unroll
              for (int q = 0; q < BM / 64; ++q) tc::tma_load_2d(a_dst + q * (BK * 128), map_a, &full[s], a_row + q * 64, k0);
            } else {
              tc::tma_load_2d(a_dst, map_a, &full[s], k0, a_row);
            }
            if (kBMn && (P.atoms[it.p] & 2)) {
              load_groups(b_dst, map_b, &full[s], b_row / 64, k0);
            } else if (kBMn) {
#pragma unroll
              for (int q = 0; q < S::kRowsB / 64; ++q) tc::tma_load_2d(b_dst + q * (BK * 128), map_b, &full[s], b_row + q * 64, k0);
            } else {
              tc::tma_load_2d(b_dst, map_b, &full[s], k0, b_row);
            }
          }
          if (++s == kStages) {
            s = 0;
            parity ^= 1u;
          }
        }
      }
      pdl_trigger();   // the last loads are on their way: the next kernel may set up beside this one's tail
      if (!ok) {
        *abort_flag = 1;
        atomicExch(g.err, 11);
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // -------------------------------------------------------- MMA issuer --
    if (rank == 0 && tc::elect_one()) {
      constexpr uint32_t idesc = tc::idesc_bf16(kTileM, BN, kAMn, kBMn);
      // 16 of K further: 32 bytes within a swizzled row, or 16 rows of 128 bytes
      constexpr uint64_t a_step = kAMn ? 128 : 2, b_step = kBMn ? 128 : 2;
      bool ok = true;
      int s = 0, i = 0;
      uint32_t parity = 0;
      for (int w = work_begin; w < work_end; ++i) {
        const Item it = item(w);
        w = it.next;
        const int kb0 = it.kb0, kb1 = it.kb1, buf = i & 1;
        if (i >= 2) {
          ok = wait(&acc_empty[buf], ((i >> 1) - 1) & 1, abort_flag);
          if (!ok) break;
          tc::fence_after_sync();
        }
        const uint32_t tmem_d = tmem_base + static_cast<uint32_t>(buf * (S::kTmem / 2));
        for (int kb = kb0; kb < kb1; ++kb) {
          ok = wait(&full[s], parity, abort_flag);
          if (!ok) break;
          tc::fence_after_sync();
          const uint8_t* a_tile = smem + s * S::kStageBytes;
          const uint64_t da = kAMn ? tc::smem_desc_mn_sw128(a_tile, BK * 128) : tc::smem_desc_k_sw128(a_tile);
          const uint64_t db = kBMn ? tc::smem_desc_mn_sw128(a_tile + S::kABytes, BK * 128) : tc::smem_desc_k_sw128(a_tile + S::kABytes);
#pragma unroll
          for (int q = 0; q < BK / UMMA_K; ++q) {
            if constexpr (kPair) mma_pair(tmem_d, da + a_step * q, db + b_step * q, idesc, q > 0 || kb != kb0);
            else tc::mma_bf16(tmem_d, da + a_step * q, db + b_step * q, idesc, q > 0 || kb != kb0);
          }
          if constexpr (kPair) commit_pair(&empty[s]);
          else tc::mma_commit(&empty[s]);
          if (++s == kStages) {
            s = 0;
            parity ^= 1u;
          }
        }
        if (!ok) break;
        if constexpr (kPair) commit_pair(&acc_full[buf]);
        else tc::mma_commit(&acc_full[buf]);
      }
      if (!ok) {
        *abort_flag = 1;
        atomicExch(g.err, 12);
      }
    }
    __syncwarp();
  } else {
    // ----------------------------------------------------------- epilogue --
    const int e = warp - 2, quarter = warp & 3, part = e >> 2;
    uint8_t* stage = smem + S::kStagingOff + e * 4096;
    uint64_t* xfull = extra_full + e;
    const bool has_bias = !kF32 && !kScaled && (g.epilogue == EPI_BIAS || g.epilogue == EPI_BIAS_GELU || g.epilogue == EPI_BIAS_GELU_D);
    const bool has_extra = kBf16 && (g.mul != nullptr || g.residual != nullptr);
    const bool multiply = g.mul != nullptr;
    const bool gelu_d = g.epilogue == EPI_BIAS_GELU_D || g.epilogue == EPI_GELU_D;
    bool ok = true;
    int i = 0;
    uint32_t xparity = 0;
    if constexpr (kMax > 1) finish_sums<S::kEpiWarps>(P.sums, reinterpret_cast<float*>(smem + S::kStagingOff), e, lane);
    float alpha = 1.f;
    if constexpr (kScaled) alpha = __ldg(g.alpha);
    for (int w = work_begin; w < work_end; ++i) {
      const Item it = item(w);
      w = it.next;
      const CUtensorMap* map_d = &P.d[it.p];
      const int m = P.m[it.p], n = P.n[it.p];
      const int buf = i & 1;
      const bool stamp = warp == 2 && lane == 0 && tl_detail(g.tl);
      const unsigned long long ts0 = stamp ? tl_now() : 0ull;
      const int col0 = it.n_blk * kTileN + part * kCols;
      const int row0 = it.m_blk * kTileM + static_cast<int>(rank) * BM + quarter * 32;
      const bool inside = row0 < m && col0 < n;   // uniform over the warp
      auto load_gate_up = [&](int col) {
        tc::mbar_expect_tx(xfull, 4096);
        tc::tma_load_2d(stage, &P.x, xfull, col, row0);
        tc::tma_load_2d(stage + 2048, &P.x, xfull, n + col, row0);
      };
      // the staging buffers are free again; fetch what the epilogue will need while the MMAs of the tile still run
      if (tc::elect_one()) {
        bulk_wait_read<0>();
        if (has_extra && inside) {
          tc::mbar_expect_tx(xfull, 4096);
          tc::tma_load_2d(stage, &P.x, xfull, col0, row0);
        }
        if (kOut == OUT_SWIGLU_GRAD && inside) load_gate_up(col0);
      }
      // lane l keeps the bias of columns [col0 + 4 l, col0 + 4 l + 4); the loop below spreads it by shuffles
      float4 bias4 = make_float4(0.f, 0.f, 0.f, 0.f);
      if (has_bias && 4 * lane < S::kCols && col0 + 4 * lane < n) bias4 = __ldg(reinterpret_cast<const float4*>(g.bias + col0 + 4 * lane));
      __syncwarp();
      ok = wait(&acc_full[buf], (i >> 1) & 1, abort_flag);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tc::fence_after_sync();
      const unsigned long long ts1 = stamp ? tl_now() : 0ull;
      const uint32_t taddr = tmem_base + static_cast<uint32_t>(buf * (S::kTmem / 2) + part * kCols) + (static_cast<uint32_t>(quarter * 32) << 16);
      auto last_read = [&]() {
        // every column of this warp's part is in registers: hand the buffer back to the MMA thread
        tc::fence_before_sync();
        if (lane == 0) {
          if constexpr (kPair) arrive_cluster(leader_addr(&acc_empty[buf]));
          else tc::mbar_arrive(&acc_empty[buf]);
        }
      };
      if constexpr (kF32) {
        [[maybe_unused]] const bool add = g.atomic_add || g.accumulate;
#pragma unroll 1
        for (int c = 0; c < S::kCols; c += 32) {
          uint32_t r[32];
          tc::tmem_ld_32x32(taddr + static_cast<uint32_t>(c), r);
          tc::tmem_ld_wait();
          if (c + 32 >= S::kCols) last_read();
          if (row0 >= m || col0 + c >= n) continue;
          if (tc::elect_one()) bulk_wait_read<0>();
          __syncwarp();
          if constexpr (kScaled) {
#pragma unroll
            for (int j = 0; j < 32; ++j) r[j] = __float_as_uint(__uint_as_float(r[j]) * alpha);
          }
#pragma unroll
          for (int j = 0; j < 8; ++j) *stage_unit(stage, lane, j) = make_uint4(r[4 * j], r[4 * j + 1], r[4 * j + 2], r[4 * j + 3]);
          fence_async_smem();
          __syncwarp();
          if (tc::elect_one()) {
            if constexpr (kOut == OUT_F32_SLABS) store_2d(map_d, stage, col0 + c, it.piece * g.slab_rows + row0);
            else if (add) reduce_add_2d(map_d, stage, col0 + c, row0);
            else store_2d(map_d, stage, col0 + c, row0);
            bulk_commit();
          }
          __syncwarp();
        }
      } else if constexpr (kOut == OUT_GELU) {
        uint32_t r[32];
        tc::tmem_ld_32x32(taddr, r);
        tc::tmem_ld_wait();
        last_read();
        if (inside) {
          uint8_t* stage2 = stage + 2048;
          const bool second = g.aux != nullptr;
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            float v[8], dv[8];
#pragma unroll
            for (int q = 0; q < 8; ++q) v[q] = __uint_as_float(r[j * 8 + q]);
            if (has_bias) {
              v[0] += __shfl_sync(0xffffffffu, bias4.x, 2 * j);
              v[1] += __shfl_sync(0xffffffffu, bias4.y, 2 * j);
              v[2] += __shfl_sync(0xffffffffu, bias4.z, 2 * j);
              v[3] += __shfl_sync(0xffffffffu, bias4.w, 2 * j);
              v[4] += __shfl_sync(0xffffffffu, bias4.x, 2 * j + 1);
              v[5] += __shfl_sync(0xffffffffu, bias4.y, 2 * j + 1);
              v[6] += __shfl_sync(0xffffffffu, bias4.z, 2 * j + 1);
              v[7] += __shfl_sync(0xffffffffu, bias4.w, 2 * j + 1);
            }
            if (!gelu_d && second) *stage_unit64(stage2, lane, j) = pack8(v);
            // value and derivative share one exponential; the derivative is what backward needs, so it is saved instead of z
#pragma unroll
            for (int q = 0; q < 8; q += 2) gelu_two<true>(v[q], v[q + 1], dv[q], dv[q + 1]);
            *stage_unit64(stage, lane, j) = pack8(v);
            if (gelu_d && second) *stage_unit64(stage2, lane, j) = pack8(dv);
          }
          fence_async_smem();
          __syncwarp();
          if (tc::elect_one()) {
            store_2d(map_d, stage, col0, row0);
            if (second) store_2d(&P.x, stage2, col0, row0);
            bulk_commit();
          }
          __syncwarp();
        }
      } else if constexpr (kGated) {
        uint32_t rg[32], ru[32];
        tc::tmem_ld_32x32(taddr, rg);
        tc::tmem_ld_32x32(taddr + static_cast<uint32_t>(BN / 2), ru);
        tc::tmem_ld_wait();
        last_read();
        if (inside) {
          const bool both = g.aux != nullptr;
          uint4 h[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            float gate[8], up[8];
#pragma unroll
            for (int q = 0; q < 8; ++q) gate[q] = __uint_as_float(rg[j * 8 + q]), up[q] = __uint_as_float(ru[j * 8 + q]);
            const uint4 pg = pack8(gate), pu = pack8(up);
            if (both) {
              *stage_unit64(stage, lane, j) = pg;
              *stage_unit64(stage + 2048, lane, j) = pu;
            }
            // rounded where a product and an activation of their own would round
            unpack8(pg, gate);
            unpack8(pu, up);
#pragma unroll
            for (int q = 0; q < 8; ++q) gate[q] = __bfloat162float(__float2bfloat16_rn(__fdividef(gate[q], 1.f + __expf(-gate[q])))) * up[q];
            h[j] = pack8(gate);
          }
          if (both) {
            fence_async_smem();
            __syncwarp();
            if (tc::elect_one()) {
              store_2d(&P.x, stage, col0, row0);
              store_2d(&P.x, stage + 2048, n + col0, row0);
              bulk_commit();
              bulk_wait_read<0>();
            }
            __syncwarp();
          }
#pragma unroll
          for (int j = 0; j < 4; ++j) *stage_unit64(stage, lane, j) = h[j];
          fence_async_smem();
          __syncwarp();
          if (tc::elect_one()) {
            store_2d(map_d, stage, col0, row0);
            bulk_commit();
          }
          __syncwarp();
        }
      } else if constexpr (kOut == OUT_SWIGLU_GRAD) {
#pragma unroll 1
        for (int c = 0; c < S::kCols; c += 32) {   // gate and up of 32 columns fill the staging buffer
          const int col = col0 + c;
          const bool here = row0 < m && col < n;
          if (here) {
            if (c > 0) {
              if (tc::elect_one()) {
                bulk_wait_read<0>();
                load_gate_up(col);
              }
              __syncwarp();
            }
            ok = wait(xfull, xparity, abort_flag);
            ok = __all_sync(0xffffffffu, ok);
            xparity ^= 1u;
            if (!ok) break;
          }
          uint32_t r[32];
          tc::tmem_ld_32x32(taddr + static_cast<uint32_t>(c), r);
          tc::tmem_ld_wait();
          if (c + 32 >= S::kCols) last_read();
          if (!here) continue;
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            float d[8], gate[8], up[8];
#pragma unroll
            for (int q = 0; q < 8; ++q) d[q] = __uint_as_float(r[j * 8 + q]);
            unpack8(pack8(d), d);   // rounded where a product of its own would round
            unpack8(*stage_unit64(stage, lane, j), gate);
            unpack8(*stage_unit64(stage + 2048, lane, j), up);
#pragma unroll
            for (int q = 0; q < 8; ++q) {
              const float s = __fdividef(1.f, 1.f + __expf(-gate[q]));
              const float dg = d[q] * up[q] * s * (1.f + gate[q] * (1.f - s));
              up[q] = d[q] * gate[q] * s;
              gate[q] = dg;
            }
            *stage_unit64(stage, lane, j) = pack8(gate);
            *stage_unit64(stage + 2048, lane, j) = pack8(up);
          }
          fence_async_smem();
          __syncwarp();
          if (tc::elect_one()) {
            store_2d(map_d, stage, col, row0);
            store_2d(map_d, stage + 2048, n + col, row0);
            bulk_commit();
          }
          __syncwarp();
        }
        if (!ok) break;
      } else {
        if (has_extra && inside) {
          ok = wait(xfull, xparity, abort_flag);
          ok = __all_sync(0xffffffffu, ok);
          xparity ^= 1u;
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          uint32_t r[32];
          tc::tmem_ld_32x32(taddr + static_cast<uint32_t>(32 * h), r);
          tc::tmem_ld_wait();
          if (h == 1) last_read();
          if (!inside) continue;
          [[maybe_unused]] float sums[32];
#pragma unroll
          for (int jj = 0; jj < 4; ++jj) {
            const int j = 4 * h + jj;
            float v[8];
#pragma unroll
            for (int q = 0; q < 8; ++q) v[q] = kScaled ? __uint_as_float(r[jj * 8 + q]) * alpha : __uint_as_float(r[jj * 8 + q]);
            if (has_bias) {
              const int src = 2 * j;
              v[0] += __shfl_sync(0xffffffffu, bias4.x, src);
              v[1] += __shfl_sync(0xffffffffu, bias4.y, src);
              v[2] += __shfl_sync(0xffffffffu, bias4.z, src);
              v[3] += __shfl_sync(0xffffffffu, bias4.w, src);
              v[4] += __shfl_sync(0xffffffffu, bias4.x, src + 1);
              v[5] += __shfl_sync(0xffffffffu, bias4.y, src + 1);
              v[6] += __shfl_sync(0xffffffffu, bias4.z, src + 1);
              v[7] += __shfl_sync(0xffffffffu, bias4.w, src + 1);
            }
            if (has_extra) {
              float x[8];
              unpack8(*stage_unit(stage, lane, j), x);
              if (multiply) {
#pragma unroll
                for (int q = 0; q < 8; ++q) v[q] *= x[q];
              } else {
#pragma unroll
                for (int q = 0; q < 8; ++q) v[q] += x[q];
              }
            }
            *stage_unit(stage, lane, j) = pack8(v);
            if constexpr (kSum) {
#pragma unroll
              for (int q = 0; q < 8; ++q) sums[jj * 8 + q] = v[q];
            }
          }
          if constexpr (kSum) {
            const float sum = column_sum32(sums, lane);   // over the warp's 32 rows
            if (col0 + 32 * h + lane < n) {
              if constexpr (kOut == OUT_BF16_PARTS) g.colsum[static_cast<size_t>(row0 >> 5) * n + col0 + 32 * h + lane] = sum;
              else atomicAdd(g.colsum + col0 + 32 * h + lane, sum);
            }
          }
        }
        if (inside) {
          fence_async_smem();
          __syncwarp();
          if (tc::elect_one()) {
            store_2d(map_d, stage, col0, row0);
            bulk_commit();
          }
          __syncwarp();
        }
        if (!ok) break;
      }
      if (stamp) {
        const unsigned long long ts2 = tl_now();   // before the records below: their atomics take a microsecond
        tl_mark(g.tl, ts0, ts1, TL_GEMM_PHASE, (1u << 24) | static_cast<uint32_t>(i));
        tl_mark(g.tl, ts1, ts2, TL_GEMM_PHASE, (2u << 24) | static_cast<uint32_t>(i));
      }
    }
    if (tc::elect_one()) bulk_wait_read<0>();   // the stores have read this warp's staging; kernel completion publishes them
    if (!ok && lane == 0) {
      *abort_flag = 1;
      atomicExch(g.err, 13);
    }
    __syncwarp();
  }
  tc::fence_before_sync();
  __syncthreads();
  if (*abort_flag) {
    // a wait ran out somewhere: loads still in flight get time to land before shared memory is given up
    const unsigned long long t0 = now_ns();
    while (now_ns() - t0 < 50000ull) __nanosleep(1000);
  }
  // nothing of the peer is touched after this: its shared memory (operands the MMAs read) and barriers (remote arrives)
  if constexpr (kPair) cluster_sync_all();
  if (warp == 1) {
    tc::fence_after_sync();
    if constexpr (kPair) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(S::kTmem) : "memory");
    else tc::tmem_dealloc(tmem_base, S::kTmem);
  }
  tl_end(g.tl, tl_t0, TL_GEMM, (static_cast<uint32_t>(tiles / P.n_tiles[0] * (kPair ? 2 : 1)) << 16) | static_cast<uint32_t>(P.n_tiles[0]));
}

// MN-major operand [K, cols] as [cols / 64][K][64], a box being `groups` groups x BK rows.  (A load costs the TMA unit 50 clocks
// and its bytes 80 per 8 KB: with one load per group an MN-major 256 x 256 k-block took 650-730 clocks against 515.)
inline bool encode_groups(CUtensorMap* map, const void* base, int k, int cols, int ld_elems, int groups) {
  const CuDriver& cu = CuDriver::get();
  if (!cu.loaded || !cu.TensorMapEncodeTiled) return false;
  int device = 0;
  cudaGetDevice(&device);
  cu.ensure_context(device);
  cuuint64_t dims[3] = {64, static_cast<cuuint64_t>(k), static_cast<cuuint64_t>(cols / 64)};
  cuuint64_t strides[2] = {static_cast<cuuint64_t>(ld_elems) * 2, 128};
  cuuint32_t box[3] = {64, static_cast<cuuint32_t>(BK), static_cast<cuuint32_t>(groups)};
  cuuint32_t estr[3] = {1, 1, 1};
  return cu.TensorMapEncodeTiled(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims, strides, box, estr,
                                 CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                                 CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Launches `workers` CTAs (pairs) over the tiles of `count` products with the same K, which is cut into `splits` (0: equal
// runs of k-blocks; with anything but 1, fp32 sums are added into D, or go to slabs).
template <int BN, bool kPair, bool kAMn, bool kBMn, int kOut, int kMax>
cudaError_t launch_tiles(const GemmArgs* args, int count, int workers, int splits, cudaStream_t stream, const PartSums* sums = nullptr) {
  using S = Shape<BN, kPair, kOut == OUT_GELU>;
  auto kernel = gemm_tile_kernel<BN, kPair, kAMn, kBMn, kOut, kMax>;
  static std::atomic<bool> configured{false};
  if (!configured.load(std::memory_order_acquire)) {
    cudaError_t rc = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, S::kTotal);
    if (rc != cudaSuccess) return rc;
    configured.store(true, std::memory_order_release);
  }
  Problems<kMax> P;
  if constexpr (kMax > 1) {
    P.sums.count = P.sums.first[0] = 0;
    if (sums) P.sums = *sums;
  }
  P.count = count;
  P.first[0] = 0;
  for (int p = 0; p < count; ++p) {
    const GemmArgs& a = args[p];
    // K-major: boxes of 64 of K x the tile's rows; MN-major: boxes of 64 columns x 64 of K (zero fill past K)
    P.atoms[p] = (kAMn && a.m % 64 == 0 ? 1 : 0) | (kBMn && a.n % 64 == 0 && S::kRowsB > 64 ? 2 : 0);
    const bool oka = P.atoms[p] & 1 ? encode_groups(&P.a[p], a.a, a.k, a.m, a.lda, BM / 64)
                     : kAMn ? encode_map(&P.a[p], a.a, a.k, a.m, a.lda, BK) : encode_map(&P.a[p], a.a, a.m, a.k, a.lda, BM);
    const bool okb = P.atoms[p] & 2 ? encode_groups(&P.b[p], a.b, a.k, a.n, a.ldb, S::kRowsB / 64)
                     : kBMn ? encode_map(&P.b[p], a.b, a.k, a.n, a.ldb, BK) : encode_map(&P.b[p], a.b, kOut == OUT_SWIGLU ? 2 * a.n : a.n, a.k, a.ldb, S::kRowsB);
    const int slab_rows = (a.m + 31) / 32 * 32;
    if (!oka || !okb || !encode_out_map(&P.d[p], a.d, kOut == OUT_F32_SLABS ? slab_rows * splits : a.m, kOut == OUT_SWIGLU_GRAD ? 2 * a.n : a.n, a.ldd, fp32_out(kOut), half_boxes(kOut))) return cudaErrorNotSupported;
    P.m[p] = a.m;
    P.n[p] = a.n;
    constexpr int kTileN = kOut == OUT_SWIGLU ? BN / 2 : BN;
    P.n_tiles[p] = (a.n + kTileN - 1) / kTileN;
    P.first[p + 1] = P.first[p] + P.n_tiles[p] * ((a.m + (kPair ? 2 * BM : BM) - 1) / (kPair ? 2 * BM : BM));
    // partial sums are added into the output: start from zero unless the caller accumulates anyway
    if (splits != 1 && !a.accumulate && kOut != OUT_F32_SLABS) {
      cudaError_t rc = cudaMemsetAsync(a.d, 0, static_cast<size_t>(a.m) * a.n * sizeof(float), stream);
      if (rc != cudaSuccess) return rc;
    }
  }
  const GemmArgs& a = args[0];
  const void* x = half_boxes(kOut) ? a.aux : (fp32_out(kOut) ? nullptr : (a.mul ? a.mul : a.residual));
  if (x == nullptr) P.x = P.d[0];   // never used
  else if (kOut == OUT_SWIGLU || kOut == OUT_SWIGLU_GRAD ? !encode_out_map(&P.x, x, a.m, 2 * a.n, 2 * a.n, false, true)
                                                         : !encode_out_map(&P.x, x, a.m, a.n, a.ldd, false, half_boxes(kOut))) return cudaErrorNotSupported;
  GemmDev g;
  g.d = a.d;
  g.aux = a.aux;
  g.bias = a.bias;
  g.residual = a.residual;
  g.mul = a.mul;
  g.colsum = a.colsum;
  g.alpha = a.alpha;
  g.m = a.m;
  g.n = a.n;
  g.k = a.k;
  g.ldd = a.ldd;
  g.d_fp32 = fp32_out(kOut) ? 1 : 0;
  g.accumulate = a.accumulate ? 1 : 0;
  g.epilogue = a.epilogue;
  g.atomic_add = splits != 1 ? 1 : 0;
  g.slab_rows = (a.m + 31) / 32 * 32;
  g.err = gemm_error_device_ptr();
  if (!g.err) return cudaErrorNotSupported;
  g.tl = timeline_device_ptr();
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(kPair ? 2 * workers : workers));
  cfg.blockDim = dim3(S::kThreads);
  cfg.dynamicSmemBytes = S::kTotal;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  cfg.attrs = attr;
  if (kPair) {
    attr[cfg.numAttrs].id = cudaLaunchAttributeClusterDimension;
    attr[cfg.numAttrs].val.clusterDim.x = 2;
    attr[cfg.numAttrs].val.clusterDim.y = attr[cfg.numAttrs].val.clusterDim.z = 1;
    ++cfg.numAttrs;
  }
  if (pdl_enabled()) {
    attr[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[cfg.numAttrs].val.programmaticStreamSerializationAllowed = 1;
    ++cfg.numAttrs;
  }
  cudaLaunchKernelEx(&cfg, kernel, P, g, splits);
  ::mccl::launch_record("gemm_tile_kernel", __FILE__, __LINE__, cfg.gridDim, cfg.blockDim, S::kTotal, stream);
  count_launch();
  return ::mccl::launch_status();
}

// Pairs of this instantiation that can be resident at once (GPCs with an odd number of free SMs leave one SM out).
template <int BN, bool kAMn, bool kBMn, int kOut, int kMax>
int max_pairs() {
  using S = Shape<BN, true>;
  static std::atomic<int> cached{0};
  int n = cached.load(std::memory_order_relaxed);
  if (n > 0) return n;
  auto kernel = gemm_tile_kernel<BN, true, kAMn, kBMn, kOut, kMax>;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(2 * 74);
  cfg.blockDim = dim3(S::kThreads);
  cfg.dynamicSmemBytes = S::kTotal;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, S::kTotal) != cudaSuccess ||
      cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess || n <= 0) {
    (void)cudaGetLastError();
    n = gemm_sm_count() / 2 - 2;
  }
  cached.store(n, std::memory_order_relaxed);
  return n;
}

}  // namespace tiles
}  // namespace ops
}  // namespace mccl
