// Causal self-attention for sm_100a, forward and backward, on the 5th-generation tensor cores.
//
// Operands come straight from the fused QKV projection: qkv is [B, S, 3, H, hd] bf16 (the projection's output
// viewed, not copied), so q, k and v tiles of a (batch, head) are boxes of one tensor map,
// fetched by TMA into 128-byte-swizzled shared memory.  The output is written as [B, S, H, hd], which is the layout the output projection reads, and backward produces the gradient of the whole
// qkv tensor in one piece.  Nothing is transposed, sliced or concatenated around the kernels.
//
// Sequences of up to 256 and head dimensions of up to 64 (multiples of 8), which is what the models train with:
//   Forward, one CTA of two warpgroups per (batch, head, block of 128 queries).  A row of scores is at most 256 wide, so
//   all of them fit tensor memory: one S = Q K^T for every key, one softmax without running rescale (the warpgroups take
//   half of the columns each and exchange maximum and sum), one O = P V.  P overwrites Q and K in shared memory and O the
//   scores in tensor memory, so two CTAs share an SM.
//   Backward, one CTA of two warpgroups per (batch, head); per block pair (i, j <= i):
//     S = Q_i K_j^T and dP = dO_i V_j^T together,  P = exp2(S*c - L_i),  dS = P (dP - delta_i) c,
//     dV_j += P^T dO_i,  dK_j += dS^T Q_i,  dQ_i += dS K_j
//   The next pair's S and dP are issued ahead of this pair's gradient products, so the tensor cores work on them while
//   the gradients finish.  The transposed products read P / dS from the same tile through an MN-major descriptor.  Column
//   sums of the qkv gradient (the projection's bias gradient) are taken on the way out.
//   Both are bound by the latency of one CTA's chain (load, MMA, exponentials, MMA, store), not by any rate: at batch 16,
//   8 heads, 256 x 64 the tensor cores would need 1 us forward and 3 backward.  Hence two threads per row, MMAs issued
//   under elect.sync, no online rescale, and one wait where the products allow it.
//   A tile row past the sequence or a column past the head dimension is zero fill of the TMA load, so ragged sizes take
//   the same path.
// Longer sequences and wider heads are the caller's business.
//
// The reference has no attention kernel (its models call PyTorch's); this one exists because attention and the
// copies around it are a tenth of the headline training step.  Every wait is bounded: on a timeout the kernel sets
// the GEMM error word, frees its tensor memory and returns.
#include "../core/launch.hpp"
#include "gemm_common.cuh"

#include <atomic>
#include <climits>

namespace mccl {
namespace ops {

namespace {

constexpr int kBlk = 128;       // queries per CTA block, keys per inner block
constexpr int kHd = 64;         // head dimension
constexpr int kTile = kBlk * kHd * 2;   // bytes of a [128 x 64] bf16 tile: 16 KiB

// Byte offset of 16-byte chunk `c` (0..7) of row `r` inside a [rows x 64] bf16 tile stored the way a TMA load with
// the 128-byte swizzle stores it: rows of 128 bytes, 8-row groups of 1024 bytes, chunk index XORed with the row.
__device__ __forceinline__ uint32_t sw128_offset(int r, int c) {
  return static_cast<uint32_t>((r >> 3) * 1024 + (r & 7) * 128 + ((c ^ (r & 7)) << 4));
}

__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float (&v)[32]) {
  uint32_t r[32];
  tc::tmem_ld_32x32(taddr, r);
  tc::tmem_ld_wait();
#pragma unroll
  for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}

// ------------------------------------------------- forward, up to 256 keys --
struct AttnArgs {
  float* lse;                 // [B, H, S], log2 domain: m + log2(l)
  float* colsum;              // optional: column sums of dqkv are added here, fp32 [3 * H * hd]
  int colsum_ld;              // when set: the sums of every 32 rows go to a row of their own of colsum, this many elements apart
  int S, H, hd;
  float scale, scale_log2;
  int* err;
};

// Box [128 rows of the sequence x 64 columns] of part `slot` (head, or part * H + head): zero fill past S and past hd.
__device__ __forceinline__ void load_tile(void* dst, const CUtensorMap* map, uint64_t* bar, int slot, int row, int b) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];"
      ::"r"(tc::smem_u32(dst)), "l"(reinterpret_cast<uint64_t>(map)), "r"(tc::smem_u32(bar)), "r"(0), "r"(slot), "r"(row), "r"(b)
      : "memory");
}

// Store of 32 rows x 64 columns of a part from a tile in shared memory (clipped past S and past hd).  A thread that stored
// its own row touched 32 lines per instruction: 1.6 us for dK and dV of one block, 3.7 us for the rest.
__device__ __forceinline__ void store_rows32(const CUtensorMap* map, const void* src, int slot, int row, int b) {
  asm volatile("cp.async.bulk.tensor.4d.global.shared::cta.bulk_group [%0, {%2, %3, %4, %5}], [%1];"
               ::"l"(reinterpret_cast<uint64_t>(map)), "r"(tc::smem_u32(src)), "r"(0), "r"(slot), "r"(row), "r"(b)
               : "memory");
  asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}
__device__ __forceinline__ void stores_read() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }

__global__ void __launch_bounds__(256, 2) attn_fwd_kernel(const __grid_constant__ CUtensorMap tm_qkv, const __grid_constant__ CUtensorMap tm_o,
                                                          AttnArgs a) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint8_t* sK = smem;                // 2 tiles
  uint8_t* sQ = smem + 2 * kTile;    // then one tile of room: P, up to four [128 x 64] sub-tiles, overwrites K, Q and this
  uint8_t* sP = smem;
  uint8_t* sV = smem + 4 * kTile;    // 2 tiles
  float* s_max = reinterpret_cast<float*>(smem + 6 * kTile);   // [2][128]
  float* s_sum = s_max + 256;                                  // [2][128]
  uint64_t* qk_full = reinterpret_cast<uint64_t*>(s_sum + 256);
  uint64_t* v_full = qk_full + 1;
  uint64_t* s_done = v_full + 1;
  uint64_t* o_done = s_done + 1;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(o_done + 1);
  volatile int* bad = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  // one grid dimension: the others end at 65535, which a batch of short sequences passes
  const int last = a.S > kBlk ? 1 : 0, unit = static_cast<int>(blockIdx.x) >> last;
  const int qi = last - (static_cast<int>(blockIdx.x) & last);   // long rows first
  const int b = unit / a.H, h = unit - b * a.H, nblk = qi + 1, nk = nblk * kBlk;
  if (warp == 0 && tc::elect_one()) {
    tc::mbar_init(qk_full, 1);
    tc::mbar_init(v_full, 1);
    tc::mbar_init(s_done, 1);
    tc::mbar_init(o_done, 1);
    *bad = 0;
    tc::mbar_init_fence();
    tc::tma_prefetch_desc(&tm_qkv);
    pdl_wait();
    tc::mbar_expect_tx(qk_full, static_cast<uint32_t>((1 + nblk) * kTile));
    load_tile(sQ, &tm_qkv, qk_full, h, qi * kBlk, b);
    for (int j = 0; j < nblk; ++j) load_tile(sK + j * kTile, &tm_qkv, qk_full, a.H + h, j * kBlk, b);
    tc::mbar_expect_tx(v_full, static_cast<uint32_t>(nblk * kTile));
    for (int j = 0; j < nblk; ++j) load_tile(sV + j * kTile, &tm_qkv, v_full, 2 * a.H + h, j * kBlk, b);
  }
  __syncwarp();
  if (warp == 1) tc::tmem_alloc(tmem_slot, 256);
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = *tmem_slot;
  pdl_wait();

  if (warp == 0) {
    bool w = tc::mbar_wait(qk_full, 0);
    w = __all_sync(0xffffffffu, w);
    tc::fence_after_sync();
    if (tc::elect_one()) {
      if (w) {
        const uint64_t da = tc::smem_desc_k_sw128(sQ), db = tc::smem_desc_k_sw128(sK);
        const uint32_t idesc = nblk == 2 ? tc::idesc_bf16(kBlk, 256) : tc::idesc_bf16(kBlk, 128);
#pragma unroll
        for (int k4 = 0; k4 < kHd / UMMA_K; ++k4) tc::mma_bf16(tmem, da + 2 * k4, db + 2 * k4, idesc, k4 != 0);
      } else {
        *bad = 1;
      }
      tc::mma_commit(s_done);   // also on the failure path: releases the waiters below
    }
    __syncwarp();
  }
  bool ok = tc::mbar_wait(s_done, 0);
  ok = __all_sync(0xffffffffu, ok);
  tc::fence_after_sync();

  pdl_trigger();
  const int wg = warp >> 2, row = (warp & 3) * 32 + lane;      // two threads per query row, half of the keys each
  // Groups of 32 keys before `diag` are seen by all of the warp's queries, those after it by none.
  const int diag = qi * kBlk + (warp & 3) * 32, cols = nk >> 1, c_begin = wg * cols, c_end = min(c_begin + cols, diag + 32);
  const uint32_t lane_base = tmem + (static_cast<uint32_t>((warp & 3) * 32) << 16);
  float mx = -INFINITY;
#pragma unroll 1
  for (int c0 = c_begin; c0 < c_end; c0 += 64) {
    uint32_t r0[32], r1[32];
    tc::tmem_ld_32x32(lane_base + static_cast<uint32_t>(c0), r0);
    tc::tmem_ld_32x32(lane_base + static_cast<uint32_t>(c0 + 32), r1);
    tc::tmem_ld_wait();
    auto group_max = [&](const uint32_t (&r)[32], int c) {
      if (c < diag) {
#pragma unroll
        for (int e = 0; e < 32; ++e) mx = fmaxf(mx, __uint_as_float(r[e]));
      } else if (c == diag) {
#pragma unroll
        for (int e = 0; e < 32; ++e) mx = e <= lane ? fmaxf(mx, __uint_as_float(r[e])) : mx;
      }
    };
    group_max(r0, c0);
    group_max(r1, c0 + 32);
  }
  s_max[wg * 128 + row] = mx;
  __syncthreads();
  const float m = fmaxf(s_max[row], s_max[128 + row]) * a.scale_log2;   // key 0 is never masked: finite
  float sum = 0.f;
#pragma unroll 1
  for (int c0 = c_begin; c0 < c_begin + cols; c0 += 32) {
    uint8_t* sub = sP + (c0 >> 6) * kTile;
    const int chunk0 = (c0 & 63) >> 3;
    if (c0 > diag) {
#pragma unroll
      for (int c8 = 0; c8 < 4; ++c8) *reinterpret_cast<uint4*>(sub + sw128_offset(row, chunk0 + c8)) = make_uint4(0u, 0u, 0u, 0u);
      continue;
    }
    float s[32];
    tmem_ld32(lane_base + static_cast<uint32_t>(c0), s);
#pragma unroll
    for (int e = 0; e < 32; ++e) s[e] = exp2f(s[e] * a.scale_log2 - m);
    if (c0 == diag) {
#pragma unroll
      for (int e = 0; e < 32; ++e) s[e] = e <= lane ? s[e] : 0.f;
    }
#pragma unroll
    for (int c8 = 0; c8 < 4; ++c8) {
      uint4 pk;
      __nv_bfloat162* hp = reinterpret_cast<__nv_bfloat162*>(&pk);
#pragma unroll
      for (int e2 = 0; e2 < 4; ++e2) {
        hp[e2] = __floats2bfloat162_rn(s[c8 * 8 + e2 * 2], s[c8 * 8 + e2 * 2 + 1]);
        // the sum uses the rounded values: they are what multiplies V
        const float2 back = __bfloat1622float2(hp[e2]);
        sum += back.x + back.y;
      }
      *reinterpret_cast<uint4*>(sub + sw128_offset(row, chunk0 + c8)) = pk;
    }
  }
  s_sum[wg * 128 + row] = sum;
  fence_async_smem();          // the MMA reads P through the async proxy
  tc::fence_before_sync();
  __syncthreads();             // P is complete and everybody has read S: O may overwrite it
  if (warp == 0) {
    bool w = tc::mbar_wait(v_full, 0);
    w = __all_sync(0xffffffffu, w);
    tc::fence_after_sync();
    if (tc::elect_one()) {
      if (w) {
        constexpr uint32_t idesc = tc::idesc_bf16(kBlk, kHd, false, true);
        const uint64_t dv = tc::smem_desc_mn_sw128(sV, kTile), dp = tc::smem_desc_k_sw128(sP);
        for (int t = 0; t < 2 * nblk; ++t) {
#pragma unroll
          for (int q = 0; q < 4; ++q)
            tc::mma_bf16(tmem, dp + (kTile >> 4) * t + 2 * q, dv + 512 * t + 128 * q, idesc, t + q != 0);
        }
      } else {
        *bad = 1;
      }
      tc::mma_commit(o_done);
    }
    __syncwarp();
  }
  ok = tc::mbar_wait(o_done, 0) && ok;
  ok = __all_sync(0xffffffffu, ok);
  tc::fence_after_sync();
  {
    float o[32];
    tmem_ld32(lane_base + static_cast<uint32_t>(wg * 32), o);
    const int q_row = qi * kBlk + row;
    const float l = s_sum[row] + s_sum[128 + row], inv = 1.f / l;
#pragma unroll
    for (int c8 = 0; c8 < 4; ++c8) {   // V has been read: its first tile takes the output on its way to memory
      uint4 pk;
      __nv_bfloat162* hp = reinterpret_cast<__nv_bfloat162*>(&pk);
#pragma unroll
      for (int e2 = 0; e2 < 4; ++e2) hp[e2] = __floats2bfloat162_rn(o[c8 * 8 + 2 * e2] * inv, o[c8 * 8 + 2 * e2 + 1] * inv);
      *reinterpret_cast<uint4*>(sV + sw128_offset(row, wg * 4 + c8)) = pk;
    }
    if (wg == 0 && q_row < a.S && ok) a.lse[(static_cast<size_t>(b) * a.H + h) * a.S + q_row] = m + log2f(l);
  }
  fence_async_smem();
  tc::fence_before_sync();
  __syncthreads();
  if (ok && *bad == 0 && warp < 4 && qi * kBlk + warp * 32 < a.S) {
    if (tc::elect_one()) {
      store_rows32(&tm_o, sV + warp * 4096, h, qi * kBlk + warp * 32, b);
      stores_read();
    }
    __syncwarp();
  }
  if ((!ok || *bad) && tid == 0) {
    atomicExch(a.err, 11);
    tc::mbar_wait(qk_full, 0, 1u << 20);   // loads that were issued must land before the CTA retires
    tc::mbar_wait(v_full, 0, 1u << 20);
  }
  if (warp == 1) {   // everybody's tensor-memory reads were before the barrier above
    tc::fence_after_sync();
    tc::tmem_dealloc(tmem, 256);
  }
}

constexpr int kFwdSmem = 6 * kTile + 2048 + 64 + 1024;   // 99 KiB: two CTAs per SM

// ------------------------------------------------ backward, up to 256 keys --
// Tensor memory, 512 columns: [0,128) S  [128,256) dP  [256,384) dQ_0, dQ_1  [384,448) dK_j  [448,512) dV_j
__global__ void __launch_bounds__(256, 1) attn_bwd_kernel(const __grid_constant__ CUtensorMap tm_qkv,
                                                          const __grid_constant__ CUtensorMap tm_do,
                                                          const __grid_constant__ CUtensorMap tm_o,
                                                          const __grid_constant__ CUtensorMap tm_dqkv, AttnArgs a) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint8_t* sQ = smem;                 // [2] tiles each
  uint8_t* sK = sQ + 2 * kTile;
  uint8_t* sV = sK + 2 * kTile;
  uint8_t* sDO = sV + 2 * kTile;
  uint8_t* sP = sDO + 2 * kTile;      // two [128 x 64] sub-tiles each
  uint8_t* sDS = sP + 2 * kTile;
  float* s_delta = reinterpret_cast<float*>(sDS + 2 * kTile);   // [256]
  float* s_lse = s_delta + 256;                                 // [256]
  uint64_t* in_full = reinterpret_cast<uint64_t*>(s_lse + 256);   // [2]: one per block
  uint64_t* s_done = in_full + 2;
  uint64_t* g_done = s_done + 1;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(g_done + 1);
  volatile int* bad = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int nblk = (a.S + kBlk - 1) / kBlk;   // 1 or 2
  const int b = static_cast<int>(blockIdx.x) / a.H, h = static_cast<int>(blockIdx.x) - b * a.H;
  if (warp == 0 && tc::elect_one()) {
    tc::mbar_init(&in_full[0], 1);
    tc::mbar_init(&in_full[1], 1);
    tc::mbar_init(s_done, 1);
    tc::mbar_init(g_done, 2);   // two issuing threads
    *bad = 0;
    tc::mbar_init_fence();
    tc::tma_prefetch_desc(&tm_qkv);
    tc::tma_prefetch_desc(&tm_do);
    tc::tma_prefetch_desc(&tm_o);
    tc::tma_prefetch_desc(&tm_dqkv);
    pdl_wait();
    for (int i = nblk - 1; i >= 0; --i) {   // the last block first: its pair is the first one computed
      tc::mbar_expect_tx(&in_full[i], 5 * kTile);
      load_tile(sQ + i * kTile, &tm_qkv, &in_full[i], h, i * kBlk, b);
      load_tile(sK + i * kTile, &tm_qkv, &in_full[i], a.H + h, i * kBlk, b);
      load_tile(sDO + i * kTile, &tm_do, &in_full[i], h, i * kBlk, b);
      load_tile(sV + i * kTile, &tm_qkv, &in_full[i], 2 * a.H + h, i * kBlk, b);
      load_tile(sP + i * kTile, &tm_o, &in_full[i], h, i * kBlk, b);   // the output waits where P will go
    }
  }
  __syncwarp();
  if (warp == 1) tc::tmem_alloc(tmem_slot, 512);
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  pdl_wait();
  const uint32_t tmem = *tmem_slot;
  const uint32_t tm_dq = tmem + 256, tm_dk = tmem + 384, tm_dv = tmem + 448;
  const int wg = warp >> 2, row = (warp & 3) * 32 + lane;
  const uint32_t lane_base = static_cast<uint32_t>((warp & 3) * 32) << 16;

  constexpr uint32_t idesc_qk = tc::idesc_bf16(kBlk, kBlk, false, false);    // S, dP: both operands K-major
  constexpr uint32_t idesc_tt = tc::idesc_bf16(kBlk, kHd, true, true);       // dV, dK: A transposed (MN-major), B MN-major
  constexpr uint32_t idesc_nt = tc::idesc_bf16(kBlk, kHd, false, true);      // dQ: A K-major, B MN-major
  // pairs in order: (1,1), (1,0), (0,0) for two blocks, (0,0) for one
  const int pairs = nblk == 2 ? 3 : 1;
  auto pair_i = [&](int p) { return nblk == 2 && p < 2 ? 1 : 0; };
  auto pair_j = [&](int p) { return nblk == 2 && p < 1 ? 1 : 0; };
  auto issue_scores = [&](int i, int j) {   // elected thread of warp 0
    const uint64_t dq = tc::smem_desc_k_sw128(sQ + i * kTile), dk = tc::smem_desc_k_sw128(sK + j * kTile);
#pragma unroll
    for (int k4 = 0; k4 < kHd / UMMA_K; ++k4) tc::mma_bf16(tmem, dq + 2 * k4, dk + 2 * k4, idesc_qk, k4 != 0);
    const uint64_t dd = tc::smem_desc_k_sw128(sDO + i * kTile), dv = tc::smem_desc_k_sw128(sV + j * kTile);
#pragma unroll
    for (int k4 = 0; k4 < kHd / UMMA_K; ++k4) tc::mma_bf16(tmem + 128, dd + 2 * k4, dv + 2 * k4, idesc_qk, k4 != 0);
    tc::mma_commit(s_done);
  };
  // one row of 32 gradient columns [c0, c0 + 32) of part t (0: dQ, 1: dK, 2: dV) out of tensor memory into a tile that is
  // no longer needed; then the warp's 32 rows leave for block blk
  auto stage_out = [&](uint8_t* tile, uint32_t taddr, int t, int c0, int blk) {
    float v[32];
    tmem_ld32(taddr + lane_base + static_cast<uint32_t>(c0), v);
#pragma unroll
    for (int c8 = 0; c8 < 4; ++c8) {
      uint4 pk;
      __nv_bfloat162* hp = reinterpret_cast<__nv_bfloat162*>(&pk);
#pragma unroll
      for (int e2 = 0; e2 < 4; ++e2) hp[e2] = __floats2bfloat162_rn(v[c8 * 8 + 2 * e2], v[c8 * 8 + 2 * e2 + 1]);
      *reinterpret_cast<uint4*>(tile + sw128_offset(row, (c0 >> 3) + c8)) = pk;
    }
    if (a.colsum != nullptr && c0 < a.hd) {   // rows past the sequence are zero
      const float sum = column_sum32(v, lane);
      if (c0 + lane < a.hd) {
        float* to = a.colsum + static_cast<size_t>((b * nblk + blk) * 4 + (warp & 3)) * a.colsum_ld + (t * a.H + h) * a.hd + c0 + lane;
        if (a.colsum_ld != 0) *to = sum;
        else atomicAdd(to, sum);
      }
    }
  };
  auto send_out = [&](const uint8_t* tile, int t, int blk) {
    fence_async_smem();
    __syncwarp();
    const int q = warp & 3;
    if (blk * kBlk + q * 32 < a.S && tc::elect_one()) store_rows32(&tm_dqkv, tile + q * 4096, t * a.H + h, blk * kBlk + q * 32, b);
    __syncwarp();
  };
  auto key_block_out = [&](int j) {   // one warpgroup takes dK_j, the other dV_j; K_j and V_j have been read for the last time
    uint8_t* tile = (wg == 0 ? sK : sV) + j * kTile;
    stage_out(tile, wg == 0 ? tm_dk : tm_dv, 1 + wg, 0, j);
    stage_out(tile, wg == 0 ? tm_dk : tm_dv, 1 + wg, 32, j);
    tc::fence_before_sync();
    send_out(tile, 1 + wg, j);
  };

  if (warp == 0) {
    bool w = tc::mbar_wait(&in_full[nblk - 1], 0);
    w = __all_sync(0xffffffffu, w);
    tc::fence_after_sync();
    if (tc::elect_one()) {
      if (!w) *bad = 1;
      issue_scores(nblk - 1, nblk - 1);
    }
    __syncwarp();
  }
  pdl_trigger();
  bool ok = true;
  {
    // delta[row] = sum_d dO[row, d] * O[row, d] and the row's log-sum-exp, one row per thread.  Rows past the sequence get an
    // infinite one: P = 0.
    const int blk = tid >> 7, r = tid & 127;
    float acc = 0.f, l = INFINITY;
    if (tid < a.S) l = a.lse[(static_cast<size_t>(b) * a.H + h) * a.S + tid];
    if (blk < nblk) {
      ok = tc::mbar_wait(&in_full[blk], 0);
#pragma unroll
      for (int c = 0; c < kHd / 8; ++c) {
        const uint4 vo = *reinterpret_cast<const uint4*>(sP + blk * kTile + sw128_offset(r, c));
        const uint4 vd = *reinterpret_cast<const uint4*>(sDO + blk * kTile + sw128_offset(r, c));
        const __nv_bfloat162* ho = reinterpret_cast<const __nv_bfloat162*>(&vo);
        const __nv_bfloat162* hd = reinterpret_cast<const __nv_bfloat162*>(&vd);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float2 x = __bfloat1622float2(ho[e]), y = __bfloat1622float2(hd[e]);
          acc += x.x * y.x + x.y * y.y;
        }
      }
    }
    s_delta[tid] = acc;
    s_lse[tid] = l;
    if (!ok) *bad = 1;
  }
#pragma unroll 1
  for (int p = 0; p < pairs; ++p) {
    const int i = pair_i(p), j = pair_j(p);
    ok = tc::mbar_wait(s_done, p & 1);
    if (!__syncthreads_and((ok && *bad == 0) ? 1 : 0)) {
      ok = false;
      break;
    }
    tc::fence_after_sync();
    const float lse = s_lse[i * kBlk + row], delta = s_delta[i * kBlk + row] * a.scale;
    // Groups of 32 keys before `diag` are seen by all of the warp's queries, those after it by none.
    const int diag = i == j ? (warp & 3) * 32 : kBlk;
    uint4 pk[8], dk[8];   // kept until the gradient products of the pair before have read the shared tiles
#pragma unroll
    for (int g = 0; g < 2; ++g) {
      const int c0 = wg * 64 + g * 32;
      if (c0 > diag) {
#pragma unroll
        for (int c8 = 0; c8 < 4; ++c8) pk[g * 4 + c8] = dk[g * 4 + c8] = make_uint4(0u, 0u, 0u, 0u);
        continue;
      }
      uint32_t rs[32], rd[32];
      tc::tmem_ld_32x32(tmem + lane_base + static_cast<uint32_t>(c0), rs);
      tc::tmem_ld_32x32(tmem + lane_base + static_cast<uint32_t>(128 + c0), rd);
      tc::tmem_ld_wait();
      float pr[32];
#pragma unroll
      for (int e = 0; e < 32; ++e) pr[e] = exp2f(__uint_as_float(rs[e]) * a.scale_log2 - lse);
      if (c0 == diag) {
#pragma unroll
        for (int e = 0; e < 32; ++e) pr[e] = e <= lane ? pr[e] : 0.f;
      }
#pragma unroll
      for (int c8 = 0; c8 < 4; ++c8) {
        __nv_bfloat162* hp = reinterpret_cast<__nv_bfloat162*>(&pk[g * 4 + c8]);
        __nv_bfloat162* hs = reinterpret_cast<__nv_bfloat162*>(&dk[g * 4 + c8]);
#pragma unroll
        for (int e2 = 0; e2 < 4; ++e2) {
          const int e = c8 * 8 + e2 * 2;
          hp[e2] = __floats2bfloat162_rn(pr[e], pr[e + 1]);
          hs[e2] = __floats2bfloat162_rn(pr[e] * (__uint_as_float(rd[e]) * a.scale - delta), pr[e + 1] * (__uint_as_float(rd[e + 1]) * a.scale - delta));
        }
      }
    }
    if (p > 0) {
      ok = tc::mbar_wait(g_done, (p - 1) & 1);   // P and dS may be overwritten, the last pair's gradients are in tensor memory
      ok = __all_sync(0xffffffffu, ok);
      tc::fence_after_sync();
      if (ok && *bad == 0 && pair_j(p - 1) != j) key_block_out(pair_j(p - 1));
    }
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      const uint32_t off = wg * kTile + sw128_offset(row, c);
      *reinterpret_cast<uint4*>(sP + off) = pk[c];
      *reinterpret_cast<uint4*>(sDS + off) = dk[c];
    }
    fence_async_smem();
    tc::fence_before_sync();
    __syncthreads();   // P and dS are complete, and nobody reads the score columns any more
    // Two threads issue: an MMA takes its issuer some 50 clocks, and these 24 would be 0.7 us of the chain for one.
    if (warp == 0) {
      bool w = true;
      if (p + 1 < pairs && p == 0) w = tc::mbar_wait(&in_full[0], 0);   // the second pair is the first to need block 0
      w = __all_sync(0xffffffffu, w);
      tc::fence_after_sync();
      if (tc::elect_one()) {
        if (!w) *bad = 1;
        if (p + 1 < pairs) issue_scores(pair_i(p + 1), pair_j(p + 1));
        const uint64_t dpt = tc::smem_desc_mn_sw128(sP, kTile), ddo = tc::smem_desc_mn_sw128(sDO + i * kTile, kTile);
        const bool add = p == 2;   // dV_0: pairs (1,0), (0,0)
#pragma unroll
        for (int kk = 0; kk < kBlk / UMMA_K; ++kk) tc::mma_bf16(tm_dv, dpt + 128 * kk, ddo + 128 * kk, idesc_tt, kk != 0 || add);
        tc::mma_commit(g_done);
      }
      __syncwarp();
    } else if (warp == 4) {
      tc::fence_after_sync();
      if (tc::elect_one()) {
        const uint64_t dst = tc::smem_desc_mn_sw128(sDS, kTile), dq = tc::smem_desc_mn_sw128(sQ + i * kTile, kTile);
        const uint64_t dkm = tc::smem_desc_mn_sw128(sK + j * kTile, kTile), dsn = tc::smem_desc_k_sw128(sDS);
        const bool add_k = p == 2, add_q = p == 1;   // dK_0: pairs (1,0), (0,0); dQ_1: pairs (1,1), (1,0)
#pragma unroll
        for (int kk = 0; kk < kBlk / UMMA_K; ++kk) tc::mma_bf16(tm_dk, dst + 128 * kk, dq + 128 * kk, idesc_tt, kk != 0 || add_k);
#pragma unroll
        for (int kk = 0; kk < kBlk / UMMA_K; ++kk)
          tc::mma_bf16(tm_dq + static_cast<uint32_t>(i * kHd), dsn + (kk >> 2) * (kTile >> 4) + 2 * (kk & 3), dkm + 128 * kk, idesc_nt, kk != 0 || add_q);
        tc::mma_commit(g_done);
      }
      __syncwarp();
    }
  }
  if (ok) {
    ok = tc::mbar_wait(g_done, (pairs - 1) & 1);
    ok = __all_sync(0xffffffffu, ok);
    tc::fence_after_sync();
    if (ok && *bad == 0) key_block_out(0);
  }
  ok = __syncthreads_and((ok && *bad == 0) ? 1 : 0) != 0;
  if (ok) {
    if (nblk == 2) {   // one query block per warpgroup
      stage_out(sQ + wg * kTile, tm_dq + static_cast<uint32_t>(wg * kHd), 0, 0, wg);
      stage_out(sQ + wg * kTile, tm_dq + static_cast<uint32_t>(wg * kHd), 0, 32, wg);
      send_out(sQ + wg * kTile, 0, wg);
    } else {           // half of the columns per warpgroup
      stage_out(sQ, tm_dq, 0, wg * 32, 0);
      fence_async_smem();
      __syncthreads();
      if (wg == 0) send_out(sQ, 0, 0);
    }
    if (tc::elect_one()) stores_read();   // the thread that sent this warp's rows
    __syncwarp();
  } else if (tid == 0) {
    atomicExch(a.err, 12);
    for (int i = 0; i < nblk; ++i) tc::mbar_wait(&in_full[i], 0, 1u << 20);   // issued loads must land before the CTA retires
  }
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 1) {
    tc::fence_after_sync();
    tc::tmem_dealloc(tmem, 512);
  }
}

constexpr int kBwdSmem = 12 * kTile + 2048 + 64 + 1024;   // 195 KiB

// [B, S, slots, hd] with contiguous hd as boxes of box_rows rows x 64 columns of one (batch, slot).
bool encode_slots(CUtensorMap* map, const void* base, int B, int S, int slots, int hd, int box_rows = kBlk) {
  const CuDriver& cu = CuDriver::get();
  if (!cu.loaded || !cu.TensorMapEncodeTiled) return false;
  int device = 0;
  cudaGetDevice(&device);
  cu.ensure_context(device);
  const cuuint64_t row = static_cast<cuuint64_t>(slots) * hd * 2;
  cuuint64_t dims[4] = {static_cast<cuuint64_t>(hd), static_cast<cuuint64_t>(slots), static_cast<cuuint64_t>(S), static_cast<cuuint64_t>(B)};
  cuuint64_t strides[3] = {static_cast<cuuint64_t>(hd) * 2, row, row * S};
  cuuint32_t box[4] = {kHd, 1, static_cast<cuuint32_t>(box_rows), 1};
  cuuint32_t estr[4] = {1, 1, 1, 1};
  return cu.TensorMapEncodeTiled(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(base), dims, strides, box, estr,
                                 CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                                 CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <typename K>
cudaError_t allow_smem(K kernel, int bytes, std::atomic<bool>& done) {
  if (done.load(std::memory_order_acquire)) return cudaSuccess;
  cudaError_t rc = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (rc == cudaSuccess) done.store(true, std::memory_order_release);
  return rc;
}

}  // namespace

static_assert(2 * kBlk == 256, "one or two blocks of queries");
bool attention_supported(int S, int hd) { return S >= 1 && S <= 2 * kBlk && hd >= 8 && hd <= kHd && hd % 8 == 0; }

int attention_bwd_parts(int B, int S) { return B * ((S + kBlk - 1) / kBlk) * 4; }

cudaError_t attention_bwd(const __nv_bfloat16* qkv, const __nv_bfloat16* o, const __nv_bfloat16* d_o, const float* lse,
                          __nv_bfloat16* dqkv, float* colsum, int B, int S, int H, int hd, float softmax_scale, cudaStream_t stream, bool in_order) {
  if (!attention_supported(S, hd) || B <= 0 || H <= 0 || static_cast<long long>(B) * H > INT_MAX) return cudaErrorNotSupported;
  if ((reinterpret_cast<uintptr_t>(qkv) | reinterpret_cast<uintptr_t>(o) | reinterpret_cast<uintptr_t>(d_o) |
       reinterpret_cast<uintptr_t>(dqkv)) & 15u)
    return cudaErrorNotSupported;
  static std::atomic<bool> configured{false};
  cudaError_t rc = allow_smem(attn_bwd_kernel, kBwdSmem, configured);
  if (rc != cudaSuccess) return rc;
  CUtensorMap tq, tdo, to, tdqkv;
  if (!encode_slots(&tq, qkv, B, S, 3 * H, hd) || !encode_slots(&tdo, d_o, B, S, H, hd) || !encode_slots(&to, o, B, S, H, hd) ||
      !encode_slots(&tdqkv, dqkv, B, S, 3 * H, hd, 32))
    return cudaErrorNotSupported;
  (void)cudaGetLastError();
  AttnArgs a = {};
  a.lse = const_cast<float*>(lse);
  a.colsum = colsum;
  a.colsum_ld = in_order ? 3 * H * hd : 0;
  a.S = S;
  a.H = H;
  a.hd = hd;
  a.scale = softmax_scale;
  a.scale_log2 = softmax_scale * 1.4426950408889634f;
  a.err = gemm_error_device_ptr();
  if (!a.err) return cudaErrorNotSupported;
  MCCL_LAUNCH_PDL(attn_bwd_kernel, H * B, 256, kBwdSmem, stream, tq, tdo, to, tdqkv, a);
  count_launch();
  return launch_status();
}

cudaError_t attention_fwd(const __nv_bfloat16* qkv, __nv_bfloat16* o, float* lse, int B, int S, int H, int hd, float softmax_scale,
                          cudaStream_t stream) {
  const int blocks = (S + kBlk - 1) / kBlk;
  if (!attention_supported(S, hd) || B <= 0 || H <= 0 || static_cast<long long>(B) * H * blocks > INT_MAX) return cudaErrorNotSupported;
  if ((reinterpret_cast<uintptr_t>(qkv) | reinterpret_cast<uintptr_t>(o)) & 15u) return cudaErrorNotSupported;
  static std::atomic<bool> configured{false};
  cudaError_t rc = allow_smem(attn_fwd_kernel, kFwdSmem, configured);
  if (rc != cudaSuccess) return rc;
  CUtensorMap tq, to;
  if (!encode_slots(&tq, qkv, B, S, 3 * H, hd) || !encode_slots(&to, o, B, S, H, hd, 32)) return cudaErrorNotSupported;
  (void)cudaGetLastError();
  AttnArgs a = {};
  a.lse = lse;
  a.S = S;
  a.H = H;
  a.hd = hd;
  a.scale = softmax_scale;
  a.scale_log2 = softmax_scale * 1.4426950408889634f;
  a.err = gemm_error_device_ptr();
  if (!a.err) return cudaErrorNotSupported;
  MCCL_LAUNCH_PDL(attn_fwd_kernel, blocks * H * B, 256, kFwdSmem, stream, tq, to, a);
  count_launch();
  return launch_status();
}

}  // namespace ops
}  // namespace mccl
