// Element-wise parts of the RMSNorm / RoPE / SwiGLU family: rotary embedding of the fused QKV projection's output and
// the gated activation of the fused gate / up projection's output, forward and backward.
//
// All four kernels are bound by memory: every operand is read once and every result written once, 16 bytes per thread
// and access, consecutive threads on consecutive addresses.  They replace chains of strided element-wise operators that
// went over fp32 intermediates (even / odd slices, stack, cast, chunk, concatenation).
#include "../core/launch.hpp"
#include "bf16x8.cuh"
#include "ops.hpp"

namespace mccl {
namespace ops {

namespace {

constexpr int kThreads = 256;

__device__ __forceinline__ float round_bf16(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }

int blocks_for(long long units) {
  long long blocks = (units + kThreads - 1) / kThreads;
  if (blocks > 148 * 16) blocks = 148 * 16;
  return blocks < 1 ? 1 : static_cast<int>(blocks);
}

// Rotates the four (even, odd) pairs of one 8-element unit; `inverse` turns the other way (the backward).  Products
// are rounded before they are added, as separate multiply and add operators do.
template <bool kInverse>
__device__ __forceinline__ void rotate8(float (&f)[8], const float* cos_row, const float* sin_row) {
  const float4 c = __ldg(reinterpret_cast<const float4*>(cos_row)), s = __ldg(reinterpret_cast<const float4*>(sin_row));
  const float cc[4] = {c.x, c.y, c.z, c.w};
  const float ss[4] = {kInverse ? -s.x : s.x, kInverse ? -s.y : s.y, kInverse ? -s.z : s.z, kInverse ? -s.w : s.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float a = f[2 * i], b = f[2 * i + 1];
    f[2 * i] = __fsub_rn(__fmul_rn(a, cc[i]), __fmul_rn(b, ss[i]));
    f[2 * i + 1] = __fadd_rn(__fmul_rn(a, ss[i]), __fmul_rn(b, cc[i]));
  }
}

// qkv [tokens, 3, H, hd] -> qk [tokens, 2, H, hd]: q and k of every token rotated by its position.  The two parts of
// a token are contiguous in both tensors, so a unit of 8 keeps its place within the row.  4 x 1024 tokens, 16 heads
// of 64: 8 us against 130 us for the operators it replaces.
__global__ void __launch_bounds__(kThreads) rope_qk_fwd_kernel(const __nv_bfloat16* __restrict__ qkv, const float* __restrict__ cos_t,
                                                               const float* __restrict__ sin_t, __nv_bfloat16* __restrict__ qk,
                                                               long long units, int seq, int row_units, int hd8) {
  ::mccl::pdl_wait();
  ::mccl::pdl_trigger();
  for (long long i = blockIdx.x * static_cast<long long>(kThreads) + threadIdx.x; i < units; i += static_cast<long long>(gridDim.x) * kThreads) {
    const long long t = i / (2 * row_units);
    const int u = static_cast<int>(i - t * (2 * row_units));   // unit within the token's q and k
    const int pos = static_cast<int>(t % seq), d8 = u % hd8;
    float f[8];
    unpack8(__ldg(reinterpret_cast<const uint4*>(qkv) + t * (3 * row_units) + u), f);
    const size_t at = (static_cast<size_t>(pos) * hd8 + d8) * 4;
    rotate8<false>(f, cos_t + at, sin_t + at);
    reinterpret_cast<uint4*>(qk)[i] = pack8(f);
  }
}

struct GradView {
  const __nv_bfloat16* p;
  long long sb, ss, sh;   // strides of batch, position and head in elements; the head dimension is contiguous
};

// Gradients of the rotated q, the rotated k and v, each in whatever layout the attention's backward left it, gathered
// into the gradient of qkv [tokens, 3, H, hd]; q and k are turned back on the way.
__global__ void __launch_bounds__(kThreads) rope_qkv_bwd_kernel(GradView dq, GradView dk, GradView dv, const float* __restrict__ cos_t,
                                                                const float* __restrict__ sin_t, __nv_bfloat16* __restrict__ dqkv,
                                                                long long units, int seq, int row_units, int hd8) {
  ::mccl::pdl_wait();
  ::mccl::pdl_trigger();
  for (long long i = blockIdx.x * static_cast<long long>(kThreads) + threadIdx.x; i < units; i += static_cast<long long>(gridDim.x) * kThreads) {
    const long long t = i / (3 * row_units);
    const int u = static_cast<int>(i - t * (3 * row_units));
    const int part = u / row_units, r = u - part * row_units;
    const int h = r / hd8, d8 = r - h * hd8;
    const long long b = t / seq;
    const int pos = static_cast<int>(t - b * seq);
    const GradView& g = part == 0 ? dq : (part == 1 ? dk : dv);
    uint4 raw = __ldg(reinterpret_cast<const uint4*>(g.p + b * g.sb + pos * g.ss + h * g.sh) + d8);
    if (part < 2) {
      float f[8];
      unpack8(raw, f);
      const size_t at = (static_cast<size_t>(pos) * hd8 + d8) * 4;
      rotate8<true>(f, cos_t + at, sin_t + at);
      raw = pack8(f);
    }
    reinterpret_cast<uint4*>(dqkv)[i] = raw;
  }
}

// gu [rows, 2 F] = [gate | up] -> h [rows, F] = silu(gate) * up.  silu(gate) is rounded to bf16 before the product,
// as the two separate operators do, so results do not depend on which path ran.
__global__ void __launch_bounds__(kThreads) swiglu_fwd_kernel(const __nv_bfloat16* __restrict__ gu, __nv_bfloat16* __restrict__ h,
                                                              long long units, int f8) {
  ::mccl::pdl_wait();
  ::mccl::pdl_trigger();
  for (long long i = blockIdx.x * static_cast<long long>(kThreads) + threadIdx.x; i < units; i += static_cast<long long>(gridDim.x) * kThreads) {
    const long long row = i / f8;
    const uint4* g_row = reinterpret_cast<const uint4*>(gu) + row * f8 + i;   // row * 2 f8 + (i - row * f8)
    float g[8], u[8], o[8];
    unpack8(__ldg(g_row), g);
    unpack8(__ldg(g_row + f8), u);
#pragma unroll
    for (int k = 0; k < 8; ++k) o[k] = round_bf16(__fdividef(g[k], 1.f + __expf(-g[k]))) * u[k];
    reinterpret_cast<uint4*>(h)[i] = pack8(o);
  }
}

// d(gate) = dh * up * silu'(gate), d(up) = dh * silu(gate), written side by side as the gradient of gu.
__global__ void __launch_bounds__(kThreads) swiglu_bwd_kernel(const __nv_bfloat16* __restrict__ dh, const __nv_bfloat16* __restrict__ gu,
                                                              __nv_bfloat16* __restrict__ dgu, long long units, int f8) {
  ::mccl::pdl_wait();
  ::mccl::pdl_trigger();
  for (long long i = blockIdx.x * static_cast<long long>(kThreads) + threadIdx.x; i < units; i += static_cast<long long>(gridDim.x) * kThreads) {
    const long long row = i / f8;
    const long long at = row * f8 + i;
    float d[8], g[8], u[8], dg[8], du[8];
    unpack8(__ldg(reinterpret_cast<const uint4*>(dh) + i), d);
    unpack8(__ldg(reinterpret_cast<const uint4*>(gu) + at), g);
    unpack8(__ldg(reinterpret_cast<const uint4*>(gu) + at + f8), u);
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const float s = __fdividef(1.f, 1.f + __expf(-g[k]));
      dg[k] = d[k] * u[k] * s * (1.f + g[k] * (1.f - s));
      du[k] = d[k] * g[k] * s;
    }
    reinterpret_cast<uint4*>(dgu)[at] = pack8(dg);
    reinterpret_cast<uint4*>(dgu)[at + f8] = pack8(du);
  }
}

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

}  // namespace

cudaError_t rope_qk_fwd(const __nv_bfloat16* qkv, const float* cos_t, const float* sin_t, __nv_bfloat16* qk, long long tokens, int seq,
                        int heads, int head_dim, cudaStream_t stream) {
  if (tokens <= 0) return cudaSuccess;
  if (head_dim % 8 != 0 || !aligned16(qkv) || !aligned16(qk) || !aligned16(cos_t) || !aligned16(sin_t)) return cudaErrorNotSupported;
  const int row_units = heads * head_dim / 8;
  const long long units = tokens * 2 * row_units;
  MCCL_LAUNCH_PDL(rope_qk_fwd_kernel, blocks_for(units), kThreads, 0, stream, qkv, cos_t, sin_t, qk, units, seq, row_units, head_dim / 8);
  count_launch();
  return ::mccl::launch_status();
}

cudaError_t rope_qkv_bwd(const StridedGrad (&d)[3], const float* cos_t, const float* sin_t, __nv_bfloat16* dqkv, long long tokens, int seq,
                         int heads, int head_dim, cudaStream_t stream) {
  if (tokens <= 0) return cudaSuccess;
  if (head_dim % 8 != 0 || !aligned16(dqkv) || !aligned16(cos_t) || !aligned16(sin_t)) return cudaErrorNotSupported;
  GradView v[3];
  for (int i = 0; i < 3; ++i) {
    if (!aligned16(d[i].p) || (d[i].sb | d[i].ss | d[i].sh) % 8 != 0) return cudaErrorNotSupported;
    v[i] = GradView{d[i].p, d[i].sb, d[i].ss, d[i].sh};
  }
  const int row_units = heads * head_dim / 8;
  const long long units = tokens * 3 * row_units;
  MCCL_LAUNCH_PDL(rope_qkv_bwd_kernel, blocks_for(units), kThreads, 0, stream, v[0], v[1], v[2], cos_t, sin_t, dqkv, units, seq, row_units,
                  head_dim / 8);
  count_launch();
  return ::mccl::launch_status();
}

cudaError_t swiglu_fwd(const __nv_bfloat16* gu, __nv_bfloat16* h, long long rows, int f, cudaStream_t stream) {
  if (rows <= 0) return cudaSuccess;
  if (f % 8 != 0 || !aligned16(gu) || !aligned16(h)) return cudaErrorNotSupported;
  const long long units = rows * (f / 8);
  MCCL_LAUNCH_PDL(swiglu_fwd_kernel, blocks_for(units), kThreads, 0, stream, gu, h, units, f / 8);
  count_launch();
  return ::mccl::launch_status();
}

cudaError_t swiglu_bwd(const __nv_bfloat16* dh, const __nv_bfloat16* gu, __nv_bfloat16* dgu, long long rows, int f, cudaStream_t stream) {
  if (rows <= 0) return cudaSuccess;
  if (f % 8 != 0 || !aligned16(dh) || !aligned16(gu) || !aligned16(dgu)) return cudaErrorNotSupported;
  const long long units = rows * (f / 8);
  MCCL_LAUNCH_PDL(swiglu_bwd_kernel, blocks_for(units), kThreads, 0, stream, dh, gu, dgu, units, f / 8);
  count_launch();
  return ::mccl::launch_status();
}

}  // namespace ops
}  // namespace mccl
