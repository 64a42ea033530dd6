// Eight bf16 values of one 16-byte access, and sums of columns over a warp that holds a row per lane.
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>

namespace mccl {
namespace ops {

__device__ __forceinline__ void unpack8(const uint4& raw, float (&f)[8]) {
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 t = __bfloat1622float2(h[i]);
    f[2 * i] = t.x;
    f[2 * i + 1] = t.y;
  }
}
__device__ __forceinline__ uint4 pack8(const float (&f)[8]) {
  uint4 raw;
  __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&raw);
#pragma unroll
  for (int i = 0; i < 4; ++i) h[i] = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
  return raw;
}

// Sum of each of 32 per-lane values over the warp's lanes, by halving (31 shuffles): lane l returns column l.
__device__ __forceinline__ float column_sum32(float (&v)[32], int lane) {
#pragma unroll
  for (int o = 16; o >= 1; o >>= 1) {
#pragma unroll
    for (int q = 0; q < o; ++q) {
      const float lo = v[q], hi = v[q + o];
      const float other = __shfl_xor_sync(0xffffffffu, (lane & o) ? lo : hi, o);
      v[q] = ((lane & o) ? hi : lo) + other;
    }
  }
  return v[0];
}

}  // namespace ops
}  // namespace mccl
