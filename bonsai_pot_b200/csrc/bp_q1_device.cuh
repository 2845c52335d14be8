// Device functions shared by the Q1_0 operators: the fixed exp, silu, and the reductions in the shaders' order.
#pragma once
#include <cuda_fp16.h>
#include <stdint.h>

namespace bp {

constexpr unsigned FULL = 0xffffffffu;

__device__ __forceinline__ float exp_det(float x) {  // the restatement's orc_exp_det, operation for operation
  x = fminf(fmaxf(x, -87.3f), 88.7f);
  const float n = rintf(__fmul_rn(x, 1.44269504088896341f));
  float r = __fmaf_rn(n, -0.693359375f, x);
  r = __fmaf_rn(n, 2.12194440e-4f, r);
  float p = __fmaf_rn(r, 1.0f / 720.0f, 1.0f / 120.0f);
  p = __fmaf_rn(r, p, 1.0f / 24.0f);
  p = __fmaf_rn(r, p, 1.0f / 6.0f);
  p = __fmaf_rn(r, p, 0.5f);
  p = __fmaf_rn(r, p, 1.0f);
  p = __fmaf_rn(r, p, 1.0f);
  return ldexpf(p, static_cast<int>(n));
}

// f16(g / (1 + exp(-g))) * up, in f16 (silu_mul.wgsl:22-26)
__device__ __forceinline__ __half silu_times_up(__half gate, __half up) {
  const float g = __half2float(gate);
  const float s = __fdiv_rn(g, __fadd_rn(1.0f, exp_det(-g)));
  return __hmul(__float2half_rn(s), up);
}

// subgroupAdd of a 32-lane subgroup: xor butterfly 16, 8, 4, 2, 1
__device__ __forceinline__ float butterfly32(float v) {
#pragma unroll
  for (int off = 16; off >= 1; off >>= 1) v = __fadd_rn(v, __shfl_xor_sync(FULL, v, off));
  return v;
}

// Workgroup sum of rms_norm.wgsl:62-78 / matvec_q1_0_fused_normed.wgsl:131-146 for a CTA of NW warps:
// per-warp butterfly, partial of warp s into lane s of warp 0 (zero elsewhere), butterfly again.
template <uint32_t NW>
__device__ __forceinline__ float workgroup_sum(float v, float* part /* shared, 32 floats */) {
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const float s = butterfly32(v);
  if (lane == 0) part[warp] = s;
  __syncthreads();
  if (warp == 0) {
    const float c = lane < NW ? part[lane] : 0.0f;
    const float f = butterfly32(c);
    if (lane == 0) part[0] = f;
  }
  __syncthreads();
  const float total = part[0];
  __syncthreads();
  return total;
}

}  // namespace bp
