// fp8 e4m3 blocks of 1x128 with one fp32 scale, as every dispatch and every requantising epilogue makes them.
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp8.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace umdk {

__device__ __forceinline__ uint32_t pack_fp8x4(float a, float b, float c, float d) {
  const __nv_fp8x2_storage_t lo = __nv_cvt_float2_to_fp8x2(make_float2(a, b), __NV_SATFINITE, __NV_E4M3);
  const __nv_fp8x2_storage_t hi = __nv_cvt_float2_to_fp8x2(make_float2(c, d), __NV_SATFINITE, __NV_E4M3);
  return (uint32_t)lo | ((uint32_t)hi << 16);
}
__device__ __forceinline__ void bf16x8_to_float(const int4& v, float* f) {
  const __nv_bfloat162* p = reinterpret_cast<const __nv_bfloat162*>(&v);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 t = __bfloat1622float2(p[i]);
    f[2 * i] = t.x;
    f[2 * i + 1] = t.y;
  }
}

// Quantises 16 consecutive elements held by this lane; 8 lanes share a 1x128 block. Returns the packed fp8 and
// writes the block scale to *scale (same value on the 8 lanes).
__device__ __forceinline__ int4 quant16(const float* f, float* scale) {
  float amax = 0.f;
#pragma unroll
  for (int i = 0; i < 16; ++i) amax = fmaxf(amax, fabsf(f[i]));
  amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
  amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 2));
  amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 4));
  amax = fmaxf(amax, 1e-4f);
  *scale = amax * (1.f / 448.f);
  const float inv = 448.f / amax;
  int4 q;
  q.x = pack_fp8x4(f[0] * inv, f[1] * inv, f[2] * inv, f[3] * inv);
  q.y = pack_fp8x4(f[4] * inv, f[5] * inv, f[6] * inv, f[7] * inv);
  q.z = pack_fp8x4(f[8] * inv, f[9] * inv, f[10] * inv, f[11] * inv);
  q.w = pack_fp8x4(f[12] * inv, f[13] * inv, f[14] * inv, f[15] * inv);
  return q;
}

// v / (1 + exp(-v)) without the branches of the division (a zero, as rows behind a tile's own hold, takes the slowest of them: 14000
// cycles for 32 tokens a thread): the quotient is rounded once more through its remainder (Markstein). That is the rounded
// quotient if the reciprocal is; this one may be a unit off, and then the result can be the rounded quotient's neighbour where
// the quotient lies next to a rounding boundary. So at most one unit in the last place from the division; 16384 values over all
// exponents, with infinities and NaN, gave the division's bits (test_swiglu_quotient_against_the_division). A remainder that is not a
// number (v or the divisor infinite) leaves the first quotient as it is.
__device__ __forceinline__ float silu(float v) {
  const float d = 1.f + __expf(-v);
  float r;
  asm("rcp.approx.f32 %0, %1;" : "=f"(r) : "f"(d));
  const float q = v * r, e = fmaf(-q, d, v);
  return fmaf(e == e ? e : -0.f, r, q);
}

}  // namespace umdk
