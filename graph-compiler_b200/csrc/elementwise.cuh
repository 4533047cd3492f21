// The scalar functions of the elementwise operations, shared by the step kernels and the fused runs.
#pragma once
#include <cuda_fp16.h>

#include "sm100_ptx.cuh"

namespace gcb {

// element types: 0 f32, 1 bf16, 2 f16
__device__ __forceinline__ float ew_load(const void *p, long long i, int dt) {
  if (dt == 0) return reinterpret_cast<const float *>(p)[i];
  if (dt == 1) return bf16_bits_to_f32(reinterpret_cast<const uint16_t *>(p)[i]);
  return __half2float(reinterpret_cast<const __half *>(p)[i]);
}
// Every bf16/f16 op rounds once on store: the reference evaluates low-precision
// elementwise ops as extf -> f32 op -> truncf (lib/gc/Transforms/Pipeline.cpp:81-90).
__device__ __forceinline__ void ew_store(void *p, long long i, int dt, float v) {
  if (dt == 0) reinterpret_cast<float *>(p)[i] = v;
  else if (dt == 1) reinterpret_cast<uint16_t *>(p)[i] = uint16_t(f32_to_bf16_bits(v));
  else reinterpret_cast<__half *>(p)[i] = __float2half_rn(v);
}
// The value a store of this type would leave in memory.
__device__ __forceinline__ float ew_round(float v, int dt) {
  if (dt == 1) return bf16_bits_to_f32(f32_to_bf16_bits(v));
  if (dt == 2) return __half2float(__float2half_rn(v));
  return v;
}
__device__ __forceinline__ float ew_binary(int fn, float x, float y) {
  switch (fn) {
  case 0: return __fadd_rn(x, y);
  case 1: return __fsub_rn(x, y);
  case 2: return __fmul_rn(x, y);
  default: return __fdiv_rn(x, y);
  }
}
__device__ __forceinline__ float ew_unary(int fn, float beta, float x) {
  switch (fn) {
  case 0: return (x != x) ? x : (x > 0.f ? x : 0.f);        // max(x, 0), NaN propagates
  case 1: return __fdiv_rn(1.f, __fadd_rn(1.f, expf(-x)));  // 1 / (1 + exp(-x))
  case 2:
    if (beta == 2.f) return __fmul_rn(x, x);
    if (beta == 1.f) return x;
    if (beta == 0.5f) return sqrtf(x);
    if (beta == 3.f) return __fmul_rn(__fmul_rn(x, x), x);
    return powf(x, beta);
  case 4: return expf(x);
  case 5: return -x;
  default: return x;
  }
}

} // namespace gcb
