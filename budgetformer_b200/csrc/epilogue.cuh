// Element-wise pieces of the GEMM epilogues: 16-bit pairs, the hash dropout mask, GELU.
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <stdint.h>

#include "f32x2.cuh"

namespace {

__device__ __forceinline__ f2 add2(f2 a, f2 b) {
  f2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}

// two 16-bit floats of one word, widened
template <bool FP16> __device__ __forceinline__ f2 widen16(uint32_t w) {
  if (FP16) {
    const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w));
    return pack2(f.x, f.y);
  }
  return pack2(__uint_as_float(w << 16), __uint_as_float(w & 0xFFFF0000u));
}
template <bool FP16> __device__ __forceinline__ uint32_t narrow16(float a, float b) {
  if (FP16) {
    const __half2 h = __floats2half2_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&h);
  }
  const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&h);
}

// Keep decision of element (row, col): hash(row * kHashRow + col * kHashCol + seed) >= thresh, ops.gemm.hash_keep_mask in Python.
// The hash ends in y ^ (y >> 16), whose upper half is y's: only where that equals the upper half t of the threshold does the lower
// half count, and there it is y's lower half ^ t.  So y ^ t >= thresh decides the same without the shift.
constexpr uint32_t kHashRow = 0x9E3779B1u, kHashCol = 0x85EBCA77u;
__device__ __forceinline__ bool hash_keep(uint32_t x, uint32_t thresh, uint32_t thresh_hi) {
  x = (x ^ (x >> 16)) * 0x7FEB352Du;
  x = (x ^ (x >> 15)) * 0x846CA68Bu;
  return (x ^ thresh_hi) >= thresh;
}

__device__ __forceinline__ float gelu_erf_f32(float x) { return 0.5f * x * (1.f + erff(x * 0.70710678118654752f)); }
// d/dx of the above: Phi(x) + x * phi(x)
__device__ __forceinline__ float gelu_erf_grad_f32(float x) {
  return 0.5f * (1.f + erff(x * 0.70710678118654752f)) + x * 0.3989422804014327f * __expf(-0.5f * x * x);
}

}  // namespace
