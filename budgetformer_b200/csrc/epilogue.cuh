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

// bits |= bit where pred holds, on the multiply-add pipe (one: 1, in a register that the compiler does not see through).  The hash,
// the selection and the packing of an element fill the ALU pipe, which takes a warp's instruction every two cycles: 20.6 cycles an element
// and scheduler with an OR, 18.4 with this.
__device__ __forceinline__ void set_bit(uint32_t& bits, bool pred, uint32_t bit, uint32_t one) {
  if (pred) asm("mad.lo.u32 %0, %1, %2, %0;" : "+r"(bits) : "r"(one), "r"(bit));
}

// GELU x * Phi(x) with the exact normal distribution function, by its lower tail: Phi(-m) = 2^-T(m), m = |x|.  T is smooth (close to
// quadratic) and was fitted by a polynomial of degree 10 on [0, 8], least squares reweighted towards the largest error (Lawson's
// method); it goes on rising up to the clamp at 30, where the tail is 0 in fp32.  Largest error of GELU over [-12, 12] 2.4e-7 (0.5 x (1 + erff)
// 4.5e-7), relative 1.7e-5 down to x = -8 (1, since 1 + erff cancels).  Half the instructions of erff.  Of its derivative 2.7e-7 (with an erff
// of no error 1.0e-7; relative from -8 to -1 2e-6 and 3e-2): of gradients rounded to bf16 one in 8,000 falls the other way than with
// erff, and their error against 64 bits is the same to six digits (1.66e-3).
__device__ __forceinline__ float ex2_approx(float x) {
  float r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
// min(|x|, 30), NaN of NaN (fminf would give 30, and GELU then 0)
__device__ __forceinline__ float tail_arg(float x) {
  float r;
  asm("min.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(fabsf(x)), "f"(30.f));
  return r;
}
__device__ __forceinline__ float2 normal_tail2(float m0, float m1) {
  const f2 m = pack2(m0, m1);
  const float c[11] = {-1.f, -1.1511205434799194f, -0.4590774476528168f, -0.05285348370671272f, 0.007505788933485746f, -0.0004156184149906039f,
                       -9.749212040333077e-05f, 2.8189317163196392e-05f, -3.3729777442204067e-06f, 2.059425554534755e-07f, -5.215246012824082e-09f};
  f2 t = pack2(c[10], c[10]);
#pragma unroll
  for (int k = 9; k >= 0; --k) t = fma2(t, m, pack2(c[k], c[k]));
  const float2 e = unpack2(t);
  return make_float2(ex2_approx(e.x), ex2_approx(e.y));
}
__device__ __forceinline__ f2 gelu2(f2 v) {
  const float2 x = unpack2(v);
  const float m0 = tail_arg(x.x), m1 = tail_arg(x.y);
  const float2 e = normal_tail2(m0, m1);
  // x >= 0: x - m e;  x < 0: x e (also where |x| is past the clamp);  NaN: e is
  return fma2(pack2(fminf(x.x, -m0), fminf(x.y, -m1)), pack2(e.x, e.y), pack2(fmaxf(x.x, 0.f), fmaxf(x.y, 0.f)));
}
// d/dx of the above: Phi(x) + x * phi(x)
__device__ __forceinline__ f2 gelu_grad2(f2 v) {
  const float2 x = unpack2(v);
  const float2 e = normal_tail2(tail_arg(x.x), tail_arg(x.y));
  const float2 q = unpack2(mul2(mul2(v, v), pack2(-0.72134752f, -0.72134752f)));      // -x^2 / 2 in powers of two
  const f2 phi = mul2(pack2(0.3989422804f, 0.3989422804f), pack2(ex2_approx(q.x), ex2_approx(q.y)));
  return fma2(v, phi, pack2(x.x < 0.f ? e.x : 1.f - e.x, x.y < 0.f ? e.y : 1.f - e.y));
}

}  // namespace
