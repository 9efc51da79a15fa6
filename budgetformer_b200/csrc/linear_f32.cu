// Weight and bias gradient of a linear layer in fp32: dW[N, K] = dY[M, N]^T X[M, K], db[N] = column sums of dY.
//
// M (rows of the activation) is 10^2 to 10^6, N and K are layer widths: the output is a few 64 x 64 tiles (for many, the library's
// GEMM is faster: ops/gemm.py::f32_gradient_pays), so one tile per block leaves the chip empty, and a library GEMM that splits no
// further takes one block's walk over all rows.  Here the rows are cut into slices until every SM has two blocks; each block
// leaves its 64 x 64 partial sum, and a second kernel
// adds the slices in a fixed order (no atomics: the gradients are bit-reproducible).  The bias gradient rides on the blocks of
// the first column of tiles, which hold dY in shared memory anyway.  All sums are plain fp32 multiply-adds, two per instruction;
// cutting the rows shortens the chains: against 64 bits dW is 1.7e-7 off at 40 k rows of 64 x 64 (one long sum: 8.3e-7).
// 40,009 rows, dW and db, us: 64 x 64 23 (library GEMM and column sum 137), 128 x 128 50 (172).  Bound by the shared-memory reads
// and issue of the 64 multiply-adds per thread and row.
#include <cuda_runtime.h>
#include <stdint.h>

#include "bf_kernels.h"
#include "f32x2.cuh"

namespace {

// BYTES from src, or zeros
template <int BYTES> __device__ __forceinline__ void copy_or_zero(void* dst, const void* src, bool ok) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
  const int n = ok ? BYTES : 0;
  if constexpr (BYTES == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(n) : "memory");
  else asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d), "l"(src), "r"(n) : "memory");
}

constexpr int TILE = 64, ROWS = 32, STAGES = 3, THREADS = 256;

// VEC: floats per copy (4 when rows of both operands are 16-byte aligned and N, K are multiples of 4)
template <int VEC>
__device__ __forceinline__ void load_stage(float (*dst)[TILE], const float* src, long long ld, long long row0, long long row_end,
                                           int col0, int cols) {
  constexpr int PER_ROW = TILE / VEC;
  for (int i = threadIdx.x; i < ROWS * PER_ROW; i += THREADS) {
    const int r = i / PER_ROW, c = (i % PER_ROW) * VEC;
    const bool ok = row0 + r < row_end && col0 + c < cols;
    copy_or_zero<4 * VEC>(&dst[r][c], ok ? src + (row0 + r) * ld + col0 + c : src, ok);
  }
}

// grid (slices, N tiles * K tiles).  256 threads = 4 groups of 64, group g takes the rows g, g + 4, ... of every stage; a thread
// holds an 8 x 8 piece of the tile (rows ty * 8 .., columns tx * 4 .. and 32 + tx * 4 ..: both operands are read from shared
// memory 16 bytes at a time without bank conflicts, 4 reads for 64 multiply-adds).
template <int VEC>
__global__ void __launch_bounds__(THREADS, 2) f32_dw_kernel(const float* __restrict__ dy, long long lddy, const float* __restrict__ x,
                                                            long long ldx, long long M, int N, int K, long long rows_per,
                                                            float* __restrict__ partial, int want_bias) {
  __shared__ __align__(16) float sm[STAGES][2][ROWS][TILE];
  const int k_tiles = (K + TILE - 1) / TILE;
  const int n0 = (blockIdx.y / k_tiles) * TILE, k0 = (blockIdx.y % k_tiles) * TILE;
  const long long beg = blockIdx.x * rows_per, end = min(M, beg + rows_per);
  const int g = threadIdx.x >> 6, t = threadIdx.x & 63, ty = t >> 3, tx = t & 7;
  const bool bias = want_bias && k0 == 0;
  f2 acc[8][4], bs[4];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = pack2(0.f, 0.f);
#pragma unroll
  for (int j = 0; j < 4; ++j) bs[j] = pack2(0.f, 0.f);
  const int n_st = beg < end ? (int)((end - beg + ROWS - 1) / ROWS) : 0;
  auto fetch = [&](int s) {
    if (s < n_st) {
      const long long r0 = beg + (long long)s * ROWS;
      load_stage<VEC>(sm[s % STAGES][0], dy, lddy, r0, end, n0, N);
      load_stage<VEC>(sm[s % STAGES][1], x, ldx, r0, end, k0, K);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
#pragma unroll
  for (int s = 0; s < STAGES - 1; ++s) fetch(s);
  const f2 one = pack2(1.f, 1.f);
  for (int s = 0; s < n_st; ++s) {
    asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
    __syncthreads();                          // stage s has landed for everyone, and stage s - 1 is free
    fetch(s + STAGES - 1);
    const float(*a)[TILE] = sm[s % STAGES][0];
    const float(*b)[TILE] = sm[s % STAGES][1];
#pragma unroll 2
    for (int r = g; r < ROWS; r += 4) {
      const float4 a0 = *reinterpret_cast<const float4*>(&a[r][ty * 8]), a1 = *reinterpret_cast<const float4*>(&a[r][ty * 8 + 4]);
      const float4 b0 = *reinterpret_cast<const float4*>(&b[r][tx * 4]), b1 = *reinterpret_cast<const float4*>(&b[r][32 + tx * 4]);
      const f2 bv[4] = {pack2(b0.x, b0.y), pack2(b0.z, b0.w), pack2(b1.x, b1.y), pack2(b1.z, b1.w)};
      const float av[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const f2 aa = pack2(av[i], av[i]);
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fma2(aa, bv[j], acc[i][j]);
      }
      if (bias) {
#pragma unroll
        for (int j = 0; j < 4; ++j) bs[j] = fma2(pack2(av[2 * j], av[2 * j + 1]), one, bs[j]);
      }
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  // the groups meet: 1 to 3 leave their piece, the threads add the four in group order
  float* red = &sm[0][0][0][0];               // [3][64][64], exactly the stages
  static_assert(STAGES * 2 * ROWS * TILE >= 3 * TILE * TILE, "reduction fits the stages");
  if (g > 0) {
    float* p = red + (size_t)(g - 1) * TILE * TILE;
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int c = (j < 2 ? 0 : 32) + tx * 4 + (j & 1) * 2;
        *reinterpret_cast<f2*>(p + (ty * 8 + i) * TILE + c) = acc[i][j];
      }
  }
  __syncthreads();
  const long long out_size = (long long)N * K + (want_bias ? N : 0);
  float* out = partial + blockIdx.x * out_size;
  if (g == 0) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int n = n0 + ty * 8 + i;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int c = (j < 2 ? 0 : 32) + tx * 4 + (j & 1) * 2;
        float2 v = unpack2(acc[i][j]);
#pragma unroll
        for (int q = 0; q < 3; ++q) {
          const float2 w = *reinterpret_cast<const float2*>(red + (size_t)q * TILE * TILE + (ty * 8 + i) * TILE + c);
          v.x += w.x; v.y += w.y;
        }
        if (n < N && k0 + c < K) out[(long long)n * K + k0 + c] = v.x;
        if (n < N && k0 + c + 1 < K) out[(long long)n * K + k0 + c + 1] = v.y;
      }
    }
  }
  if (bias) {                                 // the whole block (blockIdx.y): barriers are uniform
    __syncthreads();
    if (tx == 0) {
#pragma unroll
      for (int j = 0; j < 4; ++j) *reinterpret_cast<f2*>(red + g * TILE + ty * 8 + 2 * j) = bs[j];
    }
    __syncthreads();
    if (threadIdx.x < TILE && n0 + threadIdx.x < N) {
      const float* p = red + threadIdx.x;
      out[(long long)N * K + n0 + threadIdx.x] = ((p[0] + p[TILE]) + p[2 * TILE]) + p[3 * TILE];
    }
  }
}

// out[i] = sum over the slices, slice order fixed: 8 warps of a block take every 8th slice of 32 outputs
__global__ void __launch_bounds__(256) f32_dw_reduce_kernel(const float* __restrict__ partial, long long size, int slices,
                                                            float* __restrict__ out) {
  __shared__ float s[8][32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const long long i = (long long)blockIdx.x * 32 + lane;
  float v = 0.f;
  if (i < size) {
#pragma unroll 8
    for (int q = w; q < slices; q += 8) v += partial[q * size + i];
  }
  s[w][lane] = v;
  __syncthreads();
  if (w == 0 && i < size) out[i] = ((s[0][lane] + s[1][lane]) + (s[2][lane] + s[3][lane])) + ((s[4][lane] + s[5][lane]) + (s[6][lane] + s[7][lane]));
}

}  // namespace

// Row slices for (M, N, K): two blocks per SM over all tiles, at least 64 rows a slice.
extern "C" int bf_f32_dw_slices(long long M, int N, int K) {
  const long long tiles = (long long)((N + TILE - 1) / TILE) * ((K + TILE - 1) / TILE);
  long long s = (2 * 148 + tiles - 1) / tiles;
  const long long most = (M + 63) / 64;
  if (s > most) s = most;
  return (int)(s < 1 ? 1 : s);
}

extern "C" int bf_f32_dw(const float* dy, long long lddy, const float* x, long long ldx, long long M, int N, int K, int want_bias,
                         float* partial, float* out, cudaStream_t st) {
  if (M <= 0 || N <= 0 || K <= 0) return (int)cudaErrorInvalidValue;
  const long long tiles = (long long)((N + TILE - 1) / TILE) * ((K + TILE - 1) / TILE);
  if (tiles > 65535) return (int)cudaErrorInvalidValue;
  const int slices = bf_f32_dw_slices(M, N, K);
  const long long rows_per = (M + slices - 1) / slices;
  const bool vec = ((uintptr_t)dy % 16 == 0) && ((uintptr_t)x % 16 == 0) && lddy % 4 == 0 && ldx % 4 == 0 && N % 4 == 0 && K % 4 == 0;
  const dim3 grid((unsigned)slices, (unsigned)tiles);
  if (vec) f32_dw_kernel<4><<<grid, THREADS, 0, st>>>(dy, lddy, x, ldx, M, N, K, rows_per, partial, want_bias);
  else f32_dw_kernel<1><<<grid, THREADS, 0, st>>>(dy, lddy, x, ldx, M, N, K, rows_per, partial, want_bias);
  const long long size = (long long)N * K + (want_bias ? N : 0);
  f32_dw_reduce_kernel<<<(unsigned)((size + 31) / 32), 256, 0, st>>>(partial, size, slices, out);
  return (int)cudaGetLastError();
}
