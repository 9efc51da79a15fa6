// The small per-step work on parameters and their gradients, one launch each for all tensors of a model:
//   bf_weight_copies   16-bit copies of the fp32 weights as the GEMMs take them (as they are, transposed, several packed into one), and
//                      packed fp32 biases
//   bf_gather_f32      gradients of all parameters into a flat bucket, zeros where a parameter has none
// Both are bound by launches, not by bytes (a few MB): a four-layer model took some 60 and 72 launches of PyTorch's operators for them, 4 us
// of host time each.  The tables travel as kernel arguments.
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "bf_kernels.h"

namespace {

constexpr int kItems = 64;              // table entries of one launch (a multiple of launches takes more)

struct CopyTable {
  bf_copy_item item[kItems];
  int first_tile[kItems + 1];           // prefix sums of the items' 32 x 32 tiles
  int n;
};

template <typename F> __device__ __forceinline__ void store_as(void* dst, long long at, float v, F dtype) {
  if (dtype == BF_BF16) static_cast<__nv_bfloat16*>(dst)[at] = __float2bfloat16_rn(v);
  else if (dtype == BF_FP16) static_cast<__half*>(dst)[at] = __float2half_rn(v);
  else static_cast<float*>(dst)[at] = v;
}

__global__ void __launch_bounds__(256) weight_copies_kernel(const __grid_constant__ CopyTable t) {
  __shared__ float s[32][33];
  int k = 0;
  while (k + 1 < t.n && (int)blockIdx.x >= t.first_tile[k + 1]) ++k;
  const bf_copy_item& it = t.item[k];
  const int tile = (int)blockIdx.x - t.first_tile[k], across = (it.cols + 31) / 32;
  const int r0 = tile / across * 32, c0 = tile % across * 32;
  const int x = threadIdx.x & 31, y = threadIdx.x >> 5;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int r = r0 + y + 8 * i, c = c0 + x;
    const float v = r < it.rows && c < it.cols ? it.src[(long long)r * it.ld_src + c] : 0.f;
    if (it.transpose) s[y + 8 * i][x] = v;
    else if (r < it.rows && c < it.cols) store_as(it.dst, (long long)r * it.ld_dst + c, v, it.dtype);
  }
  if (!it.transpose) return;            // the same for the whole block
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int c = c0 + y + 8 * i, r = r0 + x;
    if (r < it.rows && c < it.cols) store_as(it.dst, (long long)c * it.ld_dst + r, s[x][y + 8 * i], it.dtype);
  }
}

struct GatherTable {
  bf_gather_item item[kItems];
  int first_block[kItems + 1];
  int n;
};
constexpr int kGatherBlock = 4096;      // elements a block moves

__global__ void __launch_bounds__(256) gather_f32_kernel(const __grid_constant__ GatherTable t, float* __restrict__ dst) {
  int k = 0;
  while (k + 1 < t.n && (int)blockIdx.x >= t.first_block[k + 1]) ++k;
  const bf_gather_item& it = t.item[k];
  const long long b = (long long)((int)blockIdx.x - t.first_block[k]) * kGatherBlock;
  const long long e = b + kGatherBlock < it.count ? b + kGatherBlock : it.count;
  float* d = dst + it.offset;
  if (((reinterpret_cast<uintptr_t>(it.src) | reinterpret_cast<uintptr_t>(d)) & 15) == 0) {
    long long i = b + 4 * threadIdx.x;
    for (; i + 4 <= e; i += 1024)
      *reinterpret_cast<float4*>(d + i) = it.src ? *reinterpret_cast<const float4*>(it.src + i) : make_float4(0.f, 0.f, 0.f, 0.f);
    for (; i < e; ++i) d[i] = it.src ? it.src[i] : 0.f;           // the thread whose four elements the end cuts
  } else {
    for (long long i = b + threadIdx.x; i < e; i += 256) d[i] = it.src ? it.src[i] : 0.f;
  }
}

}  // namespace

extern "C" int bf_weight_copies(const bf_copy_item* items, int n, cudaStream_t st) {
  for (int at = 0; at < n; at += kItems) {
    CopyTable t;
    t.n = n - at < kItems ? n - at : kItems;
    int tiles = 0;
    for (int k = 0; k < t.n; ++k) {
      const bf_copy_item& it = items[at + k];
      if (it.rows < 1 || it.cols < 1 || !it.src || !it.dst) return (int)cudaErrorInvalidValue;
      t.item[k] = it;
      t.first_tile[k] = tiles;
      tiles += ((it.rows + 31) / 32) * ((it.cols + 31) / 32);
    }
    t.first_tile[t.n] = tiles;
    weight_copies_kernel<<<(unsigned)tiles, 256, 0, st>>>(t);
  }
  return (int)cudaGetLastError();
}

extern "C" int bf_gather_f32(const bf_gather_item* items, int n, float* dst, cudaStream_t st) {
  for (int at = 0; at < n; at += kItems) {
    GatherTable t;
    t.n = n - at < kItems ? n - at : kItems;
    int blocks = 0;
    for (int k = 0; k < t.n; ++k) {
      t.item[k] = items[at + k];
      t.first_block[k] = blocks;
      blocks += (int)((items[at + k].count + kGatherBlock - 1) / kGatherBlock);
    }
    t.first_block[t.n] = blocks;
    if (blocks > 0) gather_f32_kernel<<<(unsigned)blocks, 256, 0, st>>>(t, dst);
  }
  return (int)cudaGetLastError();
}
