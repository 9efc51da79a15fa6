// By-key view of the per-epoch attention graph and the balanced dK/dV work list, built on the device.
//
// The attention graph is a CSR over queries (rowptr, col = key per edge).  The dK/dV pass of the edge attention
// walks it by key, so every epoch needs
//   t_rowptr [n+1]   edges per key (prefix sums),
//   t_eid    [E]     edge positions grouped by key, query order kept inside a key (stable => reproducible sums),
//   t_row    [E]     the query of each of those edges,
//   tasks    [T, 4]  (key, first, end, partial slot) work items of at most `chunk` edges,
//   splits   [S, 3]  (key, first slot, number of slots) for keys cut into several items.
// Steps: row id per edge, LSD radix sort of (key, edge id) pairs over only the bits a node id
// needs (cub::DeviceRadixSort: 3 passes for 2.9 M nodes instead of 8 for 64-bit keys), key boundaries read off the
// sorted keys, and two compaction kernels driven by prefix sums.  The reference has no
// counterpart (its attention runs on COO with scatter reductions, e.g. models/gt_dist_node_level.py:224-262).
#include <cuda_runtime.h>
#include <stdint.h>

#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_scan.cuh>

#include "bf_kernels.h"

namespace {

// erow[e] = row of edge e, iota[e] = e.  A block takes 256 rows; where they hold at most kStaged edges (an attention graph has 5 to 30
// a row) and no row more than 64, its threads mark their rows' edges in shared memory and the block writes them out along memory (a
// thread that marks a row of 4,000 holds the block up: 12 us for 4 k nodes, 3 otherwise).  In other blocks eight lanes
// take a row, and rows above 64 edges (the virtual node's holds every node) are left to the whole block, one after the other.  Bound by the
// bytes written: 15 M edges 83 us with eight lanes a row everywhere, 31 now; 169 k nodes and a row of all of them 44 us with that row on one
// warp, 34 now.
constexpr int kStaged = 8192;
__global__ void __launch_bounds__(256) edge_rows_kernel(const int* __restrict__ rowptr, int n, int* __restrict__ erow, int* __restrict__ iota) {
  __shared__ uint8_t s_row[kStaged];
  const int r0 = blockIdx.x * 256, rows = min(256, n - r0);
  const int b0 = rowptr[r0], b1 = rowptr[r0 + rows];
  const int lane = threadIdx.x & 31;
  int own = 0, own_end = 0;
  if ((int)threadIdx.x < rows) { own = rowptr[r0 + threadIdx.x] - b0; own_end = rowptr[r0 + threadIdx.x + 1] - b0; }
  if (__syncthreads_and(b1 - b0 <= kStaged && own_end - own <= 64)) {
    for (int e = own; e < own_end; ++e) s_row[e] = (uint8_t)threadIdx.x;
    __syncthreads();
    for (int e = threadIdx.x; e < b1 - b0; e += 256) { erow[b0 + e] = r0 + s_row[e]; iota[b0 + e] = b0 + e; }
    return;
  }
  __shared__ int s_wide[256], s_n;
  if (threadIdx.x == 0) s_n = 0;
  __syncthreads();
  for (int r = threadIdx.x >> 3; r < rows; r += 32) {
    const int beg = rowptr[r0 + r], end = rowptr[r0 + r + 1];
    if (end - beg > 64) {
      if ((lane & 7) == 0) s_wide[atomicAdd(&s_n, 1)] = r0 + r;
    } else {
      for (int e = beg + (lane & 7); e < end; e += 8) { erow[e] = r0 + r; iota[e] = e; }
    }
  }
  __syncthreads();
  for (int w = 0; w < s_n; ++w) {
    const int r = s_wide[w];
    const unsigned end = (unsigned)rowptr[r + 1];     // below 2^31: no step past it wraps around
#pragma unroll 4
    for (unsigned e = (unsigned)rowptr[r] + threadIdx.x; e < end; e += 256) { erow[e] = r; iota[e] = (int)e; }
  }
}

// t_rowptr[k] = first position in the sorted key array whose key is >= k: position i is that boundary for every key
// in (keys[i-1], keys[i]] (several when keys without edges lie in between); i = n_edges closes the array.  Four positions a thread
// (15 M edges 51 us with one, 27 now).
__global__ void key_offsets_kernel(const int* __restrict__ keys_sorted, long long n_edges, int n, int* __restrict__ t_rowptr) {
  const long long i0 = 4 * ((long long)blockIdx.x * blockDim.x + threadIdx.x);
  if (i0 > n_edges) return;
  int k[5];
  k[0] = i0 == 0 ? -1 : keys_sorted[i0 - 1];
  if (i0 + 4 <= n_edges) {
    const int4 v = *reinterpret_cast<const int4*>(keys_sorted + i0);
    k[1] = v.x; k[2] = v.y; k[3] = v.z; k[4] = v.w;
  } else {
#pragma unroll
    for (int j = 0; j < 4; ++j) k[j + 1] = i0 + j < n_edges ? keys_sorted[i0 + j] : n;
  }
#pragma unroll
  for (int j = 0; j < 4; ++j)
    if (i0 + j <= n_edges)
      for (int t = k[j] + 1; t <= k[j + 1]; ++t) t_rowptr[t] = (int)(i0 + j);
}

// Four gathers in flight a thread: 15 M edges 94 us with one, 75 now (32 lines a request).
__global__ void gather_rows_kernel(const int* __restrict__ erow, const int* __restrict__ t_eid, long long n_edges,
                                   int* __restrict__ t_row) {
  const long long i0 = 4 * ((long long)blockIdx.x * blockDim.x + threadIdx.x);
  if (i0 + 4 <= n_edges) {
    const int4 e = *reinterpret_cast<const int4*>(t_eid + i0);
    *reinterpret_cast<int4*>(t_row + i0) = make_int4(__ldg(erow + e.x), __ldg(erow + e.y), __ldg(erow + e.z), __ldg(erow + e.w));
  } else {
    for (long long i = i0; i < n_edges; ++i) t_row[i] = erow[t_eid[i]];
  }
}

// Partial slots of every key's items (0: not cut, one item) in the low half and 1 per cut key in the high half, so that one prefix
// sum serves both; rows with more than `min_split` edges are cut.  first[0] = 0 is the start of that sum.
__global__ void task_counts_kernel(const int* __restrict__ t_rowptr, int n, int chunk, int min_split,
                                   unsigned long long* __restrict__ counts, unsigned long long* __restrict__ first,
                                   int* __restrict__ length_key, int* __restrict__ ids) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k == 0) first[0] = 0;
  if (k >= n) return;
  const int deg = t_rowptr[k + 1] - t_rowptr[k];
  const bool cut = deg > min_split;
  counts[k] = cut ? (1ull << 32) | (unsigned)((deg + chunk - 1) / chunk) : 0ull;
  if (length_key != nullptr) {
    length_key[k] = cut ? min_split + 1 : min_split - deg;
    ids[k] = k;
  }
}

// The list starts with the items of all split keys in key order (full-length items: the long work is scheduled first and runs
// side by side in a warp); an item of a split key sits at its partial-slot index.  A lane looks at one key, and the warp writes the
// items of those that are split one key after the other, 32 items at a time (hub keys own thousands).  With `singles` the one item
// of every other key (an empty one too: its zero gradient has to be written) follows behind them in key order.
__global__ void task_fill_kernel(const int* __restrict__ t_rowptr, const unsigned long long* __restrict__ first, int n, int chunk,
                                 int max_tasks, int max_splits, bool singles, int4* __restrict__ tasks, int* __restrict__ splits) {
  const long long gt = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int lane = threadIdx.x & 31;
  int s0 = 0, cnt = 0, split = 0;
  if (gt < n) {
    const unsigned long long f = first[gt];
    s0 = (int)(unsigned)f;
    split = (int)(f >> 32);
    cnt = (int)(unsigned)first[gt + 1] - s0;
    if (singles && cnt == 0) {
      const int at = (int)(unsigned)first[n] + (int)gt - split;
      if (at < max_tasks) tasks[at] = make_int4((int)gt, t_rowptr[gt], t_rowptr[gt + 1], -1);
    }
  }
  unsigned left = __ballot_sync(0xffffffffu, cnt > 0);
  while (left != 0) {
    const int src = __ffs(left) - 1;
    left &= left - 1;
    const int at = __shfl_sync(0xffffffffu, s0, src), m = __shfl_sync(0xffffffffu, cnt, src), s = __shfl_sync(0xffffffffu, split, src);
    const int k = (int)(gt - lane) + src;
    const int beg = t_rowptr[k], end = t_rowptr[k + 1];
    for (int c = lane; c < m && at + c < max_tasks; c += 32) {
      const int b = beg + c * chunk;
      tasks[at + c] = make_int4(k, b, min(b + chunk, end), at + c);
    }
    if (lane == 0 && s < max_splits) { splits[3 * s] = k; splits[3 * s + 1] = at; splits[3 * s + 2] = m; }
  }
}

// The single items, longest first instead (key order among equals): the lane groups of a warp that work on neighbouring items finish
// together.  Sorting 2.9 M keys by their 7-bit length is one radix pass.
__global__ void task_singles_kernel(const int* __restrict__ t_rowptr, const unsigned long long* __restrict__ first,
                                    const int* __restrict__ keys, int n, int max_tasks, int4* __restrict__ tasks) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const unsigned long long total = first[n];
  if (i >= n - (int)(total >> 32)) return;
  const int k = keys[i], at = (int)(unsigned)total + i;
  if (at < max_tasks) tasks[at] = make_int4(k, t_rowptr[k], t_rowptr[k + 1], -1);
}

int bits_for(int n) {
  int b = 1;
  while (b < 31 && (1ll << b) < (long long)n) ++b;
  return b;
}

}  // namespace

// Bytes of scratch `bf_graph_transpose` needs for (n, n_edges); the caller allocates it.
extern "C" size_t bf_graph_transpose_scratch(int n, long long n_edges) {
  size_t sort_bytes = 0;
  cub::DeviceRadixSort::SortPairs(nullptr, sort_bytes, (const int*)nullptr, (int*)nullptr, (const int*)nullptr,
                                  (int*)nullptr, n_edges, 0, bits_for(n));
  // keys_out + iota + erow (rounded up to 256 bytes), then the sort's own temporary storage
  return ((3 * (size_t)n_edges * sizeof(int) + 255) & ~(size_t)255) + ((sort_bytes + 255) & ~(size_t)255) + 256;
}

extern "C" int bf_graph_transpose(const int* rowptr, const int* col, int n, long long n_edges, int* t_rowptr, int* t_row,
                                  int* t_eid, void* scratch, size_t scratch_bytes, cudaStream_t st) {
  if (n_edges == 0) return (int)cudaMemsetAsync(t_rowptr, 0, sizeof(int) * ((size_t)n + 1), st);
  int* keys_out = static_cast<int*>(scratch);
  int* iota = keys_out + n_edges;
  int* erow = iota + n_edges;
  const size_t head = (3 * (size_t)n_edges * sizeof(int) + 255) & ~(size_t)255;
  void* sort_tmp = static_cast<uint8_t*>(scratch) + head;
  size_t sort_bytes = scratch_bytes - head;
  if (((reinterpret_cast<uintptr_t>(t_eid) | reinterpret_cast<uintptr_t>(t_row) | reinterpret_cast<uintptr_t>(scratch)) & 15) != 0)
    return (int)cudaErrorMisalignedAddress;
  const unsigned eb = (unsigned)((n_edges / 4 + 1 + 255) / 256);   // four positions a thread, n_edges itself among them
  edge_rows_kernel<<<(unsigned)(((long long)n + 255) / 256), 256, 0, st>>>(rowptr, n, erow, iota);
  cudaError_t e = cub::DeviceRadixSort::SortPairs(sort_tmp, sort_bytes, col, keys_out, iota, t_eid, n_edges, 0,
                                                  bits_for(n), st);
  if (e != cudaSuccess) return (int)e;
  key_offsets_kernel<<<eb, 256, 0, st>>>(keys_out, n_edges, n, t_rowptr);
  gather_rows_kernel<<<eb, 256, 0, st>>>(erow, t_eid, n_edges, t_row);
  return (int)cudaGetLastError();
}

extern "C" size_t bf_row_tasks_scratch(int n, int singles) {
  size_t tmp = 0;
  cub::DeviceScan::InclusiveSum(nullptr, tmp, (const unsigned long long*)nullptr, (unsigned long long*)nullptr, n);
  size_t arrays = (size_t)n * sizeof(unsigned long long);
  if (singles == 2) {
    size_t sort_bytes = 0;
    cub::DeviceRadixSort::SortPairs(nullptr, sort_bytes, (const int*)nullptr, (int*)nullptr, (const int*)nullptr, (int*)nullptr, n);
    if (sort_bytes > tmp) tmp = sort_bytes;
    arrays += 4 * (size_t)n * sizeof(int);
  }
  return ((arrays + 255) & ~(size_t)255) + ((tmp + 255) & ~(size_t)255) + 256;
}

extern "C" int bf_row_tasks(const int* rowptr, int n, int chunk, int min_split, int singles, int max_tasks, int max_splits,
                            unsigned long long* first, int* tasks, int* splits, void* scratch, size_t scratch_bytes, cudaStream_t st) {
  if (n <= 0 || chunk < 1 || min_split < chunk) return (int)cudaErrorInvalidValue;
  // scratch: counts [n]; sorted singles: length keys, their sorted copy, ids and sorted ids [n] each; temporary storage of CUB
  unsigned long long* counts = static_cast<unsigned long long*>(scratch);
  int* key_in = reinterpret_cast<int*>(counts + n);
  int *key_out = key_in + n, *ids = key_out + n, *by_length = ids + n;
  const size_t arrays = (size_t)n * sizeof(unsigned long long) + (singles == 2 ? 4 * (size_t)n * sizeof(int) : 0);
  const size_t head = (arrays + 255) & ~(size_t)255;
  void* tmp = static_cast<uint8_t*>(scratch) + head;
  const unsigned blocks = (unsigned)(((long long)n + 255) / 256);
  task_counts_kernel<<<blocks, 256, 0, st>>>(rowptr, n, chunk, min_split, counts, first, singles == 2 ? key_in : nullptr, ids);
  size_t bytes = scratch_bytes - head;
  cudaError_t e = cub::DeviceScan::InclusiveSum(tmp, bytes, counts, first + 1, n, st);
  if (e != cudaSuccess) return (int)e;
  int4* out = reinterpret_cast<int4*>(tasks);
  task_fill_kernel<<<blocks, 256, 0, st>>>(rowptr, first, n, chunk, max_tasks, max_splits, singles == 1, out, splits);
  if (singles == 2) {
    bytes = scratch_bytes - head;
    e = cub::DeviceRadixSort::SortPairs(tmp, bytes, key_in, key_out, ids, by_length, n, 0, bits_for(min_split + 2), st);
    if (e != cudaSuccess) return (int)e;
    task_singles_kernel<<<blocks, 256, 0, st>>>(rowptr, first, by_length, n, max_tasks, out);
  }
  return (int)cudaGetLastError();
}
