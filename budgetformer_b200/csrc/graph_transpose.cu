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

// erow[e] = row of edge e, iota[e] = e.  Eight lanes per row (an attention graph holds 5 to 30 edges a row); rows above 64 edges
// (the virtual node's holds every node) are left to the whole warp, one after the other.
__global__ void edge_rows_kernel(const int* __restrict__ rowptr, int n, int* __restrict__ erow, int* __restrict__ iota) {
  const long long gt = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long row = gt >> 3;
  const int lane = threadIdx.x & 31;
  int beg = 0, end = 0;
  if (row < n) { beg = rowptr[row]; end = rowptr[row + 1]; }
  const bool wide = end - beg > 64;
  if (!wide)
    for (int e = beg + (lane & 7); e < end; e += 8) { erow[e] = (int)row; iota[e] = e; }
  unsigned left = __ballot_sync(0xffffffffu, wide && (lane & 7) == 0);
  while (left != 0) {
    const int src = __ffs(left) - 1;
    left &= left - 1;
    const int b = __shfl_sync(0xffffffffu, beg, src), e1 = __shfl_sync(0xffffffffu, end, src);
    const int r = (int)((gt >> 5) * 4 + (src >> 3));
    for (int e = b + lane; e < e1; e += 32) { erow[e] = r; iota[e] = e; }
  }
}

// t_rowptr[k] = first position in the sorted key array whose key is >= k: position i is that boundary for every key
// in (keys[i-1], keys[i]] (several when keys without edges lie in between); i = n_edges closes the array.
__global__ void key_offsets_kernel(const int* __restrict__ keys_sorted, long long n_edges, int n, int* __restrict__ t_rowptr) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i > n_edges) return;
  const int prev = i == 0 ? -1 : keys_sorted[i - 1];
  const int cur = i == n_edges ? n : keys_sorted[i];
  for (int k = prev + 1; k <= cur; ++k) t_rowptr[k] = (int)i;
}

__global__ void gather_rows_kernel(const int* __restrict__ erow, const int* __restrict__ t_eid, long long n_edges,
                                   int* __restrict__ t_row) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n_edges) t_row[i] = erow[t_eid[i]];
}

// items per key (at least one, so that keys without edges still get their zero gradient written) and partial slots; only
// rows with more than `min_split` edges are cut
__global__ void task_counts_kernel(const int* __restrict__ t_rowptr, int n, int chunk, int min_split, int* __restrict__ n_items,
                                   int* __restrict__ n_slots, int* __restrict__ is_split, int* __restrict__ length_key,
                                   int* __restrict__ ids) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  const int deg = t_rowptr[k + 1] - t_rowptr[k];
  const int c = deg <= min_split ? 1 : (deg + chunk - 1) / chunk;
  n_items[k] = c;
  n_slots[k] = c > 1 ? c : 0;
  is_split[k] = c > 1 ? 1 : 0;
  if (length_key != nullptr) {
    length_key[k] = c > 1 ? min_split + 1 : min_split - deg;
    ids[k] = k;
  }
}

// The list starts with the items of all split keys in key order (full-length items: the long work is scheduled first and runs
// side by side in a warp); an item of a split key sits at its partial-slot index.  A lane looks at one key, and the warp writes the
// items of those that are split one key after the other, 32 items at a time (hub keys own thousands).
__global__ void task_fill_kernel(const int* __restrict__ t_rowptr, const int* __restrict__ slot_first,
                                 const int* __restrict__ split_first, int n, int chunk, int max_tasks, int max_splits,
                                 int4* __restrict__ tasks, int* __restrict__ splits) {
  const long long gt = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int lane = threadIdx.x & 31;
  int s0 = 0, cnt = 0;
  if (gt < n) { s0 = slot_first[gt]; cnt = slot_first[gt + 1] - s0; }
  unsigned left = __ballot_sync(0xffffffffu, cnt > 0);
  while (left != 0) {
    const int src = __ffs(left) - 1;
    left &= left - 1;
    const int first = __shfl_sync(0xffffffffu, s0, src), m = __shfl_sync(0xffffffffu, cnt, src);
    const int k = (int)(gt - lane) + src;
    const int beg = t_rowptr[k], end = t_rowptr[k + 1];
    for (int c = lane; c < m && first + c < max_tasks; c += 32) {
      const int b = beg + c * chunk;
      tasks[first + c] = make_int4(k, b, min(b + chunk, end), first + c);
    }
    const int s = split_first[k];
    if (lane == 0 && s < max_splits) { splits[3 * s] = k; splits[3 * s + 1] = first; splits[3 * s + 2] = m; }
  }
}

// Behind them the single item of every other key, longest first (key order among equals): the lane groups of a warp that work
// on neighbouring items finish together.  Sorting 2.9 M keys by their 7-bit length is one radix pass; a thread per key instead
// of a warp writes the list in a tenth of the time.
__global__ void task_singles_kernel(const int* __restrict__ t_rowptr, const int* __restrict__ slot_first,
                                    const int* __restrict__ split_first, const int* __restrict__ keys, int n, int max_tasks,
                                    int4* __restrict__ tasks) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n - split_first[n]) return;
  const int k = keys[i], at = slot_first[n] + i;
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
  const unsigned eb = (unsigned)((n_edges + 255) / 256);
  edge_rows_kernel<<<(unsigned)(((long long)n * 8 + 255) / 256), 256, 0, st>>>(rowptr, n, erow, iota);
  cudaError_t e = cub::DeviceRadixSort::SortPairs(sort_tmp, sort_bytes, col, keys_out, iota, t_eid, n_edges, 0,
                                                  bits_for(n), st);
  if (e != cudaSuccess) return (int)e;
  key_offsets_kernel<<<(unsigned)((n_edges + 1 + 255) / 256), 256, 0, st>>>(keys_out, n_edges, n, t_rowptr);
  gather_rows_kernel<<<eb, 256, 0, st>>>(erow, t_eid, n_edges, t_row);
  return (int)cudaGetLastError();
}

// Phase 1 of the work list: per-key counts and their exclusive prefix sums ([n+1] each, last element = total), and with
// `by_length` the keys sorted by the length of their row, longest first, split keys behind all others ([n]).
extern "C" int bf_kv_task_counts(const int* t_rowptr, int n, int chunk, int min_split, int* item_first, int* slot_first,
                                 int* split_first, int* by_length, void* scratch, size_t scratch_bytes, cudaStream_t st) {
  // scratch: six int[n] arrays (three counts; length keys, their sorted copy, ids) followed by the temporary storage of CUB
  int* n_items = static_cast<int*>(scratch);
  int* n_slots = n_items + n;
  int* is_split = n_slots + n;
  int* key_in = is_split + n;
  int* key_out = key_in + n;
  int* ids = key_out + n;
  const size_t head = (6 * (size_t)n * sizeof(int) + 255) & ~(size_t)255;
  void* tmp = static_cast<uint8_t*>(scratch) + head;
  size_t tmp_bytes = scratch_bytes - head;
  if (chunk < 1 || min_split < chunk) return (int)cudaErrorInvalidValue;
  task_counts_kernel<<<(n + 255) / 256, 256, 0, st>>>(t_rowptr, n, chunk, min_split, n_items, n_slots, is_split,
                                                      by_length != nullptr ? key_in : nullptr, ids);
  cudaError_t e;
  // exclusive prefix sums with the total appended: out[0] = 0, out[1..n] = inclusive sums
  for (int which = 0; which < 3; ++which) {
    const int* in = which == 0 ? n_items : which == 1 ? n_slots : is_split;
    int* out = which == 0 ? item_first : which == 1 ? slot_first : split_first;
    e = cudaMemsetAsync(out, 0, sizeof(int), st);
    if (e != cudaSuccess) return (int)e;
    size_t bytes = tmp_bytes;
    e = cub::DeviceScan::InclusiveSum(tmp, bytes, in, out + 1, n, st);
    if (e != cudaSuccess) return (int)e;
  }
  if (by_length != nullptr) {
    size_t bytes = tmp_bytes;
    e = cub::DeviceRadixSort::SortPairs(tmp, bytes, key_in, key_out, ids, by_length, n, 0, bits_for(min_split + 2), st);
    if (e != cudaSuccess) return (int)e;
  }
  return (int)cudaGetLastError();
}

extern "C" size_t bf_kv_task_scratch(int n) {
  size_t scan_bytes = 0, sort_bytes = 0;
  cub::DeviceScan::InclusiveSum(nullptr, scan_bytes, (const int*)nullptr, (int*)nullptr, n);
  cub::DeviceRadixSort::SortPairs(nullptr, sort_bytes, (const int*)nullptr, (int*)nullptr, (const int*)nullptr, (int*)nullptr, n);
  const size_t tmp = scan_bytes > sort_bytes ? scan_bytes : sort_bytes;
  return ((6 * (size_t)n * sizeof(int) + 255) & ~(size_t)255) + ((tmp + 255) & ~(size_t)255) + 256;
}

// Phase 2: write the items and the split list.  The totals are read on the device, so the caller can read them back last: then
// the list is complete when the host knows its length, whatever stream uses it.  With `by_length` (of phase 1) the keys that are
// not split get their single items; without it they get none.
extern "C" int bf_kv_task_fill(const int* t_rowptr, const int* slot_first, const int* split_first, const int* by_length, int n,
                               int chunk, int max_tasks, int max_splits, int* tasks, int* splits, cudaStream_t st) {
  if (n <= 0) return 0;
  int4* out = reinterpret_cast<int4*>(tasks);
  const unsigned blocks = (unsigned)(((long long)n + 255) / 256);
  if (max_splits > 0) task_fill_kernel<<<blocks, 256, 0, st>>>(t_rowptr, slot_first, split_first, n, chunk, max_tasks, max_splits, out, splits);
  if (by_length != nullptr) task_singles_kernel<<<blocks, 256, 0, st>>>(t_rowptr, slot_first, split_first, by_length, n, max_tasks, out);
  return (int)cudaGetLastError();
}
