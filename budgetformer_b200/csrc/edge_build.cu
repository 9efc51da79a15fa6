// Per-epoch attention-graph construction on the GPU: one thread per query node (for few queries several lanes, pick_form).
//   1. real edges: the thread streams the query's in-edge row and keeps the smallest (hash, src) in a sorted register list;
//      rows of more than kWideRow edges are ranked by the whole warp, rows of more than BF_BUILD_HUB_DEGREE by a cluster of
//      blocks ahead of this kernel (no global sort);
//   2. random walks: the same thread runs the query's walks, two or eight at a time (Philox counter RNG, dead ends stay), and ranks the
//      W*L candidates into a second list;
//   3. merge: sorted unique union by key id (Exphormer: typed concatenation + self loop), staged in shared memory and
//      written as a fixed-width row [cap] plus a count; ell_to_csr compacts rows after a prefix sum.
// Replaces the reference's argsort / scatter_reduce rounds / coalesce pipeline
// (utils/fullgraph_sp_support.py:975-1192, gt_sp/utils.py:1198-1248, :877-887) and is bit-identical
// to cpu/edge_builder.cpp and graph/builder_spec.py.
//
// What bounds it: instructions.  A row holds some 5 real candidates and W*L walk candidates, each a hash, a 10-round Philox and an
// insertion of a few dozen instructions on one query's own data; with a group of lanes per query most lanes of those steps idle.
// Selection, us, before (eight lanes, above budgets of 8 a warp per query) and now: 2.9 M nodes, 4 + 4, walks 2 x 4: 1471 / 224; 612 k nodes
// of some 50 in-edges, 8 + 8, 4 x 6: 1135 / 338; 392 k nodes of 170, 16 + 16: 1452 / 287; 1 M nodes, 3 + 11, 6 x 8: 4122 / 659; 5 k nodes 9.0 / 8.7
// (the walks' chain of reads).  Few queries leave most of the GPU idle that way: see pick_form.
#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <cub/device/device_scan.cuh>

#include "bf_kernels.h"
#include "edge_spec.h"

namespace {

namespace cg = cooperative_groups;

constexpr uint64_t kInf = ~0ull;
constexpr uint32_t kNone = ~0u;               // no node: ids are below 2^31
constexpr unsigned kAll = 0xffffffffu;

// Insert the warp's candidates (valid, comp) into the sorted list that lane i holds the i-th smallest composite of (k <= 32).
__device__ __forceinline__ void warp_insert(uint64_t& list, int k, bool valid, uint64_t comp, int lane) {
  const unsigned kmask = k >= 32 ? kAll : ((1u << k) - 1u);
  for (int guard = 0; guard <= 32; ++guard) {
    const uint64_t kth = __shfl_sync(kAll, list, k - 1);
    const unsigned ball = __ballot_sync(kAll, valid && comp < kth);
    if (ball == 0) break;
    const int src_lane = __ffs(ball) - 1;
    const uint64_t c = __shfl_sync(kAll, comp, src_lane);
    const int p = __popc(__ballot_sync(kAll, list <= c) & kmask);
    const uint64_t up = __shfl_up_sync(kAll, list, 1);
    if (lane == p) list = c;
    else if (lane > p && lane < k) list = up;
    if (lane == src_lane) valid = false;
  }
}

// Composites below this hold the `want` smallest of `deg` candidates with room to spare, as far as their hashes are spread evenly:
// whoever filters by it counts what is left and starts over without it where that is too little.  `room` pass on average, with a
// deviation of its root: 48 at most, so that of kPassed slots neither more are needed nor fewer than 32 filled but in one or two rows of a hundred.
constexpr int kPassed = 64;                       // candidates below rank_bound that a warp sorts
__device__ __forceinline__ uint64_t rank_bound(int want, int deg) {
  const uint64_t room = (uint64_t)min(want + 4 * (int)ceilf(sqrtf((float)want)) + 4, 48);
  const uint64_t h = (room << 31) / (uint64_t)deg;
  return h >= (1ull << 31) ? kInf : h << 32;
}

// one thread's sorted list of the K smallest composites
template <int K> __device__ __forceinline__ void list_take(uint64_t (&list)[K], uint64_t c) {
  if (c >= list[K - 1]) return;
  bool below[K];
#pragma unroll
  for (int i = 0; i < K; ++i) below[i] = c < list[i];
#pragma unroll
  for (int i = K - 1; i > 0; --i) list[i] = below[i - 1] ? list[i - 1] : (below[i] ? c : list[i]);
  list[0] = below[0] ? c : list[0];
}

// ascending sort of N values in registers: Batcher's odd-even merge sort (Knuth, The Art of Computer Programming 3, 5.2.2)
template <int N, int P, int D> __device__ __forceinline__ void sort_pass(uint32_t (&x)[N]) {
#pragma unroll
  for (int i = 0; i + D < N; ++i)
    if (i >= D % P && (i - D % P) / D % 2 == 0 && i / (2 * P) == (i + D) / (2 * P)) {
      const uint32_t lo = min(x[i], x[i + D]), hi = max(x[i], x[i + D]);
      x[i] = lo; x[i + D] = hi;
    }
  if constexpr (D > 1) sort_pass<N, P, D / 2>(x);
  else if constexpr (2 * P < N) sort_pass<N, 2 * P, 2 * P>(x);
}
template <int N> __device__ __forceinline__ void sort_values(uint32_t (&x)[N]) { sort_pass<N, 1, 1>(x); }

struct BuildArgs {
  const int *in_rowptr, *in_src, *out_rowptr, *out_col;
  int n;
  int row_begin;       // first query of this launch; rows are stored at index (query - row_begin)
  int b_real, b_rw, walks, walk_len;
  long long seed;
  int cap;
  int* ell_col;        // [n, cap]
  uint8_t* ell_type;   // [n, cap] or null
  int* ell_cnt;        // [n]
  unsigned long long* totals;  // [2] selected real / rw edges (with multiplicity)
  const int* hub_rows;         // ascending ids of queries with more than BF_BUILD_HUB_DEGREE in-edges, or null
  int n_hub;
  unsigned long long* hub_top; // [n_hub, 32] ranked real candidates of those queries
};

// Real-edge ranking of the longest rows: a cluster of eight blocks per listed query.  Each of its 64 warps keeps the b_real smallest
// composites of its share of the row that are below the row's rank_bound (about none of them), the blocks' first warps merge those
// lists, and the first block's the eight results.  Where the bound left too few the pass is repeated without it.  The b_real smallest
// of a multiset do not depend on the order of insertion, so the result equals the stream of one thread.
// A row's time is the latency of its share: at 612 k nodes the longest has 10^5 edges, and one block
// took 422 us for what a cluster does in 49 (392 k nodes, 66 M edges: 782 / 55).
constexpr int kHubBlocks = 8, kHubWarps = 8, kHubLoads = 4;
__global__ void __cluster_dims__(kHubBlocks, 1, 1) __launch_bounds__(kHubWarps * 32) budget_hub_topk_kernel(BuildArgs a) {
  __shared__ uint64_t s_list[kHubWarps][32];
  __shared__ uint64_t s_block[32];
  cg::cluster_group cluster = cg::this_cluster();
  const int part = (int)cluster.block_rank();
  const int hub = blockIdx.x / kHubBlocks;
  const int row = a.hub_rows[hub];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const bool mine = row >= a.row_begin && (long long)row < (long long)a.row_begin + a.n;   // uniform over the cluster
  if (mine) {
    const int beg = a.in_rowptr[row], end = a.in_rowptr[row + 1];
    const int64_t rs = a.seed + BF_REAL_SEED_OFFSET;
    uint64_t bound = rank_bound(a.b_real, end - beg);
    while (true) {
      uint64_t list = kInf;
      const long long step = (long long)kHubBlocks * kHubWarps * 32 * kHubLoads;
      for (long long base = (long long)beg + (long long)(part * kHubWarps + warp) * 32 * kHubLoads; base < end; base += step) {
        uint64_t c[kHubLoads];
        bool any = false;
#pragma unroll
        for (int j = 0; j < kHubLoads; ++j) {
          const long long e = base + j * 32 + lane;
          c[j] = e < end ? bf_edge_composite((uint32_t)__ldg(a.in_src + e), (uint32_t)row, rs) : kInf;
        }
#pragma unroll
        for (int j = 0; j < kHubLoads; ++j) any |= c[j] < bound;
        if (__any_sync(kAll, any)) {
#pragma unroll
          for (int j = 0; j < kHubLoads; ++j) warp_insert(list, a.b_real, c[j] < bound, c[j], lane);
        }
      }
      s_list[warp][lane] = lane < a.b_real ? list : kInf;
      __syncthreads();
      if (warp == 0) {
        for (int w = 1; w < kHubWarps; ++w) {
          const uint64_t c = s_list[w][lane];
          warp_insert(list, a.b_real, c != kInf, c, lane);
        }
        s_block[lane] = lane < a.b_real ? list : kInf;
      }
      cluster.sync();
      uint64_t got[kHubBlocks];                   // every block merges all eight, so that all of them see whether the pass sufficed
      if (warp == 0) {
#pragma unroll
        for (int b = 0; b < kHubBlocks; ++b) got[b] = cluster.map_shared_rank(s_block, b)[lane];
        list = kInf;
#pragma unroll
        for (int b = 0; b < kHubBlocks; ++b) warp_insert(list, a.b_real, got[b] != kInf, got[b], lane);
        s_list[0][lane] = list;
      }
      cluster.sync();                             // also: no block leaves or starts over while another reads its list
      if (bound == kInf || s_list[0][a.b_real - 1] != kInf) {
        if (part == 0 && warp == 0) a.hub_top[(long long)hub * 32 + lane] = lane < a.b_real ? list : kInf;
        break;
      }
      bound = kInf;
      __syncthreads();
    }
  }
}

// Rows of more than kWideRow edges may be ranked by the whole warp instead of their threads.  A lane that is alone with its long row holds
// the warp up for some 20 + 6 K instructions an edge (K: list length; some lane inserts in nearly every step); the warp takes about 250 a
// row and 25 for 32 edges.  So a few long rows among short ones go to the warp, and so do rows of some hundred edges; a warp
// whose rows all have 33 to 100 keeps them (100 k rows of 60, 8 + 4: 41 us, 113 when all went to the warp).
constexpr int kWideRow = 32;
constexpr int kSelectThreads = 128, kSelectWarps = kSelectThreads / 32;

// The b_real smallest composites of one row, by all lanes: what passes rank_bound is collected in shared memory and ranked by
// counting; s_top[0 .. b_real) holds them in order afterwards.
__device__ __forceinline__ void warp_rank_row(const BuildArgs& a, uint32_t q, int beg, int end, uint64_t* s_pass, uint64_t* s_top, int lane) {
  const int64_t rs = a.seed + BF_REAL_SEED_OFFSET;
  const uint64_t bound = rank_bound(a.b_real, end - beg);
  int passed = 0;
  for (unsigned base = (unsigned)beg; base < (unsigned)end; base += 128) {      // below 2^31: no step past it wraps around
    uint64_t c[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const unsigned e = base + j * 32 + lane;
      c[j] = e < (unsigned)end ? bf_edge_composite((uint32_t)__ldg(a.in_src + e), q, rs) : kInf;
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const bool take = c[j] < bound;
      const unsigned ball = __ballot_sync(kAll, take);
      const int at = passed + __popc(ball & ((1u << lane) - 1u));
      if (take && at < kPassed) s_pass[at] = c[j];
      passed += __popc(ball);
    }
  }
  __syncwarp();
  if (passed >= a.b_real && passed <= kPassed) {
    const uint64_t x0 = lane < passed ? s_pass[lane] : kInf, x1 = lane + 32 < passed ? s_pass[lane + 32] : kInf;
    int r0 = 0, r1 = 0;
    for (int t = 0; t < passed; ++t) {
      const uint64_t y = s_pass[t];
      r0 += (y < x0 || (y == x0 && t < lane)) ? 1 : 0;
      r1 += (y < x1 || (y == x1 && t < lane + 32)) ? 1 : 0;
    }
    if (lane < passed && r0 < a.b_real) s_top[r0] = x0;
    if (lane + 32 < passed && r1 < a.b_real) s_top[r1] = x1;
  } else {                                        // hashes in lumps (repeated sources): rank all of them
    uint64_t list = kInf;
    for (unsigned base = (unsigned)beg; base < (unsigned)end; base += 32) {
      const unsigned e = base + lane;
      const bool in = e < (unsigned)end;
      warp_insert(list, a.b_real, in, in ? bf_edge_composite((uint32_t)__ldg(a.in_src + e), q, rs) : kInf, lane);
    }
    if (lane < a.b_real) s_top[lane] = list;
  }
  __syncwarp();
}

// place of query v among the rows that budget_hub_topk_kernel has ranked, -1: not one of them
__device__ __forceinline__ int hub_index(const BuildArgs& a, int v, int deg) {
  if (a.n_hub <= 0 || deg <= BF_BUILD_HUB_DEGREE) return -1;
  int lo = 0, hi = a.n_hub - 1;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (a.hub_rows[mid] < v) lo = mid + 1; else hi = mid;
  }
  return a.hub_rows[lo] == v ? lo : -1;
}

// K: list length, the larger budget rounded up to 4, 8, 16 or 32; W: walks that a thread has under way
template <int K, bool TYPED, int W>
__global__ void __launch_bounds__(kSelectThreads) budget_select_kernel(BuildArgs a) {
  extern __shared__ int s_rows[];                 // [kSelectThreads][cap | 1]: odd pitch, lanes of a column in different banks
  __shared__ uint64_t s_pass[kSelectWarps][kPassed], s_top[kSelectWarps][32];
  __shared__ unsigned s_tot[2];
  __shared__ unsigned short s_cnt[kSelectThreads];
  __shared__ uint8_t s_typed[TYPED ? kSelectThreads : 1][2];   // real and walk edges of a row
  if (threadIdx.x < 2) s_tot[threadIdx.x] = 0;
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const long long slot = (long long)blockIdx.x * kSelectThreads + threadIdx.x;         // row of the output
  const bool live = slot < a.n;
  const int v = live ? (int)(slot + a.row_begin) : 0;                                  // query node
  const uint32_t q = (uint32_t)v;
  uint64_t list[K];
#pragma unroll
  for (int i = 0; i < K; ++i) list[i] = kInf;
  // ---- real edges ----
  int beg = 0, deg = 0;
  if (live && a.b_real > 0) { beg = a.in_rowptr[v]; deg = a.in_rowptr[v + 1] - beg; }
  const int r_cnt = min(deg, a.b_real), hub = hub_index(a, v, deg);
  if (hub >= 0) {
#pragma unroll
    for (int i = 0; i < K; ++i)
      if (i < a.b_real) list[i] = (uint64_t)a.hub_top[(long long)hub * 32 + i];
  }
  bool wide = deg > kWideRow && hub < 0;
  if (__any_sync(kAll, wide)) {
    const int len = wide ? min(deg, 1 << 20) : 0, rows = __popc(__ballot_sync(kAll, wide));
    const int most = (int)__reduce_max_sync(kAll, (unsigned)len), sum = (int)__reduce_add_sync(kAll, (unsigned)len);
    wide = wide && 250 * rows + sum < (most - kWideRow) * (20 + 6 * K);
  }
  if (!wide && hub < 0) {
    const int64_t rs = a.seed + BF_REAL_SEED_OFFSET;
    for (unsigned e = 0; e < (unsigned)deg; e += 4) {
      uint32_t src[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) src[j] = e + j < (unsigned)deg ? (uint32_t)__ldg(a.in_src + beg + (int)(e + j)) : kNone;
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (src[j] != kNone) list_take<K>(list, bf_edge_composite(src[j], q, rs));
    }
  }
  __syncwarp();
  unsigned left = __ballot_sync(kAll, wide);
  while (left != 0) {
    const int owner = __ffs(left) - 1;
    left &= left - 1;
    const int b = __shfl_sync(kAll, beg, owner), d = __shfl_sync(kAll, deg, owner), row = __shfl_sync(kAll, v, owner);
    warp_rank_row(a, (uint32_t)row, b, b + d, s_pass[warp], s_top[warp], lane);
    if (lane == owner) {
#pragma unroll
      for (int i = 0; i < K; ++i)
        if (i < a.b_real) list[i] = s_top[warp][i];
    }
    __syncwarp();
  }
  uint32_t id[2 * K];
#pragma unroll
  for (int i = 0; i < K; ++i) { id[i] = i < r_cnt ? (uint32_t)list[i] : kNone; list[i] = kInf; }
  // ---- random walks, W at a time so that their dependent reads overlap ----
  int w_cnt = 0;
  if (live && a.b_rw > 0 && a.walks > 0 && a.walk_len > 0) {
    const int64_t ws = a.seed + BF_RW_SEED_OFFSET;
    for (int w = 0; w < a.walks; w += W) {
      const uint64_t walk_id = (uint64_t)v * (uint64_t)a.walks + (uint64_t)w;
      int cur[W];
#pragma unroll
      for (int t = 0; t < W; ++t) cur[t] = v;
      for (int d = 1; d <= a.walk_len; ++d) {
        int ob[W], oe[W], next[W];
#pragma unroll
        for (int t = 0; t < W; ++t) {
          ob[t] = oe[t] = 0;
          if (W == 2 || w + t < a.walks) { ob[t] = a.out_rowptr[cur[t]]; oe[t] = a.out_rowptr[cur[t] + 1]; }
        }
#pragma unroll
        for (int t = 0; t < W; ++t) {
          const uint32_t n_out = (uint32_t)(oe[t] - ob[t]);
          next[t] = cur[t];
          if (n_out > 0)
            next[t] = __ldg(a.out_col + ob[t] + (int)bf_mulhi32(bf_walk_uniform32(walk_id + t, (uint32_t)d, (uint64_t)a.seed), n_out));
        }
#pragma unroll
        for (int t = 0; t < W; ++t) {
          if ((t == 0 || w + t < a.walks) && (d == 1 || next[t] != cur[t])) {
            ++w_cnt;
            list_take<K>(list, bf_edge_composite((uint32_t)next[t], q, ws));
          }
          cur[t] = next[t];
        }
      }
    }
    w_cnt = min(w_cnt, a.b_rw);
  }
#pragma unroll
  for (int i = 0; i < K; ++i) id[K + i] = i < w_cnt ? (uint32_t)list[i] : kNone;
  // ---- merge ----
  const int pitch = a.cap | 1;
  int* row = s_rows + threadIdx.x * pitch;
  int total = 0;
  if (TYPED) {
    uint32_t side[K];
#pragma unroll
    for (int i = 0; i < K; ++i) side[i] = id[i];
    sort_values<K>(side);
#pragma unroll
    for (int i = 0; i < K; ++i)
      if (i < r_cnt) row[i] = (int)side[i];
#pragma unroll
    for (int i = 0; i < K; ++i) side[i] = id[K + i];
    sort_values<K>(side);
#pragma unroll
    for (int i = 0; i < K; ++i)
      if (i < w_cnt) row[r_cnt + i] = (int)side[i];
    row[r_cnt + w_cnt] = v;
    total = r_cnt + w_cnt + 1;
    s_typed[threadIdx.x][0] = (uint8_t)r_cnt;
    s_typed[threadIdx.x][1] = (uint8_t)w_cnt;
  } else {
    sort_values<2 * K>(id);
    uint32_t prev = kNone;
#pragma unroll
    for (int i = 0; i < 2 * K; ++i) {
      if (id[i] != kNone && id[i] != prev) row[total++] = (int)id[i];
      prev = id[i];
    }
  }
  if (live) a.ell_cnt[slot] = total;
  s_cnt[threadIdx.x] = (unsigned short)(live ? total : 0);
  const unsigned sum_r = __reduce_add_sync(kAll, live ? (unsigned)r_cnt : 0u), sum_w = __reduce_add_sync(kAll, (unsigned)w_cnt);
  if (lane == 0) { atomicAdd(&s_tot[0], sum_r); atomicAdd(&s_tot[1], sum_w); }
  __syncwarp();
  // ---- the warp's 32 rows are one contiguous piece of the output ----
  const long long out0 = (slot - lane) * (long long)a.cap;
  const unsigned inv = (1u << 20) / (unsigned)a.cap + 1u;      // i / cap for i < 32 * cap <= 2080: i * (inv * cap - 2^20) < 2^20
  for (int i = lane; i < 32 * a.cap; i += 32) {
    const int r = (int)(((unsigned)i * inv) >> 20), c = i - r * a.cap, at = warp * 32 + r;
    if (c < s_cnt[at]) {
      a.ell_col[out0 + i] = s_rows[at * pitch + c];
      if (TYPED) a.ell_type[out0 + i] = (uint8_t)(c >= s_typed[at][0] && c < s_typed[at][0] + s_typed[at][1] ? 1 : 0);
    }
  }
  __syncthreads();
  if (threadIdx.x < 2 && s_tot[threadIdx.x]) atomicAdd(a.totals + threadIdx.x, (unsigned long long)s_tot[threadIdx.x]);
}

// L lanes (8 or 32) a query: lane w runs walk w, and the lists lie one entry a lane.  Most lanes idle in most steps, but a query takes the
// latency of one walk and of its row's chunks only: for few queries, whose threads would not fill the GPU (see pick_form).  Groups of one
// warp go their own ways; every warp-wide operation names the group's lanes.
template <int L> __device__ __forceinline__ unsigned group_mask(int lane) { return L == 32 ? kAll : ((1u << (L & 31)) - 1u) << (lane & ~(L - 1)); }
template <int L> __device__ __forceinline__ unsigned group_ballot(unsigned gm, int lane, bool pred) {
  const unsigned b = __ballot_sync(gm, pred);
  return L == 32 ? b : (b >> (lane & ~(L - 1))) & ((1u << (L & 31)) - 1u);
}
__device__ __forceinline__ uint64_t exchange(uint64_t v, int j, bool want_min, unsigned gm) {
  const uint64_t o = __shfl_xor_sync(gm, v, j);
  return ((o < v) == want_min) ? o : v;
}
// The k smallest of the sorted list and one candidate a lane (kInf: none) into the list.  Eight lanes sort the candidates and merge them
// bitonically, ten exchanges for all groups of the warp alike; a warp inserts one after the other, since few of its candidates still matter.
template <int L> __device__ __forceinline__ void group_take(uint64_t& list, int k, uint64_t c, int gl, unsigned gm, int lane) {
  if constexpr (L == 32) {
    warp_insert(list, k, c != kInf, c, lane);
  } else {
    const uint64_t kth = __shfl_sync(gm, list, k - 1, L);
    if (group_ballot<L>(gm, lane, c < kth) == 0) return;
#pragma unroll
    for (int m = 2; m <= L; m <<= 1)
#pragma unroll
      for (int j = m >> 1; j > 0; j >>= 1) c = exchange(c, j, ((gl & j) == 0) != ((gl & m) != 0 && m < L), gm);
    const uint64_t rev = __shfl_sync(gm, c, L - 1 - gl, L);
    uint64_t v = rev < list ? rev : list;         // the L smallest of both, bitonic
#pragma unroll
    for (int j = L >> 1; j > 0; j >>= 1) v = exchange(v, j, (gl & j) == 0, gm);
    list = v;
  }
}

template <int L>
__global__ void __launch_bounds__(256) budget_select_group_kernel(BuildArgs a, bool typed) {
  __shared__ unsigned s_tot[2];
  if (threadIdx.x < 2) s_tot[threadIdx.x] = 0;
  __syncthreads();
  const int lane = threadIdx.x & 31, gl = lane & (L - 1);
  const unsigned gm = group_mask<L>(lane);
  const long long slot = ((long long)blockIdx.x * blockDim.x + threadIdx.x) / L;       // row of the output
  if (slot < a.n) {
    const int v = (int)(slot + a.row_begin);
    const uint32_t q = (uint32_t)v;
    // ---- real edges ----
    uint64_t real = kInf, walked = kInf;
    int r_cnt = 0;
    if (a.b_real > 0) {
      const int beg = a.in_rowptr[v], deg = a.in_rowptr[v + 1] - beg, hub = hub_index(a, v, deg);
      if (hub >= 0) {
        real = gl < a.b_real ? (uint64_t)a.hub_top[(long long)hub * 32 + gl] : kInf;
      } else {
        const int64_t rs = a.seed + BF_REAL_SEED_OFFSET;
        for (unsigned e0 = 0; e0 < (unsigned)deg; e0 += L) {
          const unsigned e = e0 + gl;
          group_take<L>(real, a.b_real, e < (unsigned)deg ? bf_edge_composite((uint32_t)__ldg(a.in_src + beg + (int)e), q, rs) : kInf, gl, gm, lane);
        }
      }
      r_cnt = min(deg, a.b_real);
    }
    // ---- random walks; where they are fewer than half the lanes of a small group, the candidates of several steps are ranked together:
    // lane t * walks + w holds walk w's of the batch's step t ----
    int w_cnt = 0;
    if (a.b_rw > 0 && a.walks > 0 && a.walk_len > 0) {
      const int64_t ws = a.seed + BF_RW_SEED_OFFSET;
      const int batch = L == 32 ? 1 : max(1, min(a.walk_len, L / a.walks));
      const int step = batch > 1 ? gl / a.walks : 0, from = batch > 1 ? gl - step * a.walks : gl;
      for (int w0 = 0; w0 < a.walks; w0 += L) {
        const bool active = w0 + gl < a.walks;
        const uint64_t walk_id = (uint64_t)v * (uint64_t)a.walks + (uint64_t)(w0 + gl);
        uint64_t held = kInf;
        int cur = v, in_batch = 0;
        for (int d = 1; d <= a.walk_len; ++d) {
          int next = cur;
          if (active) {
            const int ob = a.out_rowptr[cur];
            const uint32_t n_out = (uint32_t)(a.out_rowptr[cur + 1] - ob);
            if (n_out > 0) next = __ldg(a.out_col + ob + (int)bf_mulhi32(bf_walk_uniform32(walk_id, (uint32_t)d, (uint64_t)a.seed), n_out));
          }
          const bool emit = active && (d == 1 || next != cur);
          cur = next;
          w_cnt += __popc(group_ballot<L>(gm, lane, emit));
          uint64_t c = emit ? bf_edge_composite((uint32_t)next, q, ws) : kInf;
          if (batch > 1) {
            c = __shfl_sync(gm, c, from, L);
            if (step == in_batch) held = c;
            if (++in_batch < batch && d < a.walk_len) continue;
            c = held;
            held = kInf;
            in_batch = 0;
          }
          group_take<L>(walked, a.b_rw, c, gl, gm, lane);
        }
      }
      w_cnt = min(w_cnt, a.b_rw);
    }
    // ---- merge: every lane finds the place of its two sources ----
    const uint32_t sr = gl < r_cnt ? (uint32_t)real : kNone, sw = gl < w_cnt ? (uint32_t)walked : kNone;
    int* row = a.ell_col + slot * a.cap;
    int at_r = 0, at_w = 0, total;
    if (typed) {
      for (int t = 0; t < L; ++t) {
        const uint32_t yr = __shfl_sync(gm, sr, t, L), yw = __shfl_sync(gm, sw, t, L);
        at_r += yr < sr || (yr == sr && t < gl) ? 1 : 0;
        at_w += yw < sw || (yw == sw && t < gl) ? 1 : 0;
      }
      uint8_t* types = a.ell_type + slot * a.cap;
      if (gl < r_cnt) { row[at_r] = (int)sr; types[at_r] = 0; }
      if (gl < w_cnt) { row[r_cnt + at_w] = (int)sw; types[r_cnt + at_w] = 1; }
      if (gl == 0) { row[r_cnt + w_cnt] = v; types[r_cnt + w_cnt] = 0; }
      total = r_cnt + w_cnt + 1;
    } else {
      bool keep_r = sr != kNone, keep_w = sw != kNone;
      for (int t = 0; t < L; ++t) {
        const uint32_t yr = __shfl_sync(gm, sr, t, L), yw = __shfl_sync(gm, sw, t, L);
        if (t < gl && yr == sr) keep_r = false;
        if (yr == sw || (t < gl && yw == sw)) keep_w = false;
      }
      for (int t = 0; t < L; ++t) {                        // what is not kept comes last: kNone
        const uint32_t yr = __shfl_sync(gm, keep_r ? sr : kNone, t, L), yw = __shfl_sync(gm, keep_w ? sw : kNone, t, L);
        at_r += (yr < sr ? 1 : 0) + (yw < sr ? 1 : 0);
        at_w += (yr < sw ? 1 : 0) + (yw < sw ? 1 : 0);
      }
      if (keep_r) row[at_r] = (int)sr;
      if (keep_w) row[at_w] = (int)sw;
      total = __popc(group_ballot<L>(gm, lane, keep_r)) + __popc(group_ballot<L>(gm, lane, keep_w));
    }
    if (gl == 0) { a.ell_cnt[slot] = total; atomicAdd(&s_tot[0], (unsigned)r_cnt); atomicAdd(&s_tot[1], (unsigned)w_cnt); }
  }
  __syncthreads();
  if (threadIdx.x < 2 && s_tot[threadIdx.x]) atomicAdd(a.totals + threadIdx.x, (unsigned long long)s_tot[threadIdx.x]);
}

// Compaction: a block takes 256 rows, its threads the row slots in order, so that reads and the writes of what is kept run along memory.
// Bound by those bytes; the division of a slot index by the capacity is a multiplication (a 64-bit division a slot took 106 us
// at 2.9 M rows of 8, this takes 34).
constexpr int kCompactRows = 256;
template <bool TYPED>
__global__ void __launch_bounds__(256) ell_to_csr_kernel(const int* __restrict__ ell_col, const uint8_t* __restrict__ ell_type,
                                                         const int* __restrict__ rowptr, int n, int cap, int* __restrict__ col,
                                                         uint8_t* __restrict__ etype) {
  __shared__ int s_beg[kCompactRows + 1];
  const int r0 = blockIdx.x * kCompactRows, rows = min(kCompactRows, n - r0);
  for (int i = threadIdx.x; i <= rows; i += 256) s_beg[i] = rowptr[r0 + i];
  __syncthreads();
  const unsigned inv = (1u << 22) / (unsigned)cap + 1u;      // i / cap for i < 256 * cap, cap <= 128: i * (inv * cap - 2^22) < 2^22
  const bool narrow = cap <= 128;
  const long long base = (long long)r0 * cap;
  for (int i = threadIdx.x; i < rows * cap; i += 256) {
    const int r = narrow ? (int)(((unsigned long long)(unsigned)i * inv) >> 22) : i / cap, c = i - r * cap;
    const int beg = s_beg[r];
    if (c < s_beg[r + 1] - beg) {
      col[beg + c] = ell_col[base + i];
      if (TYPED) etype[beg + c] = ell_type[base + i];
    }
  }
}

using SelectKernel = void (*)(BuildArgs);
template <int K, int W> SelectKernel select_kernel(bool typed) { return typed ? budget_select_kernel<K, true, W> : budget_select_kernel<K, false, W>; }

// Lanes of a query: 1 (a thread), 8 or 32, whichever is estimated to be done first.  us: a group takes the latency of one walk and of its row's
// chunks, and throughput that grows with the queries; a thread takes the latency of all its walks' candidates and of its warp's long rows, one
// after the other, however few queries there are, and little more for many.  Measured, a thread (its better form) / a group (8 lanes where budgets and
// walks fit, else 32); budgets, walks x length, nodes: 8 + 8, 4 x 6: 2 k 13 / 11, 10 k 15 / 13, 20 k 17 / 23; 8 + 8, 8 x 8: 5 k 24 / 15, 20 k 30 / 30, 40 k
// 39 / 47; 16 + 16, 6 x 8: 2 k 24 / 16, 5 k 26 / 31; 16 x 10: 10 k 68 / 66, 20 k 91 / 123; 32 + 32, 4 x 6: 2 k 24 / 13, 5 k 27 / 25; 4 + 4, 2 x 4: 500 6.4 / 7.8.  Rows of 1,000
// edges, 8 + 4: 5 k nodes 107 / 44 (32 lanes), 20 k 189 / 181; of 3,000, 3 k nodes 254 / 41.
int pick_form(const bf_build_params* p, int n, int most) {
  const bool walk = p->b_rw > 0 && p->walks > 0;
  const double len = walk ? p->walk_len : 0, candidates = walk ? (double)p->walks * p->walk_len : 0, k = n * 1e-3;
  const double row = p->b_real > 0 && p->n > 0 ? (double)p->in_edges / p->n : 0;
  double thread;
  if (!walk || p->walks <= 2 || most > 16) thread = 4.0 + 0.35 * candidates + (most <= 4 ? -1.0 : most <= 8 ? 0.0 : most <= 16 ? 2.0 : 8.0);
  else thread = 8.8 + (most <= 8 ? 0.2 : 0.31) * candidates;
  thread = thread * (1.0 + 0.02 * k) + (row > 200 ? 0.077 * (250.0 + row) : 0.0);
  const double warp = 7.0 + k * (1.0 + 0.5 * len + 0.008 * row);
  const double eight = most <= 8 && p->walks <= 8 ? 3.0 + 1.2 * len + (k > 5 ? (k - 5) * (0.04 + 0.12 * len) : 0.0) + 0.056 * row : 1e9;
  return thread <= warp && thread <= eight ? 1 : eight <= warp ? 8 : 32;
}

}  // namespace

extern "C" int bf_budget_select(const bf_build_params* p, cudaStream_t st) {
  if (p->b_real > BF_MAX_SIDE_BUDGET || p->b_rw > BF_MAX_SIDE_BUDGET || p->walk_len > BF_MAX_WALK_LEN)
    return (int)cudaErrorInvalidValue;
  BuildArgs a;
  a.in_rowptr = p->in_rowptr; a.in_src = p->in_src; a.out_rowptr = p->out_rowptr; a.out_col = p->out_col;
  a.n = p->row_count > 0 ? p->row_count : p->n; a.row_begin = p->row_count > 0 ? p->row_begin : 0;
  if (a.row_begin < 0 || (long long)a.row_begin + a.n > p->n) return (int)cudaErrorInvalidValue;
  a.b_real = p->b_real; a.b_rw = p->b_rw; a.walks = p->walks; a.walk_len = p->walk_len;
  a.seed = p->seed; a.cap = p->cap;
  a.ell_col = p->ell_col; a.ell_type = p->ell_type; a.ell_cnt = p->ell_cnt;
  a.totals = reinterpret_cast<unsigned long long*>(p->totals);
  const long long blocks = ((long long)a.n + kSelectThreads - 1) / kSelectThreads;
  const bool hubs = p->hub_rows != nullptr && p->hub_top != nullptr && p->n_hub > 0 && p->b_real > 0;
  a.hub_rows = hubs ? p->hub_rows : nullptr; a.n_hub = hubs ? p->n_hub : 0; a.hub_top = hubs ? p->hub_top : nullptr;
  if (blocks == 0) return (int)cudaSuccess;
  if (hubs) budget_hub_topk_kernel<<<(unsigned)p->n_hub * kHubBlocks, kHubWarps * 32, 0, st>>>(a);
  const int most = p->b_real > p->b_rw ? p->b_real : p->b_rw;
  const bool typed = p->exphormer != 0;
  const size_t smem = (size_t)kSelectThreads * (size_t)(a.cap | 1) * sizeof(int);
  const int lanes = pick_form(p, a.n, most);
  if (lanes > 1) {
    const unsigned grid = (unsigned)(((long long)a.n * lanes + 255) / 256);
    if (lanes == 8) budget_select_group_kernel<8><<<grid, 256, 0, st>>>(a, typed);
    else budget_select_group_kernel<32><<<grid, 256, 0, st>>>(a, typed);
    return (int)cudaGetLastError();
  }
  // Eight walks under way instead of two cost registers and save latency, which is what few queries wait for: 8 + 8, 8 x 8, 10 k nodes 33 / 25 us,
  // 40 k 44 / 39, 100 k 81 / 76; 16 + 16, 6 x 8, 40 k 50 / 47, 100 k 88 / 93; 4 + 4, 2 x 4, 40 k 8.9 / 10.
  const bool deep = p->walks > 2 && a.n <= 65536;
  auto kern = most <= 4    ? (deep ? select_kernel<4, 8>(typed) : select_kernel<4, 2>(typed))
              : most <= 8  ? (deep ? select_kernel<8, 8>(typed) : select_kernel<8, 2>(typed))
              : most <= 16 ? (deep ? select_kernel<16, 8>(typed) : select_kernel<16, 2>(typed))
                           : select_kernel<32, 2>(typed);
  kern<<<(unsigned)blocks, kSelectThreads, smem, st>>>(a);
  return (int)cudaGetLastError();
}

extern "C" int bf_ell_to_csr(const int* ell_col, const uint8_t* ell_type, const int* rowptr, int n, int cap, int* col,
                             uint8_t* etype, cudaStream_t st) {
  const unsigned blocks = (unsigned)(((long long)n + kCompactRows - 1) / kCompactRows);
  if (blocks == 0 || cap < 1) return (int)cudaSuccess;
  if (etype) ell_to_csr_kernel<true><<<blocks, 256, 0, st>>>(ell_col, ell_type, rowptr, n, cap, col, etype);
  else ell_to_csr_kernel<false><<<blocks, 256, 0, st>>>(ell_col, ell_type, rowptr, n, cap, col, etype);
  return (int)cudaGetLastError();
}

// rowptr[0 .. n] of the counts: an inclusive prefix sum behind a leading zero.
extern "C" size_t bf_count_offsets_scratch(int n) {
  size_t bytes = 0;
  cub::DeviceScan::InclusiveSum(nullptr, bytes, (const int*)nullptr, (int*)nullptr, n);
  return bytes + 1;
}
extern "C" int bf_count_offsets(const int* counts, int n, int* rowptr, void* scratch, size_t scratch_bytes, cudaStream_t st) {
  cudaError_t e = cudaMemsetAsync(rowptr, 0, sizeof(int), st);
  if (e == cudaSuccess && n > 0) e = cub::DeviceScan::InclusiveSum(scratch, scratch_bytes, counts, rowptr + 1, n, st);
  return (int)e;
}
