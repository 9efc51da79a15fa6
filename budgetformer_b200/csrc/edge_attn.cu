// Budgeted sparse edge attention for sm_100a: forward, dK/dV pass (over the transposed graph) and
// dQ pass (over queries), each in two forms that a rule on size, type and shape chooses between.
// Gather-only on regular rows: every query owns <= B sampled in-edges, so one lane group streams
// them and keeps the running numerator / normaliser in registers.  Rows longer than BF_LONG_ROW (the Graphormer virtual node,
// hubs of a graph without a budget, popular keys in the transposed graph) are cut into work items of
// BF_LONG_CHUNK edges, one warp each, whose fp32 partial sums are added in a fixed order by two small
// kernels: no atomics, bit-reproducible.  (The gradient of the edge-type table, a sum over all edges, does meet in atomics, one
// set per thread block.)
//
// Math (reference: models/graphormer_dist_node_level.py:231-263, models/gt_dist_node_level.py:
// 224-262, models/graphgps_dist_node_level.py:151-177, models/exphormer_dist_node_level.py:92-121):
//   s = clamp(<q_i,k_j>/sqrt(hn) [*E_type], -5, 5);  w = exp(s);  Z_i = sum w
//   plain/exphormer: out_i = sum w v_j / (Z_i + 1e-6)
//   gps:             out_i = sum (w/(Z_i+1e-6)) * keep/(1-p) * v_j
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdlib.h>
#include <string.h>

#include "bf_kernels.h"
#include "f32x2.cuh"

namespace {

constexpr float kEps = 1e-6f;
constexpr float kClamp = 5.0f;

template <typename T> struct Vec;
template <> struct Vec<__nv_bfloat16> { static constexpr int N = 8; };
template <> struct Vec<__half> { static constexpr int N = 8; };
template <> struct Vec<float> { static constexpr int N = 4; };

template <typename T> __device__ __forceinline__ void load_vec(const T* p, float* f);
template <> __device__ __forceinline__ void load_vec<__nv_bfloat16>(const __nv_bfloat16* p, float* f) {
  uint4 u = __ldg(reinterpret_cast<const uint4*>(p));
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
  for (int i = 0; i < 4; ++i) { float2 t = __bfloat1622float2(h[i]); f[2 * i] = t.x; f[2 * i + 1] = t.y; }
}
template <> __device__ __forceinline__ void load_vec<__half>(const __half* p, float* f) {
  uint4 u = __ldg(reinterpret_cast<const uint4*>(p));
  const __half2* h = reinterpret_cast<const __half2*>(&u);
#pragma unroll
  for (int i = 0; i < 4; ++i) { float2 t = __half22float2(h[i]); f[2 * i] = t.x; f[2 * i + 1] = t.y; }
}
template <> __device__ __forceinline__ void load_vec<float>(const float* p, float* f) {
  float4 u = __ldg(reinterpret_cast<const float4*>(p));
  f[0] = u.x; f[1] = u.y; f[2] = u.z; f[3] = u.w;
}
template <typename T> __device__ __forceinline__ void store_vec(T* p, const float* f);
template <> __device__ __forceinline__ void store_vec<__nv_bfloat16>(__nv_bfloat16* p, const float* f) {
  uint4 u; __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&u);
#pragma unroll
  for (int i = 0; i < 4; ++i) h[i] = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
  *reinterpret_cast<uint4*>(p) = u;
}
template <> __device__ __forceinline__ void store_vec<__half>(__half* p, const float* f) {
  uint4 u; __half2* h = reinterpret_cast<__half2*>(&u);
#pragma unroll
  for (int i = 0; i < 4; ++i) h[i] = __floats2half2_rn(f[2 * i], f[2 * i + 1]);
  *reinterpret_cast<uint4*>(p) = u;
}
template <> __device__ __forceinline__ void store_vec<float>(float* p, const float* f) {
  *reinterpret_cast<float4*>(p) = make_float4(f[0], f[1], f[2], f[3]);
}

// One 16-byte slice of a row, kept packed until used.
template <typename T> struct Raw;
template <> struct Raw<__nv_bfloat16> {
  uint4 u;
  __device__ __forceinline__ void load(const __nv_bfloat16* p) { u = *reinterpret_cast<const uint4*>(p); }
  __device__ __forceinline__ void load_if(bool on, const __nv_bfloat16* p) { u = make_uint4(0u, 0u, 0u, 0u); if (on) u = *reinterpret_cast<const uint4*>(p); }
  __device__ __forceinline__ float get(int i) const {
    const uint32_t w = (i >> 1) == 0 ? u.x : (i >> 1) == 1 ? u.y : (i >> 1) == 2 ? u.z : u.w;
    return (i & 1) ? __uint_as_float(w & 0xFFFF0000u) : __uint_as_float(w << 16);
  }
};
template <> struct Raw<__half> {
  uint4 u;
  __device__ __forceinline__ void load(const __half* p) { u = *reinterpret_cast<const uint4*>(p); }
  __device__ __forceinline__ void load_if(bool on, const __half* p) { u = make_uint4(0u, 0u, 0u, 0u); if (on) u = *reinterpret_cast<const uint4*>(p); }
  __device__ __forceinline__ float get(int i) const {
    const uint32_t w = (i >> 1) == 0 ? u.x : (i >> 1) == 1 ? u.y : (i >> 1) == 2 ? u.z : u.w;
    return __half2float(__ushort_as_half((unsigned short)((i & 1) ? (w >> 16) : (w & 0xFFFFu))));
  }
};
template <> struct Raw<float> {
  float4 f;
  __device__ __forceinline__ void load(const float* p) { f = *reinterpret_cast<const float4*>(p); }
  __device__ __forceinline__ void load_if(bool on, const float* p) { f = make_float4(0.f, 0.f, 0.f, 0.f); if (on) f = *reinterpret_cast<const float4*>(p); }
  __device__ __forceinline__ float get(int i) const { return i == 0 ? f.x : i == 1 ? f.y : i == 2 ? f.z : f.w; }
};

template <typename T> __device__ __forceinline__ void load_vec_if(bool on, const T* p, float* f) {
  Raw<T> r;
  r.load_if(on, p);
#pragma unroll
  for (int i = 0; i < 16 / (int)sizeof(T); ++i) f[i] = r.get(i);
}

// One 16-byte slice of a row widened to fp32 pairs.
template <typename T> __device__ __forceinline__ void widen(const uint4& u, f2* p);
template <> __device__ __forceinline__ void widen<__nv_bfloat16>(const uint4& u, f2* p) {
  const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) p[i] = pack2(__uint_as_float(w[i] << 16), __uint_as_float(w[i] & 0xFFFF0000u));
}
template <> __device__ __forceinline__ void widen<__half>(const uint4& u, f2* p) {
  const __half2* h = reinterpret_cast<const __half2*>(&u);
#pragma unroll
  for (int i = 0; i < 4; ++i) { const float2 t = __half22float2(h[i]); p[i] = pack2(t.x, t.y); }
}
template <> __device__ __forceinline__ void widen<float>(const uint4& u, f2* p) {
  p[0] = pack2(__uint_as_float(u.x), __uint_as_float(u.y));
  p[1] = pack2(__uint_as_float(u.z), __uint_as_float(u.w));
}
template <int NP> __device__ __forceinline__ float dot2(const f2* a, const f2* b) {
  f2 t = mul2(a[0], b[0]);
#pragma unroll
  for (int i = 1; i < NP; ++i) t = fma2(a[i], b[i], t);
  const float2 r = unpack2(t);
  return r.x + r.y;
}
template <typename T, int NP> __device__ __forceinline__ void store_pairs(T* dst, const f2* p) {
  float f[2 * NP];
#pragma unroll
  for (int i = 0; i < NP; ++i) { const float2 t = unpack2(p[i]); f[2 * i] = t.x; f[2 * i + 1] = t.y; }
  store_vec<T>(dst, f);
}

// Asynchronous copies into shared memory (both addresses a multiple of the size).  Every lane copies the bytes that it alone
// reads back, so waiting for its own groups is enough: no barrier.
template <int BYTES> __device__ __forceinline__ void copy_async(void* dst, const void* src) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
  // .ca: through L1.  A lane's two slices share a 32-byte sector, which L2 would otherwise deliver twice, and rows that
  // everyone gathers (the virtual node, hubs) would queue at one L2 slice.
  if constexpr (BYTES == 16) asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
  else if constexpr (BYTES == 8) asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(d), "l"(src) : "memory");
  else asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void copy_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

template <typename T> __device__ __forceinline__ T from_float(float x);
template <> __device__ __forceinline__ __nv_bfloat16 from_float<__nv_bfloat16>(float x) { return __float2bfloat16_rn(x); }
template <> __device__ __forceinline__ __half from_float<__half>(float x) { return __float2half_rn(x); }
template <> __device__ __forceinline__ float from_float<float>(float x) { return x; }

__device__ __forceinline__ bool keep_edge(uint32_t seed, uint32_t eid, uint32_t head, uint32_t thresh) {
  uint32_t x = eid * 0x9E3779B1u + head * 0x85EBCA77u + seed;
  x = (x ^ (x >> 16)) * 0x7FEB352Du;
  x = (x ^ (x >> 15)) * 0x846CA68Bu;
  x ^= x >> 16;
  return x >= thresh;
}

template <int HN> __host__ __device__ constexpr float inv_sqrt_hn() {
  return HN == 8 ? 0.35355339059327373f : HN == 16 ? 0.25f : HN == 32 ? 0.17677669529663687f
       : HN == 64 ? 0.125f : 0.08838834764831845f;
}

// Lane-group geometry: LPH lanes cover one head (HN elements, 16 bytes per lane); a task is one
// (row, head chunk) handled by TL = LPH*HPT lanes, 32/TL tasks per warp.
struct Geo {
  int lph, hpt, tl, n_hc;
};
template <typename T, int HN> __host__ __device__ inline Geo make_geo(int hl) {
  Geo g;
  g.lph = HN / Vec<T>::N;
  int cap = 32 / g.lph;
  int hpt = 1;
  while (hpt * 2 <= cap && hpt * 2 <= hl) hpt *= 2;
  g.hpt = hpt;
  g.tl = g.lph * hpt;
  g.n_hc = (hl + hpt - 1) / hpt;
  return g;
}

// Sum over the LPH lanes of one head.  The mask names only those lanes: they always share
// control flow (same row, same head), so no wider convergence is needed.
template <int LPH> __device__ __forceinline__ unsigned head_mask() {
  const unsigned lane = threadIdx.x & 31u;
  return LPH >= 32 ? 0xffffffffu : (((1u << LPH) - 1u) << (lane & ~(unsigned)(LPH - 1)));
}
template <int LPH> __device__ __forceinline__ float head_sum(float x, unsigned m) {
#pragma unroll
  for (int o = LPH / 2; o > 0; o >>= 1) x += __shfl_xor_sync(m, x, o);
  return x;
}

// Routed rows: the result row of query / key `row` belongs to the rank that owns that node (row / rows_per) and is
// stored straight into that rank's buffer - the heads->nodes all-to-all of sequence parallelism done by the stores of
// the kernel that produces the rows.  Every destination holds one slab of `rows_per` rows per source rank
// ([n_dest * rows_per, ld] elements); `slab_row0` = this rank's slab.  n_dest == 0: off.
struct Route {
  unsigned long long base[BF_MAX_PEERS];   // buffer base address on every destination (peer mappings)
  int n_dest;
  int rows_per;
  long long ld;                            // row stride of the destination buffers (elements)
  long long slab_row0;                     // source rank * rows_per
};

template <typename T>
__device__ __forceinline__ T* routed(const Route& r, long long row, int col) {
  const int d = (int)(row / r.rows_per);
  const long long lr = row - (long long)d * r.rows_per + r.slab_row0;
  return reinterpret_cast<T*>(r.base[d]) + lr * r.ld + col;
}

struct AttnArgs {
  const void *q, *k, *v;       // [n, Hl, HN] with row strides ldq/ldk/ldv (elements)
  long long ldq, ldk, ldv;
  void* out;                   // [n, Hl, HN] contiguous
  float* z;                    // [n, Hl]
  const int* rowptr;           // [n+1]
  const int* col;              // [E]
  const uint8_t* etype;        // [E] or null
  const float* etab;           // [T, Hl, HN] fp32 or null
  int n, hl;
  int variant;                 // 0 plain, 1 gps, 2 exphormer
  float inv_keep;              // 1/(1-p)
  uint32_t thresh, seed;
  int long_row;                // rows with more edges are left to the long-row kernels (0: every row is walked here)
  // long rows as work items (see bf_long_rows)
  const int4* long_task;       // [n_long_task]: row, first edge, end edge, slot
  int n_long_task;
  const int* long_split;       // [n_long_split, 3]: row, first slot, slot count
  int n_long_split;
  float* long_partial;         // [n_long_task, forward: fwd_pitch(Hl*HN, Hl); backward: Hl*HN]
  // long rows of the allocation-free entry point: fixed scratch, atomics
  const int* hub_rows;         // [n_hub]
  int n_hub, hub_chunk;
  float* hub_scratch;          // [n_hub, Hl*HN + Hl]
  // fused dropout on the stored output (out_thresh == 0: off)
  uint32_t out_thresh, out_seed;
  float out_inv_keep, out_keep;
  int out_rows_local, out_col0;
  Route route_out;             // second copy of every output row, delivered to the row's owner (n_dest == 0: none)
};

// keep decision of ops.gemm.hash_keep_mask / bf_hash_dropout for element (row, col)
__device__ __forceinline__ bool keep_out(const AttnArgs& a, int row, int c) {
  const uint32_t r = (uint32_t)(a.out_rows_local > 0 ? row % a.out_rows_local : row);
  uint32_t x = r * 0x9E3779B1u + (uint32_t)(a.out_col0 + c) * 0x85EBCA77u + a.out_seed;
  x = (x ^ (x >> 16)) * 0x7FEB352Du;
  x = (x ^ (x >> 15)) * 0x846CA68Bu;
  x ^= x >> 16;
  return x >= a.out_thresh;
}

// Two edges of one query for one task lane (second one optional: absent, it is zeros, since weight 0 times an infinity is NaN).
template <typename T, int HN>
__device__ __forceinline__ void fwd_pair(const AttnArgs& a, int head, int off, int e0, int e1, bool has1, unsigned hm,
                                         const float* qs0, const float* qs1, float* acc, float& zsum) {
  constexpr int VN = Vec<T>::N;
  constexpr int LPH = HN / VN;
  const T* kp = static_cast<const T*>(a.k);
  const T* vp = static_cast<const T*>(a.v);
  const int j0 = __ldg(a.col + e0);
  const int j1 = has1 ? __ldg(a.col + e1) : j0;
  float k0[VN], v0[VN], k1[VN], v1[VN];
  load_vec<T>(kp + (long long)j0 * a.ldk + off, k0);
  load_vec_if<T>(has1, kp + (long long)j1 * a.ldk + off, k1);
  load_vec<T>(vp + (long long)j0 * a.ldv + off, v0);
  load_vec_if<T>(has1, vp + (long long)j1 * a.ldv + off, v1);
  int t0 = 0, t1 = 0;
  if (a.variant == 2) { t0 = a.etype[e0]; t1 = has1 ? a.etype[e1] : 0; }
  float d0 = 0.f, d1 = 0.f;
#pragma unroll
  for (int i = 0; i < VN; ++i) { d0 += (t0 ? qs1[i] : qs0[i]) * k0[i]; d1 += (t1 ? qs1[i] : qs0[i]) * k1[i]; }
  d0 = head_sum<LPH>(d0, hm);
  d1 = head_sum<LPH>(d1, hm);
  float w0 = __expf(fminf(fmaxf(d0, -kClamp), kClamp));
  float w1 = has1 ? __expf(fminf(fmaxf(d1, -kClamp), kClamp)) : 0.f;
  zsum += w0 + w1;
  if (a.variant == 1 && a.thresh) {
    if (!keep_edge(a.seed, (uint32_t)e0, (uint32_t)head, a.thresh)) w0 = 0.f;
    if (has1 && !keep_edge(a.seed, (uint32_t)e1, (uint32_t)head, a.thresh)) w1 = 0.f;
  }
#pragma unroll
  for (int i = 0; i < VN; ++i) acc[i] += w0 * v0[i] + w1 * v1[i];
}

template <typename T, int HN>
__device__ __forceinline__ void load_q_scaled(const AttnArgs& a, int row, int head, int off, float* qs0, float* qs1) {
  constexpr int VN = Vec<T>::N;
  const float scale = inv_sqrt_hn<HN>();
  float qf[VN];
  load_vec<T>(static_cast<const T*>(a.q) + (long long)row * a.ldq + off, qf);
#pragma unroll
  for (int i = 0; i < VN; ++i) { qs0[i] = qf[i] * scale; qs1[i] = qs0[i]; }
  if (a.variant == 2) {
    const int hlhn = a.hl * HN;
#pragma unroll
    for (int i = 0; i < VN; ++i) {
      qs0[i] = qf[i] * scale * a.etab[off + i];
      qs1[i] = qf[i] * scale * a.etab[hlhn + off + i];
    }
  }
}

// Forward over the rows, one lane group (16 bytes a lane) per (row, head chunk), two edges' gathers in flight in registers.  Many
// small lane groups and few registers: the better form where the gathered rows come out of L2 (see rows_forward).
template <typename T, int HN>
__global__ void __launch_bounds__(256) edge_attn_fwd_rows_kernel(AttnArgs a) {
  constexpr int VN = Vec<T>::N;
  constexpr int LPH = HN / VN;
  const Geo g = make_geo<T, HN>(a.hl);
  const int lane = threadIdx.x & 31;
  const long long warp = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const long long task = warp * (32 / g.tl) + lane / g.tl;
  const int lt = lane % g.tl;
  const bool live = task < (long long)a.n * g.n_hc;
  const int row = live ? (int)(task / g.n_hc) : 0;
  const int hc = live ? (int)(task % g.n_hc) : 0;
  const int head = hc * g.hpt + lt / LPH;
  const bool head_ok = live && head < a.hl;
  const int hsafe = head_ok ? head : 0;
  const int off = hsafe * HN + (lt % LPH) * VN;
  int beg = 0, end = 0;
  if (head_ok) { beg = a.rowptr[row]; end = a.rowptr[row + 1]; }
  const bool cut = a.long_row > 0 && end - beg > a.long_row;          // left to the long-row kernels
  if (cut) end = beg;
  float qs0[VN], qs1[VN], acc[VN];
  float zsum = 0.f;
#pragma unroll
  for (int i = 0; i < VN; ++i) acc[i] = 0.f;
  load_q_scaled<T, HN>(a, row, hsafe, off, qs0, qs1);
  const unsigned hm = head_mask<LPH>();
  for (int e = beg; e < end; e += 2) fwd_pair<T, HN>(a, hsafe, off, e, e + 1, e + 1 < end, hm, qs0, qs1, acc, zsum);
  if (head_ok && !cut) {
    float inv = 1.f / (zsum + kEps);
    if (a.variant == 1) inv *= a.inv_keep;
    float o[VN];
#pragma unroll
    for (int i = 0; i < VN; ++i) o[i] = acc[i] * inv;
    if (a.out_thresh) {
#pragma unroll
      for (int i = 0; i < VN; ++i) o[i] = keep_out(a, row, off + i) ? o[i] * a.out_inv_keep : 0.f;
    }
    store_vec<T>(static_cast<T*>(a.out) + (long long)row * a.hl * HN + off, o);
    if (a.route_out.n_dest) store_vec<T>(routed<T>(a.route_out, row, off), o);
    if ((lt % LPH) == 0) a.z[(long long)row * a.hl + head] = zsum;
  }
}

// ---------------------------------------------------------------------------------------------
// Streams.  A warp holds 32 / TL lane groups of TL lanes; each group owns one segment (a query row, or a key work item) at a
// time and `per` of them in all.  The groups of a warp step together: segment r of every group starts at the same step and
// lasts as long as the longest of them, so all control flow is uniform over the warp.  The rows that the edges name are copied
// into a shared-memory ring kRing - 1 steps ahead of the arithmetic, across segment ends: a short segment costs no latency of
// its own, and the gathers in flight take no registers.  A lane holds 32 bytes of a row where the head is wide enough, which
// halves the scalar work per edge (score, exponential, cursor) against 16 bytes; the arithmetic runs in fp32 pairs.
// Without this (two 16-byte gathers a step in registers, one row per lane group) issue slots and latency, not memory, bound the
// kernels where the rows come from DRAM: it stood at 36 (forward), 40 (dK/dV) and 42 % (dQ), now 46 and 56 %, and 37 % in a dQ that gathers
// half the rows and is bound by issue.  2.9 M nodes, 15.3 M edges, 8 heads x 16 bf16, us, without and with streams: forward 2060 / 1460,
// dK/dV 3470 / 2680, dQ 2200 / 860 and 250 for the row terms; 612 k nodes, 8.8 M edges, 8 x 32 with dropout: 1370 / 1220, 2610 / 2230,
// 1500 / 690; typed (392 k nodes, 9.1 M edges): dK/dV 4560 / 3190, dQ 5440 / 1490.  Where the rows stay in L2 the picture turns: see
// rows_forward and recomputed_backward.  Six blocks an SM in the forward pass instead of four: 17 % slower; two in the dK/dV pass instead
// of three: 15 %.
// ---------------------------------------------------------------------------------------------
constexpr int kRing = 4;
constexpr int kStreamThreads = 128;
constexpr unsigned kFull = 0xffffffffu;

// elements of a row that one lane holds: 32 bytes, or a whole narrower head
template <typename T, int HN> constexpr int wide_elems() { return HN < 32 / (int)sizeof(T) ? HN : 32 / (int)sizeof(T); }

// 2^ltl lanes per group, blockIdx.y = head chunk
struct StreamGeo {
  int ltl;
  int per;                     // segments per lane group
};

// One lane's part of a row in the ring: VN elements as 16-byte slices, slice-major so that a warp's accesses do not collide.
template <typename T, int VN> struct Slices {
  static constexpr int N = VN * (int)sizeof(T) / 16;
  static constexpr int PP = 8 / (int)sizeof(T);             // pairs per slice
  static __device__ __forceinline__ void copy(uint4 (*dst)[kStreamThreads], int tid, const char* src) {
#pragma unroll
    for (int i = 0; i < N; ++i) copy_async<16>(&dst[i][tid], src + 16 * i);
  }
  static __device__ __forceinline__ void read(const uint4 (*src)[kStreamThreads], int tid, f2* p) {
#pragma unroll
    for (int i = 0; i < N; ++i) widen<T>(src[i][tid], p + PP * i);
  }
  static __device__ __forceinline__ void load(const T* src, uint4* u) {
#pragma unroll
    for (int i = 0; i < N; ++i) u[i] = __ldg(reinterpret_cast<const uint4*>(src) + i);
  }
  static __device__ __forceinline__ void put(T* dst, const uint4* u) {
#pragma unroll
    for (int i = 0; i < N; ++i) reinterpret_cast<uint4*>(dst)[i] = u[i];
  }
  static __device__ __forceinline__ void spread(const uint4* u, f2* p) {
#pragma unroll
    for (int i = 0; i < N; ++i) widen<T>(u[i], p + PP * i);
  }
  static __device__ __forceinline__ void store(T* dst, const f2* p) {
#pragma unroll
    for (int i = 0; i < N; ++i) store_pairs<T, PP>(dst + 16 / (int)sizeof(T) * i, p + PP * i);
  }
};

// the segments of a lane group that are rows of a CSR: row(r) = base + r * stride, long rows and rows past the end are empty
struct Rows {
  long long base;
  int stride, n;
  bool on;
  // of the group, whether or not this lane's head exists
  __device__ __forceinline__ bool extent(const AttnArgs& a, int r, int& beg, int& len) const {
    beg = len = 0;
    const long long row = base + (long long)r * stride;
    if (row >= n) return false;
    beg = __ldg(a.rowptr + row);
    len = __ldg(a.rowptr + row + 1) - beg;
    if (a.long_row > 0 && len > a.long_row) { len = 0; return false; }
    return true;
  }
  // of the lane
  __device__ __forceinline__ bool bounds(const AttnArgs& a, int r, int& beg, int& len) const {
    if (on && extent(a, r, beg, len)) return true;
    beg = len = 0;
    return false;
  }
};

// every segment takes at least one step, so that the ring never runs more than kRing segments ahead
__device__ __forceinline__ int steps_of(int len) { return max(1, (int)__reduce_max_sync(kFull, (unsigned)len)); }

// What a lane group reads of its edges ahead of them, one edge a lane: the chunk that the stream is in, the chunk behind it, and the first
// chunk of the next segment.  A step takes its edge by a shuffle.  (With a load for every edge, one step ahead, each trip to memory for
// a new sector of the list held all groups of the warp up: dK/dV and dQ of eight heads of 16, bf16, 300 k
// nodes of ten edges 1070 us then and 902 now; 700 k packed nodes of eight 7431 and 6949 with the forward pass, twice over.  dQ of 612 k
// nodes of 16 edges 8 x 32 bf16, 793 and 734; on a power-law graph of that size, whose dQ pass is bound by what L2 holds, 695 and 702.)
// The shuffle's own width folds the edge into its group: with the lane computed, that pass took 2 % longer.
struct Chunk {
  int now, next, other;
  __device__ __forceinline__ int at(int i, int lanes) const { return __shfl_sync(kFull, now, i, lanes); }      // i modulo the group's lanes
};

// The fetching side of a stream over rows, one warp-uniform step at a time: edge i of segment r, its key (and type).  The bounds
// are read two segments ahead and the first keys of a segment one segment ahead: a chain of row pointer, key, row would
// otherwise stall every segment for two trips to memory.
template <bool TYPED> struct RowFetch {
  int r, i, m, beg, len, beg1, len1, beg2, len2;
  int lt, mask;                  // lane in its group, group size - 1
  Chunk key_, type_;
  __device__ __forceinline__ void read(const AttnArgs& a, int b, int n, int from, int& key, int& type) const {
    if (from + lt < n) { key = __ldg(a.col + b + from + lt); if (TYPED) type = a.etype[b + from + lt]; }
  }
  __device__ __forceinline__ void start(const AttnArgs& a, const Rows& rows, int n_seg, int lane, int ltl) {
    mask = (1 << ltl) - 1;
    lt = lane & mask;
    r = i = 0;
    rows.extent(a, 0, beg, len);
    beg1 = len1 = beg2 = len2 = 0;
    if (1 < n_seg) rows.extent(a, 1, beg1, len1);
    if (2 < n_seg) rows.extent(a, 2, beg2, len2);
    m = steps_of(len);
    key_.now = key_.next = key_.other = type_.now = type_.next = type_.other = 0;
    read(a, beg, len, 0, key_.now, type_.now);
    read(a, beg, len, mask + 1, key_.next, type_.next);
    read(a, beg1, len1, 0, key_.other, type_.other);
  }
  __device__ __forceinline__ bool has() const { return i < len; }
  __device__ __forceinline__ int edge() const { return beg + i; }
  __device__ __forceinline__ int key() const { return key_.at(i, mask + 1); }           // by all lanes of the warp
  __device__ __forceinline__ int type() const { return TYPED ? type_.at(i, mask + 1) : 0; }
  __device__ __forceinline__ void advance(const AttnArgs& a, const Rows& rows, int n_seg) {
    if (r >= n_seg) return;
    if (++i == m) {
      i = 0;
      ++r;
      beg = beg1; len = len1; key_.now = key_.other; type_.now = type_.other;      // empty past the last segment
      beg1 = beg2; len1 = len2;
      beg2 = len2 = 0;
      read(a, beg, len, mask + 1, key_.next, type_.next);
      read(a, beg1, len1, 0, key_.other, type_.other);
      if (r + 2 < n_seg) rows.extent(a, r + 2, beg2, len2);
      if (r < n_seg) m = steps_of(len);
    } else if ((i & mask) == 0) {
      key_.now = key_.next; type_.now = type_.next;
      read(a, beg, len, i + mask + 1, key_.next, type_.next);
    }
  }
};

template <typename T, int HN, bool GPS>
__global__ void __launch_bounds__(kStreamThreads, 4) edge_attn_fwd_kernel(AttnArgs a, StreamGeo sg) {
  constexpr int VN = wide_elems<T, HN>(), NP = VN / 2, LPH = HN / VN;
  using S = Slices<T, VN>;
  __shared__ uint4 ring[kRing][2][S::N][kStreamThreads];
  const int tid = threadIdx.x, lane = tid & 31, lt = lane & ((1 << sg.ltl) - 1), groups = 32 >> sg.ltl;
  const int head = blockIdx.y * ((1 << sg.ltl) / LPH) + lt / LPH;
  const long long warp0 = ((long long)blockIdx.x * (kStreamThreads / 32) + (tid >> 5)) * groups * sg.per;
  if (warp0 >= a.n) return;                     // the whole warp
  const int n_seg = (int)min((long long)sg.per, (a.n - warp0 + groups - 1) / groups);
  const Rows rows{warp0 + (lane >> sg.ltl), groups, a.n, head < a.hl};
  const int off = (rows.on ? head * HN : 0) + (lt % LPH) * VN;
  const char* kb = reinterpret_cast<const char*>(static_cast<const T*>(a.k) + off);
  const char* vb = reinterpret_cast<const char*>(static_cast<const T*>(a.v) + off);
  const T* qb = static_cast<const T*>(a.q) + off;
  const unsigned long long skb = (unsigned long long)a.ldk * sizeof(T), svb = (unsigned long long)a.ldv * sizeof(T);

  RowFetch<false> f;
  f.start(a, rows, n_seg, lane, sg.ltl);
  auto issue = [&](int slot) {
    const unsigned key = (unsigned)f.key();
    if (rows.on && f.has()) {
      S::copy(ring[slot][0], tid, kb + key * skb);
      S::copy(ring[slot][1], tid, vb + key * svb);
    }
    copy_commit();
    f.advance(a, rows, n_seg);
  };
#pragma unroll
  for (int s = 0; s < kRing - 1; ++s) issue(s);

  int beg, len, nbeg = 0, nlen = 0;
  bool stored = rows.bounds(a, 0, beg, len), nstored = false;
  uint4 qn[S::N];
#pragma unroll
  for (int i = 0; i < S::N; ++i) qn[i] = make_uint4(0, 0, 0, 0);
  if (stored) S::load(qb + rows.base * a.ldq, qn);
  int slot = 0;
  for (int r = 0; r < n_seg; ++r) {
    const long long row = rows.base + (long long)r * groups;
    f2 q0[NP], acc[NP];
    const float scale = inv_sqrt_hn<HN>();
    const f2 sc = pack2(scale, scale);
    S::spread(qn, q0);
#pragma unroll
    for (int i = 0; i < NP; ++i) { q0[i] = mul2(q0[i], sc); acc[i] = pack2(0.f, 0.f); }
    if (r + 1 < n_seg) {
      nstored = rows.bounds(a, r + 1, nbeg, nlen);
      if (nstored) S::load(qb + (row + groups) * a.ldq, qn);
    }
    const int m = steps_of(len);
    float zsum = 0.f;
    for (int i = 0; i < m; ++i) {
      issue((slot + kRing - 1) & (kRing - 1));
      copy_wait<kRing - 1>();
      f2 x[NP];
      S::read(ring[slot][0], tid, x);
      const float d = head_sum<LPH>(dot2<NP>(q0, x), kFull);
      float w = __expf(fminf(fmaxf(d, -kClamp), kClamp));
      S::read(ring[slot][1], tid, x);
      if (i < len) {                            // a group whose segment is over holds a stale slot: nothing of it is added
        zsum += w;
        if (GPS && a.thresh && !keep_edge(a.seed, (uint32_t)(beg + i), (uint32_t)head, a.thresh)) w = 0.f;
        const f2 ww = pack2(w, w);
#pragma unroll
        for (int u = 0; u < NP; ++u) acc[u] = fma2(ww, x[u], acc[u]);
      }
      slot = (slot + 1) & (kRing - 1);
    }
    if (stored) {
      float inv = 1.f / (zsum + kEps);
      if (GPS) inv *= a.inv_keep;
      const f2 iv = pack2(inv, inv);
#pragma unroll
      for (int i = 0; i < NP; ++i) acc[i] = mul2(acc[i], iv);
      if (a.out_thresh) {
#pragma unroll
        for (int i = 0; i < NP; ++i) {
          const float2 t = unpack2(acc[i]);
          acc[i] = pack2(keep_out(a, (int)row, off + 2 * i) ? t.x * a.out_inv_keep : 0.f,
                         keep_out(a, (int)row, off + 2 * i + 1) ? t.y * a.out_inv_keep : 0.f);
        }
      }
      S::store(static_cast<T*>(a.out) + row * a.hl * HN + off, acc);
      if (a.route_out.n_dest) S::store(routed<T>(a.route_out, row, off), acc);
      if ((lt % LPH) == 0) a.z[row * a.hl + head] = zsum;
    }
    beg = nbeg; len = nlen; stored = nstored;
  }
  copy_wait<0>();
}

// Long rows.  One warp per (work item, head chunk): the 32 / TL lane groups take consecutive quarters (halves, ...) of the
// item's edges and meet in shuffles; the item's numerator and normaliser go to its slot of the scratch.  An item is
// BF_LONG_CHUNK = 64 edges, so a virtual node over 169 k nodes is 2,646 warps side by side (18 per SM, each 16 dependent
// gathers deep) instead of the 21 blocks of 8,192 edges it used to be: 25 us against 340 us (8 heads x 16, bf16), the dQ
// pass 24 against 421 us, and a 720 k-edge power-law graph without a budget (4 heads x 64, fp32) 31 against 781 us.
__host__ __device__ inline int fwd_pitch(int w, int hl) { return w + ((hl + 3) & ~3); }

// lanes of the first lane group receive the sum over the warp's lane groups (tl a power of two)
__device__ __forceinline__ float group_total(float x, int tl) {
  for (int o = tl; o < 32; o <<= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  return x;
}

template <typename T, int HN>
__global__ void __launch_bounds__(256) edge_attn_fwd_long_kernel(AttnArgs a) {
  constexpr int VN = Vec<T>::N;
  constexpr int LPH = HN / VN;
  const Geo g = make_geo<T, HN>(a.hl);
  const int lane = threadIdx.x & 31;
  const long long warp = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (warp >= (long long)a.n_long_task * g.n_hc) return;
  const int tpw = 32 / g.tl, sub = lane / g.tl, lt = lane % g.tl;
  const int item = (int)(warp / g.n_hc), hc = (int)(warp % g.n_hc);
  const int head = hc * g.hpt + lt / LPH;
  const bool head_ok = head < a.hl;
  const int hsafe = head_ok ? head : 0;
  const int off = hsafe * HN + (lt % LPH) * VN;
  const int4 it = __ldg(a.long_task + item);
  const int per = (it.z - it.y + tpw - 1) / tpw;
  const int beg = it.y + sub * per, end = min(it.z, beg + per);
  float qs0[VN], qs1[VN], acc[VN];
  float zsum = 0.f;
#pragma unroll
  for (int i = 0; i < VN; ++i) acc[i] = 0.f;
  load_q_scaled<T, HN>(a, it.x, hsafe, off, qs0, qs1);
  const unsigned hm = head_mask<LPH>();
  for (int e = beg; e < end; e += 2) fwd_pair<T, HN>(a, hsafe, off, e, e + 1, e + 1 < end, hm, qs0, qs1, acc, zsum);
  __syncwarp();
#pragma unroll
  for (int i = 0; i < VN; ++i) acc[i] = group_total(acc[i], g.tl);
  zsum = group_total(zsum, g.tl);
  if (sub == 0 && head_ok) {
    const int w = a.hl * HN;
    float* pp = a.long_partial + (long long)it.w * fwd_pitch(w, a.hl);
#pragma unroll
    for (int i = 0; i < VN; i += 4) *reinterpret_cast<float4*>(pp + off + i) = make_float4(acc[i], acc[i + 1], acc[i + 2], acc[i + 3]);
    if ((lt % LPH) == 0) pp[w + head] = zsum;
  }
}

// Hub rows of the allocation-free entry point: grid = (n_hub * chunks_per_hub) blocks; each warp strides over its block's chunk.
template <typename T, int HN>
__global__ void __launch_bounds__(256) edge_attn_fwd_hub_kernel(AttnArgs a, int chunks_per_hub) {
  constexpr int VN = Vec<T>::N;
  constexpr int LPH = HN / VN;
  const Geo g = make_geo<T, HN>(a.hl);
  const int hub_i = blockIdx.x / chunks_per_hub;
  const int row = a.hub_rows[hub_i];
  const int rbeg = a.rowptr[row], rend = a.rowptr[row + 1];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
  const int tpw = 32 / g.tl;
  const int lt = lane % g.tl;
  const int sub_task = lane / g.tl;            // parallel edge streams inside the warp
  const int streams = nwarp * tpw;
  const int stream = warp * tpw + sub_task;
  float* scratch = a.hub_scratch + (long long)hub_i * (a.hl * HN + a.hl);
  // a block walks the row's chunks with stride chunks_per_hub: a row longer than the caller's bound costs parallelism,
  // never edges
  for (int chunk = blockIdx.x % chunks_per_hub; (long long)chunk * a.hub_chunk < rend - rbeg; chunk += chunks_per_hub) {
  const int cbeg = rbeg + chunk * a.hub_chunk;
  const int cend = min(rend, cbeg + a.hub_chunk);
  for (int hc = 0; hc < g.n_hc; ++hc) {
    const int head = hc * g.hpt + lt / LPH;
    const bool head_ok = head < a.hl;
    const int hsafe = head_ok ? head : 0;
    const int off = hsafe * HN + (lt % LPH) * VN;
    float qs0[VN], qs1[VN], acc[VN];
    float zsum = 0.f;
#pragma unroll
    for (int i = 0; i < VN; ++i) acc[i] = 0.f;
    load_q_scaled<T, HN>(a, row, hsafe, off, qs0, qs1);
    const unsigned hm = head_mask<LPH>();
    if (head_ok)
      for (int e = cbeg + stream; e < cend; e += 2 * streams)
        fwd_pair<T, HN>(a, hsafe, off, e, e + streams, e + streams < cend, hm, qs0, qs1, acc, zsum);
    if (head_ok) {
#pragma unroll
      for (int i = 0; i < VN; ++i) atomicAdd(scratch + off + i, acc[i]);
      if ((lt % LPH) == 0) atomicAdd(scratch + a.hl * HN + head, zsum);
    }
  }
  }
}

template <typename T, int HN>
__global__ void edge_attn_fwd_hub_finalize(AttnArgs a) {
  const int hub_i = blockIdx.x;
  const int row = a.hub_rows[hub_i];
  const int w = a.hl * HN;
  const float* scratch = a.hub_scratch + (long long)hub_i * (w + a.hl);
  for (int c = threadIdx.x; c < w; c += blockDim.x) {
    const int head = c / HN;
    const float zs = scratch[w + head];
    float inv = 1.f / (zs + kEps);
    if (a.variant == 1) inv *= a.inv_keep;
    float ov = scratch[c] * inv;
    if (a.out_thresh) ov = keep_out(a, row, c) ? ov * a.out_inv_keep : 0.f;
    static_cast<T*>(a.out)[(long long)row * w + c] = from_float<T>(ov);
    if (a.route_out.n_dest) *routed<T>(a.route_out, row, c) = from_float<T>(ov);
    if ((c % HN) == 0) a.z[(long long)row * a.hl + head] = zs;
  }
}

// ---------------------------------------------------------------------------------------------
// Backward
// ---------------------------------------------------------------------------------------------
struct BwdArgs {
  AttnArgs f;
  const void* dout;            // [n, Hl, HN] contiguous
  void *dq, *dk, *dv;          // [n, Hl, HN], row stride ldg (elements)
  long long ldg;
  float2* zd;                  // [n, Hl]: (1/(Z+eps), D = <dout,out>)
  float* ds;                   // [E, Hl]: score gradient / sqrt(hn), left by the dK/dV pass for the dQ pass; null: computed twice
  const int *t_row, *t_eid;    // by key: query and position of every edge
  float* detab;                // [T, Hl, HN] fp32 or null
  // balanced dK/dV work list
  const int4* kv_task;         // [n_kv_task]: key row, first edge, end edge, partial slot (-1 = direct store)
  int n_kv_task;
  const int* kv_split;         // [n_kv_split, 3]: key row, first slot, number of slots
  int n_kv_split, n_kv_slots;
  float* kv_partial;           // [n_kv_slots, 2*Hl*HN] fp32
  // Packed query records for narrow rows (optional): the first kernel writes q and dout of every (row, head) next to each other
  // and the dK/dV pass gathers one contiguous record per edge instead of two short rows, which matters when a row of q is only 32
  // or 64 bytes.  Where dQ takes its score gradients from that pass, dout goes in as it is: dout / (Z + eps) rounded to 16 bits would
  // enter <dout, v> but not D, and the score gradient is a difference of the two (1.5 times the error in dQ).
  void* qg;                    // [n, Hl, 2, HN] in the operand dtype, or null
  // Routed gradients (route.n_dest > 0): dq / dk / dv rows go to the owner of the row instead of the local buffers, at
  // column offsets cq / ck / cv of the destination's packed row
  Route route;
  int cq, ck, cv;
};

// first element of gradient row `row`: in the local buffer, or in the row owner's slab when the gradients are routed
template <typename T>
__device__ __forceinline__ T* grad_row(const BwdArgs& b, void* local, int col0, long long row) {
  if (b.route.n_dest == 0) return static_cast<T*>(local) + row * b.ldg;
  return routed<T>(b.route, row, col0);
}

// What the dK/dV pass needs of every query: 1 / (Z + eps) and D = <dout, out>, and the packed records of narrow rows.
template <typename T, int HN>
__global__ void __launch_bounds__(kStreamThreads) edge_attn_bwd_delta_kernel(BwdArgs b, StreamGeo sg) {
  constexpr int VN = wide_elems<T, HN>(), NP = VN / 2, LPH = HN / VN;
  using S = Slices<T, VN>;
  const AttnArgs& a = b.f;
  const int tid = threadIdx.x, lt = tid & ((1 << sg.ltl) - 1);
  const int head = blockIdx.y * ((1 << sg.ltl) / LPH) + lt / LPH;
  const long long row = ((long long)blockIdx.x * kStreamThreads + tid) >> sg.ltl;
  const bool on = row < a.n && head < a.hl;
  const int off = (on ? head * HN : 0) + (lt % LPH) * VN;
  const long long rs = on ? row : 0, at = rs * a.hl * HN + off, hz = rs * a.hl + (on ? head : 0);
  uint4 gu[S::N], ou[S::N];
  S::load(static_cast<const T*>(b.dout) + at, gu);
  S::load(static_cast<const T*>(a.out) + at, ou);
  const float invz = 1.f / (__ldg(a.z + hz) + kEps);
  f2 g[NP], o[NP];
  S::spread(gu, g);
  S::spread(ou, o);
  float dterm = head_sum<LPH>(dot2<NP>(g, o), kFull);
  if (!on) return;
  if (a.out_thresh) dterm *= a.out_keep;        // the stored output is the dropped one, rescaled by 1 / (1 - p)
  if (b.qg != nullptr) {
    T* rec = static_cast<T*>(b.qg) + hz * 2 * HN + (lt % LPH) * VN;
    S::load(static_cast<const T*>(a.q) + row * a.ldq + off, ou);
    S::put(rec, ou);
    S::put(rec + HN, gu);
  }
  if ((lt % LPH) == 0) b.zd[hz] = make_float2(invz, dterm);
}

// s0 * E_0 + s1 * E_1 into s0, of the edge types that were met (bit t of `seen`)
template <int NP> __device__ __forceinline__ void typed_sum(const float* et, int w_row, unsigned seen, f2* s0, const f2* s1) {
  if (seen & 1u) {
#pragma unroll
    for (int i = 0; i < NP; ++i) s0[i] = mul2(s0[i], pack2(__ldg(et + 2 * i), __ldg(et + 2 * i + 1)));
  }
  if (seen & 2u) {
#pragma unroll
    for (int i = 0; i < NP; ++i) s0[i] = fma2(s1[i], pack2(__ldg(et + w_row + 2 * i), __ldg(et + w_row + 2 * i + 1)), s0[i]);
  }
}

// dK/dV over the balanced work list, first of the two passes over the edges.  It gathers q, dout and (1/Z, D) of each query and
// leaves the score gradient of every (edge, head) in `ds` (fp32, at the edge's own position), so that the dQ pass gathers k alone.
// The list holds the items of split keys (64 edges each), then the rest sorted by length.
template <typename T, int HN, int VAR, bool PACKED>
__global__ void __launch_bounds__(kStreamThreads, 3) edge_attn_bwd_kv_kernel(BwdArgs b, StreamGeo sg) {
  constexpr bool EXPH = VAR == 2;
  constexpr int VN = wide_elems<T, HN>(), NP = VN / 2, LPH = HN / VN;
  using S = Slices<T, VN>;
  const AttnArgs& a = b.f;
  __shared__ uint4 ring[kRing][2][S::N][kStreamThreads];
  __shared__ float2 ring_zd[kRing][kStreamThreads];
  __shared__ int ring_eid[kRing][kStreamThreads];
  __shared__ uint4 s_et[EXPH ? 2 : 1][EXPH ? VN / 4 : 1][32];       // the type table's part of this block's heads: slices of four, by lane
  const int tid = threadIdx.x, lane = tid & 31, lt = lane & ((1 << sg.ltl) - 1), groups = 32 >> sg.ltl;
  const int head = blockIdx.y * ((1 << sg.ltl) / LPH) + lt / LPH;
  const bool on = head < a.hl;
  // the list is sorted by length: a group takes every `stride`-th item, so that every warp gets its share of the long ones, and
  // the groups of a warp hold neighbours
  const long long warp = (long long)blockIdx.x * (kStreamThreads / 32) + (tid >> 5);
  const long long stride = (long long)gridDim.x * (kStreamThreads / 32) * groups;
  const long long warp0 = warp * groups, item0 = warp0 + (lane >> sg.ltl);
  if (EXPH) {
    for (int i = tid; i < 2 * (VN / 4) << sg.ltl; i += kStreamThreads) {
      const int l = i & ((1 << sg.ltl) - 1), sl = (i >> sg.ltl) % (VN / 4), t = (i >> sg.ltl) / (VN / 4);
      const int h = blockIdx.y * ((1 << sg.ltl) / LPH) + l / LPH;
      if (h < a.hl) s_et[t][sl][l] = __ldg(reinterpret_cast<const uint4*>(a.etab + (long long)t * a.hl * HN + h * HN + (l % LPH) * VN) + sl);
    }
    __syncthreads();
  }
  if (warp0 >= b.n_kv_task) return;             // the whole warp
  const int n_seg = (int)((b.n_kv_task - warp0 + stride - 1) / stride);
  auto item = [&](int r) {                      // key row, first edge, length, partial slot (-2: none)
    const long long t = item0 + r * stride;
    if (!on || t >= b.n_kv_task) return make_int4(0, 0, 0, -2);
    int4 it = __ldg(b.kv_task + t);
    it.z -= it.y;
    return it;
  };
  const int hsafe = on ? head : 0, off = hsafe * HN + (lt % LPH) * VN, w_row = a.hl * HN;
  // (the record form as a template argument: chosen at run time it cost the other one 5 % in registers)
  const char *qb, *gb;
  unsigned long long sq, sgr;
  if (PACKED) {
    qb = reinterpret_cast<const char*>(static_cast<const T*>(b.qg) + (long long)hsafe * 2 * HN + (lt % LPH) * VN);
    gb = qb + HN * sizeof(T);
    sq = sgr = (unsigned long long)w_row * 2 * sizeof(T);
  } else {
    qb = reinterpret_cast<const char*>(static_cast<const T*>(a.q) + off); sq = (unsigned long long)a.ldq * sizeof(T);
    gb = reinterpret_cast<const char*>(static_cast<const T*>(b.dout) + off); sgr = (unsigned long long)w_row * sizeof(T);
  }
  const char* zb = reinterpret_cast<const char*>(b.zd + hsafe);
  const unsigned long long szd = (unsigned long long)a.hl * sizeof(float2);
  // fetching side: items two segments ahead, the first queries of a segment one segment ahead (see RowFetch); with edge types, whose
  // place in memory comes from the list, a segment more
  constexpr int AHEAD = EXPH ? 3 : 2;
  const int mask = (1 << sg.ltl) - 1;
  int fr = 0, fi = 0, fbeg[AHEAD + 1], flen[AHEAD + 1];
  auto extent = [&](int r, int& beg, int& len) {
    const long long t = item0 + r * stride;
    beg = len = 0;
    if (t < b.n_kv_task) { const int4 x = __ldg(b.kv_task + t); beg = x.y; len = x.z - x.y; }
  };
#pragma unroll
  for (int s = 0; s <= AHEAD; ++s) extent(s, fbeg[s], flen[s]);
  int fm = steps_of(flen[0]);
  Chunk rowc{0, 0, 0}, eidc{0, 0, 0}, typec{0, 0, 0};
  int row2 = 0, eid2 = 0;                       // typed: first chunk of the segment after the next
  auto read = [&](int beg, int len, int from, int& row, int& eid) {
    if (from + lt < len) { row = __ldg(b.t_row + beg + from + lt); eid = __ldg(b.t_eid + beg + from + lt); }
  };
  auto read_type = [&](int len, int from, int eid, int& type) {
    if (EXPH && from + lt < len) type = __ldg(a.etype + eid);
  };
  read(fbeg[0], flen[0], 0, rowc.now, eidc.now);
  read(fbeg[0], flen[0], mask + 1, rowc.next, eidc.next);
  read(fbeg[1], flen[1], 0, rowc.other, eidc.other);
  read_type(flen[0], 0, eidc.now, typec.now);
  if (EXPH) {
    if (mask == 0) read_type(flen[0], 1, eidc.next, typec.next);
    read(fbeg[2], flen[2], 0, row2, eid2);
    read_type(flen[1], 0, eidc.other, typec.other);
  }
  unsigned types = 0;                           // edge type of every ring slot
  auto issue = [&](int slot) {
    const unsigned i_row = (unsigned)rowc.at(fi, mask + 1);
    const int eid = eidc.at(fi, mask + 1);
    const int ty = EXPH ? typec.at(fi, mask + 1) : 0;
    if (on && fi < flen[0]) {
      S::copy(ring[slot][0], tid, qb + i_row * sq);
      S::copy(ring[slot][1], tid, gb + i_row * sgr);
      copy_async<8>(&ring_zd[slot][tid], zb + i_row * szd);
      ring_eid[slot][tid] = eid;
      if (EXPH) types = (types & ~(1u << slot)) | ((ty ? 1u : 0u) << slot);
    }
    copy_commit();
    if (fr >= n_seg) return;
    if (++fi == fm) {
      fi = 0;
      ++fr;
      rowc.now = rowc.other; eidc.now = eidc.other; typec.now = typec.other;
#pragma unroll
      for (int s = 0; s < AHEAD; ++s) { fbeg[s] = fbeg[s + 1]; flen[s] = flen[s + 1]; }
      read(fbeg[0], flen[0], mask + 1, rowc.next, eidc.next);
      if (EXPH) {
        if (mask == 0) read_type(flen[0], 1, eidc.next, typec.next);
        rowc.other = row2; eidc.other = eid2;
        read_type(flen[1], 0, eidc.other, typec.other);
        read(fbeg[2], flen[2], 0, row2, eid2);
      } else {
        read(fbeg[1], flen[1], 0, rowc.other, eidc.other);
      }
      extent(fr + AHEAD, fbeg[AHEAD], flen[AHEAD]);
      if (fr < n_seg) fm = steps_of(flen[0]);
    } else if ((fi & mask) == 0) {
      rowc.now = rowc.next; eidc.now = eidc.next; typec.now = typec.next;
      read(fbeg[0], flen[0], fi + mask + 1, rowc.next, eidc.next);
      if (EXPH && mask == 0) read_type(flen[0], fi + 1, eidc.next, typec.next);
    } else if (EXPH && (fi & mask) == ((mask + 1) >> 1)) {
      read_type(flen[0], (fi & ~mask) + mask + 1, eidc.next, typec.next);      // the next chunk's, half a chunk ahead
    }
  };
#pragma unroll
  for (int s = 0; s < kRing - 1; ++s) issue(s);

  const T* kb = static_cast<const T*>(a.k) + off;
  const T* vb = static_cast<const T*>(a.v) + off;
  int4 it = item(0), itn = item(1);
  uint4 kn[S::N], vn[S::N];
#pragma unroll
  for (int i = 0; i < S::N; ++i) kn[i] = vn[i] = make_uint4(0, 0, 0, 0);
  if (it.w != -2) { S::load(kb + (long long)it.x * a.ldk, kn); S::load(vb + (long long)it.x * a.ldv, vn); }
  int slot = 0;
  for (int r = 0; r < n_seg; ++r) {
    f2 kf[NP], vf[NP], dk[NP], dv[NP];
    const float scale = inv_sqrt_hn<HN>();
    S::spread(kn, kf);
    S::spread(vn, vf);
#pragma unroll
    for (int i = 0; i < NP; ++i) dk[i] = dv[i] = pack2(0.f, 0.f);
    const int4 cur = it;
    it = itn;
    itn = item(r + 2);
    if (it.w != -2) { S::load(kb + (long long)it.x * a.ldk, kn); S::load(vb + (long long)it.x * a.ldv, vn); }
    const int m = steps_of(cur.z);
    for (int i = 0; i < m; ++i) {
      issue((slot + kRing - 1) & (kRing - 1));
      copy_wait<kRing - 1>();
      f2 qf[NP], gf[NP];
      S::read(ring[slot][0], tid, qf);
      S::read(ring[slot][1], tid, gf);
      const int eid = ring_eid[slot][tid];
      const float2 zd = ring_zd[slot][tid];
      if (EXPH) {                               // q * E of the edge's type enters the score and dK alike
        const uint4 (*et)[32] = s_et[(types >> slot) & 1u];
#pragma unroll
        for (int u = 0; u < NP; u += 2) {
          const uint4 e = et[u / 2][lt];
          qf[u] = mul2(qf[u], pack2(__uint_as_float(e.x), __uint_as_float(e.y)));
          qf[u + 1] = mul2(qf[u + 1], pack2(__uint_as_float(e.z), __uint_as_float(e.w)));
        }
      }
      const float d = head_sum<LPH>(dot2<NP>(qf, kf), kFull) * scale;
      const float dotv = head_sum<LPH>(dot2<NP>(gf, vf), kFull);
      if (i < cur.z) {                          // a group whose item is over holds a stale slot: nothing of it is used
        const bool inr = (d > -kClamp) && (d < kClamp);
        const float w = __expf(fminf(fmaxf(d, -kClamp), kClamp)) * zd.x;
        float mf = 1.f;
        if (VAR == 1) mf = (a.thresh && !keep_edge(a.seed, (uint32_t)eid, (uint32_t)head, a.thresh)) ? 0.f : a.inv_keep;
        const float dss = inr ? (dotv * mf - zd.y) * w * scale : 0.f;
        const float wn = w * mf;
        if ((lt % LPH) == 0) b.ds[(long long)eid * a.hl + head] = dss;
        const f2 s2 = pack2(dss, dss), w2 = pack2(wn, wn);
#pragma unroll
        for (int u = 0; u < NP; ++u) dk[u] = fma2(s2, qf[u], dk[u]);
#pragma unroll
        for (int u = 0; u < NP; ++u) dv[u] = fma2(w2, gf[u], dv[u]);
      }
      slot = (slot + 1) & (kRing - 1);
    }
    if (cur.w == -1) {
      S::store(grad_row<T>(b, b.dk, b.ck, cur.x) + off, dk);
      S::store(grad_row<T>(b, b.dv, b.cv, cur.x) + off, dv);
    } else if (cur.w >= 0) {
      float* pp = b.kv_partial + (long long)cur.w * 2 * w_row + off;
#pragma unroll
      for (int i = 0; i < NP; i += 2) { store_pairs<float, 2>(pp + 2 * i, dk + i); store_pairs<float, 2>(pp + w_row + 2 * i, dv + i); }
    }
  }
  copy_wait<0>();
}

// dQ, the second pass: dq_i = sum over the row's edges of ds * k_j [* E_type].  With the typed sums S_t = sum of ds * k_j over the
// edges of type t, dq = S_0 * E_0 + S_1 * E_1 and dE_t += q_i * S_t: one product per edge and a few per row.
template <typename T, int HN, bool EXPH>
__global__ void __launch_bounds__(kStreamThreads, EXPH ? 3 : 7) edge_attn_bwd_q_kernel(BwdArgs b, StreamGeo sg) {
  constexpr int VN = wide_elems<T, HN>(), NP = VN / 2, LPH = HN / VN;
  using S = Slices<T, VN>;
  const AttnArgs& a = b.f;
  __shared__ uint4 ring[kRing][S::N][kStreamThreads];
  __shared__ float ring_ds[kRing][kStreamThreads];
  extern __shared__ float s_detab[];            // [2, Hl*HN] when exphormer
  const int w_row = a.hl * HN;
  if (EXPH) {
    for (int i = threadIdx.x; i < 2 * w_row; i += blockDim.x) s_detab[i] = 0.f;
    __syncthreads();
  }
  const int tid = threadIdx.x, lane = tid & 31, lt = lane & ((1 << sg.ltl) - 1), groups = 32 >> sg.ltl;
  const int head = blockIdx.y * ((1 << sg.ltl) / LPH) + lt / LPH;
  const long long warp0 = ((long long)blockIdx.x * (kStreamThreads / 32) + (tid >> 5)) * groups * sg.per;
  const int n_seg = warp0 >= a.n ? 0 : (int)min((long long)sg.per, (a.n - warp0 + groups - 1) / groups);
  const Rows rows{warp0 + (lane >> sg.ltl), groups, a.n, head < a.hl};
  const int hsafe = rows.on ? head : 0, off = hsafe * HN + (lt % LPH) * VN;
  const char* kb = reinterpret_cast<const char*>(static_cast<const T*>(a.k) + off);
  const T* qb = static_cast<const T*>(a.q) + off;
  const unsigned long long skb = (unsigned long long)a.ldk * sizeof(T);
  const float* dsb = b.ds + hsafe;
  if (n_seg > 0) {
    RowFetch<EXPH> f;
    f.start(a, rows, n_seg, lane, sg.ltl);
    unsigned types = 0;
    auto issue = [&](int slot) {
      const unsigned key = (unsigned)f.key();
      const int type = f.type();
      if (rows.on && f.has()) {
        S::copy(ring[slot], tid, kb + key * skb);
        copy_async<4>(&ring_ds[slot][tid], dsb + (long long)f.edge() * a.hl);
        if (EXPH) types = (types & ~(1u << slot)) | ((type ? 1u : 0u) << slot);
      }
      copy_commit();
      f.advance(a, rows, n_seg);
    };
#pragma unroll
    for (int s = 0; s < kRing - 1; ++s) issue(s);
    int beg, len, nbeg = 0, nlen = 0;
    bool stored = rows.bounds(a, 0, beg, len), nstored = false;
    f2 de0[NP], de1[NP];
    uint4 qn[S::N];
#pragma unroll
    for (int i = 0; i < NP; ++i) de0[i] = de1[i] = pack2(0.f, 0.f);
#pragma unroll
    for (int i = 0; i < S::N; ++i) qn[i] = make_uint4(0, 0, 0, 0);
    if (EXPH && stored) S::load(qb + rows.base * a.ldq, qn);
    int slot = 0;
    for (int r = 0; r < n_seg; ++r) {
      const long long row = rows.base + (long long)r * groups;
      f2 s0[NP], s1[NP], qf[NP];
      if (EXPH) S::spread(qn, qf);
#pragma unroll
      for (int i = 0; i < NP; ++i) { s0[i] = pack2(0.f, 0.f); s1[i] = pack2(0.f, 0.f); }
      if (r + 1 < n_seg) {
        nstored = rows.bounds(a, r + 1, nbeg, nlen);
        if (EXPH && nstored) S::load(qb + (row + groups) * a.ldq, qn);
      }
      const int m = steps_of(len);
      unsigned seen = 0;                        // edge types of the row (see the dK/dV pass)
      for (int i = 0; i < m; ++i) {
        issue((slot + kRing - 1) & (kRing - 1));
        copy_wait<kRing - 1>();
        if (i < len) {
          f2 kf[NP];
          S::read(ring[slot], tid, kf);
          const float dss = ring_ds[slot][tid];
          const f2 d2 = pack2(dss, dss);
          if (EXPH) {
            const bool t1 = (types >> slot) & 1u;
            seen |= t1 ? 2u : 1u;
            if (t1) {
#pragma unroll
              for (int u = 0; u < NP; ++u) s1[u] = fma2(d2, kf[u], s1[u]);
            } else {
#pragma unroll
              for (int u = 0; u < NP; ++u) s0[u] = fma2(d2, kf[u], s0[u]);
            }
          } else {
#pragma unroll
            for (int u = 0; u < NP; ++u) s0[u] = fma2(d2, kf[u], s0[u]);
          }
        }
        slot = (slot + 1) & (kRing - 1);
      }
      if (stored) {
        if (EXPH) {
          if (seen & 1u) {
#pragma unroll
            for (int i = 0; i < NP; ++i) de0[i] = fma2(qf[i], s0[i], de0[i]);
          }
          if (seen & 2u) {
#pragma unroll
            for (int i = 0; i < NP; ++i) de1[i] = fma2(qf[i], s1[i], de1[i]);
          }
          typed_sum<NP>(a.etab + off, w_row, seen, s0, s1);
        }
        S::store(grad_row<T>(b, b.dq, b.cq, row) + off, s0);
      }
      beg = nbeg; len = nlen; stored = nstored;
    }
    copy_wait<0>();
    if (EXPH && rows.on) {
#pragma unroll
      for (int i = 0; i < NP; ++i) {
        const float2 x = unpack2(de0[i]), y = unpack2(de1[i]);
        atomicAdd(&s_detab[off + 2 * i], x.x); atomicAdd(&s_detab[off + 2 * i + 1], x.y);
        atomicAdd(&s_detab[w_row + off + 2 * i], y.x); atomicAdd(&s_detab[w_row + off + 2 * i + 1], y.y);
      }
    }
  }
  if (EXPH) {
    __syncthreads();
    for (int i = threadIdx.x; i < 2 * w_row; i += blockDim.x)
      if (s_detab[i] != 0.f) atomicAdd(b.detab + i, s_detab[i]);
  }
}

// Long rows of the dQ pass: work items as in edge_attn_fwd_long_kernel, partial dQ rows to the scratch.  The type table's gradient
// of a block's eight items meets in shared memory first, as in the regular kernel: every item would otherwise add 2 * Hl * HN
// values to the same addresses.
template <typename T, int HN, bool EXPH>
__global__ void __launch_bounds__(256, EXPH ? 3 : 4) edge_attn_bwd_q_long_kernel(BwdArgs b) {
  constexpr int VN = Vec<T>::N, NP = VN / 2, LPH = HN / VN, NB = 4;
  const AttnArgs& a = b.f;
  const Geo g = make_geo<T, HN>(a.hl);
  const int w_row = a.hl * HN;
  const int lane = threadIdx.x & 31;
  const long long warp = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const bool work = warp < (long long)a.n_long_task * g.n_hc;         // the whole warp
  extern __shared__ float s_detab[];            // [2, Hl*HN] when exphormer
  if (EXPH) {
    for (int i = threadIdx.x; i < 2 * w_row; i += blockDim.x) s_detab[i] = 0.f;
    __syncthreads();
  } else if (!work) {
    return;
  }
  if (work) {
    const int tpw = 32 / g.tl, sub = lane / g.tl, lt = lane % g.tl;
    const int item = (int)(warp / g.n_hc), hc = (int)(warp % g.n_hc);
    const int head = hc * g.hpt + lt / LPH;
    const bool head_ok = head < a.hl;
    const int hsafe = head_ok ? head : 0;
    const int off = hsafe * HN + (lt % LPH) * VN;
    const int4 it = __ldg(a.long_task + item);
    const int per = (it.z - it.y + tpw - 1) / tpw;
    const int beg = it.y + sub * per, end = min(it.z, beg + per);
    f2 s0[NP], s1[NP];
    unsigned seen = 0;                            // edge types of the item (see the dK/dV pass)
#pragma unroll
    for (int i = 0; i < NP; ++i) { s0[i] = pack2(0.f, 0.f); s1[i] = pack2(0.f, 0.f); }
    for (int e = beg; e < end; e += NB) {
      uint4 kr[NB];
      float ds[NB];
      bool t1[NB];
#pragma unroll
      for (int u = 0; u < NB; ++u) {
        const bool ok = e + u < end;
        const int j = ok ? __ldg(a.col + e + u) : 0;
        kr[u] = __ldg(reinterpret_cast<const uint4*>(static_cast<const T*>(a.k) + (long long)j * a.ldk + off));
        ds[u] = ok ? __ldg(b.ds + (long long)(e + u) * a.hl + hsafe) : 0.f;
        t1[u] = EXPH && ok && a.etype[e + u] != 0;
      }
#pragma unroll
      for (int u = 0; u < NB; ++u) {
        // an absent edge reads key 0 with weight 0: nothing may be added from it, not even 0 * inf
        if (e + u >= end) break;
        f2 kf[NP];
        widen<T>(kr[u], kf);
        const f2 d2 = pack2(ds[u], ds[u]);
        if (EXPH) seen |= t1[u] ? 2u : 1u;
        if (EXPH && t1[u]) {
#pragma unroll
          for (int i = 0; i < NP; ++i) s1[i] = fma2(d2, kf[i], s1[i]);
        } else {
#pragma unroll
          for (int i = 0; i < NP; ++i) s0[i] = fma2(d2, kf[i], s0[i]);
        }
      }
    }
    __syncwarp();
    if (EXPH) seen = __reduce_or_sync(kFull, seen);
    float x0[VN], x1[VN];
#pragma unroll
    for (int i = 0; i < NP; ++i) {
      const float2 t = unpack2(s0[i]);
      x0[2 * i] = group_total(t.x, g.tl); x0[2 * i + 1] = group_total(t.y, g.tl);
      if (EXPH) {
        const float2 y = unpack2(s1[i]);
        x1[2 * i] = group_total(y.x, g.tl); x1[2 * i + 1] = group_total(y.y, g.tl);
      }
    }
    if (sub == 0 && head_ok) {
      float* pp = a.long_partial + (long long)it.w * w_row;
      if (EXPH) {
        float qf[VN];
        load_vec<T>(static_cast<const T*>(a.q) + (long long)it.x * a.ldq + off, qf);
#pragma unroll
        for (int i = 0; i < VN; ++i) {
          if (seen & 1u) atomicAdd(&s_detab[off + i], qf[i] * x0[i]);
          if (seen & 2u) atomicAdd(&s_detab[w_row + off + i], qf[i] * x1[i]);
          x0[i] = ((seen & 1u) ? x0[i] * __ldg(a.etab + off + i) : 0.f) + ((seen & 2u) ? x1[i] * __ldg(a.etab + w_row + off + i) : 0.f);
        }
      }
#pragma unroll
      for (int i = 0; i < VN; i += 4) *reinterpret_cast<float4*>(pp + off + i) = make_float4(x0[i], x0[i + 1], x0[i + 2], x0[i + 3]);
    }
  }
  if (EXPH) {
    __syncthreads();
    for (int i = threadIdx.x; i < 2 * w_row; i += blockDim.x)
      if (s_detab[i] != 0.f) atomicAdd(b.detab + i, s_detab[i]);
  }
}

// ---------------------------------------------------------------------------------------------
// The backward pass without streams (untyped edges; see recomputed_backward): dQ first, over the queries, which also leaves the row
// terms and records, then dK/dV over the work list.  Both compute the score gradients, so none are kept: `ds` is not used.
// ---------------------------------------------------------------------------------------------
// what a query's gradient needs beside its edges
template <typename T, int HN> struct QueryTerms {
  float qs[Vec<T>::N], dof[Vec<T>::N], invz, dterm;
  __device__ __forceinline__ void load(const BwdArgs& b, int row, int head, int off, unsigned hm) {
    constexpr int VN = Vec<T>::N;
    const AttnArgs& a = b.f;
    const long long at = (long long)row * a.hl * HN + off;
    float of[VN], unused[VN];
    load_q_scaled<T, HN>(a, row, head, off, qs, unused);
    load_vec<T>(static_cast<const T*>(b.dout) + at, dof);
    load_vec<T>(static_cast<const T*>(a.out) + at, of);
    dterm = 0.f;
#pragma unroll
    for (int i = 0; i < VN; ++i) dterm += dof[i] * of[i];
    dterm = head_sum<HN / VN>(dterm, hm);
    if (a.out_thresh) dterm *= a.out_keep;      // the stored output is the dropped one, rescaled by 1 / (1 - p)
    invz = 1.f / (a.z[(long long)row * a.hl + head] + kEps);
  }
};

// two edges of one query; an absent second one is zeros (no branch between them: their sums overlap)
template <typename T, int HN>
__device__ __forceinline__ void dq_pair(const BwdArgs& b, int e, int end, int head, int off, const QueryTerms<T, HN>& t, float* dq,
                                        unsigned hm) {
  constexpr int VN = Vec<T>::N, LPH = HN / VN;
  const AttnArgs& a = b.f;
  const int j0 = __ldg(a.col + e), j1 = e + 1 < end ? __ldg(a.col + e + 1) : j0;
  Raw<T> kr[2], vr[2];
  kr[0].load(static_cast<const T*>(a.k) + (long long)j0 * a.ldk + off);
  vr[0].load(static_cast<const T*>(a.v) + (long long)j0 * a.ldv + off);
  kr[1].load_if(e + 1 < end, static_cast<const T*>(a.k) + (long long)j1 * a.ldk + off);
  vr[1].load_if(e + 1 < end, static_cast<const T*>(a.v) + (long long)j1 * a.ldv + off);
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    float d = 0.f, dv = 0.f;
#pragma unroll
    for (int i = 0; i < VN; ++i) { d += t.qs[i] * kr[u].get(i); dv += t.dof[i] * vr[u].get(i); }
    d = head_sum<LPH>(d, hm);
    dv = head_sum<LPH>(dv, hm);
    const bool inr = (d > -kClamp) && (d < kClamp) && (u == 0 || e + 1 < end);
    const float w = __expf(fminf(fmaxf(d, -kClamp), kClamp));
    float mf = 1.f;
    if (a.variant == 1) mf = (a.thresh && !keep_edge(a.seed, (uint32_t)(e + u), (uint32_t)head, a.thresh)) ? 0.f : a.inv_keep;
    const float dss = inr ? (dv * mf - t.dterm) * t.invz * w * inv_sqrt_hn<HN>() : 0.f;
#pragma unroll
    for (int i = 0; i < VN; ++i) dq[i] += dss * kr[u].get(i);
  }
}

template <typename T, int HN>
__global__ void __launch_bounds__(256, 4) edge_attn_bwd_q_rows_kernel(BwdArgs b) {
  constexpr int VN = Vec<T>::N, LPH = HN / VN;
  const AttnArgs& a = b.f;
  const Geo g = make_geo<T, HN>(a.hl);
  const int lane = threadIdx.x & 31, lt = lane % g.tl;
  const long long warp = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const long long task = warp * (32 / g.tl) + lane / g.tl;
  const bool live = task < (long long)a.n * g.n_hc;
  const int row = live ? (int)(task / g.n_hc) : 0, hc = live ? (int)(task % g.n_hc) : 0;
  const int head = hc * g.hpt + lt / LPH;
  if (!live || head >= a.hl) return;            // whole heads leave together; shuffles use head masks
  const int off = head * HN + (lt % LPH) * VN;
  const int beg = a.rowptr[row];
  int end = a.rowptr[row + 1];
  const bool cut = a.long_row > 0 && end - beg > a.long_row;
  if (cut) end = beg;
  const unsigned hm = head_mask<LPH>();
  QueryTerms<T, HN> t;
  t.load(b, row, head, off, hm);
  const long long hz = (long long)row * a.hl + head;
  if (b.qg != nullptr) {
    // narrow rows: [q | dout / (Z + eps)] and D / (Z + eps), which only dK and dV see here (4 bytes of row terms instead of 8: 7 % of
    // the dK/dV pass at 1 x 16 and 2.9 M rows)
    T* rec = static_cast<T*>(b.qg) + hz * 2 * HN + (lt % LPH) * VN;
    float gz[VN];
#pragma unroll
    for (int i = 0; i < VN; ++i) gz[i] = t.dof[i] * t.invz;
    *reinterpret_cast<uint4*>(rec) = __ldg(reinterpret_cast<const uint4*>(static_cast<const T*>(a.q) + (long long)row * a.ldq + off));
    store_vec<T>(rec + HN, gz);
    if ((lt % LPH) == 0) reinterpret_cast<float*>(b.zd)[hz] = t.dterm * t.invz;
  } else if ((lt % LPH) == 0) {
    b.zd[hz] = make_float2(t.invz, t.dterm);
  }
  float dq[VN];
#pragma unroll
  for (int i = 0; i < VN; ++i) dq[i] = 0.f;
  for (int e = beg; e < end; e += 2) dq_pair<T, HN>(b, e, end, head, off, t, dq, hm);
  if (!cut) store_vec<T>(grad_row<T>(b, b.dq, b.cq, row) + off, dq);
}

// its long rows: work items as in edge_attn_fwd_long_kernel
template <typename T, int HN>
__global__ void __launch_bounds__(256, 3) edge_attn_bwd_q_items_kernel(BwdArgs b) {
  constexpr int VN = Vec<T>::N, LPH = HN / VN;
  const AttnArgs& a = b.f;
  const Geo g = make_geo<T, HN>(a.hl);
  const int lane = threadIdx.x & 31;
  const long long warp = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (warp >= (long long)a.n_long_task * g.n_hc) return;
  const int tpw = 32 / g.tl, sub = lane / g.tl, lt = lane % g.tl;
  const int head = (int)(warp % g.n_hc) * g.hpt + lt / LPH;
  const bool head_ok = head < a.hl;
  const int hsafe = head_ok ? head : 0, off = hsafe * HN + (lt % LPH) * VN;
  const int4 it = __ldg(a.long_task + warp / g.n_hc);
  const int per = (it.z - it.y + tpw - 1) / tpw;
  const int beg = it.y + sub * per, end = min(it.z, beg + per);
  const unsigned hm = head_mask<LPH>();
  QueryTerms<T, HN> t;
  t.load(b, it.x, hsafe, off, hm);
  float dq[VN];
#pragma unroll
  for (int i = 0; i < VN; ++i) dq[i] = 0.f;
  for (int e = beg; e < end; e += 2) dq_pair<T, HN>(b, e, end, hsafe, off, t, dq, hm);
  __syncwarp();
#pragma unroll
  for (int i = 0; i < VN; ++i) dq[i] = group_total(dq[i], g.tl);
  if (sub == 0 && head_ok) {
    float* pp = a.long_partial + (long long)it.w * a.hl * HN + off;
#pragma unroll
    for (int i = 0; i < VN; i += 4) *reinterpret_cast<float4*>(pp + i) = make_float4(dq[i], dq[i + 1], dq[i + 2], dq[i + 3]);
  }
}

// one lane group per (work item, head chunk), two edges at a time: four 16-byte gathers in flight
template <typename T, int HN, bool PACKED>
__global__ void __launch_bounds__(256, 4) edge_attn_bwd_kv_rows_kernel(BwdArgs b) {
  constexpr int VN = Vec<T>::N, LPH = HN / VN;
  const AttnArgs& a = b.f;
  const Geo g = make_geo<T, HN>(a.hl);
  const int w_row = a.hl * HN;
  const int lane = threadIdx.x & 31, lt = lane % g.tl;
  const long long warp = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const long long task = warp * (32 / g.tl) + lane / g.tl;
  const bool live = task < (long long)b.n_kv_task * g.n_hc;
  const int item = live ? (int)(task / g.n_hc) : 0, hc = live ? (int)(task % g.n_hc) : 0;
  const int head = hc * g.hpt + lt / LPH;
  if (!live || head >= a.hl) return;            // whole heads leave together; shuffles use head masks
  const int off = head * HN + (lt % LPH) * VN;
  const int4 it = __ldg(b.kv_task + item);
  const T* qb = PACKED ? static_cast<const T*>(b.qg) + (long long)head * 2 * HN + (lt % LPH) * VN : static_cast<const T*>(a.q) + off;
  const T* gb = PACKED ? qb + HN : static_cast<const T*>(b.dout) + off;
  const long long sq = PACKED ? 2 * (long long)w_row : a.ldq, sg = PACKED ? sq : w_row;
  Raw<T> kf, vf;                                // this key's k | v slice stays packed for the whole item
  kf.load(static_cast<const T*>(a.k) + (long long)it.x * a.ldk + off);
  vf.load(static_cast<const T*>(a.v) + (long long)it.x * a.ldv + off);
  float dk[VN], dv[VN];
#pragma unroll
  for (int i = 0; i < VN; ++i) { dk[i] = 0.f; dv[i] = 0.f; }
  const unsigned hm = head_mask<LPH>();
  const float scale = inv_sqrt_hn<HN>();
  for (int e = it.y; e < it.z; e += 2) {
    int row[2], eid[2];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int at = min(e + u, it.z - 1);
      row[u] = __ldg(b.t_row + at);
      eid[u] = a.variant == 1 ? __ldg(b.t_eid + at) : 0;
    }
    Raw<T> qr[2], gr[2];
    float2 zd[2];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      qr[u].load_if(e + u < it.z, qb + row[u] * sq);
      gr[u].load_if(e + u < it.z, gb + row[u] * sg);
      const long long hz = (long long)row[u] * a.hl + head;
      zd[u] = PACKED ? make_float2(1.f, __ldg(reinterpret_cast<const float*>(b.zd) + hz)) : __ldg(b.zd + hz);
    }
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      float d = 0.f, dotv = 0.f;
#pragma unroll
      for (int i = 0; i < VN; ++i) { d += qr[u].get(i) * kf.get(i); dotv += gr[u].get(i) * vf.get(i); }
      d = head_sum<LPH>(d, hm) * scale;
      dotv = head_sum<LPH>(dotv, hm);
      const bool ok = u == 0 || e + 1 < it.z;   // an absent second edge is zeros, with the first's row terms
      const bool inr = (d > -kClamp) && (d < kClamp) && ok;
      const float w = __expf(fminf(fmaxf(d, -kClamp), kClamp)) * zd[u].x;
      float mf = 1.f;
      if (a.variant == 1) mf = (a.thresh && !keep_edge(a.seed, (uint32_t)eid[u], (uint32_t)head, a.thresh)) ? 0.f : a.inv_keep;
      const float dss = inr ? (dotv * mf - zd[u].y) * w * scale : 0.f, wn = ok ? w * mf : 0.f;
#pragma unroll
      for (int i = 0; i < VN; ++i) { dk[i] += dss * qr[u].get(i); dv[i] += wn * gr[u].get(i); }
    }
  }
  if (it.w < 0) {
    store_vec<T>(grad_row<T>(b, b.dk, b.ck, it.x) + off, dk);
    store_vec<T>(grad_row<T>(b, b.dv, b.cv, it.x) + off, dv);
  } else {
    float* pp = b.kv_partial + (long long)it.w * 2 * w_row + off;
#pragma unroll
    for (int i = 0; i < VN; i += 4) {
      *reinterpret_cast<float4*>(pp + i) = make_float4(dk[i], dk[i + 1], dk[i + 2], dk[i + 3]);
      *reinterpret_cast<float4*>(pp + w_row + i) = make_float4(dv[i], dv[i + 1], dv[i + 2], dv[i + 3]);
    }
  }
}

// ---------------------------------------------------------------------------------------------
// Rows cut into work items: their partial sums lie side by side in slot order.  Pass 1 gives every window of SPLIT_WINDOW
// slots to a block.  A warp takes 128 columns of one row's slots inside the window, four columns a lane, or every eighth slot of them
// where there are more than eight, adds them and finishes the row if it lies in the window whole; of a row that goes on, the window's sum replaces its first slot there.  Pass 2 adds those window sums for the rows that cross a window's end.  The association depends on the
// slot numbers alone: bit-reproducible.  A row of 10^6 edges (16 k slots) is thus 244 blocks and one short tail instead of
// one block's walk, and 10^4 rows of two or three slots are a few hundred blocks instead of 10^4 (each of 1,024 threads):
// both passes over the dK/dV slots take 103 us a layer on a 612 k-node power-law graph at h = 256 (113 with a block that walks its
// window's rows, 632 with a block per row), 22 us at 700 k nodes / h = 128 (41, 78).
// ---------------------------------------------------------------------------------------------
constexpr int SPLIT_WINDOW = 64;
constexpr int SPLIT_WARPS = 16;
constexpr int SPLIT_THREADS = 256;               // of the second pass
constexpr int SPLIT_FWD = 0, SPLIT_DQ = 1, SPLIT_KV = 2;

// s[0 .. ncol) holds the finished sums of row `row`
template <typename T, int MODE>
__device__ __forceinline__ void split_finish(const BwdArgs& b, int row, int w, int hn, const float* s) {
  const AttnArgs& a = b.f;
  if (MODE == SPLIT_FWD) {
    for (int c = threadIdx.x; c < w; c += blockDim.x) {
      const int head = c / hn;
      const float zs = s[w + head];
      float inv = 1.f / (zs + kEps);
      if (a.variant == 1) inv *= a.inv_keep;
      float ov = s[c] * inv;
      if (a.out_thresh) ov = keep_out(a, row, c) ? ov * a.out_inv_keep : 0.f;
      static_cast<T*>(a.out)[(long long)row * w + c] = from_float<T>(ov);
      if (a.route_out.n_dest) *routed<T>(a.route_out, row, c) = from_float<T>(ov);
      if (c % hn == 0) a.z[(long long)row * a.hl + head] = zs;
    }
  } else if (MODE == SPLIT_DQ) {
    T* dst = grad_row<T>(b, b.dq, b.cq, row);
    for (int c = threadIdx.x; c < w; c += blockDim.x) dst[c] = from_float<T>(s[c]);
  } else {
    T* dk = grad_row<T>(b, b.dk, b.ck, row);
    T* dv = grad_row<T>(b, b.dv, b.cv, row);
    for (int c = threadIdx.x; c < 2 * w; c += blockDim.x) (c < w ? dk + c : dv + (c - w))[0] = from_float<T>(s[c]);
  }
}

// four columns from c on (all of one head) of the finished sums of row `row`; z: the head's sum of weights (forward)
template <typename T> __device__ __forceinline__ void store4(T* p, const float* f) {
  if constexpr (sizeof(T) == 4) {
    *reinterpret_cast<float4*>(p) = make_float4(f[0], f[1], f[2], f[3]);
  } else {
    uint2 u;
    T* t = reinterpret_cast<T*>(&u);
#pragma unroll
    for (int i = 0; i < 4; ++i) t[i] = from_float<T>(f[i]);
    *reinterpret_cast<uint2*>(p) = u;
  }
}
template <typename T, int MODE>
__device__ __forceinline__ void split_finish4(const BwdArgs& b, int row, int w, int hn, int c, float* f, float z) {
  const AttnArgs& a = b.f;
  if (MODE == SPLIT_FWD) {
    float inv = 1.f / (z + kEps);
    if (a.variant == 1) inv *= a.inv_keep;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      f[i] *= inv;
      if (a.out_thresh) f[i] = keep_out(a, row, c + i) ? f[i] * a.out_inv_keep : 0.f;
    }
    store4<T>(static_cast<T*>(a.out) + (long long)row * w + c, f);
    if (a.route_out.n_dest) store4<T>(routed<T>(a.route_out, row, c), f);
    if (c % hn == 0) a.z[(long long)row * a.hl + c / hn] = z;
  } else if (MODE == SPLIT_DQ) {
    store4<T>(grad_row<T>(b, b.dq, b.cq, row) + c, f);
  } else if (c < w) {
    store4<T>(grad_row<T>(b, b.dk, b.ck, row) + c, f);
  } else {
    store4<T>(grad_row<T>(b, b.dv, b.cv, row) + c - w, f);
  }
}

// Bound by the latency of a row's reads where there are few windows: with the block walking its rows one after the other, two barriers
// each, a call took 20 to 35 us however few slots it had: 60 k nodes, 4 x 64 fp32, the three of a pass 99 us then and 31 now; 700 k nodes, 8 x 16
// bf16, four dK/dV calls 141 and 64; one row of 41 windows 9 and 4.4.  (A long row's window by the warps of its columns alone: 31.)  Heads are of 128 columns at most, so that a warp's columns hold them whole.
template <typename T, int MODE>
__global__ void __launch_bounds__(SPLIT_WARPS * 32) split_window_kernel(BwdArgs b, const int4* __restrict__ task, int n_slots,
                                                                        float* partial, int pitch, int w, int hn) {
  __shared__ int s_key[SPLIT_WINDOW], s_run[SPLIT_WINDOW + 1], s_first[2];
  static_assert(SPLIT_WINDOW == 64 && SPLIT_WARPS % 8 == 0, "two warps look for the rows' first slots, eight share a long one");
  const int s0 = blockIdx.x * SPLIT_WINDOW, n = min(SPLIT_WINDOW, n_slots - s0);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, t = threadIdx.x;
  const int before = s0 > 0 ? task[s0 - 1].x : -1, after = s0 + n < n_slots ? task[s0 + n].x : -1;
  unsigned firsts = 0;
  if (warp < 2) {
    const int key = t < n ? task[s0 + t].x : 0;
    s_key[t] = key;
    const bool first = t < n && (t == 0 || task[s0 + t - 1].x != key);
    firsts = __ballot_sync(kFull, first);
    if (lane == 0) s_first[warp] = __popc(firsts);
  }
  __syncthreads();
  const int runs = s_first[0] + s_first[1];
  if (warp < 2 && (firsts >> lane & 1u)) s_run[(warp ? s_first[0] : 0) + __popc(firsts & ((1u << lane) - 1u))] = t;
  if (t == 0) s_run[runs] = n;
  __syncthreads();
  const int width = MODE == SPLIT_KV ? 2 * w : w, chunks = (width + 127) / 128;
  auto total = [](float x0, float x1, float x2, float x3, float x4, float x5, float x6, float x7) {
    return ((x0 + x4) + (x2 + x6)) + ((x1 + x5) + (x3 + x7));
  };
  // the sums over the eight residues of the slot number in its run, in x, to the row or to the run's first slot
  auto finish = [&](int i, int j, int c, const float4 (&x)[8], const float (&xz)[8]) {
    const int key = s_key[i];
    float f[4] = {total(x[0].x, x[1].x, x[2].x, x[3].x, x[4].x, x[5].x, x[6].x, x[7].x),
                  total(x[0].y, x[1].y, x[2].y, x[3].y, x[4].y, x[5].y, x[6].y, x[7].y),
                  total(x[0].z, x[1].z, x[2].z, x[3].z, x[4].z, x[5].z, x[6].z, x[7].z),
                  total(x[0].w, x[1].w, x[2].w, x[3].w, x[4].w, x[5].w, x[6].w, x[7].w)};
    const float z = MODE == SPLIT_FWD ? total(xz[0], xz[1], xz[2], xz[3], xz[4], xz[5], xz[6], xz[7]) : 0.f;
    if (!(i == 0 && before == key) && !(j == n && after == key)) {
      split_finish4<T, MODE>(b, key, w, hn, c, f, z);
    } else {
      float* first = partial + (long long)(s0 + i) * pitch;
      *reinterpret_cast<float4*>(first + c) = make_float4(f[0], f[1], f[2], f[3]);
      if (MODE == SPLIT_FWD && c % hn == 0) first[w + c / hn] = z;
    }
  };
  for (int unit = warp; unit < runs * chunks; unit += SPLIT_WARPS) {
    const int run = unit / chunks, c = (unit - run * chunks) * 128 + 4 * lane;
    const int i = s_run[run], j = s_run[run + 1];
    if (j - i > 8) continue;
    float4 x[8];
    float xz[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const float* pp = partial + (long long)(s0 + i + u) * pitch;
      const bool on = c < width && u < j - i;
      x[u] = on ? *reinterpret_cast<const float4*>(pp + c) : make_float4(0.f, 0.f, 0.f, 0.f);
      xz[u] = MODE == SPLIT_FWD && on ? pp[w + c / hn] : 0.f;
    }
    __syncwarp();                               // all lanes of a head have read its sum of weights
    if (c < width) finish(i, j, c, x, xz);
  }
  __shared__ float4 s_x[SPLIT_WARPS][32];
  __shared__ float s_z[MODE == SPLIT_FWD ? SPLIT_WARPS : 1][32];
  for (int run = 0; run < runs; ++run) {
    const int i = s_run[run], j = s_run[run + 1];
    if (j - i <= 8) continue;
    for (int part = 0; part < chunks; part += SPLIT_WARPS / 8) {
      const int c = (part + (warp >> 3)) * 128 + 4 * lane;
      float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
      float sz = 0.f;
      if (c < width) {
        const float* pp = partial + (long long)(s0 + i) * pitch;
#pragma unroll
        for (int k = 0; k < SPLIT_WINDOW / 8; ++k) {
          const int slot = 8 * k + (warp & 7);
          if (slot < j - i) {
            const float4 x = *reinterpret_cast<const float4*>(pp + (long long)slot * pitch + c);
            sum.x += x.x; sum.y += x.y; sum.z += x.z; sum.w += x.w;
            if (MODE == SPLIT_FWD) sz += pp[(long long)slot * pitch + w + c / hn];
          }
        }
      }
      s_x[warp][lane] = sum;
      if (MODE == SPLIT_FWD) s_z[warp][lane] = sz;
      __syncthreads();
      if ((warp & 7) == 0 && c < width) {
        float4 x[8];
        float xz[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) { x[u] = s_x[warp + u][lane]; xz[u] = MODE == SPLIT_FWD ? s_z[warp + u][lane] : 0.f; }
        finish(i, j, c, x, xz);
      }
      __syncthreads();
    }
  }
}

template <typename T, int MODE>
__global__ void __launch_bounds__(SPLIT_THREADS) split_cross_kernel(BwdArgs b, const int* __restrict__ split, int n_split,
                                                                    const float* partial, int pitch, int ncol, int w, int hn) {
  extern __shared__ float s_sum[];            // [ncol]
  for (int s = blockIdx.x; s < n_split; s += gridDim.x) {
    const int first = split[3 * s + 1];
    const int w0 = first / SPLIT_WINDOW, w1 = (first + split[3 * s + 2] - 1) / SPLIT_WINDOW;
    if (w0 == w1) continue;                   // finished by its window
    for (int c = threadIdx.x; c < ncol; c += blockDim.x) {
      float acc[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) acc[u] = 0.f;
      const float* pp = partial + c;
      int k = w0 + 1;
      for (; k + 7 <= w1; k += 8) {
#pragma unroll
        for (int u = 0; u < 8; ++u) acc[u] += pp[(long long)(k + u) * SPLIT_WINDOW * pitch];
      }
      for (; k <= w1; ++k) acc[0] += pp[(long long)k * SPLIT_WINDOW * pitch];
      s_sum[c] = pp[(long long)first * pitch] + ((acc[0] + acc[4]) + (acc[2] + acc[6])) + ((acc[1] + acc[5]) + (acc[3] + acc[7]));
    }
    __syncthreads();
    split_finish<T, MODE>(b, split[3 * s], w, hn, s_sum);
    __syncthreads();
  }
}

template <typename T, int MODE>
void launch_split(const BwdArgs& b, const int4* task, int n_slots, const int* split, int n_split, float* partial, int pitch,
                  int ncol, int w, int hn, cudaStream_t st) {
  // Rows above some 6,100 elements (dK | dV; 12,000 otherwise) need more than a block's default 48 KB.  (Taking the columns in parts
  // instead, by a loop or a grid dimension, made the reduction of popular keys 15 to 65 % slower: 86 to 142 us a layer at 612 k nodes,
  // h = 256.)
  const size_t smem = sizeof(float) * ncol;
  if (smem > 48 * 1024) cudaFuncSetAttribute(split_cross_kernel<T, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  split_window_kernel<T, MODE><<<(n_slots + SPLIT_WINDOW - 1) / SPLIT_WINDOW, SPLIT_WARPS * 32, 0, st>>>(b, task, n_slots, partial, pitch, w, hn);
  split_cross_kernel<T, MODE><<<n_split < 148 * 8 ? n_split : 148 * 8, SPLIT_THREADS, smem, st>>>(b, split, n_split, partial, pitch, ncol, w, hn);
}

// Lanes of a group (VN elements each, whole heads, at most a warp), and how many segments each group takes: as many as leave two
// full loads of the chip (every SM holding `blocks_per_sm` blocks), at most `most`.
template <int HN, int VN>
StreamGeo stream_geo(int hl, long long segments, int blocks_per_sm, int most) {
  constexpr int lph = HN / VN;
  StreamGeo s;
  int tl = lph;
  while (tl * 2 <= 32 && tl / lph * 2 <= hl) tl *= 2;
  s.ltl = 0;
  while ((1 << s.ltl) < tl) ++s.ltl;
  const int chunks = (hl + tl / lph - 1) / (tl / lph);
  const long long resident = 148ll * blocks_per_sm * (kStreamThreads >> s.ltl);
  const long long per = segments * chunks / (2 * resident);
  s.per = (int)(per < 1 ? 1 : per > most ? most : per);
  return s;
}
template <int HN, int VN>
dim3 stream_grid(int hl, long long warps, const StreamGeo& s) {
  const int heads = (1 << s.ltl) / (HN / VN);
  return dim3((unsigned)((warps + kStreamThreads / 32 - 1) / (kStreamThreads / 32)), (unsigned)((hl + heads - 1) / heads));
}
// warps over n segments
inline long long stream_warps(long long n, const StreamGeo& s, int per) {
  const long long each = (32ll >> s.ltl) * per;
  return (n + each - 1) / each;
}

template <typename T, int HN, int VAR>
void launch_kv(const BwdArgs& b, cudaStream_t st) {
  constexpr int VN = wide_elems<T, HN>();
  const StreamGeo s = stream_geo<HN, VN>(b.f.hl, b.n_kv_task, 3, 8);
  const dim3 grid = stream_grid<HN, VN>(b.f.hl, stream_warps(b.n_kv_task, s, s.per), s);
  if (b.qg) edge_attn_bwd_kv_kernel<T, HN, VAR, true><<<grid, kStreamThreads, 0, st>>>(b, s);
  else edge_attn_bwd_kv_kernel<T, HN, VAR, false><<<grid, kStreamThreads, 0, st>>>(b, s);
}

// Whether the forward pass takes edge_attn_fwd_rows_kernel.  Streams hide the latency of DRAM; where the gathered rows stay in L2
// (126 MB, shared with everything else) they cost more instructions per edge than they save.  Measured, us, rows against streams:
// - fp32, 8 x 16: 10 k nodes 14 / 18, 50 k (51 MB of k and v) 76 / 117, 170 k (174 MB) 297 / 354, 300 k 406 / 410, 2 M 2155 / 1975;
//   8 x 8: 300 k (154 MB) 225 / 232, 600 k 472 / 453; 4 x 64: 60 k (123 MB) 189 / 224, 170 k (348 MB) 450 / 418
// - 16 bits, rows of up to 64 bytes (little work per lane): 1 x 16 600 k (38 MB) 60 / 96, 2.9 M (186 MB) 339 / 363; 2 x 16 600 k
//   (77 MB) 118 / 138, 2.9 M (371 MB) 681 / 624
// - 16 bits, heads of 8 (a head is one lane's 16 bytes): 8 x 8 170 k (44 MB) 83 / 98, 300 k (77 MB) 151 / 159, 600 k 222 / 206
// - 16 bits otherwise, 16 edges a row: 4 x 16 170 k (44 MB) 95 / 105, 8 x 32 50 k (51 MB) with dropout 153 / 178, 8 x 16 170 k (87 MB)
//   198 / 186; 5 to 8 edges a row: 4 x 16 110 k 57 / 49, 8 x 16 50 k 36 / 31, 8 x 32 50 k 63 / 58 (longer rows pay the streams' cost
//   per edge, short ones the other kernel's cost per row)
// - with dropout on the stored output (a hash per element, for which the streams have no issue slots left): 8 x 16, 5 edges a row, 2 k
//   5.2 / 6.2, 50 k 35 / 41, 170 k (87 MB) 128 / 144, 300 k (154 MB) 231 / 221; 8 x 32, 110 k (113 MB) 148 / 153, 170 k (174 MB) 233 / 235, 300 k 420 /
//   399; 8 x 8, 700 k (179 MB) 279 / 302
// - typed edges (two scaled queries, a select per element): 8 x 32, 25 edges, 50 k 167 / 201, 390 k (400 MB) 1879 / 1893
//
// The figures above, and the rule for them, are for query rows of much the same length (a budgeted graph: the builder's bound on the
// row length is known, or only a few virtual nodes' rows exceed it).  A lane group of a stream walks several rows one after another and a warp
// waits for its longest group, so rows that differ (an edge list with Poisson degrees, say: no bound is known) cost the streams 10 to
// 30 % that a warp of one row does not lose.  Measured there with a cold L2, us, rows against streams; 4 / 10 / 20 edges a row:
// - fp32, 4 x 64: 60 k (123 MB) 92 / 108, 143 / 225, 294 / 456; 150 k (307 MB) 223 / 192, 360 / 379, 652 / 767; 400 k (819 MB) 604 / 496, 1012 / 994,
//   1783 / 1914; 8 x 8: 150 k (77 MB) 68 / 91, 102 / 199, 210 / 349; 400 k (205 MB) 174 / 143, 276 / 311, 495 / 540
// - 16 bits, 8 x 8: 150 k (38 MB) 50 / 78, 76 / 164, 159 / 284; 400 k (102 MB) 123 / 120, 197 / 234, 353 / 386; 4 x 64: 60 k (61 MB) 66 / 79,
//   103 / 154, 228 / 314; 150 k (154 MB) 155 / 119, 252 / 256, 480 / 470
inline bool rows_forward(int dtype, long long n, int hl, int hn, int variant, bool out_dropout, long long n_edges, bool irregular) {
  const long long row = (long long)hl * hn * (dtype == BF_FP32 ? 4 : 2), gathered = 2 * n * row;
  if (variant == 2) return true;
  if (irregular) {
    const bool deep = n_edges >= 8 * n;
    if (dtype == BF_FP32) return n_edges >= 16 * n || gathered <= (deep ? 320'000'000 : 200'000'000);
    if (row <= 64) return gathered <= 200'000'000;
    if (hn == 8) return gathered <= (deep ? 250'000'000 : out_dropout ? 200'000'000 : 120'000'000);
    return gathered <= (out_dropout ? 120'000'000 : deep ? 100'000'000 : 64'000'000);
  }
  if (dtype == BF_FP32 || row <= 64 || (hn == 8 && out_dropout)) return gathered <= 200'000'000;
  if (hn == 8) return gathered <= 100'000'000;
  if (out_dropout) return gathered <= 120'000'000;
  return n_edges >= 12 * n && gathered <= 64'000'000;
}

template <typename T, int HN>
cudaError_t launch_fwd_t(const AttnArgs& a, bool rows, int chunks_per_hub, cudaStream_t st) {
  const Geo g = make_geo<T, HN>(a.hl);
  if (a.n > 0 && rows) {
    const int tpw = 32 / g.tl;
    const long long warps = ((long long)a.n * g.n_hc + tpw - 1) / tpw;
    edge_attn_fwd_rows_kernel<T, HN><<<(unsigned)((warps + 7) / 8), 256, 0, st>>>(a);
  } else if (a.n > 0) {
    constexpr int VN = wide_elems<T, HN>();
    const StreamGeo s = stream_geo<HN, VN>(a.hl, a.n, 4, 8);
    const dim3 grid = stream_grid<HN, VN>(a.hl, stream_warps(a.n, s, s.per), s);
    if (a.variant == 1) edge_attn_fwd_kernel<T, HN, true><<<grid, kStreamThreads, 0, st>>>(a, s);
    else edge_attn_fwd_kernel<T, HN, false><<<grid, kStreamThreads, 0, st>>>(a, s);
  }
  if (a.n_long_task > 0) {
    edge_attn_fwd_long_kernel<T, HN><<<(unsigned)(((long long)a.n_long_task * g.n_hc + 7) / 8), 256, 0, st>>>(a);
    BwdArgs b{};
    b.f = a;
    const int w = a.hl * HN, pitch = fwd_pitch(w, a.hl);
    launch_split<T, SPLIT_FWD>(b, a.long_task, a.n_long_task, a.long_split, a.n_long_split, a.long_partial, pitch, w + a.hl, w, HN, st);
  }
  if (a.n_hub > 0) {
    edge_attn_fwd_hub_kernel<T, HN><<<a.n_hub * chunks_per_hub, 256, 0, st>>>(a, chunks_per_hub);
    edge_attn_fwd_hub_finalize<T, HN><<<a.n_hub, 256, 0, st>>>(a);
  }
  return cudaGetLastError();
}

// shared memory for the gradient of the two rows of the type table
inline size_t type_table_bytes(int w_row) { return sizeof(float) * 2 * (size_t)w_row; }

// Whether the backward pass computes the score gradients twice instead of keeping them in `ds` (untyped edges).  `ds` holds 4 bytes
// per edge and head, and the dK/dV pass writes them edge by edge in another order than they lie in: with one or two heads every
// write is a sector of its own.  Measured, us, dQ and dK/dV of this form against row terms, dK/dV and dQ of the streams:
// - rows of 32 bytes: 1 x 16 bf16, 50 k 44 / 47, 170 k 78 / 84, 600 k 217 / 274, 2.9 M 963 / 1233
// - rows of 64 bytes: 2 x 16 bf16, 170 k (22 MB of k and v) 104 / 98, 300 k (38 MB) 205 / 188, 600 k (77 MB) 375 / 400, 2.9 M 1557 / 1654
// - fp32, rows of 512 bytes and more that stay in L2 (the dK/dV stream holds 12 warps an SM, this form 32): 8 x 16, 2 k 26 / 32, 10 k
//   41 / 43, 50 k (51 MB) with 16 edges a row 219 / 253 and with five 121 / 111, 110 k (113 MB) 356 / 311; 4 x 64, 10 k (20 MB) 61 / 66,
//   50 k (102 MB) 248 / 190; 8 x 8, 10 k 37 / 32, 50 k 136 / 117
//
// As in rows_forward, those are rows of much the same length.  Where no bound is known, with a cold L2, 4 / 10 / 20 edges a row:
// - fp32, 8 x 8 (256 bytes): 60 k (31 MB) 103 / 97, 144 / 141, 257 / 254; 150 k (77 MB) 201 / 202, 305 / 322, 519 / 558; 4 x 64: 20 k (41 MB)
//   136 / 142, 202 / 229, 309 / 375; 60 k (123 MB) 314 / 316, 457 / 513, 739 / 854 (416 / 400 where degrees are even); 150 k (307 MB) 687 / 604,
//   1097 / 1027, 1798 / 1746
// - 16 bits, 3 x 16 (96 bytes): 20 k 87 / 97, 97 / 111, 143 / 157; 400 k (77 MB) 336 / 408, 546 / 817, 921 / 1503; 8 x 8: 150 k (38 MB) 142 / 169,
//   215 / 288, 368 / 472; 400 k (102 MB) 315 / 360, 514 / 603, 874 / 993; 4 x 64: 20 k (20 MB) 114 / 110, 136 / 134, 292 / 280; 60 k (61 MB)
//   217 / 197, 317 / 301, 604 / 630; 400 k (410 MB) 1099 / 811, 1862 / 1411, 3301 / 2666
// Heads that leave lanes of the streams' groups idle (12 x 16 in groups of 8 heads) are counted by what the groups hold.
inline bool recomputed_backward(int dtype, long long n, int hl, int hn, int variant, long long n_edges, bool irregular) {
  const long long row = (long long)hl * hn * (dtype == BF_FP32 ? 4 : 2), gathered = 2 * n * row;
  if (variant == 2) return false;
  if (irregular) {
    const bool deep = n_edges >= 8 * n;
    if (row <= 96) return true;
    if (dtype == BF_FP32) return row <= 128 || gathered <= (deep ? 110'000'000 : 60'000'000);
    if (hn == 8) return gathered <= 160'000'000;
    const int lanes = hn / 16;                                                  // of a head: 32 bytes each
    int heads = 1;                                                              // of a group
    while (2 * heads * lanes <= 32 && 2 * heads <= hl) heads *= 2;
    if (5 * ((hl + heads - 1) / heads * heads) > 6 * hl) return gathered <= (deep ? 110'000'000 : 30'000'000);
    return gathered <= 10'000'000;
  }
  if (row <= 32) return true;
  if (row <= 64) return gathered > 64'000'000;
  return dtype == BF_FP32 && row >= 512 && gathered <= 64'000'000;
}

template <typename T, int HN>
cudaError_t launch_recomputed_bwd_t(const BwdArgs& b, cudaStream_t st) {
  const AttnArgs& a = b.f;
  const Geo g = make_geo<T, HN>(a.hl);
  const int w_row = a.hl * HN, tpw = 32 / g.tl;
  auto blocks = [&](long long rows) { return (unsigned)(((rows * g.n_hc + tpw - 1) / tpw + 7) / 8); };
  if (a.n > 0) edge_attn_bwd_q_rows_kernel<T, HN><<<blocks(a.n), 256, 0, st>>>(b);
  if (a.n_long_task > 0) {
    edge_attn_bwd_q_items_kernel<T, HN><<<(unsigned)(((long long)a.n_long_task * g.n_hc + 7) / 8), 256, 0, st>>>(b);
    launch_split<T, SPLIT_DQ>(b, a.long_task, a.n_long_task, a.long_split, a.n_long_split, a.long_partial, w_row, w_row, w_row, HN, st);
  }
  if (b.n_kv_task > 0) {
    if (b.qg) edge_attn_bwd_kv_rows_kernel<T, HN, true><<<blocks(b.n_kv_task), 256, 0, st>>>(b);
    else edge_attn_bwd_kv_rows_kernel<T, HN, false><<<blocks(b.n_kv_task), 256, 0, st>>>(b);
  }
  if (b.n_kv_split > 0)
    launch_split<T, SPLIT_KV>(b, b.kv_task, b.n_kv_slots, b.kv_split, b.n_kv_split, b.kv_partial, 2 * w_row, 2 * w_row, w_row, HN, st);
  return cudaGetLastError();
}

template <typename T, int HN>
cudaError_t launch_bwd_t(const BwdArgs& b, cudaStream_t st) {
  const AttnArgs& a = b.f;
  const Geo g = make_geo<T, HN>(a.hl);
  const int w_row = a.hl * HN;
  if (b.ds == nullptr) return launch_recomputed_bwd_t<T, HN>(b, st);
  if (a.n > 0) {
    constexpr int VN = wide_elems<T, HN>();
    const StreamGeo s = stream_geo<HN, VN>(a.hl, 0, 1, 1);
    edge_attn_bwd_delta_kernel<T, HN><<<stream_grid<HN, VN>(a.hl, stream_warps(a.n, s, 1), s), kStreamThreads, 0, st>>>(b, s);
  }
  if (b.n_kv_task > 0) {
    if (a.variant == 2) launch_kv<T, HN, 2>(b, st);
    else if (a.variant == 1) launch_kv<T, HN, 1>(b, st);
    else launch_kv<T, HN, 0>(b, st);
  }
  // the items of split keys come first in the list, so item i of them is slot i
  if (b.n_kv_split > 0)
    launch_split<T, SPLIT_KV>(b, b.kv_task, b.n_kv_slots, b.kv_split, b.n_kv_split, b.kv_partial, 2 * w_row, 2 * w_row, w_row, HN, st);
  if (a.n > 0) {
    if (a.variant == 2) {
      // every block ends in 2 * Hl * HN atomics: longer streams where the rows allow it
      constexpr int VN = wide_elems<T, HN>();
      const StreamGeo s = stream_geo<HN, VN>(a.hl, a.n, 3, 32);
      constexpr size_t ring = kRing * kStreamThreads * (VN * sizeof(T) + sizeof(float));
      if (type_table_bytes(w_row) + ring > 48 * 1024 && type_table_bytes(w_row) <= 48 * 1024) {
        // beside the ring (10 or 18 KB) the type table's gradient of wide rows goes over the default 48 KB of a block
        const cudaError_t e = cudaFuncSetAttribute(edge_attn_bwd_q_kernel<T, HN, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, 48 * 1024);
        if (e != cudaSuccess) return e;
      }
      edge_attn_bwd_q_kernel<T, HN, true><<<stream_grid<HN, VN>(a.hl, stream_warps(a.n, s, s.per), s), kStreamThreads, type_table_bytes(w_row), st>>>(b, s);
    } else {
      constexpr int VN = wide_elems<T, HN>();
      const StreamGeo s = stream_geo<HN, VN>(a.hl, a.n, 7, 8);
      edge_attn_bwd_q_kernel<T, HN, false><<<stream_grid<HN, VN>(a.hl, stream_warps(a.n, s, s.per), s), kStreamThreads, 0, st>>>(b, s);
    }
  }
  if (a.n_long_task > 0) {
    const unsigned lb = (unsigned)(((long long)a.n_long_task * g.n_hc + 7) / 8);
    if (a.variant == 2) edge_attn_bwd_q_long_kernel<T, HN, true><<<lb, 256, type_table_bytes(w_row), st>>>(b);
    else edge_attn_bwd_q_long_kernel<T, HN, false><<<lb, 256, 0, st>>>(b);
    launch_split<T, SPLIT_DQ>(b, a.long_task, a.n_long_task, a.long_split, a.n_long_split, a.long_partial, w_row, w_row, w_row, HN, st);
  }
  return cudaGetLastError();
}

AttnArgs to_args(const bf_attn_params& p) {
  AttnArgs a;
  a.q = p.q; a.k = p.k; a.v = p.v; a.ldq = p.ldq; a.ldk = p.ldk; a.ldv = p.ldv;
  a.out = p.out; a.z = p.z; a.rowptr = p.rowptr; a.col = p.col; a.etype = p.etype; a.etab = p.etab;
  a.n = p.n; a.hl = p.hl; a.variant = p.variant;
  a.inv_keep = p.dropout_p > 0.f ? 1.f / (1.f - p.dropout_p) : 1.f;
  a.thresh = p.dropout_p > 0.f ? (uint32_t)(p.dropout_p * 4294967296.0) : 0u;
  a.seed = p.dropout_seed;
  a.out_thresh = p.out_dropout_p > 0.f ? (uint32_t)(p.out_dropout_p * 4294967296.0) : 0u;
  a.out_seed = p.out_dropout_seed;
  a.out_keep = 1.f - p.out_dropout_p;
  a.out_inv_keep = p.out_dropout_p > 0.f ? 1.f / (1.f - p.out_dropout_p) : 1.f;
  a.out_rows_local = p.out_rows_local; a.out_col0 = p.out_col0;
  a.hub_rows = p.hub_rows; a.n_hub = p.n_hub; a.hub_chunk = BF_HUB_CHUNK; a.hub_scratch = p.hub_scratch;
  a.long_row = p.n_hub > 0 ? BF_HUB_DEGREE : 0;
  a.long_task = nullptr; a.n_long_task = 0; a.long_split = nullptr; a.n_long_split = 0; a.long_partial = nullptr;
  memset(&a.route_out, 0, sizeof(a.route_out));
  return a;
}

// A caller's list of long rows (false: reject the call).  It replaces the hub list.
bool take_long_rows(const bf_long_rows* r, AttnArgs* a) {
  if (r == nullptr || r->n_task <= 0) return true;
  if (r->task == nullptr || ((uintptr_t)r->task) % 16 != 0 || r->split == nullptr || r->n_split <= 0 || r->partial == nullptr ||
      ((uintptr_t)r->partial) % 16 != 0 || r->min_degree <= 0 || a->n_hub > 0)
    return false;
  a->long_row = r->min_degree;
  a->long_task = reinterpret_cast<const int4*>(r->task); a->n_long_task = r->n_task;
  a->long_split = r->split; a->n_long_split = r->n_split; a->long_partial = r->partial;
  return true;
}

// Validated copy of a caller's route for `n` rows of `width` elements each; false = reject the call.
bool to_route(const bf_attn_route* r, int n, long long width, Route* out) {
  memset(out, 0, sizeof(*out));
  if (r == nullptr || r->n_dest <= 0) return true;
  if (r->n_dest > BF_MAX_PEERS || r->rows_per <= 0 || (long long)r->rows_per * r->n_dest != n || r->ld < width || r->ld % 8 != 0 ||
      r->slab_row0 < 0 || r->slab_row0 + r->rows_per > (long long)r->rows_per * r->n_dest)
    return false;
  for (int i = 0; i < r->n_dest; ++i) {
    if (r->base[i] == nullptr || ((uintptr_t)r->base[i]) % 16 != 0) return false;
    out->base[i] = (unsigned long long)(uintptr_t)r->base[i];
  }
  out->n_dest = r->n_dest; out->rows_per = r->rows_per; out->ld = r->ld; out->slab_row0 = r->slab_row0;
  return true;
}

}  // namespace

#define BF_DISPATCH(DT, HN, CALL)                                                           \
  do {                                                                                      \
    if (DT == BF_BF16) {                                                                    \
      if (HN == 16) return CALL(__nv_bfloat16, 16); if (HN == 32) return CALL(__nv_bfloat16, 32); \
      if (HN == 64) return CALL(__nv_bfloat16, 64); if (HN == 8) return CALL(__nv_bfloat16, 8);   \
      if (HN == 128) return CALL(__nv_bfloat16, 128);                                       \
    } else if (DT == BF_FP16) {                                                             \
      if (HN == 16) return CALL(__half, 16); if (HN == 32) return CALL(__half, 32);         \
      if (HN == 64) return CALL(__half, 64); if (HN == 8) return CALL(__half, 8);           \
      if (HN == 128) return CALL(__half, 128);                                              \
    } else if (DT == BF_FP32) {                                                             \
      if (HN == 16) return CALL(float, 16); if (HN == 32) return CALL(float, 32);           \
      if (HN == 64) return CALL(float, 64); if (HN == 8) return CALL(float, 8);             \
      if (HN == 128) return CALL(float, 128);                                               \
    }                                                                                       \
  } while (0)

extern "C" size_t bf_attn_fwd_long_pitch(int hl, int hn) { return (size_t)fwd_pitch(hl * hn, hl); }

extern "C" int bf_edge_attn_fwd_routed(const bf_attn_params* p, const bf_attn_route* route, const bf_long_rows* long_rows,
                                       long long n_edges, int irregular, cudaStream_t st) {
  AttnArgs a = to_args(*p);
  if (!take_long_rows(long_rows, &a)) return (int)cudaErrorInvalidValue;
  if (!to_route(route, p->n, (long long)p->hl * p->hn, &a.route_out)) return (int)cudaErrorInvalidValue;
  const int chunks = p->max_hub_degree > 0 ? (p->max_hub_degree + BF_HUB_CHUNK - 1) / BF_HUB_CHUNK : 1;
  const bool rows = rows_forward(p->dtype, p->n, p->hl, p->hn, p->variant, p->out_dropout_p > 0.f, n_edges, irregular != 0);
#define CALL_FWD(T, H) (int)launch_fwd_t<T, H>(a, rows, chunks, st)
  BF_DISPATCH(p->dtype, p->hn, CALL_FWD);
#undef CALL_FWD
  return (int)cudaErrorInvalidValue;
}

extern "C" int bf_edge_attn_fwd(const bf_attn_params* p, cudaStream_t st) {
  AttnArgs a = to_args(*p);
  const int chunks = p->max_hub_degree > 0 ? (p->max_hub_degree + BF_HUB_CHUNK - 1) / BF_HUB_CHUNK : 1;
  const bool rows = rows_forward(p->dtype, p->n, p->hl, p->hn, p->variant, p->out_dropout_p > 0.f, -1, false);       // the number of edges is not known here
#define CALL_FWD(T, H) (int)launch_fwd_t<T, H>(a, rows, chunks, st)
  BF_DISPATCH(p->dtype, p->hn, CALL_FWD);
#undef CALL_FWD
  return (int)cudaErrorInvalidValue;
}

extern "C" int bf_attn_bwd_keeps_scores(int dtype, long long n, int hl, int hn, int variant, long long n_edges, int irregular) {
  return recomputed_backward(dtype, n, hl, hn, variant, n_edges, irregular != 0) ? 0 : 1;
}

extern "C" int bf_edge_attn_bwd(const bf_attn_params* p, const bf_attn_bwd_params* q, cudaStream_t st) {
  BwdArgs b;
  b.f = to_args(*p);
  if (b.f.n_hub > 0 || !take_long_rows(&q->long_rows, &b.f) || q->kv_task == nullptr) return (int)cudaErrorInvalidValue;
  if (p->variant == 2 && q->ds == nullptr) return (int)cudaErrorInvalidValue;
  b.dout = q->dout; b.dq = q->dq; b.dk = q->dk; b.dv = q->dv;
  b.ldg = q->ldg > 0 ? q->ldg : (long long)p->hl * p->hn;
  b.zd = reinterpret_cast<float2*>(q->zd);
  b.ds = q->ds;
  b.t_row = q->t_row; b.t_eid = q->t_eid; b.detab = q->detab;
  b.kv_task = reinterpret_cast<const int4*>(q->kv_task); b.n_kv_task = q->n_kv_task;
  b.kv_split = q->kv_split; b.n_kv_split = q->n_kv_split; b.n_kv_slots = q->n_kv_split > 0 ? q->n_kv_slots : 0; b.kv_partial = q->kv_partial;
  if (b.n_kv_split > 0 && (b.kv_split == nullptr || b.kv_partial == nullptr || b.n_kv_slots <= 0 || b.n_kv_slots > b.n_kv_task))
    return (int)cudaErrorInvalidValue;
  b.qg = q->qg;
  b.cq = q->route_cq; b.ck = q->route_ck; b.cv = q->route_cv;
  {
    // a routed row is [.. ck: dk .. cv: dv .. cq: dq ..]: every part must fit the destination's row stride
    const long long w = (long long)p->hl * p->hn;
    const long long hi = (long long)(b.cq > b.ck ? (b.cq > b.cv ? b.cq : b.cv) : (b.ck > b.cv ? b.ck : b.cv)) + w;
    if (!to_route(&q->route, p->n, q->route.n_dest > 0 ? hi : w, &b.route)) return (int)cudaErrorInvalidValue;
    if (b.route.n_dest > 0 && (b.cq < 0 || b.ck < 0 || b.cv < 0 || ((b.cq | b.ck | b.cv) % 8) != 0))
      return (int)cudaErrorInvalidValue;
  }
#define CALL_BWD(T, H) (int)launch_bwd_t<T, H>(b, st)
  BF_DISPATCH(p->dtype, p->hn, CALL_BWD);
#undef CALL_BWD
  return (int)cudaErrorInvalidValue;
}

// ---------------------------------------------------------------------------------------------------
// Allocation-free variant of the forward entry point (declared and documented in bf_noalloc.h).
// ---------------------------------------------------------------------------------------------------
#include "bf_noalloc.h"

#include <mutex>

// Scratch of the long-row kernels for callers that cannot allocate.  In host code this name is only a handle for
// the runtime (it is not a device address); the address is resolved per device below.
static __device__ __align__(256) float g_bf_noalloc_scratch[BF_NOALLOC_SCRATCH_FLOATS];

namespace {
constexpr int kMaxDevices = 64;
float* g_noalloc_ptr[kMaxDevices] = {nullptr};
std::mutex g_noalloc_mutex;

// Device address of the scratch array on the current device (looked up once per device).
int noalloc_scratch_ptr(float** out) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess || dev < 0 || dev >= kMaxDevices) return BF_NOALLOC_ERR_SETUP;
  std::lock_guard<std::mutex> lock(g_noalloc_mutex);
  if (g_noalloc_ptr[dev] == nullptr) {
    float* ptr = nullptr;
    e = cudaGetSymbolAddress(reinterpret_cast<void**>(&ptr), g_bf_noalloc_scratch);
    if (e != cudaSuccess || ptr == nullptr) return BF_NOALLOC_ERR_SETUP;
    g_noalloc_ptr[dev] = ptr;
  }
  *out = g_noalloc_ptr[dev];
  return 0;
}
}  // namespace

extern "C" int bf_edge_attn_fwd_noalloc(const bf_attn_params* p, cudaStream_t stream) {
  if (p == nullptr) return (int)cudaErrorInvalidValue;
  const long long width = (long long)p->hl * p->hn;
  if (p->n_hub < 0 || p->n_hub > BF_NOALLOC_MAX_HUBS || width > BF_NOALLOC_MAX_WIDTH || p->hl > BF_NOALLOC_MAX_HEADS)
    return BF_NOALLOC_ERR_TOO_LARGE;
  // everything the launcher would reject is rejected here, before anything is queued on the stream
  const bool hn_ok = p->hn == 8 || p->hn == 16 || p->hn == 32 || p->hn == 64 || p->hn == 128;
  const bool dtype_ok = p->dtype == BF_BF16 || p->dtype == BF_FP16 || p->dtype == BF_FP32;
  if (!hn_ok || !dtype_ok || p->n <= 0 || p->hl <= 0) return (int)cudaErrorInvalidValue;
  if (p->n_hub > 0 && (p->hub_rows == nullptr || p->max_hub_degree <= 0)) return (int)cudaErrorInvalidValue;
  bf_attn_params q = *p;
  q.hub_scratch = nullptr;
  if (p->n_hub > 0) {
    float* scratch = nullptr;
    const int rc = noalloc_scratch_ptr(&scratch);
    if (rc != 0) return rc;
    // the array keeps the previous call's sums: clear the part this call accumulates into
    const size_t bytes = sizeof(float) * (size_t)p->n_hub * (size_t)(width + p->hl);
    const cudaError_t e = cudaMemsetAsync(scratch, 0, bytes, stream);
    if (e != cudaSuccess) return (int)e;
    q.hub_scratch = scratch;
  }
  return bf_edge_attn_fwd(&q, stream);
}

extern "C" size_t bf_attn_params_size(void) { return sizeof(bf_attn_params); }

extern "C" const char* bf_noalloc_strerror(int code) {
  switch (code) {
    case 0: return "success";
    case BF_NOALLOC_ERR_TOO_LARGE:
      return "bf_edge_attn_fwd_noalloc: problem exceeds the built-in scratch (n_hub <= 64, hl*hn <= 1024, hl <= 64)";
    case BF_NOALLOC_ERR_SETUP:
      return "bf_edge_attn_fwd_noalloc: could not resolve the device address of the built-in scratch array";
    default: return code > 0 ? cudaGetErrorString((cudaError_t)code) : "unknown error";
  }
}
