// Feed-forward block with the hidden tile kept on chip, for sm_100a:
//
//     H = drop1(act(X W1^T + b1))            [128 rows x F hidden]   from tensor memory to shared memory, not to HBM
//     Y = [X | R +] drop2(H W2^T + b2)       [128 rows x D]
//
// for layers whose two weight matrices (D = 128, F = 256: 2 x 64 KB; D = 64, F = 128: 2 x 16 KB) stay in shared memory for the whole
// persistent kernel.  The hidden width is worked on in units of 128 columns, u = 0, 1, 2, ... over the CTA's tiles:
//
//   producer warp   TMA-loads X tiles (64-column panels, 128-byte swizzle) into two or four buffers, free again when GEMM1 has read them
//   MMA warp        GEMM1 of unit u + 2 into one of two accumulators once GEMM2 of unit u has read it; GEMM2 of unit u, when its hidden
//                   columns are a 16-bit operand in tensor memory, onto the tile's output accumulator (two of them)
//   16 epilogue     two teams of eight, unit u to team u & 1: tcgen05.ld -> bias, ReLU / GELU, dropout -> 16-bit -> tcgen05.st over the
//   warps           accumulator columns the warp read, from where GEMM2 takes its A operand; then a 64-column panel of the output of the team's
//                   tile before (its second product ran meanwhile): bias, dropout, residual.  The teams meet only through the products, so
//                   that one computes while the other waits for tensor memory.  What a warp stores, 32 rows x 32 columns at a time, goes
//                   through its own 2 KB of shared memory and a TMA store (64-byte swizzle): no barrier among warps anywhere.
//
// Without a backward pass the kernel moves X in and Y out.  A training forward asks for side outputs: the hidden matrix
// (stored from registers, 64 bytes a lane, it took 95 us of 235 at 800 k rows); for ReLU one bit per element (value > 0); for GELU the pre-activation, rounded, of
// which the activation is then taken (round_z: also without that output, so that evaluation and the first pass of a recomputed layer
// give what a training pass gives).  Dropout masks are the hash masks of the GEMM epilogues, so a recomputation on the
// two-GEMM path reproduces them.
//
// Bound by the ALU pipe of the epilogue: the dropout hash, selection and packing of a hidden element take a scheduler 18 cycles a warp,
// which is 2.5 us a tile of 128 x 256 against 1.5 to 3 us for its bytes.  us before (all sixteen warps on
// one unit, its operand through one shared-memory buffer, GELU by erff; bf16 128 / 256 only, the rest two GEMMs) and now, at 800 k rows 128 / 256:
// ReLU without a backward pass 182 / 137, with dropout, hidden matrix and bits 314 / 255; GELU 575 / 209, with z and hidden matrix 633 / 299; at
// 300 k rows 64 / 128: ReLU 79 / 33 and 97 / 53, GELU 136 / 47 and 144 / 64; fp16 at 50 k rows 128 / 256: ReLU 42 / 21 and 50 / 31.  Hidden operands
// in tensor-memory columns of their own (GEMM1 of unit u + 2 ahead of GEMM2 of unit u) were no faster: 142, 255, 216, 315.
// Every mbarrier wait is bounded (status word, early return, tensor memory freed).  Replaces Linear -> act -> Dropout -> Linear -> Dropout
// -> add of the reference layers (models/gt_dist_node_level.py:655-660, models/graphormer_dist_node_level.py:48-60).
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <string.h>

#include "bf_kernels.h"
#include "epilogue.cuh"
#include "sm100_ptx.cuh"

namespace {

constexpr int FF_M = 128;            // rows per tile
constexpr int FF_HC = 128;           // hidden columns of a unit
constexpr int FF_PANEL = FF_M * 128; // bytes of one 64-column panel of 128 rows
constexpr int FF_EPI_WARPS = 16;
constexpr int FF_THREADS = 32 * (2 + FF_EPI_WARPS);
constexpr int FF_MAX_X = 4;
constexpr int FF_BLOCK = 32 * 64;    // a warp's staging buffer: 32 rows of 32 columns
constexpr int FF_TEAM_WARPS = FF_EPI_WARPS / 2;

struct FfnArgs {
  int M, m_tiles;
  const float* b1;               // [F] or null
  const float* b2;               // [D] or null
  uint32_t thresh1, seed1;       // dropout on the hidden tile
  float scale1;
  uint32_t thresh2, seed2;       // dropout on the output before the residual (thresh 0 = off)
  float scale2;
  const unsigned short* res;     // residual [M, ldr] or null
  long long ldr;
  uint32_t one;                  // 1
  int* status;
  // side outputs of a training forward
  int keep_h, keep_z;
  unsigned short* bits_out;      // [F / 16, ldmb >= M] or null
  long long ldmb;
  int round_z;                   // with side outputs: GELU of the rounded pre-activation (without: ACT 3)
};

struct FfnControl {
  uint64_t w_full;
  uint64_t x_full[FF_MAX_X], x_empty[FF_MAX_X];
  uint64_t acc1_full[2];                     // GEMM1 of a unit has retired
  uint64_t hidden_full[2], hidden_done[2];   // its hidden columns are in place, GEMM2 has read them
  uint64_t acc2_full[2], acc2_empty[2];
  uint32_t tmem_base;
  int abort_flag;
};

__device__ __forceinline__ uint32_t ff_instr_desc(int n, bool fp16) {
  uint32_t d = 0;
  d |= 1u << 4;                                  // accumulator fp32
  d |= (fp16 ? 0u : 1u) << 7;                    // A format: 0 fp16, 1 bf16
  d |= (fp16 ? 0u : 1u) << 10;                   // B format
  d |= (uint32_t)(n >> 3) << 17;                 // N / 8
  d |= (uint32_t)(FF_M >> 4) << 24;              // M / 16
  return d;
}

// D (+)= A[tmem] * B[smem]: lane = row, a 32-bit column holds two neighbouring K elements
__device__ __forceinline__ void umma_f16_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc, uint32_t accum) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(tmem_d), "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accum)
      : "memory");
}
__device__ __forceinline__ void tmem_st_32x32b_x16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
      "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}
// COLS accumulator columns from TMEM column `taddr` as pairs
template <int COLS> __device__ __forceinline__ void ff_load(uint32_t taddr, f2 (&v)[COLS / 2]) {
  uint32_t r[COLS];
#pragma unroll
  for (int i = 0; i < COLS; i += 16) tmem_ld_32x32b_x16(taddr + (uint32_t)i, r + i);
  tmem_ld_wait();
#pragma unroll
  for (int i = 0; i < COLS / 2; ++i) v[i] = pack2(__uint_as_float(r[2 * i]), __uint_as_float(r[2 * i + 1]));
}
template <int COLS> __device__ __forceinline__ void ff_add_bias(const float* s_bias, f2 (&v)[COLS / 2]) {
  const ulonglong2* bp = reinterpret_cast<const ulonglong2*>(s_bias);
#pragma unroll
  for (int i = 0; i < COLS / 4; ++i) {
    const ulonglong2 b = bp[i];
    v[2 * i] = add2(v[2 * i], b.x); v[2 * i + 1] = add2(v[2 * i + 1], b.y);
  }
}

// D model width, F hidden width, ACT 1 ReLU, 2 GELU, 3 GELU of the rounded pre-activation, SIDE side outputs
template <int D, int F, bool FP16, int ACT, bool DROP1, bool SIDE>
__global__ void __launch_bounds__(FF_THREADS, 1)
ffn_fused_tcgen05_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w1,
                         const __grid_constant__ CUtensorMap map_w2, const __grid_constant__ CUtensorMap map_y,
                         const __grid_constant__ CUtensorMap map_h, const __grid_constant__ CUtensorMap map_z, const FfnArgs g) {
  constexpr int DP = D / 64;                              // panels of a row tile
  constexpr int NU = F / FF_HC;                           // units of a tile
  constexpr int NX = D == 64 ? 4 : 2;                     // X buffers
  constexpr int W1_PANEL = FF_HC * 128, W2_PANEL = D * 128;
  static_assert(NU == DP, "a team has the output panel of its units");
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* s_x = smem;                                    // [NX][DP][128 rows][128 B]
  uint8_t* s_w1 = s_x + NX * DP * FF_PANEL;               // [NU][DP][128 hidden rows][128 B]
  uint8_t* s_w2 = s_w1 + NU * DP * W1_PANEL;              // [F / 64 K panels][D output rows][128 B]
  uint8_t* s_stage = s_w2 + (F / 64) * W2_PANEL;          // [16 warps][32 rows][64 B]
  FfnControl* ctl = reinterpret_cast<FfnControl*>(s_stage + FF_EPI_WARPS * FF_BLOCK);
  float* s_b1 = reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(ctl) + ((sizeof(FfnControl) + 15) & ~size_t(15)));
  float* s_b2 = s_b1 + F;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    mbar_init(&ctl->w_full, 1);
    for (int i = 0; i < NX; ++i) { mbar_init(&ctl->x_full[i], 1); mbar_init(&ctl->x_empty[i], 1); }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&ctl->acc1_full[i], 1);
      mbar_init(&ctl->hidden_full[i], FF_TEAM_WARPS);
      mbar_init(&ctl->hidden_done[i], 1);
      mbar_init(&ctl->acc2_full[i], 1);
      mbar_init(&ctl->acc2_empty[i], FF_TEAM_WARPS * DP);
    }
    ctl->abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  for (int i = threadIdx.x; i < F; i += FF_THREADS) s_b1[i] = g.b1 != nullptr ? g.b1[i] : 0.f;
  for (int i = threadIdx.x; i < D; i += FF_THREADS) s_b2[i] = g.b2 != nullptr ? g.b2[i] : 0.f;
  if (warp == 1) {
    // two unit accumulators (columns 0-127, 128-255) and two output accumulators (D columns each from 256)
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&ctl->tmem_base)), "r"(512)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = ctl->tmem_base;
  volatile int* abort_flag = &ctl->abort_flag;
  const int tiles = (int)blockIdx.x < g.m_tiles ? (g.m_tiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;   // of this CTA
  const int units = tiles * NU;
  auto tile_of = [&](int i) { return (int)blockIdx.x + i * (int)gridDim.x; };

  if (warp == 0) {
    // ------------------------------------------------------------------ producer: first X tile, weights once, further X tiles
    if (lane == 0) {
      bool ok = true;
      for (int i = 0; i < tiles && ok; ++i) {
        const int b = i % NX;
        if (!mbar_wait(&ctl->x_empty[b], (uint32_t)((i / NX) & 1) ^ 1u, abort_flag)) { ok = false; break; }
        mbar_expect_tx(&ctl->x_full[b], (uint32_t)(DP * FF_PANEL));
        for (int p = 0; p < DP; ++p) tma_load_2d(s_x + (b * DP + p) * FF_PANEL, &map_x, &ctl->x_full[b], p * 64, tile_of(i) * FF_M);
        if (i == 0) {
          mbar_expect_tx(&ctl->w_full, (uint32_t)(NU * DP * W1_PANEL + (F / 64) * W2_PANEL));
          for (int c = 0; c < NU; ++c)
            for (int p = 0; p < DP; ++p) tma_load_2d(s_w1 + (c * DP + p) * W1_PANEL, &map_w1, &ctl->w_full, p * 64, c * FF_HC);
          for (int kp = 0; kp < F / 64; ++kp) tma_load_2d(s_w2 + kp * W2_PANEL, &map_w2, &ctl->w_full, kp * 64, 0);
        }
      }
      if (!ok) { *abort_flag = 1; atomicExch(g.status, 9); }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    if (lane == 0) {
      const uint32_t idesc1 = ff_instr_desc(FF_HC, FP16), idesc2 = ff_instr_desc(D, FP16);
      bool ok = tiles == 0 || mbar_wait(&ctl->w_full, 0, abort_flag);
      tc_fence_after();
      auto gemm1 = [&](int u) -> bool {
        const int i = u / NU, c = u % NU, b = i % NX;
        if (c == 0 && !mbar_wait(&ctl->x_full[b], (uint32_t)((i / NX) & 1), abort_flag)) return false;
        if (!mbar_wait(&ctl->hidden_done[u & 1], (uint32_t)((u >> 1) & 1) ^ 1u, abort_flag)) return false;   // unit u - 2
        tc_fence_after();
        const uint32_t d = tmem_base + (uint32_t)((u & 1) * FF_HC);
        for (int p = 0; p < DP; ++p) {
          const uint64_t adesc = make_smem_desc(smem_u32(s_x + (b * DP + p) * FF_PANEL));
          const uint64_t bdesc = make_smem_desc(smem_u32(s_w1 + (c * DP + p) * W1_PANEL));
#pragma unroll
          for (int kk = 0; kk < 4; ++kk) umma_f16(d, adesc + 2 * kk, bdesc + 2 * kk, idesc1, (p > 0 || kk > 0) ? 1u : 0u);
        }
        umma_commit(&ctl->acc1_full[u & 1]);
        if (c == NU - 1) umma_commit(&ctl->x_empty[b]);
        return true;
      };
      for (int u = 0; u < 2 && u < units && ok; ++u) ok = gemm1(u);
      for (int u = 0; u < units && ok; ++u) {
        const int i = u / NU, c = u % NU;
        if (!mbar_wait(&ctl->hidden_full[u & 1], (uint32_t)((u >> 1) & 1), abort_flag)) { ok = false; break; }
        if (c == 0 && !mbar_wait(&ctl->acc2_empty[i & 1], (uint32_t)((i >> 1) & 1) ^ 1u, abort_flag)) { ok = false; break; }
        tc_fence_after();
        const uint32_t d = tmem_base + 2u * FF_HC + (uint32_t)((i & 1) * D);
        for (int p = 0; p < 2; ++p) {
          const uint64_t bdesc = make_smem_desc(smem_u32(s_w2 + (c * 2 + p) * W2_PANEL));
          // hidden columns 32 j .. 32 j + 31 of the unit are the first 16 of the accumulator's columns 32 j .. 32 j + 31
          const uint32_t a = tmem_base + (uint32_t)((u & 1) * FF_HC + p * 64);
#pragma unroll
          for (int kk = 0; kk < 4; ++kk)
            umma_f16_ts(d, a + (uint32_t)((kk >> 1) * 32 + (kk & 1) * 8), bdesc + 2 * kk, idesc2, (c > 0 || p > 0 || kk > 0) ? 1u : 0u);
        }
        umma_commit(&ctl->hidden_done[u & 1]);
        if (c == NU - 1) umma_commit(&ctl->acc2_full[i & 1]);
        if (u + 2 < units) ok = gemm1(u + 2);
      }
      if (!ok) { *abort_flag = 1; atomicExch(g.status, 10); }
    }
  } else {
    // ------------------------------------------------------------------ epilogue warps (2..17)
    const int quarter = warp & 3;                          // TMEM lane quarter this warp may read
    const int team = (warp - 2) / FF_TEAM_WARPS;
    const int half = ((warp - 2) >> 2) & 1;                // its 64 columns of a unit, its 32 columns of an output panel
    const int r = quarter * 32 + lane;                     // row inside the tile
    const uint32_t lane_addr = (uint32_t)(quarter * 32) << 16;
    const int panel = DP == 2 ? team : 0;                  // the 64-column panel of the output this warp's team writes
    uint8_t* block = s_stage + (size_t)(warp - 2) * FF_BLOCK;
    // 32 columns of this warp's 32 rows, w[i] = columns 2 i and 2 i + 1 of row `lane`, to column `col` of a matrix; rows past M are outside
    // its map.  16-byte chunk c of row r sits at c ^ ((r >> 1) & 3).
    auto put = [&](const uint32_t (&w)[16], const CUtensorMap& map, int col, int row0) {
      if (lane == 0) tma_store_wait_read<0>();             // what the buffer held before has been read
      __syncwarp();
      uint4* p = reinterpret_cast<uint4*>(block + lane * 64);
#pragma unroll
      for (int q = 0; q < 4; ++q) p[q ^ ((lane >> 1) & 3)] = make_uint4(w[4 * q], w[4 * q + 1], w[4 * q + 2], w[4 * q + 3]);
      fence_async_smem();
      __syncwarp();
      if (lane == 0 && row0 + quarter * 32 < g.M) {
        tma_store_2d(&map, block, col, row0 + quarter * 32);
        tma_store_commit();
      }
    };
    // hidden unit: accumulator -> activation -> A operand
    auto hidden = [&](int u) -> bool {
      const int c = u % NU;
      const int row = tile_of(u / NU) * FF_M + r;
      if (!mbar_wait(&ctl->acc1_full[u & 1], (uint32_t)((u >> 1) & 1), abort_flag)) return false;
      tc_fence_after();
#pragma unroll 1
      for (int q32 = 0; q32 < 2; ++q32) {                  // 32 columns
        f2 v[16];
        const int ucol = half * 64 + q32 * 32;
        const uint32_t taddr = tmem_base + lane_addr + (uint32_t)((u & 1) * FF_HC + ucol);
        ff_load<32>(taddr, v);
        const int hcol = c * FF_HC + ucol;                   // hidden column of element 0
        ff_add_bias<32>(s_b1 + hcol, v);
        if (ACT == 3 || (SIDE && ACT == 2 && g.round_z)) {   // what the backward pass differentiates at: the rounded value
          uint32_t w[16];
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            const float2 x = unpack2(v[i]);
            w[i] = narrow16<FP16>(x.x, x.y);
            v[i] = widen16<FP16>(w[i]);
          }
          if (SIDE && g.keep_z) put(w, map_z, hcol, tile_of(u / NU) * FF_M);
        }
        if (ACT >= 2) {
#pragma unroll
          for (int i = 0; i < 16; ++i) v[i] = gelu2(v[i]);
        }
        uint32_t positive = 0;                               // one bit an element
        if (DROP1) {
          const f2 s = pack2(g.scale1, g.scale1);
          const uint32_t hash = (uint32_t)row * kHashRow + (uint32_t)hcol * kHashCol + g.seed1;
          const uint32_t thresh_hi = g.thresh1 >> 16;
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            const float2 x = unpack2(mul2(v[i], s));
            bool k0 = hash_keep(hash + (uint32_t)(2 * i) * kHashCol, g.thresh1, thresh_hi);
            bool k1 = hash_keep(hash + (uint32_t)(2 * i + 1) * kHashCol, g.thresh1, thresh_hi);
            if (ACT == 1) { k0 = k0 && x.x > 0.f; k1 = k1 && x.y > 0.f; }
            if (SIDE && ACT == 1) { set_bit(positive, k0, 1u << (2 * i), g.one); set_bit(positive, k1, 2u << (2 * i), g.one); }
            v[i] = pack2(k0 ? x.x : 0.f, k1 ? x.y : 0.f);
          }
        } else if (ACT == 1) {
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            const float2 x = unpack2(v[i]);
            if (SIDE) { set_bit(positive, x.x > 0.f, 1u << (2 * i), g.one); set_bit(positive, x.y > 0.f, 2u << (2 * i), g.one); }
            v[i] = pack2(fmaxf(x.x, 0.f), fmaxf(x.y, 0.f));
          }
        }
        if (SIDE && g.bits_out != nullptr && row < g.M) {
          if (ACT == 2) {
#pragma unroll
            for (int i = 0; i < 16; ++i) {
              const float2 x = unpack2(v[i]);
              set_bit(positive, x.x > 0.f, 1u << (2 * i), g.one);
              set_bit(positive, x.y > 0.f, 2u << (2 * i), g.one);
            }
          }
          unsigned short* bo = g.bits_out + (long long)(hcol >> 4) * g.ldmb + row;
          bo[0] = (unsigned short)positive;
          bo[g.ldmb] = (unsigned short)(positive >> 16);
        }
        uint32_t w[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          const float2 x = unpack2(v[i]);
          w[i] = narrow16<FP16>(x.x, x.y);
        }
        tmem_st_32x32b_x16(taddr, w);
        if (q32 == 1) {
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&ctl->hidden_full[u & 1]);
        }
        if (SIDE && g.keep_h) put(w, map_h, hcol, tile_of(u / NU) * FF_M);
      }
      return true;
    };
    // the team's panel of the output of tile i: accumulator -> bias, dropout, residual -> TMA store
    auto output = [&](int i) -> bool {
      const int row = tile_of(i) * FF_M + r;
      const int col = panel * 64 + half * 32;
      uint4 pre[4];
      if (g.res != nullptr) {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          pre[q] = make_uint4(0u, 0u, 0u, 0u);
          if (row < g.M) pre[q] = __ldg(reinterpret_cast<const uint4*>(g.res + (long long)row * g.ldr + col) + q);
        }
      }
      if (!mbar_wait(&ctl->acc2_full[i & 1], (uint32_t)((i >> 1) & 1), abort_flag)) return false;
      tc_fence_after();
      f2 v[16];
      ff_load<32>(tmem_base + lane_addr + (uint32_t)(2 * FF_HC + (i & 1) * D + col), v);
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&ctl->acc2_empty[i & 1]);
      ff_add_bias<32>(s_b2 + col, v);
      if (g.thresh2) {
        const f2 s = pack2(g.scale2, g.scale2);
        const uint32_t hash = (uint32_t)row * kHashRow + (uint32_t)col * kHashCol + g.seed2;
#pragma unroll
        for (int k = 0; k < 16; ++k) {
          const float2 x = unpack2(mul2(v[k], s));
          v[k] = pack2(hash_keep(hash + (uint32_t)(2 * k) * kHashCol, g.thresh2, g.thresh2 >> 16) ? x.x : 0.f,
                       hash_keep(hash + (uint32_t)(2 * k + 1) * kHashCol, g.thresh2, g.thresh2 >> 16) ? x.y : 0.f);
        }
      }
      uint32_t w[16];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        if (g.res != nullptr) {
          const uint32_t x[4] = {pre[q].x, pre[q].y, pre[q].z, pre[q].w};
#pragma unroll
          for (int k = 0; k < 4; ++k) v[4 * q + k] = add2(v[4 * q + k], widen16<FP16>(x[k]));
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const float2 x = unpack2(v[4 * q + k]);
          w[4 * q + k] = narrow16<FP16>(x.x, x.y);
        }
      }
      put(w, map_y, col, tile_of(i) * FF_M);
      return true;
    };
    // units of this team; the tile behind the last one whose output is still to come
    bool ok = true;
    int done = -1;
    for (int u = team; u < units && ok; u += 2) {
      ok = hidden(u);
      if (ok && done >= 0) ok = output(done);
      done = u / NU;
    }
    if (ok && done >= 0) ok = output(done);
    if (lane == 0) tma_store_wait_all();
    if (!ok && lane == 0) { *abort_flag = 1; atomicExch(g.status, 11); }
  }

  // ------------------------------------------------------------------ teardown
  __syncwarp();
  if (*abort_flag) {
    for (int i = 0; i < 200; ++i) __nanosleep(1000);        // copies still in flight land before shared memory is released
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512) : "memory");
  }
}

using FfnKernel = void (*)(const CUtensorMap, const CUtensorMap, const CUtensorMap, const CUtensorMap, const CUtensorMap, const CUtensorMap, const FfnArgs);

template <int D, int F, bool FP16, int ACT, bool SIDE> FfnKernel ffn_pick(bool drop1) {
  return drop1 ? (FfnKernel)ffn_fused_tcgen05_kernel<D, F, FP16, ACT, true, SIDE> : (FfnKernel)ffn_fused_tcgen05_kernel<D, F, FP16, ACT, false, SIDE>;
}
// Rounding at run time costs the form without side outputs 7 % (224 us of 210, 800 k rows of 128 / 256): an instance of its own, and, where nobody
// has ever had the unrounded one, the only one.
template <int D, int F, bool FP16> FfnKernel ffn_pick(int act, bool drop1, bool side, bool round_z) {
  if (act == 1) return side ? ffn_pick<D, F, FP16, 1, true>(drop1) : ffn_pick<D, F, FP16, 1, false>(drop1);
  if (side) return ffn_pick<D, F, FP16, 2, true>(drop1);
  if constexpr (D == 128 && !FP16) {
    if (!round_z) return ffn_pick<D, F, FP16, 2, false>(drop1);
  }
  return ffn_pick<D, F, FP16, 3, false>(drop1);
}

}  // namespace

extern "C" int bf_ffn_fused_supported(long long M, int hidden, int ffn) {
  return (M > 0 && M < (1ll << 31) - FF_M && ((hidden == 128 && ffn == 256) || (hidden == 64 && ffn == 128))) ? 1 : 0;
}

extern "C" int bf_ffn_fused_fwd(const bf_ffn_params* p, cudaStream_t st) {
  if (!bf_ffn_fused_supported(p->M, p->hidden, p->ffn)) return (int)cudaErrorInvalidValue;
  if (p->act != 1 && p->act != 2) return (int)cudaErrorInvalidValue;
  if (p->dropout1 < 0.f || p->dropout1 >= 1.f || p->dropout2 < 0.f || p->dropout2 >= 1.f) return (int)cudaErrorInvalidValue;
  const int D = p->hidden, F = p->ffn;
  const uintptr_t align = (uintptr_t)p->X | (uintptr_t)p->Y | (uintptr_t)p->W1 | (uintptr_t)p->W2 | (uintptr_t)p->b1 | (uintptr_t)p->b2 |
                          (uintptr_t)p->R | (uintptr_t)p->z_out | (uintptr_t)p->H_out;
  if (!p->X || !p->Y || !p->W1 || !p->W2 || !p->status || align % 16 != 0 || (p->ldx * 2) % 16 != 0 || (p->ldy * 2) % 16 != 0 ||
      p->ldx < D || p->ldy < D)
    return (int)cudaErrorInvalidValue;
  if (p->R && ((p->ldr * 2) % 16 != 0 || p->ldr < D || p->residual)) return (int)cudaErrorInvalidValue;
  if (p->z_out && ((p->ldz * 2) % 16 != 0 || p->ldz < F || p->act != 2)) return (int)cudaErrorInvalidValue;
  FfnArgs g;
  memset(&g, 0, sizeof(g));
  g.M = (int)p->M; g.m_tiles = (int)((p->M + FF_M - 1) / FF_M);
  g.b1 = p->b1; g.b2 = p->b2;
  g.thresh1 = p->dropout1 > 0.f ? (uint32_t)(p->dropout1 * 4294967296.0) : 0u;
  g.scale1 = p->dropout1 > 0.f ? 1.f / (1.f - p->dropout1) : 1.f;
  g.seed1 = p->seed1;
  g.thresh2 = p->dropout2 > 0.f ? (uint32_t)(p->dropout2 * 4294967296.0) : 0u;
  g.scale2 = p->dropout2 > 0.f ? 1.f / (1.f - p->dropout2) : 1.f;
  g.seed2 = p->seed2;
  g.res = static_cast<const unsigned short*>(p->R ? p->R : p->residual ? p->X : nullptr);
  g.ldr = p->R ? p->ldr : p->ldx;
  g.one = 1u;
  g.status = p->status;
  g.keep_h = p->H_out != nullptr;
  g.keep_z = p->z_out != nullptr;
  g.round_z = g.keep_z || p->round_z;
  g.bits_out = static_cast<unsigned short*>(p->relu_bits_out);
  g.ldmb = p->ldmb;
  if (g.keep_h && ((p->ldh * 2) % 16 != 0 || p->ldh < F)) return (int)cudaErrorInvalidValue;
  if (g.bits_out != nullptr && p->ldmb < p->M) return (int)cudaErrorInvalidValue;
  const bool fp16 = p->dtype == BF_FP16, side = g.keep_h || g.keep_z || g.bits_out != nullptr;
  CUtensorMap map_x, map_w1, map_w2, map_y, map_h, map_z;
  memset(&map_h, 0, sizeof(map_h));
  memset(&map_z, 0, sizeof(map_z));
  if (g.keep_h && make_map(&map_h, p->H_out, p->M, F, p->ldh, 32, fp16, 32, true) != 0) return (int)cudaErrorNotSupported;
  if (g.keep_z && make_map(&map_z, p->z_out, p->M, F, p->ldz, 32, fp16, 32, true) != 0) return (int)cudaErrorNotSupported;
  if (make_map(&map_x, p->X, p->M, D, p->ldx, FF_M, fp16) != 0) return (int)cudaErrorNotSupported;
  if (make_map(&map_w1, p->W1, F, D, D, FF_HC, fp16) != 0) return (int)cudaErrorNotSupported;
  if (make_map(&map_w2, p->W2, D, F, F, D, fp16) != 0) return (int)cudaErrorNotSupported;
  if (make_map(&map_y, p->Y, p->M, D, p->ldy, 32, fp16, 32, true) != 0) return (int)cudaErrorNotSupported;
  const size_t x_bufs = D == 64 ? 4 : 2;
  const size_t smem = 1024 + x_bufs * (D / 64) * FF_PANEL + (size_t)(F / FF_HC) * (D / 64) * (FF_HC * 128) + (size_t)(F / 64) * (D * 128) +
                      FF_EPI_WARPS * FF_BLOCK + ((sizeof(FfnControl) + 15) & ~size_t(15)) + (size_t)(F + D) * sizeof(float);
  const bool drop1 = g.thresh1 != 0, round_z = g.round_z != 0;
  const FfnKernel kern = D == 128 ? (fp16 ? ffn_pick<128, 256, true>(p->act, drop1, side, round_z) : ffn_pick<128, 256, false>(p->act, drop1, side, round_z))
                                  : (fp16 ? ffn_pick<64, 128, true>(p->act, drop1, side, round_z) : ffn_pick<64, 128, false>(p->act, drop1, side, round_z));
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  {
    constexpr int MAX_DEV = 64;
    static bool attr_set[MAX_DEV][64] = {};
    const int slot = (round_z ? 32 : 0) | (D == 128 ? 16 : 0) | (fp16 ? 8 : 0) | (p->act == 1 ? 4 : 0) | (g.thresh1 ? 2 : 0) | (side ? 1 : 0);
    if (dev < 0 || dev >= MAX_DEV || !attr_set[dev][slot]) {
      cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
      if (e != cudaSuccess) return (int)e;
      if (dev >= 0 && dev < MAX_DEV) attr_set[dev][slot] = true;
    }
  }
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int grid = g.m_tiles < sms ? g.m_tiles : sms;
  kern<<<grid, FF_THREADS, smem, st>>>(map_x, map_w1, map_w2, map_y, map_h, map_z, g);
  return (int)cudaGetLastError();
}
