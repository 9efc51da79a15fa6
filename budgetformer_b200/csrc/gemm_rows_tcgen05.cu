// Row-streaming tcgen05 GEMM for sm_100a:  C[M, N] = epilogue(A[M, K] * B[N, K]^T), a tall activation times a small weight, both
// 16-bit, into one 16-bit matrix.  The layers of this package are such products with K and N of 64 to 768: bound by the bytes of A,
// C and the residual, if the epilogue keeps up with them.
//
// * The columns are cut into panels of 64.  A CTA owns a group of panels and walks row tiles of 128; the group's rows of B are loaded
//   once and stay in shared memory (up to 128 KB; wider weights stream through the ring with A), so that the TMA ring carries A alone and
//   a row tile is read once for all panels of the group.
// * One elected thread issues tcgen05.mma into two to four accumulators of 64 to 192 columns (256 where B streams) in tensor memory.
// * Sixteen epilogue warps form four teams.  A unit of work is one panel of one row tile; units go to the teams in turn, and a warp of a
//   team takes the 32 rows of its tensor-memory quarter x 64 columns = one 4 KB block of the 128-byte-swizzled staging buffer.  It loads
//   that block of the residual (or of the pre-activation) by TMA, writes its results over it and stores it by TMA itself: warps meet
//   only at the accumulators' barriers.  (With sixteen warps on one tile and a barrier of all of them a tile, and features read at run
//   time, a 128 x 128 tile took 850 instructions a warp and 32 columns, and issue slots were half idle.)
// * Epilogue features are template parameters.  Masks, biases and activations as in gemm_tcgen05.cu, in the same order.
//
// us at 800 k rows before (gemm_tcgen05.cu) and now, and the time of its bytes at the measured copy rate (outputs x features): 384 x 128
// + bias 168 / 152 / 125; 128 x 128 + bias, dropout, residual 203 / 119 / 94; 128 x 128 + dropout 159 / 83 / 63 (without 72 / 72 / 63);
// 128 x 384 + residual 174 / 170 / 157; 256 x 128 + bit mask 173 / 123 / 98; 128 x 256 + residual 168 / 138 / 125; 256 x 128 * gelu'
// 601 / 354 / 157; 128 x 272 + dropout 161 / 124 / 98.  At 400 k rows: 768 x 256 229 / 202 / 125; 256 x 256 + residual 205 / 120 / 94; 512 x 256
// + ReLU, dropout, bits 298 / 200 / 98; 256 x 512 + residual 209 / 152 / 125; 112 x 256 215 / 58 / 45.  At 2 k rows 6 us either way.
// Every mbarrier wait is bounded: on expiry the kernel records a status word, stops issuing work, lets copies in flight land, frees its
// tensor memory and returns.
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <string.h>

#include "bf_kernels.h"
#include "epilogue.cuh"
#include "sm100_ptx.cuh"

namespace {

constexpr int kTileM = 128, kPanel = 64;
constexpr int kAStage = kTileM * kPanel * 2;        // bytes of one K panel of a row tile
constexpr int kTeams = 4;
constexpr int kThreads = 32 * (2 + 4 * kTeams);     // TMA producer, MMA issuer, epilogue
constexpr int kMaxStages = 12, kMaxAcc = 4;
constexpr int kBlockBytes = 32 * 128;               // a warp's part of a staged panel
constexpr int kMaxGroupCols = 512;                  // columns of one CTA's group

enum : int { F_BIAS = 1, F_RELU = 2, F_GELU = 4, F_DROP = 8, F_RES = 16, F_BITS_IN = 32, F_SCALE = 64, F_BITS_OUT = 128,
             F_GELU_GRAD = 256, F_KEEP_Z = 512 };

struct RowsArgs {
  int M, N, m_tiles, k_panels;
  int panels, groups, group_panels, chunk_panels;   // a group is processed in chunks (one accumulator each) of chunk_panels panels
  int n_acc, stages, resident, n_buf;
  uint32_t one;                                     // 1
  const float* bias;
  uint32_t thresh, seed;
  float keep_scale, out_scale;
  const unsigned short* bits_in;
  unsigned short* bits_out;
  long long ldmb;
  int dst_row;
  int* status;
};

struct RowsControl {
  uint64_t full[kMaxStages], empty[kMaxStages];
  uint64_t acc_full[kMaxAcc], acc_empty[kMaxAcc];
  uint64_t staged[4 * kTeams][2];                   // residual block of a warp has landed
  uint64_t b_full;
  uint32_t tmem_base;
  int abort_flag;
};

__device__ __forceinline__ void tmem_ld_32x32b_x32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, "
      "%19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
        "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]),
        "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]),
        "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}

template <bool FP16, int EPI>
__global__ void __launch_bounds__(kThreads, 1)
gemm_rows_tcgen05_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                         const __grid_constant__ CUtensorMap map_out, const __grid_constant__ CUtensorMap map_z,
                         const __grid_constant__ CUtensorMap map_in, const RowsArgs g) {
  constexpr bool STAGED = (EPI & (F_RES | F_GELU_GRAD)) != 0;     // an operand of the epilogue comes through the staging buffer
  constexpr bool KEEP_Z = (EPI & F_KEEP_Z) != 0;                  // the pre-activation goes to map_z as well
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int chunk_cols = g.chunk_panels * kPanel;
  const uint32_t b_panel = (uint32_t)chunk_cols * 128u;           // one K panel of one chunk of B
  const uint32_t stage_bytes = kAStage + (g.resident ? 0u : b_panel);
  const int chunks = g.group_panels / g.chunk_panels;
  uint8_t* s_b = smem;                                            // [chunk][K panel][chunk_cols rows][128 B]
  uint8_t* s_ring = smem + (g.resident ? (size_t)chunks * g.k_panels * b_panel : 0);
  uint8_t* s_out = s_ring + (size_t)g.stages * stage_bytes;       // [team][n_buf][4 warps][32 rows][128 B]
  RowsControl* ctl = reinterpret_cast<RowsControl*>(s_out + (size_t)kTeams * g.n_buf * 4 * kBlockBytes);
  float* s_bias = reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(ctl) + ((sizeof(RowsControl) + 15) & ~size_t(15)));

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int group = (int)blockIdx.x % g.groups;
  const int first_tile = (int)blockIdx.x / g.groups, tile_step = (int)gridDim.x / g.groups;
  const int panel0 = group * g.group_panels;

  if (threadIdx.x == 0) {
    for (int s = 0; s < g.stages; ++s) { mbar_init(&ctl->full[s], 1); mbar_init(&ctl->empty[s], 1); }
    for (int a = 0; a < g.n_acc; ++a) { mbar_init(&ctl->acc_full[a], 1); mbar_init(&ctl->acc_empty[a], 4 * g.chunk_panels); }
    for (int w = 0; w < 4 * kTeams; ++w) { mbar_init(&ctl->staged[w][0], 1); mbar_init(&ctl->staged[w][1], 1); }
    mbar_init(&ctl->b_full, 1);
    ctl->abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (EPI & F_BIAS) {
    for (int i = threadIdx.x; i < g.group_panels * kPanel; i += kThreads)
      s_bias[i] = panel0 * kPanel + i < g.N ? g.bias[panel0 * kPanel + i] : 0.f;
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&ctl->tmem_base)), "r"(512)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = ctl->tmem_base;
  volatile int* abort_flag = &ctl->abort_flag;

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    if (lane == 0) {
      uint32_t stage = 0, phase = 0;
      bool ok = true, first = true;
      for (int t = first_tile; t < g.m_tiles && ok; t += tile_step) {
        for (int kp = 0; kp < g.k_panels; ++kp) {
          if (!mbar_wait(&ctl->empty[stage], phase ^ 1u, abort_flag)) { ok = false; break; }
          uint8_t* dst = s_ring + stage * stage_bytes;
          mbar_expect_tx(&ctl->full[stage], stage_bytes);
          tma_load_2d(dst, &map_a, &ctl->full[stage], kp * kPanel, t * kTileM);
          if (!g.resident) tma_load_2d(dst + kAStage, &map_b, &ctl->full[stage], kp * kPanel, panel0 * kPanel);
          if (first) {                                            // behind the first row panel: the group's weights
            first = false;
            if (g.resident) {
              mbar_expect_tx(&ctl->b_full, (uint32_t)(chunks * g.k_panels) * b_panel);
              for (int c = 0; c < chunks; ++c)
                for (int k = 0; k < g.k_panels; ++k)
                  tma_load_2d(s_b + (size_t)(c * g.k_panels + k) * b_panel, &map_b, &ctl->b_full, k * kPanel,
                              panel0 * kPanel + c * chunk_cols);
            }
          }
          if (++stage == (uint32_t)g.stages) { stage = 0; phase ^= 1u; }
        }
      }
      if (!ok) { *abort_flag = 1; atomicExch(g.status, 21); }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    if (lane == 0) {
      const uint32_t idesc = (1u << 4) | ((FP16 ? 0u : 1u) << 7) | ((FP16 ? 0u : 1u) << 10) | ((uint32_t)(chunk_cols >> 3) << 17) |
                             ((uint32_t)(kTileM >> 4) << 24);
      uint32_t stage = 0, phase = 0, acc = 0, acc_phase = 0;
      bool ok = !g.resident || first_tile >= g.m_tiles || mbar_wait(&ctl->b_full, 0, abort_flag);
      tc_fence_after();
      for (int t = first_tile; t < g.m_tiles && ok; t += tile_step) {
        uint32_t s = stage, ph = phase;
        for (int c = 0; c < chunks && ok; ++c) {
          if (!mbar_wait(&ctl->acc_empty[acc], acc_phase ^ 1u, abort_flag)) { ok = false; break; }
          tc_fence_after();
          const uint32_t d = tmem_base + acc * (uint32_t)chunk_cols;
          s = stage; ph = phase;
          for (int kp = 0; kp < g.k_panels; ++kp) {
            if (c == 0 && !mbar_wait(&ctl->full[s], ph, abort_flag)) { ok = false; break; }
            tc_fence_after();
            const uint8_t* a = s_ring + s * stage_bytes;
            const uint64_t adesc = make_smem_desc(smem_u32(a));
            const uint64_t bdesc = make_smem_desc(smem_u32(g.resident ? s_b + (size_t)(c * g.k_panels + kp) * b_panel : a + kAStage));
#pragma unroll
            for (int kk = 0; kk < kPanel / 16; ++kk)
              umma_f16(d, adesc + 2 * kk, bdesc + 2 * kk, idesc, (kp > 0 || kk > 0) ? 1u : 0u);
            if (c == chunks - 1) umma_commit(&ctl->empty[s]);
            if (++s == (uint32_t)g.stages) { s = 0; ph ^= 1u; }
          }
          if (!ok) break;
          umma_commit(&ctl->acc_full[acc]);
          if (++acc == (uint32_t)g.n_acc) { acc = 0; acc_phase ^= 1u; }
        }
        stage = s; phase = ph;
      }
      if (!ok) { *abort_flag = 1; atomicExch(g.status, 22); }
    }
  } else {
    // ------------------------------------------------------------------ epilogue
    const int quarter = warp & 3, team = (warp - 2) >> 2;          // a warp reads the tensor-memory lanes of its quarter
    const int ew = team * 4 + quarter;
    uint8_t* block0 = s_out + (size_t)(team * g.n_buf * 4 + quarter) * kBlockBytes;   // this warp's block of its team's first buffer
    const uint32_t tlane = tmem_base + ((uint32_t)(quarter * 32) << 16);
    const int units_per_tile = g.group_panels;
    const uint32_t thresh_hi = g.thresh >> 16;
    const bool ahead = STAGED && g.n_buf == 2;
    const bool twin = !STAGED && !KEEP_Z && g.n_buf == 2;          // results alternate between two blocks
    bool ok = true;
    // unit (t, p): row tile t, panel p of the group; acc_seq counts the accumulators of this CTA up to the unit's
    int t = first_tile, p = team, seq0 = 0;
    auto settle = [&](int& tt, int& pp, int& sq) {
      while (pp >= units_per_tile) { pp -= units_per_tile; tt += tile_step; sq += chunks; }
    };
    settle(t, p, seq0);
    auto fetch = [&](int tt, int pp, int buf) {                    // lane 0: the unit's block of the staged operand
      if (tt < g.m_tiles && tt * kTileM + quarter * 32 < g.M) {
        mbar_expect_tx(&ctl->staged[ew][buf], kBlockBytes);
        tma_load_2d(block0 + (size_t)buf * 4 * kBlockBytes, &map_in, &ctl->staged[ew][buf], (panel0 + pp) * kPanel,
                    tt * kTileM + quarter * 32);
      }
    };
    if (STAGED && lane == 0) fetch(t, p, 0);
    int buf = 0;
    uint32_t buf_phase = 0;
    while (t < g.m_tiles) {
      int tn = t, pn = p + kTeams, seqn = seq0;
      settle(tn, pn, seqn);
      if (ahead && lane == 0) {
        tma_store_wait_read<0>();                                  // the other buffer's store was issued one unit ago
        fetch(tn, pn, buf ^ 1);
      }
      const int row = t * kTileM + quarter * 32 + lane;
      const bool any_row = t * kTileM + quarter * 32 < g.M;        // warp-uniform
      const bool row_ok = row < g.M;
      const int col0 = (panel0 + p) * kPanel;
      const int chunk = g.chunk_panels == 1 ? p : g.chunk_panels == 2 ? p >> 1 : p / g.chunk_panels;
      const int seq = seq0 + chunk, in_chunk = p - chunk * g.chunk_panels;
      const int acc = seq & (g.n_acc - 1);
      uint32_t bits[4] = {0u, 0u, 0u, 0u};
      if ((EPI & F_BITS_IN) && row_ok) {
#pragma unroll
        for (int q = 0; q < 4; ++q)
          if (col0 + 16 * q < g.N) bits[q] = __ldg(g.bits_in + (long long)((col0 >> 4) + q) * g.ldmb + row);
      }
      uint8_t* block = block0 + (size_t)(KEEP_Z ? 0 : buf) * 4 * kBlockBytes;
      if (STAGED && any_row && !mbar_wait(&ctl->staged[ew][buf], buf_phase, abort_flag)) { ok = false; break; }
      if (!mbar_wait(&ctl->acc_full[acc], (uint32_t)(seq / g.n_acc) & 1u, abort_flag)) { ok = false; break; }
      tc_fence_after();
      if (!STAGED) {
        if (lane == 0) {                                           // this buffer's last store
          if (twin) tma_store_wait_read<1>();
          else tma_store_wait_read<0>();
        }
        __syncwarp();
      }
      const uint32_t taddr = tlane + (uint32_t)(acc * chunk_cols + in_chunk * kPanel);
      const uint32_t hash0 = (uint32_t)row * kHashRow + (uint32_t)col0 * kHashCol + g.seed;
#pragma unroll 1
      for (int h = 0; h < 2; ++h) {                                // 32 columns
        uint32_t r[32];
        tmem_ld_32x32b_x32(taddr + 32u * h, r);
        uint4 pre[4];
        // 16-byte chunk c of row `lane` sits at c ^ (lane & 7)
        uint4* slot = reinterpret_cast<uint4*>(block + lane * 128);
        if (STAGED) {
#pragma unroll
          for (int q = 0; q < 4; ++q) pre[q] = slot[(4 * h + q) ^ (lane & 7)];
        }
        tmem_ld_wait();
        if (h == 1) {
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&ctl->acc_empty[acc]);
        }
        f2 v[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) v[i] = pack2(__uint_as_float(r[2 * i]), __uint_as_float(r[2 * i + 1]));
        if (EPI & F_SCALE) {
          const f2 s = pack2(g.out_scale, g.out_scale);
#pragma unroll
          for (int i = 0; i < 16; ++i) v[i] = mul2(v[i], s);
        }
        if (EPI & F_BIAS) {
          const ulonglong2* bp = reinterpret_cast<const ulonglong2*>(s_bias + p * kPanel + 32 * h);
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const ulonglong2 b = bp[i];
            v[2 * i] = add2(v[2 * i], b.x); v[2 * i + 1] = add2(v[2 * i + 1], b.y);
          }
        }
        if (KEEP_Z) {                                              // what the backward pass differentiates at: the rounded value
          uint4* zslot = reinterpret_cast<uint4*>(block + 4 * kBlockBytes + lane * 128);
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            uint32_t w[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const float2 x = unpack2(v[4 * q + i]);
              w[i] = narrow16<FP16>(x.x, x.y);
              v[4 * q + i] = widen16<FP16>(w[i]);
            }
            zslot[(4 * h + q) ^ (lane & 7)] = make_uint4(w[0], w[1], w[2], w[3]);
          }
        }
        if (EPI & F_GELU) {
#pragma unroll
          for (int i = 0; i < 16; ++i) v[i] = gelu2(v[i]);
        }
        uint32_t positive = 0;                                     // one bit a result (bits_out goes with ReLU)
        if (EPI & F_DROP) {
          const f2 s = pack2(g.keep_scale, g.keep_scale);
          const uint32_t hash = hash0 + (uint32_t)(32 * h) * kHashCol;
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            float2 x = unpack2(mul2(v[i], s));
            bool k0 = hash_keep(hash + (uint32_t)(2 * i) * kHashCol, g.thresh, thresh_hi);
            bool k1 = hash_keep(hash + (uint32_t)(2 * i + 1) * kHashCol, g.thresh, thresh_hi);
            if (EPI & F_RELU) { k0 = k0 && x.x > 0.f; k1 = k1 && x.y > 0.f; }
            if (EPI & F_BITS_OUT) { set_bit(positive, k0, 1u << (2 * i), g.one); set_bit(positive, k1, 2u << (2 * i), g.one); }
            v[i] = pack2(k0 ? x.x : 0.f, k1 ? x.y : 0.f);
          }
        } else if (EPI & F_RELU) {
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            const float2 x = unpack2(v[i]);
            if (EPI & F_BITS_OUT) { set_bit(positive, x.x > 0.f, 1u << (2 * i), g.one); set_bit(positive, x.y > 0.f, 2u << (2 * i), g.one); }
            v[i] = pack2(fmaxf(x.x, 0.f), fmaxf(x.y, 0.f));
          }
        }
        if (EPI & F_BITS_IN) {
          const uint32_t m = h == 0 ? (bits[0] | (bits[1] << 16)) : (bits[2] | (bits[3] << 16));
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            float2 x = unpack2(v[i]);
            x.x = (m >> (2 * i)) & 1u ? x.x : 0.f;
            x.y = (m >> (2 * i + 1)) & 1u ? x.y : 0.f;
            v[i] = pack2(x.x, x.y);
          }
        }
        if (EPI & F_BITS_OUT) {
          if (row_ok) {
            unsigned short* bo = g.bits_out + (long long)((col0 >> 4) + 2 * h) * g.ldmb + row;
            if (col0 + 32 * h < g.N) bo[0] = (unsigned short)positive;
            if (col0 + 32 * h + 16 < g.N) bo[g.ldmb] = (unsigned short)(positive >> 16);
          }
        }
        if (STAGED) {
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const uint32_t w[4] = {pre[q].x, pre[q].y, pre[q].z, pre[q].w};
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              if (EPI & F_RES) v[4 * q + i] = add2(v[4 * q + i], widen16<FP16>(w[i]));
              else v[4 * q + i] = mul2(v[4 * q + i], gelu_grad2(widen16<FP16>(w[i])));
            }
          }
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          uint32_t w[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float2 x = unpack2(v[4 * q + i]);
            w[i] = narrow16<FP16>(x.x, x.y);
          }
          slot[(4 * h + q) ^ (lane & 7)] = make_uint4(w[0], w[1], w[2], w[3]);
        }
      }
      fence_async_smem();                                          // generic-proxy accesses -> visible to the bulk copies
      __syncwarp();
      if (lane == 0) {
        if (any_row) {                                             // rows past M and columns past N are outside the maps
          tma_store_2d(&map_out, block, col0, g.dst_row + t * kTileM + quarter * 32);
          if (KEEP_Z) tma_store_2d(&map_z, block + 4 * kBlockBytes, col0, t * kTileM + quarter * 32);
        }
        tma_store_commit();
        if (STAGED && !ahead) {
          tma_store_wait_read<0>();
          fetch(tn, pn, 0);
        }
      }
      if (STAGED) {
        if (ahead) { buf ^= 1; if (buf == 0) buf_phase ^= 1u; }
        else buf_phase ^= 1u;
      }
      if (twin) buf ^= 1;
      t = tn; p = pn; seq0 = seqn;
    }
    if (lane == 0) tma_store_wait_all();
    if (!ok && lane == 0) { *abort_flag = 1; atomicExch(g.status, 23); }
  }

  // ------------------------------------------------------------------ teardown
  __syncwarp();
  if (*abort_flag) {
    for (int i = 0; i < 200; ++i) __nanosleep(1000);               // copies still in flight land before shared memory is released
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512) : "memory");
  }
}

// ---------------------------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------------------------
using RowsKernel = void (*)(const CUtensorMap, const CUtensorMap, const CUtensorMap, const CUtensorMap, const CUtensorMap, const RowsArgs);

template <int EPI> RowsKernel pick(bool fp16) {
  return fp16 ? (RowsKernel)gemm_rows_tcgen05_kernel<true, EPI> : (RowsKernel)gemm_rows_tcgen05_kernel<false, EPI>;
}

// the combinations of the layers; others stay with gemm_tcgen05.cu
RowsKernel rows_kernel(int f, bool fp16) {
  switch (f) {
    case 0: return pick<0>(fp16);
    case F_BIAS: return pick<F_BIAS>(fp16);
    case F_DROP: return pick<F_DROP>(fp16);
    case F_RES: return pick<F_RES>(fp16);
    case F_BIAS | F_DROP: return pick<F_BIAS | F_DROP>(fp16);
    case F_BIAS | F_RES: return pick<F_BIAS | F_RES>(fp16);
    case F_BIAS | F_DROP | F_RES: return pick<F_BIAS | F_DROP | F_RES>(fp16);
    case F_BIAS | F_RELU: return pick<F_BIAS | F_RELU>(fp16);
    case F_BIAS | F_GELU: return pick<F_BIAS | F_GELU>(fp16);
    case F_BIAS | F_RELU | F_BITS_OUT: return pick<F_BIAS | F_RELU | F_BITS_OUT>(fp16);
    case F_BIAS | F_RELU | F_DROP | F_BITS_OUT: return pick<F_BIAS | F_RELU | F_DROP | F_BITS_OUT>(fp16);
    case F_BITS_IN: return pick<F_BITS_IN>(fp16);
    case F_BITS_IN | F_SCALE: return pick<F_BITS_IN | F_SCALE>(fp16);
    case F_GELU_GRAD: return pick<F_GELU_GRAD>(fp16);
    case F_GELU_GRAD | F_DROP: return pick<F_GELU_GRAD | F_DROP>(fp16);
    case F_BIAS | F_GELU | F_KEEP_Z: return pick<F_BIAS | F_GELU | F_KEEP_Z>(fp16);
    case F_BIAS | F_GELU | F_DROP | F_KEEP_Z: return pick<F_BIAS | F_GELU | F_DROP | F_KEEP_Z>(fp16);
    default: return nullptr;
  }
}

// Shared-memory plan: panels of a group, chunk, ring depth, staging buffers (`twice`: two a team where they leave the ring four
// stages).  False: no plan fits.
bool plan_rows(RowsArgs& g, bool twice, bool keep_z, int sms, size_t budget) {
  const size_t panel_bytes = (size_t)g.k_panels * kPanel * 128;              // one panel's rows of B
  const size_t out_bytes = (size_t)kTeams * 4 * kBlockBytes;                 // one staging buffer a team
  auto chunk_of = [](int gp) { return gp % 2 == 0 ? 2 : gp == 3 ? 3 : 1; };
  const int few = 3;                                                         // ring stages without which the loads' latency shows
  int best = 0;
  for (int gp = g.panels; gp >= 1 && best == 0; --gp) {                      // the widest group that leaves the ring deep enough
    if (g.panels % gp != 0 || gp * kPanel > kMaxGroupCols) continue;
    const int need = gp > chunk_of(gp) ? (g.k_panels > few ? g.k_panels : few) : few;   // several chunks share a row tile's panels
    if (gp * panel_bytes + (keep_z ? 2 : 1) * out_bytes + (size_t)need * kAStage <= budget) best = gp;
  }
  // Splitting the columns reads A once per group (all but once from L2).  Groups side by side / B streamed, us at 400 k rows (outputs x
  // features): two groups 256 x 256 120 / 132, 256 x 200 91 / 129; four 768 x 256 217 / 202, 512 x 256 with a bit mask 173 / 146, 256 x 512
  // 270 / 153, 256 x 768 381 / 196.
  g.resident = best > 0 && g.panels / best <= 2;
  if (g.resident) {
    // too few row tiles for the SMs: narrower groups
    while (best > 1 && g.m_tiles * (g.panels / best) * 2 <= sms) {
      int gp = best - 1;
      while (g.panels % gp != 0) --gp;
      best = gp;
    }
    g.group_panels = best;
    g.chunk_panels = chunk_of(best);
    g.n_acc = g.chunk_panels == 3 ? 2 : 4;
    const size_t left = budget - best * panel_bytes;
    g.n_buf = keep_z ? 2 : 1;
    if (twice && left >= 2 * out_bytes + (size_t)4 * kAStage) g.n_buf = 2;
    const int deep = (int)((left - g.n_buf * out_bytes) / kAStage);
    g.stages = deep < kMaxStages ? deep : kMaxStages;
    if (g.stages < (g.group_panels > g.chunk_panels ? g.k_panels : 1)) return false;
  } else {
    g.n_buf = keep_z ? 2 : 1;
    const size_t left = budget - g.n_buf * out_bytes;
    int gp = 4;
    while (gp > 1 && (g.panels % gp != 0 || 2 * (kAStage + (size_t)gp * kPanel * 128) > left)) --gp;
    g.group_panels = g.chunk_panels = gp;
    g.n_acc = gp >= 3 ? 2 : 4;
    const size_t stage = kAStage + (size_t)gp * kPanel * 128;
    const int deep = (int)(left / stage);
    g.stages = deep < kMaxStages ? deep : kMaxStages;
  }
  g.groups = g.panels / g.group_panels;
  return true;
}

}  // namespace

// cudaErrorNotSupported: not a product of this kernel (the caller's other kernel takes it); any other value is the result.
extern "C" int bf_gemm_rows(const bf_gemm_params* p, cudaStream_t st) {
  if (p->n_src > 1 || p->n_dest != 1 || p->out_fp32 || (p->ldc * 2) % 16 != 0 || ((uintptr_t)p->dst[0]) % 16 != 0 ||
      (p->relu_mask != nullptr && (p->mask_mode != 1 || p->residual != nullptr)) || p->dst_row_offset < 0 ||
      p->dst_row_offset + p->M >= (1ll << 31) - kTileM)
    return (int)cudaErrorNotSupported;
  const bool fp16 = p->dtype == BF_FP16;
  RowsArgs g;
  memset(&g, 0, sizeof(g));
  g.out_scale = p->out_scale == 0.f ? 1.f : p->out_scale;
  g.thresh = p->dropout_p > 0.f ? (uint32_t)(p->dropout_p * 4294967296.0) : 0u;
  g.keep_scale = g.thresh ? 1.f / (1.f - p->dropout_p) : 1.f;
  const bool gelu_grad = p->relu_mask != nullptr;
  int f = 0;
  if (p->bias) f |= F_BIAS;
  if (p->act == 1) f |= F_RELU;
  if (p->act == 2) f |= F_GELU;
  if (g.thresh) f |= F_DROP;
  if (p->residual) f |= F_RES;
  if (g.out_scale != 1.f) f |= F_SCALE;
  if (p->relu_bits_in) f |= F_BITS_IN;
  if (p->relu_bits_out) f |= F_BITS_OUT;
  if (gelu_grad) f |= F_GELU_GRAD;
  if (p->z_out) f |= F_KEEP_Z;
  RowsKernel kern = rows_kernel(f, fp16);
  if (kern == nullptr) return (int)cudaErrorNotSupported;
  g.M = p->M; g.N = p->N; g.one = 1u;
  g.m_tiles = (p->M + kTileM - 1) / kTileM;
  g.k_panels = (p->K + kPanel - 1) / kPanel;
  g.panels = (p->N + kPanel - 1) / kPanel;
  g.bias = p->bias; g.seed = p->dropout_seed;
  g.bits_in = static_cast<const unsigned short*>(p->relu_bits_in);
  g.bits_out = static_cast<unsigned short*>(p->relu_bits_out);
  g.ldmb = p->ldmb;
  g.dst_row = (int)p->dst_row_offset;
  g.status = p->status;
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int group_cols = g.panels * kPanel < kMaxGroupCols ? g.panels * kPanel : kMaxGroupCols;
  const size_t tail = ((sizeof(RowsControl) + 15) & ~size_t(15)) + (p->bias ? (size_t)group_cols * 4 : 0);
  const size_t budget = 227 * 1024 - 1024 - tail;
  const bool staged = (f & (F_RES | F_GELU_GRAD)) != 0;
  // A second staging buffer lets a warp write while its last store is read: 800 k rows of 128 x 128 plain 77 -> 72 us, with a bias 78 -> 72, with
  // a bit mask 78 -> 74.  With dropout the ALU pipe is what is short, and the shallower ring costs: 76 -> 78, with ReLU and bits 90 -> 94.
  const bool twice = staged || !(f & F_DROP);
  if (!plan_rows(g, twice, (f & F_KEEP_Z) != 0, sms, budget)) return (int)cudaErrorNotSupported;
  // With no epilogue to speak of, reading A twice, streaming B or a short ring shows: bf16 goes back to the other kernel there.  us at 800 k
  // rows there / here: 256 x 256 plain 151 / 158, with a bias 154 / 162; 128 x 384 143 / 150, 144 / 150; 256 x 512 246 / 269, 246 / 280;
  // 256 x 768 334 / 357, 339 / 351.  (More columns than features: 384 x 128 152 / 141, 512 x 256 276 / 257; fp16, which has no such instance there: 256 x 256
  // 247 / 162; 50 k rows: within 1 us.)
  if (!fp16 && (f == 0 || f == F_BIAS) && p->N <= p->K && g.m_tiles >= 4 * sms && (!g.resident || g.groups > 1 || g.stages < 5))
    return (int)cudaErrorNotSupported;
  CUtensorMap map_a, map_b, map_out, map_z, map_in;
  memset(&map_z, 0, sizeof(map_z));
  memset(&map_in, 0, sizeof(map_in));
  if (make_map(&map_a, p->A, p->M, p->K, p->lda, kTileM, fp16) != 0 ||
      make_map(&map_b, p->B, p->N, p->K, p->ldb, g.chunk_panels * kPanel, fp16) != 0 ||
      make_map(&map_out, p->dst[0], p->dst_row_offset + p->M, p->N, p->ldc, 32, fp16) != 0 ||
      (p->z_out && make_map(&map_z, p->z_out, p->M, p->N, p->ldz, 32, fp16) != 0) ||
      (staged && make_map(&map_in, gelu_grad ? p->relu_mask : p->residual, p->M, p->N, gelu_grad ? p->ldm : p->ldr, 32, fp16) != 0))
    return (int)cudaErrorNotSupported;
  const size_t b_panel = (size_t)g.chunk_panels * kPanel * 128;
  const size_t smem = 1024 + (g.resident ? (size_t)(g.group_panels / g.chunk_panels) * g.k_panels * b_panel : 0) +
                      (size_t)g.stages * (kAStage + (g.resident ? 0 : b_panel)) + (size_t)kTeams * g.n_buf * 4 * kBlockBytes + tail;
  {
    // the attribute belongs to (function, device): remember it per device, not per process
    constexpr int MAX_DEV = 64;
    static bool attr_set[MAX_DEV][2048] = {};
    const int slot = f | (fp16 ? 1024 : 0);
    if (dev < 0 || dev >= MAX_DEV || !attr_set[dev][slot]) {
      cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
      if (e != cudaSuccess) return (int)e;
      if (dev >= 0 && dev < MAX_DEV) attr_set[dev][slot] = true;
    }
  }
  const int per_group = sms / g.groups;
  const int tiles = g.m_tiles < per_group ? g.m_tiles : per_group;
  if (tiles < 1) return (int)cudaErrorNotSupported;
  kern<<<tiles * g.groups, kThreads, smem, st>>>(map_a, map_b, map_out, map_z, map_in, g);
  return (int)cudaGetLastError();
}
