// Persistent, warp-specialised bf16 GEMM  D[m][n] = sum_k A[m][k] * B[n][k]  for sm_100a.
//
//   warp 0      : TMA producer (one lane elected inside the instructions), 128-byte-swizzled K-major tiles, STAGES-deep ring
//   warp 1      : tcgen05.mma issuer (one lane elected inside the instructions); owns the TMEM allocation (2 accumulators)
//   warps 2..9  : epilogue; two warps share each 32-lane quarter of the 128-row accumulator (one per
//                 half of the columns) and drain it with tcgen05.ld while the MMA warp already fills
//                 the other buffer.  Row-major outputs leave through each warp's own staging tiles
//                 and TMA stores; residual and gate tiles of the 128-wide configuration come in by TMA.
//
// The output projections, the single representation's and the diffusion transformer's projections and the per-channel
// N x N x N TriangleMultiplication contraction (batched over the 128 channels) run through this kernel; they differ only in
// the tensor maps and in the epilogue that is fused behind the accumulator.
#include <cuda_fp16.h>

#include "internal.h"
#include "umma.cuh"

namespace xf {

__device__ __forceinline__ uint32_t pack_f16x2(float lo, float hi) {
  const __half2 h = __floats2half2_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&h);
}

constexpr int BM = 128;
constexpr int BK = 64;
constexpr int GEMM_THREADS = 320;  // TMA warp, MMA warp, 8 epilogue warps

constexpr uint32_t EPI_TILE = 128 * 64 * 2;  // a residual / gate chunk: [128 rows][64 columns] bf16, 128-byte swizzled
constexpr uint32_t OUT_TILE = 32 * 32 * 2;   // a warp's part of an output chunk: [32 rows][32 columns] bf16, 64-byte swizzled

template <int BN>
struct GemmCfg {
  static constexpr int STAGES = BN == 64 ? 5 : 4;
  static constexpr uint32_t A_BYTES = BM * BK * 2;
  static constexpr uint32_t B_BYTES = BN * BK * 2;
  static constexpr uint32_t STAGE_BYTES = A_BYTES + B_BYTES;
  // after the operand ring: 2 output parts for each of 8 warps; with 128- and 64-wide tiles also 2 residual and 2 gate chunks
  static constexpr uint32_t OFF_OUT = STAGES * STAGE_BYTES;
  static constexpr uint32_t OFF_RES = OFF_OUT + 8 * 2 * OUT_TILE;
  static constexpr uint32_t OFF_GATE = OFF_RES + 2 * EPI_TILE;
  static constexpr uint32_t OFF_BAR = (BN <= 128) ? OFF_GATE + 2 * EPI_TILE : OFF_RES;
  static constexpr uint32_t SMEM_BYTES = OFF_BAR + 256 /*barriers*/ + 1024 /*align slack*/;
};

template <int BN, int EPI>
__global__ void __launch_bounds__(GEMM_THREADS, 1)
gemm_tn_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
               const __grid_constant__ CUtensorMap tmO, const __grid_constant__ CUtensorMap tmR,
               const __grid_constant__ CUtensorMap tmG, const GemmArgs p) {
  using Cfg = GemmCfg<BN>;
  constexpr int STAGES = Cfg::STAGES;
  // residual / gate chunks are prefetched by TMA
  constexpr bool EPI_LOADS = EPI == EPI_GATE_RESID;
  static_assert(!EPI_LOADS || BN <= 128, "no room for the residual / gate chunks beside 256-wide operand tiles");
  // SWIGLU weights come in groups of [128 SiLU rows | 128 linear rows]: a tile takes BN / 2 rows of either half
  constexpr bool B_SPLIT = EPI == EPI_SWIGLU && BN < 256;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw_addr = smem_u32(smem_raw);
  uint8_t* smem = smem_raw + (((raw_addr + 1023u) & ~1023u) - raw_addr);
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + Cfg::OFF_BAR);
  uint64_t* empty = full + STAGES;
  uint64_t* tfull = empty + STAGES;
  uint64_t* tempty = tfull + 2;
  uint64_t* efull = tempty + 2;   // [2] residual / gate chunk landed
  uint64_t* eempty = efull + 2;   // [2] residual / gate chunk consumed
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(eempty + 2);
  volatile int* cta_abort = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = __reduce_max_sync(0xffffffffu, threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  const AbortCtx ab{cta_abort, p.status};

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(&tfull[s], 1);
      mbar_init(&tempty[s], 8);
      mbar_init(&efull[s], 1);
      mbar_init(&eempty[s], 8);
    }
    *cta_abort = 0;
    fence_barrier_init();
    tma_prefetch_desc(&tmA);
    tma_prefetch_desc(&tmB);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 2 * BN);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = __reduce_max_sync(0xffffffffu, *tmem_slot);

  const int KB = (p.K + BK - 1) / BK;
  const long long total = (long long)p.batches * p.tiles_m * p.tiles_n;

  if (warp == 0) {
    // warp-uniform, like the issuer below
    const uint32_t go = elect_one();
    uint32_t stage = 0, phase = 0, echunk = 0;
    bool okay = true;
    (void)echunk;
    auto load_b = [&](uint8_t* sB, uint64_t* bar, int kb, int tn, int bb) {
      if constexpr (B_SPLIT) {
        const int r0 = tn * (BN / 2) / 128 * 256 + tn * (BN / 2) % 128;
        tma_load_3d_if(go, sB, &tmB, bar, kb * BK, r0, bb);
        tma_load_3d_if(go, sB + Cfg::B_BYTES / 2, &tmB, bar, kb * BK, r0 + 128, bb);
      } else {
        tma_load_3d_if(go, sB, &tmB, bar, kb * BK, tn * BN, bb);
      }
    };
    // Weights that no kernel of this call writes are fetched before the wait for the previous kernel: with a few rows
    // of activations the launch is a latency chain and the weights' trip from HBM is the longest link of it.
    int pre = 0;
    if (p.static_b && (long long)blockIdx.x < total) {
      const int b0 = p.b_batched ? int(blockIdx.x / (p.tiles_n * p.tiles_m)) : 0;
      for (; pre < STAGES && pre < KB; ++pre) {
        mbar_arrive_expect_tx_if(go, &full[pre], Cfg::STAGE_BYTES);
        load_b(smem + pre * Cfg::STAGE_BYTES + Cfg::A_BYTES, &full[pre], pre, int(blockIdx.x % p.tiles_n), b0);
      }
      // What the ring has no room for yet: into L2, so that its later stages no longer wait for HBM (diffusion step at 77
      // tokens 787 -> 762 us, 5 x 384 1700 -> 1654, 2048 2550 -> 2520).
      for (int kb = pre; kb < KB; ++kb) {
        const int tn = int(blockIdx.x % p.tiles_n);
        if constexpr (B_SPLIT) {
          const int r0 = tn * (BN / 2) / 128 * 256 + tn * (BN / 2) % 128;
          tma_prefetch_3d_if(go, &tmB, kb * BK, r0, b0);
          tma_prefetch_3d_if(go, &tmB, kb * BK, r0 + 128, b0);
        } else {
          tma_prefetch_3d_if(go, &tmB, kb * BK, tn * BN, b0);
        }
      }
    }
    pdl_wait();
    pdl_launch();
    for (long long t = blockIdx.x; t < total && okay; t += gridDim.x) {
      const int tn = int(t % p.tiles_n);
      const int tm = int((t / p.tiles_n) % p.tiles_m);
      const int b = int(t / ((long long)p.tiles_n * p.tiles_m));
      const int a1 = tm * BM, a2 = b;
      const int bb = p.b_batched ? b : 0;
      if constexpr (EPI_LOADS) {
        const uint32_t nload = (p.resid ? 1u : 0u) + (p.gate ? 1u : 0u);
        if (nload) {
          for (int c = 0; c < BN / 64 && tn * BN + c * 64 < p.N && okay; ++c, ++echunk) {
            const uint32_t eb = echunk & 1u;
            if (!mbar_wait_warp(&eempty[eb], ((echunk >> 1) & 1u) ^ 1u, ab, XF_ERR_WAIT_EMPTY)) { okay = false; break; }
            mbar_arrive_expect_tx_if(go, &efull[eb], nload * EPI_TILE);
            if (p.resid) tma_load_3d_if(go, smem + Cfg::OFF_RES + eb * EPI_TILE, &tmR, &efull[eb], tn * BN + c * 64, tm * BM, 0);
            if (p.gate) tma_load_3d_if(go, smem + Cfg::OFF_GATE + eb * EPI_TILE, &tmG, &efull[eb], tn * BN + c * 64, tm * BM, 0);
          }
          if (!okay) break;
        }
      }
      for (int kb = 0; kb < KB; ++kb) {
        uint8_t* sA = smem + stage * Cfg::STAGE_BYTES;
        if (pre > 0) {  // the first tile's first stages: announced, and B on its way
          --pre;
          tma_load_3d_if(go, sA, &tmA, &full[stage], kb * BK, a1, a2);
          if (++stage == STAGES) { stage = 0; phase ^= 1u; }
          continue;
        }
        if (!mbar_wait_warp(&empty[stage], phase ^ 1u, ab, XF_ERR_WAIT_EMPTY)) { okay = false; break; }
        mbar_arrive_expect_tx_if(go, &full[stage], Cfg::STAGE_BYTES);
        if (!p.mn_major) {
          tma_load_3d_if(go, sA, &tmA, &full[stage], kb * BK, a1, a2);
          load_b(sA + Cfg::A_BYTES, &full[stage], kb, tn, bb);
        } else {
          // operands stored [k][m] / [k][n]: one [64 k][64 m] box (8 KB, 128-byte rows) per 64 rows of the tile
#pragma unroll
          for (int x = 0; x < BM / 64; ++x) tma_load_3d_if(go, sA + x * 8192, &tmA, &full[stage], a1 + x * 64, kb * BK, a2);
#pragma unroll
          for (int x = 0; x < BN / 64; ++x)
            tma_load_3d_if(go, sA + Cfg::A_BYTES + x * 8192, &tmB, &full[stage], tn * BN + x * 64, kb * BK, bb);
        }
        if (++stage == STAGES) { stage = 0; phase ^= 1u; }
      }
    }
  } else if (warp == 1) {
    pdl_wait();
    pdl_launch();
    // Warp-uniform throughout: votes instead of per-lane branches, one elected lane predicated inside each instruction, so
    // that descriptors and addresses stay in uniform registers.
    // MN-major operands (rows of the smem tile are K indices): 64-element chunks along M / N are 8 KB apart, a step of
    // 16 along K is 16 rows of 128 B
    const uint32_t go = elect_one();
    const uint32_t idesc = p.mn_major ? make_idesc(BM, BN, 1, 1) : make_idesc(BM, BN);
    const uint32_t lbo = p.mn_major ? 8192u : 16u, kstep = p.mn_major ? 128u : 2u;
    uint32_t stage = 0, phase = 0, it = 0;
    bool okay = true;
    for (long long t = blockIdx.x; t < total && okay; t += gridDim.x, ++it) {
      const uint32_t buf = it & 1u, aphase = (it >> 1) & 1u;
      if (!mbar_wait_warp(&tempty[buf], aphase ^ 1u, ab, XF_ERR_WAIT_TMEM_EMPTY)) break;
      tc_fence_after();
      const uint32_t d = tmem_base + buf * BN;
      for (int kb = 0; kb < KB; ++kb) {
        if (!mbar_wait_warp(&full[stage], phase, ab, XF_ERR_WAIT_FULL)) { okay = false; break; }
        tc_fence_after();
        const uint32_t sA = smem_u32(smem + stage * Cfg::STAGE_BYTES);
        const uint64_t ad = make_sdesc(sA, lbo, 1024);
        const uint64_t bd = make_sdesc(sA + Cfg::A_BYTES, lbo, 1024);
#pragma unroll
        for (int k = 0; k < BK / 16; ++k)  // K-major: 16 bf16 = 32 B along K inside the swizzled row
          umma_ss_if(go, d, ad + kstep * k, bd + kstep * k, idesc, (kb | k) ? 1u : 0u);
        umma_commit_if(go, &empty[stage]);
        if (++stage == STAGES) { stage = 0; phase ^= 1u; }
      }
      if (okay) umma_commit_if(go, &tfull[buf]);
    }
  } else {
    pdl_wait();
    pdl_launch();
    const uint32_t go = elect_one();
    const int q = warp & 3;          // TMEM lane quarter this warp may read
    const int ch = (warp - 2) >> 2;  // which half of the tile's columns this warp drains
    const int row = q * 32 + lane;
    uint32_t it = 0, ochunk = 0, echunk = 0;
    (void)ochunk; (void)echunk;
    for (long long t = blockIdx.x; t < total; t += gridDim.x, ++it) {
      const int tn = int(t % p.tiles_n);
      const int tm = int((t / p.tiles_n) % p.tiles_m);
      const int b = int(t / ((long long)p.tiles_n * p.tiles_m));
      const uint32_t buf = it & 1u, aphase = (it >> 1) & 1u;
      // GATE_RESID with a gate row per (row % mod): the first chunk's gate values, fetched before the wait as well
      const bool row_gate_vec = EPI == EPI_GATE_RESID && p.row_gate && (p.ldg & 7) == 0 && (p.N & 31) == 0 &&
                                (reinterpret_cast<uintptr_t>(p.row_gate) & 15) == 0;
      uint4 rg[4];
      auto fetch_row_gate = [&](int c) {
        const long long m = (long long)tm * BM + row;
        const int col = tn * BN + c * 64 + ch * 32;
        if (m < p.M && col < p.N) {
          const uint4* src = reinterpret_cast<const uint4*>(p.row_gate + (m % p.row_gate_mod) * p.ldg + col);
#pragma unroll
          for (int g = 0; g < 4; ++g) rg[g] = src[g];
        }
      };
      if constexpr (EPI == EPI_GATE_RESID)
        if (row_gate_vec) fetch_row_gate(0);
      // COLS: this lane's element of the column vectors, likewise
      float cb = 0.f, cs = 1.f;
      auto fetch_cols = [&](int c) {
        const int col = tn * BN + c * 64 + ch * 32 + lane;
        cb = p.col_bias && col < p.N ? p.col_bias[b * p.N + col] : 0.f;
        cs = p.col_scale && col < p.N ? p.col_scale[b * p.N + col] : 1.f;
        if (col - lane < p.log2e_cols) cs *= 1.4426950408889634f;
      };
      if constexpr (EPI == EPI_COLS) fetch_cols(0);
      if (!mbar_wait(&tfull[buf], aphase, ab, XF_ERR_WAIT_TMEM_FULL)) break;
      tc_fence_after();
      const uint32_t taddr = tmem_base + buf * BN + (uint32_t(q * 32) << 16);

      // Staged epilogue: the tile leaves in 64-column chunks.  Each of the 8 warps converts its 32 rows x 32
      // columns of the chunk into a 64-byte-swizzled shared-memory tile of its own (conflict-free 16-byte stores) and
      // hands it to TMA, without waiting for the other warps.  Residual / gate chunks arrive by TMA as [128][64] tiles.
      constexpr int NCH = (EPI == EPI_SWIGLU) ? BN / 128 : BN / 64;  // output chunks per tile
      constexpr int WOUT = (EPI == EPI_SWIGLU) ? BN / 2 : BN;        // output columns per tile
      const int n_out = (EPI == EPI_SWIGLU) ? p.N / 2 : p.N;
      const long long m = (long long)tm * BM + row;
      const uint32_t rsw = uint32_t(row & 7);
      // Chunks beyond the output's last column are left out.  (A part that passes through the staging buffers commits a
      // group even if it stores nothing: the wait below counts groups, and a part without one would let the next
      // overwrite a tile that is still being read.)
      const int nch = min(NCH, (n_out - tn * WOUT + 63) / 64);
#pragma unroll 1
      for (int c = 0; c < nch; ++c, ++ochunk) {
        const int col0 = tn * WOUT + c * 64;          // first output column of the chunk
        const int colw = col0 + ch * 32;              // first output column of this warp
        uint8_t* so = smem + Cfg::OFF_OUT + ((warp - 2) * 2 + (ochunk & 1u)) * OUT_TILE;
        float v[32];
        if constexpr (EPI == EPI_SWIGLU) {
          uint32_t ra[32], rb[32];
          tmem_ld32(taddr + c * 64 + ch * 32, ra);
          tmem_ld32(taddr + BN / 2 + c * 64 + ch * 32, rb);
          tmem_ld_wait();
#pragma unroll
          for (int e = 0; e < 32; e += 2) {
            const float2 x = make_float2(__uint_as_float(ra[e]), __uint_as_float(ra[e + 1]));
            const float2 h = fmul2(fmul2(x, sigmoid2(x)), make_float2(__uint_as_float(rb[e]), __uint_as_float(rb[e + 1])));
            v[e] = h.x;
            v[e + 1] = h.y;
          }
        } else {
          uint32_t r[32];
          tmem_ld32(taddr + c * 64 + ch * 32, r);
          tmem_ld_wait();
#pragma unroll
          for (int e = 0; e < 32; ++e) v[e] = __uint_as_float(r[e]);
        }
        if constexpr (EPI == EPI_GATE_RESID) {
          // order: v * sigmoid(gate) first, residual added last
          const bool staged = p.resid || p.gate;
          const uint32_t eb = echunk & 1u;
          if (staged) {
            mbar_wait(&efull[eb], (echunk >> 1) & 1u, ab, XF_ERR_WAIT_FULL);  // (a failed wait runs through)
            ++echunk;
          }
          uint8_t* sg = smem + Cfg::OFF_GATE + eb * EPI_TILE + row * 128;
          if (p.row_gate && !row_gate_vec) {  // by element into the gate chunk's place, which only p.gate uses
#pragma unroll 1
            for (int e = 0; e < 32; ++e) {
              bf16 t = __float2bfloat16(0.f);
              if (m < p.M && colw + e < n_out) t = p.row_gate[(m % p.row_gate_mod) * p.ldg + colw + e];
              *reinterpret_cast<bf16*>(sg + ((uint32_t(ch * 4 + (e >> 3)) ^ rsw) << 4) + (e & 7) * 2) = t;
            }
          }
          if (p.gate || p.row_gate) {
#pragma unroll
            for (int g = 0; g < 4; ++g) {
              const uint4 u = row_gate_vec ? rg[g] : *reinterpret_cast<const uint4*>(sg + ((uint32_t(ch * 4 + g) ^ rsw) << 4));
              const uint32_t w4[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                const float2 x = fmul2(make_float2(v[g * 8 + 2 * e], v[g * 8 + 2 * e + 1]), sigmoid2(make_float2(bf16_lo(w4[e]), bf16_hi(w4[e]))));
                v[g * 8 + 2 * e] = x.x;
                v[g * 8 + 2 * e + 1] = x.y;
              }
            }
            if (row_gate_vec && c + 1 < nch) fetch_row_gate(c + 1);
          }
          if (p.resid) {
            const uint8_t* sr = smem + Cfg::OFF_RES + eb * EPI_TILE + row * 128;
#pragma unroll
            for (int g = 0; g < 4; ++g) {
              const uint4 u = *reinterpret_cast<const uint4*>(sr + ((uint32_t(ch * 4 + g) ^ rsw) << 4));
              const uint32_t w4[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                const float2 x = fadd2(make_float2(v[g * 8 + 2 * e], v[g * 8 + 2 * e + 1]), make_float2(bf16_lo(w4[e]), bf16_hi(w4[e])));
                v[g * 8 + 2 * e] = x.x;
                v[g * 8 + 2 * e + 1] = x.y;
              }
            }
          }
          if (staged) {
            __syncwarp();
            if (lane == 0) mbar_arrive(&eempty[eb]);
          }
        }
        // the TMA store that last used this staging buffer (two chunks ago) must have read it out
        tma_store_wait_read<1>();
        __syncwarp();
        if constexpr (EPI == EPI_COLS) {
          // Every row needs all 32 elements of the column vectors: they pass through the free staging buffer.  (Loaded by
          // every thread from global memory they cost 1.3 us more in a launch of 128 tiles, and the code for columns that do
          // not come in fours cost instruction fetches.)
          float* sv = reinterpret_cast<float*>(so);
          sv[lane] = cb;
          sv[32 + lane] = cs;
          __syncwarp();
          if (c + 1 < nch) fetch_cols(c + 1);
#pragma unroll
          for (int e = 0; e < 8; ++e) {
            const float4 fb = reinterpret_cast<const float4*>(sv)[e], fs = reinterpret_cast<const float4*>(sv)[8 + e];
            const float2 x = fmul2(fadd2(make_float2(v[4 * e], v[4 * e + 1]), make_float2(fb.x, fb.y)), make_float2(fs.x, fs.y));
            const float2 y = fmul2(fadd2(make_float2(v[4 * e + 2], v[4 * e + 3]), make_float2(fb.z, fb.w)), make_float2(fs.z, fs.w));
            v[4 * e] = x.x; v[4 * e + 1] = x.y; v[4 * e + 2] = y.x; v[4 * e + 3] = y.y;
          }
          __syncwarp();
        }
        bool as_f16 = false;
        if constexpr (EPI == EPI_COLS) as_f16 = colw >= p.f16_col0 && colw < p.f16_col1;
#pragma unroll
        for (int g = 0; g < 4; ++g) {
          uint4 u;
          if (as_f16) {
            u.x = pack_f16x2(v[g * 8 + 0], v[g * 8 + 1]);
            u.y = pack_f16x2(v[g * 8 + 2], v[g * 8 + 3]);
            u.z = pack_f16x2(v[g * 8 + 4], v[g * 8 + 5]);
            u.w = pack_f16x2(v[g * 8 + 6], v[g * 8 + 7]);
          } else {
            u.x = pack_bf16x2(v[g * 8 + 0], v[g * 8 + 1]);
            u.y = pack_bf16x2(v[g * 8 + 2], v[g * 8 + 3]);
            u.z = pack_bf16x2(v[g * 8 + 4], v[g * 8 + 5]);
            u.w = pack_bf16x2(v[g * 8 + 6], v[g * 8 + 7]);
          }
          *reinterpret_cast<uint4*>(so + lane * 64 + ((uint32_t(g) ^ uint32_t((lane >> 1) & 3)) << 4)) = u;
        }
        fence_proxy_async_smem();
        __syncwarp();
        tma_store_3d_if(colw < n_out && tm * BM + q * 32 < p.M ? go : 0u, &tmO, so, colw, tm * BM + q * 32, b);
        tma_store_commit();  // empty groups (the other lanes', parts outside the output) count too: the wait is by number
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&tempty[buf]);
    }
    tma_store_wait_all();  // written, not only read out: the next kernel may be waiting already
  }

  tc_fence_before();
  __syncthreads();
  if (*cta_abort && threadIdx.x == 0) {
    // give TMA copies that were already in flight time to land before the CTA's memory is released
    const long long t0 = clock64();
    while (clock64() - t0 < 2000000) {}
  }
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 2 * BN);
  }
}

template <int BN, int EPI>
static int launch_one(Ctx* c, const CUtensorMap& tmA, const CUtensorMap& tmB, const GemmArgs& a, cudaStream_t st) {
  using Cfg = GemmCfg<BN>;
  static bool attr_done[8] = {false};
  auto kern = gemm_tn_kernel<BN, EPI>;
  if (!attr_done[c->device & 7]) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::SMEM_BYTES);
    if (e != cudaSuccess) return fail(c, XFOLD_ERR_LAUNCH, "gemm smem attribute: %s", cudaGetErrorString(e));
    attr_done[c->device & 7] = true;
  }
  const long long total = (long long)a.batches * a.tiles_m * a.tiles_n;
  if (total <= 0) return XFOLD_OK;
  CUtensorMap tmO = tmA, tmR = tmA, tmG = tmA;  // placeholders when unused
  const int n_out = (EPI == EPI_SWIGLU) ? a.N / 2 : a.N;
  const uint64_t bstride = a.batches > 1 ? (uint64_t)a.out_batch_stride : (uint64_t)a.ldo * (uint64_t)a.M;
  if (!make_tmap_bf16_3d(&tmO, a.out, n_out, a.M, a.batches, a.ldo, bstride, 32, 32, 1, 64))
    return fail(c, XFOLD_ERR_ARG, "gemm: cannot encode the output tensor map (16-byte aligned base, ld multiple of 8?)");
  if (EPI == EPI_GATE_RESID) {
    if (a.resid && !make_tmap_bf16_3d(&tmR, a.resid, a.N, a.M, 1, a.ldr, (uint64_t)a.ldr * a.M, 64, 128, 1))
      return fail(c, XFOLD_ERR_ARG, "gemm: cannot encode the residual tensor map");
    if (a.gate && !make_tmap_bf16_3d(&tmG, a.gate, a.N, a.M, 1, a.ldg, (uint64_t)a.ldg * a.M, 64, 128, 1))
      return fail(c, XFOLD_ERR_ARG, "gemm: cannot encode the gate tensor map");
  }
  const int sms = c->gemm_sms > 0 && c->gemm_sms < c->sm_count ? c->gemm_sms : c->sm_count;
  const int grid = (int)(total < sms ? total : sms);
  const int tag = EPI == EPI_SWIGLU ? XFOLD_K_LINEAR_SWIGLU
                  : EPI == EPI_GATE_RESID ? XFOLD_K_LINEAR_GATE_RESID
                  : (EPI == EPI_PLAIN && a.batches > 1 ? XFOLD_K_TRIMUL_CONTRACT : XFOLD_K_LINEAR);
  ProfScope ps(c, tag, st);
  launch_pdl(kern, grid, GEMM_THREADS, Cfg::SMEM_BYTES, st, tmA, tmB, tmO, tmR, tmG, a);
  return check_launch(c, "gemm_tn_kernel");
}

int launch_gemm(Ctx* c, int epi, int bn, const CUtensorMap& tmA, const CUtensorMap& tmB, const GemmArgs& a,
                cudaStream_t st) {
  switch (epi * 1000 + bn) {
    case EPI_PLAIN * 1000 + 256: return launch_one<256, EPI_PLAIN>(c, tmA, tmB, a, st);
    case EPI_PLAIN * 1000 + 128: return launch_one<128, EPI_PLAIN>(c, tmA, tmB, a, st);
    case EPI_PLAIN * 1000 + 64: return launch_one<64, EPI_PLAIN>(c, tmA, tmB, a, st);
    case EPI_COLS * 1000 + 256: return launch_one<256, EPI_COLS>(c, tmA, tmB, a, st);
    case EPI_COLS * 1000 + 128: return launch_one<128, EPI_COLS>(c, tmA, tmB, a, st);
    case EPI_COLS * 1000 + 64: return launch_one<64, EPI_COLS>(c, tmA, tmB, a, st);
    case EPI_GATE_RESID * 1000 + 128: return launch_one<128, EPI_GATE_RESID>(c, tmA, tmB, a, st);
    case EPI_GATE_RESID * 1000 + 64: return launch_one<64, EPI_GATE_RESID>(c, tmA, tmB, a, st);
    case EPI_SWIGLU * 1000 + 256: return launch_one<256, EPI_SWIGLU>(c, tmA, tmB, a, st);
    case EPI_SWIGLU * 1000 + 128: return launch_one<128, EPI_SWIGLU>(c, tmA, tmB, a, st);
  }
  return fail(c, XFOLD_ERR_ARG, "gemm: unsupported tile %d / epilogue %d", bn, epi);
}

// Width of the output tiles.  A CTA's time is its number of tiles times what a tile costs, in clocks: the shared-memory
// reads of the products' operands (128 bytes per clock: 128 + BN of them per 64-wide step of K; they, not the tensor pipe,
// bound one CTA's products) or the epilogue (about 10 per column, it runs beside the next tile's products), and once the
// first tile's latency.  Wide tiles win when there are many (fewer operand reads), narrow ones when a wide tile would
// leave most SMs without work.
int gemm_tile_n(const Ctx* c, long long M, int N, int K, int batches, int widest, int narrowest) {
  const long long tm = (M + BM - 1) / BM * batches;
  const int kb = (K + BK - 1) / BK;
  int best = widest;
  double best_cost = 1e30;
  for (int bn = widest; bn >= narrowest; bn /= 2) {
    const long long tiles = tm * ((N + bn - 1) / bn), waves = (tiles + c->sm_count - 1) / c->sm_count;
    const double main_loop = double(kb) * (128 + bn), epi = 10.0 * bn;
    const double cost = waves * (main_loop > epi ? main_loop : epi) + (main_loop > epi ? epi : main_loop);
    if (cost < best_cost * 0.98) {
      best_cost = cost;
      best = bn;
    }
  }
  return best;
}

}  // namespace xf
