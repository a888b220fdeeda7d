// Output projections of the pair representation, 128 -> 128, with everything around them:
//   CM  (TriangleMultiplication): z += (LN_c(o) W^T) * sigmoid(g),  o channel-major [128][rows][tokens]
//   !CM (TriangleAttention)     : z += x W^T,                        x row-major [tokens][128]
// Bound: HBM.  CM reads o, g and z and writes z, 1024 bytes per token; !CM 768.
// CM_GZ: CM without g in memory, 768 bytes per token: g = LN(z) Wg^T is made here from the z that is loaded anyway, with the
// roundings of where it is written out (the row-shard stages).  It saves the projection kernel 256 of its 1024 bytes as well:
// projection and output of 1024 x 1024 tokens 332 + 195 -> 230 + 219 us, TriangleMultiplication of 768 tokens, both directions,
// 810 -> 720.  (The gate from the raw rows and their statistics, as for the pair bias: the same time, but its weights are
// rounded once more.)
//
// CM: the [128 channels][128 tokens] tile as it lies in memory is an MN-major operand of the tensor core, so nothing is
// transposed, and the LayerNorm over the channels enters through each token's statistics:
//     out = rstd * (D - mean * colsum) + colbias,  D = sum_c o[c] w'[n][c],  w' = bf16(w * gamma),
//     colsum[n] = sum_c w'[n][c] (of the rounded w': a constant token cancels exactly),  colbias[n] = sum_c beta[c] w[n][c]
// (As two launches -- LayerNorm with a transposing write-back, then a GEMM -- the normalised tokens made a round trip:
// 0.38 ms for 1024 x 1024 tokens, of which this kernel takes less than two thirds.)
//
// Persistent CTAs, tiles of 128 tokens through a ring of two stages {operand, z, g}:
//   warp 0        : TMA          warp 1 : tcgen05.mma issuer, one accumulator per stage
//   warps 2 - 9   : CM: token statistics from the operand tile, beside the product; CM_GZ: first LN(z) into a tile of its own
//   warps 10 - 25 : epilogue, one set of four per stage and half of the columns; a set's result replaces the z half it read
//                   and leaves by TMA
#include "internal.h"
#include "stages.h"
#include "umma.cuh"

namespace xf {

constexpr uint32_t RO_TILE = 32768;
constexpr int RO_THREADS = 26 * 32;
enum RoMode : int { RO_X = 0, RO_CM = 1, RO_CM_GZ = 2 };
template <int MODE>
struct RoCfg {
  static constexpr bool GZ = MODE == RO_CM_GZ;
  static constexpr uint32_t STAGE = (GZ ? 2 : 3) * RO_TILE;  // operand, z, g
  // GZ: the gate's weights, and a tile's normalised z
  static constexpr uint32_t OFF_W = 2 * STAGE, OFF_WG = OFF_W + RO_TILE, OFF_ZN = OFF_WG + RO_TILE,
                            OFF_CS = GZ ? OFF_ZN + RO_TILE : OFF_WG, OFF_GB = OFF_CS + 1024, OFF_BAR = OFF_GB + (GZ ? 1024 : 0),
                            SMEM = OFF_BAR + 256, TMEM = GZ ? 512 : 256;
  static_assert(SMEM <= 232448, "shared memory");
};

struct RowOutputArgs {
  const bf16* w;
  const float *gamma, *beta;
  long long tiles;
  int tiles_j;        // tiles per row (row mode), or 0: flat tokens
  int extent;         // tokens of a row
  int gate, resid, static_w;
  const float *g_gamma, *g_beta;  // GZ: the LayerNorm before the gate's projection
  int* status;
};

template <int MODE>
__global__ void __launch_bounds__(RO_THREADS, 1)
row_output_kernel(const __grid_constant__ CUtensorMap tmx, const __grid_constant__ CUtensorMap tmz,
                  const __grid_constant__ CUtensorMap tmg, const __grid_constant__ CUtensorMap tmo, const RowOutputArgs p) {
  using Cfg = RoCfg<MODE>;
  constexpr bool CM = MODE != RO_X, GZ = Cfg::GZ;
  extern __shared__ __align__(1024) uint8_t smem[];  // (no room to round up)
  float2* cs = reinterpret_cast<float2*>(smem + Cfg::OFF_CS);     // [128] (colsum, colbias)
  // a stage's token statistics (-mean, rstd) go over its operand tile once the product has read that
  auto rstat = [&](uint32_t s) { return reinterpret_cast<float2*>(smem + s * Cfg::STAGE); };
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + Cfg::OFF_BAR);  // [2]
  uint64_t* empty = full + 2;    // [2] the result has left shared memory (8 warps)
  uint64_t* t_full = empty + 2;  // [2] product complete
  uint64_t* t_empty = t_full + 2;  // [2] accumulator read (8 warps)
  uint64_t* st_full = t_empty + 2;  // [2] statistics written (8 warps)
  uint64_t* wg_full = st_full + 2;   // GZ: the gate's weights have landed
  uint64_t* zn_full = wg_full + 1;   // GZ: z of the tile normalised (8 warps)
  uint64_t* zn_empty = zn_full + 1;  // GZ: the gate's product has read it
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(zn_empty + 1);
  volatile int* cta_abort = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int warp = int(__reduce_max_sync(0xffffffffu, threadIdx.x >> 5)), lane = threadIdx.x & 31;
  const AbortCtx ab{cta_abort, p.status};

  if (threadIdx.x == 0) {
    for (int s = 0; s < 2; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 8);
      mbar_init(&t_full[s], 1);
      mbar_init(&t_empty[s], 8);
      mbar_init(&st_full[s], 8);
    }
    mbar_init(wg_full, 1);
    mbar_init(zn_full, 8);
    mbar_init(zn_empty, 1);
    *cta_abort = 0;
    fence_barrier_init();
    tma_prefetch_desc(&tmx);
    tma_prefetch_desc(&tmz);
    tma_prefetch_desc(&tmg);
    tma_prefetch_desc(&tmo);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, Cfg::TMEM);
    tmem_relinquish();
  }
  if (!p.static_w) pdl_wait();
  // Weights (times gamma) as a K-major swizzled operand; one row per half-warp, eight channels per lane.  All loads first: one
  // after the other, a row's trip behind the row's before, they were longer than a small predecessor takes.
  {
    constexpr int HW = RO_THREADS / 16, ROWS = (128 + HW - 1) / HW;
    const int l16 = lane & 15, n0 = threadIdx.x >> 4;
    uint4 u[ROWS];
    float ga[8], be[8];
#pragma unroll
    for (int i = 0; i < ROWS; ++i)
      if (n0 + i * HW < 128) u[i] = *reinterpret_cast<const uint4*>(p.w + (n0 + i * HW) * 128 + l16 * 8);
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      ga[e] = CM && p.gamma ? p.gamma[l16 * 8 + e] : 1.f;
      be[e] = CM && p.beta ? p.beta[l16 * 8 + e] : 0.f;
    }
    if (GZ && threadIdx.x < 128) {  // the input LayerNorm's scale and offset
      float* gb = reinterpret_cast<float*>(smem + Cfg::OFF_GB);
      gb[threadIdx.x] = p.g_gamma ? p.g_gamma[threadIdx.x] : 1.f;
      gb[threadIdx.x + 128] = p.g_beta ? p.g_beta[threadIdx.x] : 0.f;
    }
#pragma unroll
    for (int i = 0; i < ROWS; ++i) {
      const int n = n0 + i * HW;
      if (n < 128) {  // (the same for both half-warps of a warp: HW and 128 are even)
        const uint32_t w4[4] = {u[i].x, u[i].y, u[i].z, u[i].w};
        uint32_t o[4];
        float s = 0.f, b = 0.f;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float w0 = bf16_lo(w4[e]), w1 = bf16_hi(w4[e]);
          o[e] = CM ? pack_bf16x2(w0 * ga[2 * e], w1 * ga[2 * e + 1]) : w4[e];
          s += bf16_lo(o[e]) + bf16_hi(o[e]);
          b += w0 * be[2 * e] + w1 * be[2 * e + 1];
        }
#pragma unroll
        for (int x = 8; x > 0; x >>= 1) {
          s += __shfl_xor_sync(0xffffffffu, s, x);
          b += __shfl_xor_sync(0xffffffffu, b, x);
        }
        *reinterpret_cast<uint4*>(smem + Cfg::OFF_W + (l16 >> 3) * 16384 + n * 128 + ((uint32_t(l16 & 7) ^ uint32_t(n & 7)) << 4)) =
            make_uint4(o[0], o[1], o[2], o[3]);
        if (l16 == 0) cs[n] = make_float2(s, b);
      }
    }
  }
  fence_proxy_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = __reduce_max_sync(0xffffffffu, *tmem_slot);
  const uint32_t base = smem_u32(smem);
  if (GZ && warp == 0) {
    const uint32_t go = elect_one();
    mbar_arrive_expect_tx_if(go, wg_full, RO_TILE);
    tma_load_3d_if(go, smem + Cfg::OFF_WG, &tmg, wg_full, 0, 0, 0);
    tma_load_3d_if(go, smem + Cfg::OFF_WG + 16384, &tmg, wg_full, 64, 0, 0);
  }
  pdl_wait();
  pdl_launch();
  const int mine = p.tiles > blockIdx.x ? int((p.tiles - blockIdx.x + gridDim.x - 1) / gridDim.x) : 0;
  // token coordinates of a tile: (first token, row)
  auto coords = [&](int it, int& j, int& i) {
    const long long t = blockIdx.x + (long long)it * gridDim.x;
    if (p.tiles_j) {
      i = int(t / p.tiles_j);
      j = int(t % p.tiles_j) * 128;
    } else {
      i = 0;
      j = int(t) * 128;
    }
  };

  if (warp == 0) {
    const uint32_t go = elect_one();  // warp-uniform, like the issuers
    for (int it = 0; it < mine; ++it) {
      const uint32_t s = it & 1;
      int j, i;
      coords(it, j, i);
      if (!mbar_wait_warp(&empty[s], ((uint32_t(it) >> 1) & 1u) ^ 1u, ab, XF_ERR_WAIT_EMPTY)) break;
      mbar_arrive_expect_tx_if(go, &full[s], RO_TILE * (1 + (GZ || p.resid ? 1 : 0) + (!GZ && p.gate ? 1 : 0)));
      uint8_t* sx = smem + s * Cfg::STAGE;
      if constexpr (CM) {
#pragma unroll
        for (int kb = 0; kb < 2; ++kb)
#pragma unroll
          for (int x = 0; x < 2; ++x) tma_load_3d_if(go, sx + kb * 16384 + x * 8192, &tmx, &full[s], j + x * 64, kb * 64, i);
      } else {
        tma_load_3d_if(go, sx, &tmx, &full[s], 0, j, i);
        tma_load_3d_if(go, sx + 16384, &tmx, &full[s], 64, j, i);
      }
      if (!GZ && p.gate) {
        tma_load_3d_if(go, sx + 2 * RO_TILE, &tmg, &full[s], 0, j, i);
        tma_load_3d_if(go, sx + 2 * RO_TILE + 16384, &tmg, &full[s], 64, j, i);
      }
      if (GZ || p.resid) {
        tma_load_3d_if(go, sx + RO_TILE, &tmz, &full[s], 0, j, i);
        tma_load_3d_if(go, sx + RO_TILE + 16384, &tmz, &full[s], 64, j, i);
      }
    }
  } else if (warp == 1) {
    const uint32_t leader = elect_one() ? 1u : 0u;
    constexpr uint32_t idesc = CM ? make_idesc(128, 128, 1, 0) : make_idesc(128, 128);
    const uint64_t wd = make_sdesc(base + Cfg::OFF_W, 16, 1024);
    for (int it = 0; it < mine; ++it) {
      const uint32_t s = it & 1, ph = (uint32_t(it) >> 1) & 1u;
      if (!mbar_wait_warp(&t_empty[s], ph ^ 1u, ab, XF_ERR_WAIT_TMEM_EMPTY)) break;
      if (!mbar_wait_warp(&full[s], ph, ab, XF_ERR_WAIT_FULL)) break;
      tc_fence_after();
      // CM: K rows of 128 bytes (64 tokens); 64-token chunks 8 KB apart, 16 channels = 2 KB
      const uint64_t xd = make_sdesc(base + s * Cfg::STAGE, CM ? 8192 : 16, 1024);
#pragma unroll
      for (int kh = 0; kh < 2; ++kh)
#pragma unroll
        for (int k = 0; k < 4; ++k)
          umma_ss_if(leader, tmem_base + s * 128, xd + uint64_t(kh * 1024 + k * (CM ? 128 : 2)), wd + uint64_t(kh * 1024 + 2 * k), idesc,
                     (kh | k) ? 1u : 0u);
      if constexpr (GZ) {  // the gate's product
        if (it == 0 && !mbar_wait_warp(wg_full, 0, ab, XF_ERR_WAIT_FULL)) break;
        if (!mbar_wait_warp(zn_full, uint32_t(it) & 1u, ab, XF_ERR_WAIT_FULL)) break;
        tc_fence_after();
        const uint64_t zd = make_sdesc(base + Cfg::OFF_ZN, 16, 1024);
#pragma unroll
        for (int kh = 0; kh < 2; ++kh)
#pragma unroll
          for (int k = 0; k < 4; ++k)
            umma_ss_if(leader, tmem_base + 256 + s * 128, zd + uint64_t(kh * 1024 + 2 * k), wd + uint64_t(RO_TILE / 16 + kh * 1024 + 2 * k),
                       make_idesc(128, 128), (kh | k) ? 1u : 0u);
        umma_commit_if(leader, zn_empty);
      }
      umma_commit_if(leader, &t_full[s]);
    }
  } else if (warp < 10) {
    if constexpr (CM) {
      // 16 tokens (8 pairs) per warp; lane = (quarter of the channels, token pair)
      const int tp = (warp - 2) * 8 + (lane & 7), part = lane >> 3;  // token pair 0..63
      const uint32_t off = uint32_t(tp >> 5) * 8192, chunk = uint32_t(tp & 31) >> 2, in = uint32_t(tp & 3) * 4;
      for (int it = 0; it < mine; ++it) {
        const uint32_t s = it & 1, ph = (uint32_t(it) >> 1) & 1u;
        mbar_wait(&full[s], ph, ab, XF_ERR_WAIT_FULL);  // (a failed wait runs through: these warps meet at a barrier)
        uint32_t xr[32];
        if constexpr (GZ) {  // LN(z) first, the longer way: 16 rows per warp, two threads per row, as in the projection of a and b
          const int zrow = (warp - 2) * 16 + (lane & 15), half = lane >> 4;
          float nm, rs;
          load_half_row(smem + s * Cfg::STAGE + RO_TILE, zrow, half, xr);
          half_row_stats(xr, nm, rs);
          mbar_wait(zn_empty, (uint32_t(it) & 1u) ^ 1u, ab, XF_ERR_WAIT_EMPTY);
          store_half_row(smem + Cfg::OFF_ZN, zrow, half, xr, nm, rs, reinterpret_cast<const float*>(smem + Cfg::OFF_GB));
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) mbar_arrive(zn_full);
        }
        const uint8_t* sx = smem + s * Cfg::STAGE + (part >> 1) * 16384 + off + in;
        float2 a[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
#pragma unroll
        for (int e = 0; e < 32; ++e) {
          const uint32_t r = uint32_t(part & 1) * 32 + ((e + 2 * part) & 31);  // rotated: the four parts hit different banks
          xr[e] = *reinterpret_cast<const uint32_t*>(sx + r * 128 + ((chunk ^ (r & 7u)) << 4));
        }
#pragma unroll
        for (int e = 0; e < 32; ++e) sum2(xr[e], a[e & 1]);
        float2 m = fadd2(a[0], a[1]);
#pragma unroll
        for (int x = 8; x < 32; x <<= 1) m = fadd2(m, make_float2(__shfl_xor_sync(0xffffffffu, m.x, x), __shfl_xor_sync(0xffffffffu, m.y, x)));
        const float n0 = -m.x * (1.f / 128), n1 = -m.y * (1.f / 128);
        float2 q[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
#pragma unroll
        for (int e = 0; e < 32; ++e) {
          float2 v;
          asm("{\n\t.reg .b16 l, h;\n\tmov.b32 {l, h}, %2;\n\tadd.rn.f32.bf16 %0, l, %3;\n\tadd.rn.f32.bf16 %1, h, %4;\n\t}"
              : "=f"(v.x), "=f"(v.y) : "r"(xr[e]), "f"(n0), "f"(n1));
          q[e & 1] = ffma2(v, v, q[e & 1]);
        }
        float2 ss = fadd2(q[0], q[1]);
#pragma unroll
        for (int x = 8; x < 32; x <<= 1) ss = fadd2(ss, make_float2(__shfl_xor_sync(0xffffffffu, ss.x, x), __shfl_xor_sync(0xffffffffu, ss.y, x)));
        named_bar_sync(5, 256);  // the tile has been read by all of these warps
        mbar_wait(&t_full[s], ph, ab, XF_ERR_WAIT_TMEM_FULL);
        if (part == 0) {
          rstat(s)[2 * tp] = make_float2(n0, rsqrtf(ss.x * (1.f / 128) + 1e-5f));
          rstat(s)[2 * tp + 1] = make_float2(n1, rsqrtf(ss.y * (1.f / 128) + 1e-5f));
        }
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(&st_full[s]);
      }
    }
  } else {
    const int set = (warp - 10) >> 2, s = set & 1, half = set >> 1, quarter = warp & 3, row = quarter * 32 + lane;
    const uint32_t rsw = uint32_t(row & 7), laddr = tmem_base + s * 128 + half * 64 + (uint32_t(quarter * 32) << 16);
    uint8_t* sz = smem + s * Cfg::STAGE + RO_TILE + half * 16384 + row * 128;
    const uint32_t go = elect_one();
    const uint8_t* sg = sz + RO_TILE;
    for (int it = s; it < mine; it += 2) {
      const uint32_t ph = (uint32_t(it) >> 1) & 1u;
      mbar_wait(&full[s], ph, ab, XF_ERR_WAIT_FULL);  // (a failed wait runs through)
      if (CM) mbar_wait(&st_full[s], ph, ab, XF_ERR_WAIT_FULL);
      mbar_wait(&t_full[s], ph, ab, XF_ERR_WAIT_TMEM_FULL);
      tc_fence_after();
      float nmean = 0.f, rstd = 1.f;
      if (CM) {
        const float2 st = rstat(s)[row];
        nmean = st.x;
        rstd = st.y;
      }
      constexpr int W = GZ ? 16 : 32;  // columns at a time
#pragma unroll 1
      for (int c = 0; c < 64 / W; ++c) {
        uint32_t r[W], rg[GZ ? W : 1];
        if constexpr (GZ) {
          tmem_ld16(laddr + c * W, r);
          tmem_ld16(laddr + 256 + c * W, rg);
        } else {
          tmem_ld32(laddr + c * W, r);
        }
        tmem_ld_wait();
        if (c == 64 / W - 1) {
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&t_empty[s]);
        }
#pragma unroll
        for (int q = 0; q < W / 8; ++q) {
          const uint32_t at = (uint32_t(c * (W / 8) + q) ^ rsw) << 4;
          const uint4 zu = p.resid ? *reinterpret_cast<const uint4*>(sz + at) : make_uint4(0, 0, 0, 0);
          const uint32_t zw[4] = {zu.x, zu.y, zu.z, zu.w};
          uint4 gu = make_uint4(0, 0, 0, 0);
          if (MODE == RO_CM && p.gate) gu = *reinterpret_cast<const uint4*>(sg + at);
          const uint32_t gw[4] = {gu.x, gu.y, gu.z, gu.w};
          uint32_t o[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int n = half * 64 + c * W + q * 8 + 2 * e;
            float2 v = make_float2(__uint_as_float(r[q * 8 + 2 * e]), __uint_as_float(r[q * 8 + 2 * e + 1]));
            if constexpr (CM) {
              uint32_t g2 = gw[e];
              // (rounded as where it passes through memory, so that the stages by rows give the same bits)
              if constexpr (GZ) g2 = pack_bf16x2(__uint_as_float(rg[q * 8 + 2 * e]), __uint_as_float(rg[q * 8 + 2 * e + 1]));
              const float4 k = *reinterpret_cast<const float4*>(&cs[n]);
              v = ffma2(make_float2(rstd, rstd), ffma2(make_float2(nmean, nmean), make_float2(k.x, k.z), v), make_float2(k.y, k.w));
              v = fmul2(v, sigmoid2(make_float2(bf16_lo(g2), bf16_hi(g2))));
            }
            v = fadd2(v, make_float2(bf16_lo(zw[e]), bf16_hi(zw[e])));
            o[e] = pack_bf16x2(v.x, v.y);
          }
          *reinterpret_cast<uint4*>(sz + at) = make_uint4(o[0], o[1], o[2], o[3]);
        }
      }
      // a warp's rows leave by themselves
      fence_proxy_async_smem();
      __syncwarp();
      int j, i;
      coords(it, j, i);
      j += quarter * 32;
      tma_store_3d_if(j < p.extent ? go : 0u, &tmo, smem + s * Cfg::STAGE + RO_TILE + half * 16384 + quarter * 4096, half * 64, j, i);
      tma_store_commit();
      tma_store_wait_read<0>();
      __syncwarp();
      if (lane == 0) mbar_arrive(&empty[s]);
    }
    tma_store_wait_all();
  }

  tc_fence_before();
  __syncthreads();
  if (*cta_abort && threadIdx.x == 0) {
    const long long c0 = clock64();
    while (clock64() - c0 < 2000000) {}
  }
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, Cfg::TMEM);
  }
}

template <int MODE>
static int launch_ro(Ctx* c, const CUtensorMap& tmx, const CUtensorMap& tmz, const CUtensorMap& tmg, const CUtensorMap& tmo,
                     RowOutputArgs& a, cudaStream_t st) {
  static bool attr_done[8] = {false};
  if (!attr_done[c->device & 7]) {
    cudaError_t e = cudaFuncSetAttribute(row_output_kernel<MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, RoCfg<MODE>::SMEM);
    if (e != cudaSuccess) return fail(c, XFOLD_ERR_LAUNCH, "row output smem attribute: %s", cudaGetErrorString(e));
    if (!only_dynamic_smem(row_output_kernel<MODE>)) return fail(c, XFOLD_ERR_LAUNCH, "row output: shared memory does not start at 1 KB");
    attr_done[c->device & 7] = true;
  }
  if (reinterpret_cast<uintptr_t>(a.w) & 15) return fail(c, XFOLD_ERR_ARG, "row output: the weights must be 16-byte aligned");
  const int sms = c->gemm_sms > 0 && c->gemm_sms < c->sm_count ? c->gemm_sms : c->sm_count;
  a.static_w = c->static_weights;
  a.status = c->d_status;
  ProfScope ps(c, XFOLD_K_LINEAR_GATE_RESID, st);
  launch_pdl(row_output_kernel<MODE>, (int)(a.tiles < sms ? a.tiles : sms), RO_THREADS, RoCfg<MODE>::SMEM, st, tmx, tmz, tmg, tmo, a);
  return check_launch(c, "row_output_kernel");
}

// out = (resid or 0) + x w^T; x, resid, out: [M][128]
int launch_row_output(Ctx* c, const bf16* x, long long M, const bf16* w, const bf16* resid, bf16* out, cudaStream_t st) {
  if (M <= 0) return XFOLD_OK;
  if (M >= (1ll << 31)) return fail(c, XFOLD_ERR_ARG, "linear: too many rows");
  CUtensorMap tmx, tmz, tmo;
  if (!make_tmap_bf16_3d(&tmx, x, 128, M, 1, 128, (uint64_t)128 * M, 64, 128, 1) ||
      !make_tmap_bf16_3d(&tmz, resid ? resid : out, 128, M, 1, 128, (uint64_t)128 * M, 64, 128, 1) ||
      !make_tmap_bf16_3d(&tmo, out, 128, M, 1, 128, (uint64_t)128 * M, 64, 32, 1))
    return fail(c, XFOLD_ERR_ARG, "row output: cannot encode tensor maps");
  RowOutputArgs a = {};
  a.w = w;
  a.tiles = (M + 127) / 128;
  a.extent = (int)M;
  a.resid = resid != nullptr;
  return launch_ro<RO_X>(c, tmx, tmz, tmz, tmo, a, st);
}

// out = (resid or 0) + (LN(o) w^T) * sigmoid(g); o element (i, c, j) at i * o_rs + c * o_cs + j; g, z, out: [R * N][128].
// g null: the gate is LN(z) wg^T, computed here.  resid: z is added.
int launch_row_output_cm(Ctx* c, const bf16* o, long long o_cs, long long o_rs, int R, int N, const float* gamma, const float* beta,
                         const bf16* w, const bf16* g, const float* g_gamma, const float* g_beta, const bf16* wg, const bf16* z,
                         int resid, bf16* out, cudaStream_t st) {
  if (R <= 0 || N <= 0) return XFOLD_OK;
  if ((o_cs | o_rs) & 7) return fail(c, XFOLD_ERR_ARG, "channel LayerNorm: strides must be multiples of 8");
  // rows that follow one another without padding are one long row of tokens: no partial tiles at each row's end
  const bool flat = o_rs == N && (long long)R * N < (1ll << 31);
  const uint64_t J = flat ? (uint64_t)R * N : N, I = flat ? 1 : R;
  CUtensorMap tmx, tmz, tmg, tmo;
  if (!make_tmap_bf16_3d(&tmx, o, J, 128, I, o_cs, flat ? (uint64_t)o_cs * 128 : (uint64_t)o_rs, 64, 64, 1) ||
      !make_tmap_bf16_3d(&tmz, z ? z : out, 128, J, I, 128, 128 * J, 64, 128, 1) ||
      !(g ? make_tmap_bf16_3d(&tmg, g, 128, J, I, 128, 128 * J, 64, 128, 1) : make_tmap_bf16_3d(&tmg, wg, 128, 128, 1, 128, 128 * 128, 64, 128, 1)) ||
      !make_tmap_bf16_3d(&tmo, out, 128, J, I, 128, 128 * J, 64, 32, 1))
    return fail(c, XFOLD_ERR_ARG, "row output: cannot encode tensor maps");
  RowOutputArgs a = {};
  a.w = w;
  a.gamma = gamma;
  a.beta = beta;
  a.g_gamma = g_gamma;
  a.g_beta = g_beta;
  a.tiles_j = flat ? 0 : (N + 127) / 128;
  a.tiles = flat ? (long long)(J + 127) / 128 : (long long)a.tiles_j * R;
  a.extent = (int)J;
  a.gate = g != nullptr;
  a.resid = resid;
  return g ? launch_ro<RO_CM>(c, tmx, tmz, tmg, tmo, a, st) : launch_ro<RO_CM_GZ>(c, tmx, tmz, tmg, tmo, a, st);
}

}  // namespace xf
