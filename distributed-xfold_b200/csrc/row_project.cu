// LayerNorm of the pair representation fused with the projections behind it:
//   trimul : a, b = gated projections (channel planes)                          (512 x 128 weights),
//            for the row-shard stages also g = gating rows                        (640 x 128)
//   attn   : q, k, v, gate (row-major [rows][512]) and the 4-head pair bias     (512 x 128 weights)
//
// Bound: HBM.  256 bytes of a row come in and 512 (trimul), 768 (with g) or 1032 (attn) leave.  As two launches the
// normalised rows made an extra round trip, and the projections' epilogues -- eight warps in lock-step over two staging buffers -- left HBM half idle.
//
// Persistent CTAs keep the weights in shared memory and walk over tiles of 128 rows:
//   warp 0              : TMA (weights once, then x tiles, two in flight)
//   warp 1              : tcgen05.mma issuer; a tile's columns in units of 128 accumulator columns, a ring of NSET units
//   warps 2 - 9         : LayerNorm in place, two threads per row.  For the pair bias the tensor core first multiplies the
//                         RAW tile (exact bf16) by w * gamma; the normalisation enters through the row's statistics.
//   then NSET x 4 warps : epilogue, one set of four per unit of the ring, each set on its own: no set waits for another
// A unit is 128 weight rows; for the gated projections [64 projection rows | 64 gate rows], so that both halves of 64 outputs
// meet in one accumulator; g is two units of 64.  With few tiles the units are divided over several CTAs per tile (`parts`;
// each normalises the tile for itself), so that a short sequence still uses the whole chip.  With g there are at least two parts
// (a with half of g, b with the other half): 160 KB of weights would leave no room for a second x tile, and with one, its
// load and normalisation stood between a tile's last product and the next tile's first (11 700 clocks per tile instead of
// the 7200 that HBM needs in the attn form).
#include <cuda_fp16.h>

#include "internal.h"
#include "stages.h"
#include "umma.cuh"

namespace xf {

struct RowProjectArgs {
  const float *gamma, *beta;
  int tiles, parts, static_w;
  int norm;         // 0: the rows come normalised, nothing is done to them
  long long rows;
  int mode1, dim1;  // mode1: tile rows step along the first token axis, second axis fixed (transposed planes)
  // trimul
  bf16 *out_a, *out_b;
  long long chan_stride, row_stride;
  int ntok;
  const float* mask;
  // attn
  const float *scale, *w_bias;
  bf16* bias;
  int pitch, inner;
  long long plane;
  int* status;
};

enum RpMode : int { RP_TRIMUL = 0, RP_TRIMUL_G = 1, RP_ATTN = 2 };
template <int MODE>
struct RpCfg {
  static constexpr bool ATTN = MODE == RP_ATTN, G = MODE == RP_TRIMUL_G;
  // units: attn q, k, v, gate; trimul a0, a1, b0, b1, with g a0, a1, g0, b0, b1, g1 (g: 64 columns)
  static constexpr int UNITS = G ? 6 : 4, NSET = ATTN ? 3 : 4, MIN_PARTS = G ? 2 : 1;
  static constexpr int THREADS = (10 + 4 * NSET) * 32;
  static constexpr uint32_t W_UNIT = 32768, X_TILE = 32768;      // [2 K halves][128 rows][64], swizzled
  static constexpr uint32_t STG = ATTN || G ? 128 * 32 * 2 : 0;                  // a set's staging tiles, [32 rows][32 columns] per warp
  static constexpr uint32_t OFF_W = 0, OFF_X = OFF_W + UNITS / MIN_PARTS * W_UNIT, OFF_STG = OFF_X + 2 * X_TILE,
                            OFF_WB = OFF_STG + NSET * STG, OFF_GB = OFF_WB + (ATTN ? 4096 : 0), OFF_SC = OFF_GB + 1024,
                            OFF_CB = OFF_SC + (ATTN ? 2048 : 0), OFF_ST = OFF_CB + (ATTN ? 128 : 0),
                            OFF_BAR = OFF_ST + (ATTN ? 2048 : 0), SMEM = OFF_BAR + 256 + 1024;
  static_assert(SMEM <= 232448, "shared memory");
};

template <int MODE>
__global__ void __launch_bounds__(RpCfg<MODE>::THREADS, 1)
row_project_kernel(const __grid_constant__ CUtensorMap tmx, const __grid_constant__ CUtensorMap tmw,
                   const __grid_constant__ CUtensorMap tmo, const RowProjectArgs p) {
  using Cfg = RpCfg<MODE>;
  constexpr int NSET = Cfg::NSET, UNITS = Cfg::UNITS, PER = UNITS / 2;  // PER: units of a (or b) and its part of g
  constexpr bool ATTN = Cfg::ATTN;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw_addr = smem_u32(smem_raw);
  uint8_t* smem = smem_raw + (((raw_addr + 1023u) & ~1023u) - raw_addr);
  float* gb = reinterpret_cast<float*>(smem + Cfg::OFF_GB);      // gamma[128], beta[128]
  float* sc = reinterpret_cast<float*>(smem + Cfg::OFF_SC);      // column scales, log2(e) on the q columns
  float* colsum = reinterpret_cast<float*>(smem + Cfg::OFF_CB);  // [16], colbias[16]
  float* colbias = colsum + 16;
  uint64_t* w_full = reinterpret_cast<uint64_t*>(smem + Cfg::OFF_BAR);
  uint64_t* x_full = w_full + 1;   // [2]
  uint64_t* x_free = x_full + 2;   // [2] the tile's last product is complete
  uint64_t* n_full = x_free + 2;   // [2] normalised in place
  uint64_t* b_full = n_full + 2;   // [2] bias product complete
  uint64_t* t_full = b_full + 2;   // [NSET] a unit's accumulator is complete
  uint64_t* t_empty = t_full + NSET;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(t_empty + NSET);
  volatile int* cta_abort = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int warp = int(__reduce_max_sync(0xffffffffu, threadIdx.x >> 5)), lane = threadIdx.x & 31;
  const AbortCtx ab{cta_abort, p.status};

  if (threadIdx.x == 0) {
    mbar_init(w_full, 1);
    for (int s = 0; s < 2; ++s) {
      mbar_init(&x_full[s], 1);
      mbar_init(&x_free[s], 1);
      mbar_init(&n_full[s], 8);
      mbar_init(&b_full[s], 1);
    }
    for (int s = 0; s < NSET; ++s) {
      mbar_init(&t_full[s], 1);
      mbar_init(&t_empty[s], 4);
    }
    *cta_abort = 0;
    fence_barrier_init();
    tma_prefetch_desc(&tmx);
    tma_prefetch_desc(&tmw);
    tma_prefetch_desc(&tmo);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  if (!p.static_w) pdl_wait();  // the parameters read below may come from the kernel before
  if (threadIdx.x < 128) {
    gb[threadIdx.x] = p.gamma ? p.gamma[threadIdx.x] : 1.f;
    gb[threadIdx.x + 128] = p.beta ? p.beta[threadIdx.x] : 0.f;
  }
  if constexpr (ATTN) {
    for (int i = threadIdx.x; i < 512; i += Cfg::THREADS) sc[i] = (p.scale ? p.scale[i] : 1.f) * (i < 128 ? 1.4426950408889634f : 1.f);
    // bias weights times gamma, four heads padded to 16 rows: [2 halves][16 rows][128 B], swizzled; one head per half-warp
    if (threadIdx.x < 256) {
      const int h = threadIdx.x >> 4, l16 = lane & 15;
      float s = 0.f, b = 0.f;
      uint32_t packed[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        float w2[2];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const int c = l16 * 8 + e * 2 + u;
          const float w = h < 4 && p.w_bias ? p.w_bias[h * 128 + c] : 0.f;
          w2[u] = __bfloat162float(__float2bfloat16(w * (p.gamma ? p.gamma[c] : 1.f)));
          s += w2[u];
          b += (p.beta ? p.beta[c] : 0.f) * w;
        }
        packed[e] = pack_bf16x2(w2[0], w2[1]);
      }
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) {
        s += __shfl_xor_sync(0xffffffffu, s, o);
        b += __shfl_xor_sync(0xffffffffu, b, o);
      }
      *reinterpret_cast<uint4*>(smem + Cfg::OFF_WB + (l16 >> 3) * 2048 + h * 128 + ((uint32_t(l16 & 7) ^ uint32_t(h & 7)) << 4)) =
          make_uint4(packed[0], packed[1], packed[2], packed[3]);
      if (l16 == 0) {
        colsum[h] = s;
        colbias[h] = b;
      }
    }
    fence_proxy_async_smem();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = __reduce_max_sync(0xffffffffu, *tmem_slot);
  const uint32_t base = smem_u32(smem);
  const int part = int(blockIdx.x) % p.parts, u0 = part * UNITS / p.parts, U = (part + 1) * UNITS / p.parts - u0;
  const int t0 = int(blockIdx.x) / p.parts, step = int(gridDim.x) / p.parts;
  const int mine = t0 < p.tiles ? (p.tiles - t0 + step - 1) / step : 0;
  const bool with_bias = ATTN && part == 0 && p.w_bias;
  auto unit_g = [](int g) { return Cfg::G && g % 3 == 2; };

  if (warp == 0) {
    const uint32_t go = elect_one();  // warp-uniform, like the issuers
    uint32_t bytes = 0;
    for (int u = 0; u < U; ++u) bytes += unit_g(u0 + u) ? Cfg::W_UNIT / 2 : Cfg::W_UNIT;
    mbar_arrive_expect_tx_if(go, w_full, bytes);
    for (int u = 0; u < U; ++u) {
      uint8_t* sw = smem + Cfg::OFF_W + u * Cfg::W_UNIT;
      const int g = u0 + u;
      // first 64 and last 64 weight rows of the unit (g: 64 in all)
      const int r0 = ATTN ? g * 128 : unit_g(g) ? 512 + (g / 3) * 64 : (g / PER) * 256 + (g % PER) * 64, r1 = ATTN ? r0 + 64 : r0 + 128;
#pragma unroll
      for (int kh = 0; kh < 2; ++kh) {
        tma_load_3d_if(go, sw + kh * 16384, &tmw, w_full, kh * 64, r0, 0);
        if (!unit_g(g)) tma_load_3d_if(go, sw + kh * 16384 + 8192, &tmw, w_full, kh * 64, r1, 0);
      }
    }
    pdl_wait();
    pdl_launch();
    for (int it = 0; it < mine; ++it) {
      const int t = t0 + it * step;
      const uint32_t xb = it & 1;
      if (!mbar_wait_warp(&x_free[xb], ((uint32_t(it) >> 1) & 1u) ^ 1u, ab, XF_ERR_WAIT_EMPTY)) break;
      mbar_arrive_expect_tx_if(go, &x_full[xb], Cfg::X_TILE);
      uint8_t* sx = smem + Cfg::OFF_X + xb * Cfg::X_TILE;
      const int c1 = p.mode1 ? t % p.dim1 : t * 128, c2 = p.mode1 ? t / p.dim1 * 128 : 0;
      tma_load_3d_if(go, sx, &tmx, &x_full[xb], 0, c1, c2);
      tma_load_3d_if(go, sx + 16384, &tmx, &x_full[xb], 64, c1, c2);
    }
  } else if (warp == 1) {
    pdl_wait();
    pdl_launch();
    const uint32_t leader = elect_one() ? 1u : 0u;
    constexpr uint32_t idesc = make_idesc(128, 128), idesc_b = make_idesc(128, 16);
    const uint64_t wbd = make_sdesc(base + Cfg::OFF_WB, 16, 1024);
    uint32_t set = 0, ph = 0;
    bool okay = mbar_wait_warp(w_full, 0, ab, XF_ERR_WAIT_FULL);
    int nb = 0;  // tiles whose bias product has been issued; it runs ahead of the tile's other products
    auto bias_product = [&]() {
      tc_fence_after();
      const uint32_t xb = nb & 1;
      const uint64_t xd = make_sdesc(base + Cfg::OFF_X + xb * Cfg::X_TILE, 16, 1024);
#pragma unroll
      for (int kh = 0; kh < 2; ++kh)
#pragma unroll
        for (int j = 0; j < 4; ++j)
          umma_ss_if(leader, tmem_base + 384 + xb * 16, xd + uint64_t(kh * 1024 + 2 * j), wbd + uint64_t(kh * 128 + 2 * j), idesc_b,
                     (kh | j) ? 1u : 0u);
      umma_commit_if(leader, &b_full[xb]);
      ++nb;
    };
    for (int it = 0; it < mine && okay; ++it) {
      const uint32_t xb = it & 1, xph = (uint32_t(it) >> 1) & 1u;
      if (with_bias && nb == it) {
        if (!mbar_wait_warp(&x_full[xb], xph, ab, XF_ERR_WAIT_FULL)) break;
        bias_product();
      }
      if (!mbar_wait_warp(&n_full[xb], xph, ab, XF_ERR_WAIT_FULL)) break;
      const uint64_t xd = make_sdesc(base + Cfg::OFF_X + xb * Cfg::X_TILE, 16, 1024);
      for (int u = 0; u < U; ++u) {
        if (with_bias && nb == it + 1 && nb < mine &&
            __all_sync(0xffffffffu, mbar_test_wait(&x_full[nb & 1], (uint32_t(nb) >> 1) & 1u)))
          bias_product();
        if (!mbar_wait_warp(&t_empty[set], ph ^ 1u, ab, XF_ERR_WAIT_TMEM_EMPTY)) { okay = false; break; }
        tc_fence_after();
        const uint64_t wd = make_sdesc(base + Cfg::OFF_W + u * Cfg::W_UNIT, 16, 1024);
        const uint32_t id = unit_g(u0 + u) ? make_idesc(128, 64) : idesc;
#pragma unroll
        for (int kh = 0; kh < 2; ++kh)
#pragma unroll
          for (int j = 0; j < 4; ++j)
            umma_ss_if(leader, tmem_base + set * 128, xd + uint64_t(kh * 1024 + 2 * j), wd + uint64_t(kh * 1024 + 2 * j), id,
                       (kh | j) ? 1u : 0u);
        umma_commit_if(leader, &t_full[set]);
        if (++set == NSET) { set = 0; ph ^= 1u; }
      }
      if (okay) umma_commit_if(leader, &x_free[xb]);
    }
  } else if (warp < 10) {
    pdl_wait();
    pdl_launch();
    // 16 rows per warp; the two halves of a row in lanes l and l + 16
    const int row = (warp - 2) * 16 + (lane & 15), half = lane >> 4;
    for (int it = 0; it < mine; ++it) {
      const uint32_t xb = it & 1, xph = (uint32_t(it) >> 1) & 1u;
      mbar_wait(&x_full[xb], xph, ab, XF_ERR_WAIT_FULL);  // (a failed wait runs through: these warps may meet at a barrier)
      if (!p.norm) {
        __syncwarp();
        if (lane == 0) mbar_arrive(&n_full[xb]);
        continue;
      }
      uint8_t* sx = smem + Cfg::OFF_X + xb * Cfg::X_TILE;
      uint32_t xr[32];
      load_half_row(sx, row, half, xr);
      float nmean, rstd;
      half_row_stats(xr, nmean, rstd);
      if (with_bias) {
        // (by tile parity: a warp may be one tile ahead of the readers, not two -- the barrier is in between)
        float2* rstat = reinterpret_cast<float2*>(smem + Cfg::OFF_ST) + xb * 128;
        if (half == 0) rstat[row] = make_float2(nmean, rstd);
        named_bar_sync(NSET + 1, 256);
        mbar_wait(&b_full[xb], xph, ab, XF_ERR_WAIT_TMEM_FULL);
        if (warp < 6) {  // (warp & 3) is the quarter of tensor memory's lanes this warp may read: row = lane there
          tc_fence_after();
          uint32_t d[4];
          asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
                       : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
                       : "r"(tmem_base + 384 + xb * 16 + (uint32_t((warp & 3) * 32) << 16)) : "memory");
          tmem_ld_wait();
          tc_fence_before();
          const int rr = (warp & 3) * 32 + lane;
          const long long r = (long long)(t0 + it * step) * 128 + rr;
          if (r < p.rows) {
            const float2 st = rstat[rr];
            const int q = int(r / p.inner), k = int(r - (long long)q * p.inner);
            __half* dst = reinterpret_cast<__half*>(p.bias) + (long long)q * p.pitch + k;
#pragma unroll
            for (int h = 0; h < 4; ++h) {
              const float v = fmaf(st.y, fmaf(st.x, colsum[h], __uint_as_float(d[h])), colbias[h]) * 1.4426950408889634f;
              dst[h * p.plane] = __float2half_rn(fminf(fmaxf(v, -60000.f), 60000.f));
            }
          }
        }
      }
      store_half_row(sx, row, half, xr, nmean, rstd, gb);
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(&n_full[xb]);
    }
  } else {
    pdl_wait();
    pdl_launch();
    const int set = (warp - 10) >> 2, quarter = warp & 3, row = quarter * 32 + lane;
    const uint32_t laddr = tmem_base + set * 128 + (uint32_t(quarter * 32) << 16);
    uint8_t* stg = smem + Cfg::OFF_STG + set * Cfg::STG + quarter * 2048;
    const uint32_t go = elect_one();
    uint32_t k = 0;  // units this set has taken
    for (int n = set; n < mine * U; n += NSET, ++k) {
      const int it = n / U, g = u0 + n % U, t = t0 + it * step;
      const int c1 = p.mode1 ? t % p.dim1 : t * 128, c2 = p.mode1 ? t / p.dim1 * 128 : 0;
      const uint32_t rsw = uint32_t(lane >> 1) & 3u;  // 64-byte swizzle of the staging tile
      if (ATTN || unit_g(g)) {
        const int chunks = ATTN ? 4 : 2, col0 = ATTN ? g * 128 : (g / 3) * 64;
        mbar_wait(&t_full[set], k & 1u, ab, XF_ERR_WAIT_TMEM_FULL);  // (a failed wait runs through)
        tc_fence_after();
#pragma unroll 1
        for (int c = 0; c < chunks; ++c) {
          uint32_t r[32];
          tmem_ld32(laddr + c * 32, r);
          tmem_ld_wait();
          if (c == chunks - 1) {
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&t_empty[set]);
          }
          uint4 o4[4];
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            uint32_t o[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              float v0 = __uint_as_float(r[q * 8 + 2 * e]), v1 = __uint_as_float(r[q * 8 + 2 * e + 1]);
              if constexpr (ATTN) {
                const float2 s2 = *reinterpret_cast<const float2*>(sc + col0 + c * 32 + q * 8 + 2 * e);
                v0 *= s2.x;
                v1 *= s2.y;
              }
              const __half2 h2 = __floats2half2_rn(v0, v1);  // the v columns leave as fp16
              o[e] = ATTN && g == 2 ? *reinterpret_cast<const uint32_t*>(&h2) : pack_bf16x2(v0, v1);
            }
            o4[q] = make_uint4(o[0], o[1], o[2], o[3]);
          }
          // a warp stages and stores its own rows; its store before has mostly been read out by now
          tma_store_wait_read<0>();
          __syncwarp();
#pragma unroll
          for (int q = 0; q < 4; ++q) *reinterpret_cast<uint4*>(stg + lane * 64 + ((uint32_t(q) ^ rsw) << 4)) = o4[q];
          fence_proxy_async_smem();
          __syncwarp();
          const int y = p.mode1 ? c1 : c1 + quarter * 32, x = p.mode1 ? c2 + quarter * 32 : c2;
          const bool inside = p.mode1 ? (long long)x * p.ntok < p.rows : (long long)y < p.rows;
          tma_store_3d_if(inside ? go : 0u, &tmo, stg, col0 + c * 32, y, x);
          tma_store_commit();
        }
      } else {
        // where this thread's token goes, and its mask value, before the wait
        long long off = 0;
        bool valid;
        float mk = 1.f;
        if (!p.mode1) {
          const long long tok = (long long)c1 + row, i = tok / p.ntok;
          valid = tok < p.rows;
          off = i * p.row_stride + (tok - i * p.ntok);
          if (valid && p.mask) mk = p.mask[tok];
        } else {
          const long long i = c2 + row;
          valid = i * p.ntok < p.rows;  // rows = first axis * ntok
          off = (long long)c1 * p.row_stride + i;
          if (valid && p.mask) mk = p.mask[i * p.ntok + c1];
        }
        bf16* dst = (g < PER ? p.out_a : p.out_b) + off + (long long)(g % PER * 64) * p.chan_stride;
        mbar_wait(&t_full[set], k & 1u, ab, XF_ERR_WAIT_TMEM_FULL);
        tc_fence_after();
#pragma unroll 1
        for (int c = 0; c < 4; ++c) {
          uint32_t rp[16], rg[16];
          tmem_ld16(laddr + c * 16, rp);
          tmem_ld16(laddr + 64 + c * 16, rg);
          tmem_ld_wait();
          if (c == 3) {
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&t_empty[set]);
          }
          if (valid) {
#pragma unroll
            for (int e = 0; e < 16; e += 2) {
              const float2 v = fmul2(make_float2(__uint_as_float(rp[e]), __uint_as_float(rp[e + 1])), make_float2(mk, mk));
              const float2 s = fmul2(v, sigmoid2(make_float2(__uint_as_float(rg[e]), __uint_as_float(rg[e + 1]))));
              const uint32_t o = pack_bf16x2(s.x, s.y);
              *dst = __ushort_as_bfloat16((unsigned short)o);
              dst += p.chan_stride;
              *dst = __ushort_as_bfloat16((unsigned short)(o >> 16));
              dst += p.chan_stride;
            }
          }
        }
      }
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
    tmem_dealloc(tmem_base, 512);
  }
}

template <int MODE>
static int launch_row_project(Ctx* c, const CUtensorMap& tmx, const CUtensorMap& tmw, const CUtensorMap& tmo, RowProjectArgs& a,
                              cudaStream_t st) {
  using Cfg = RpCfg<MODE>;
  static bool attr_done[8] = {false};
  if (!attr_done[c->device & 7]) {
    cudaError_t e = cudaFuncSetAttribute(row_project_kernel<MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::SMEM);
    if (e != cudaSuccess) return fail(c, XFOLD_ERR_LAUNCH, "row projection smem attribute: %s", cudaGetErrorString(e));
    attr_done[c->device & 7] = true;
  }
  const int sms = c->gemm_sms > 0 && c->gemm_sms < c->sm_count ? c->gemm_sms : c->sm_count;
  // units divided over CTAs as long as a tile per CTA group leaves SMs without work
  const int spread = sms / a.tiles;
  a.parts = spread < Cfg::MIN_PARTS ? Cfg::MIN_PARTS : spread > Cfg::UNITS ? Cfg::UNITS : spread;
  const int groups = a.tiles < sms / a.parts ? a.tiles : sms / a.parts;
  a.static_w = c->static_weights;
  a.status = c->d_status;
  ProfScope ps(c, Cfg::ATTN ? XFOLD_K_LINEAR : XFOLD_K_TRIMUL_PROJ, st);
  launch_pdl(row_project_kernel<MODE>, groups * a.parts, Cfg::THREADS, Cfg::SMEM, st, tmx, tmw, tmo, a);
  return check_launch(c, "row_project_kernel");
}

// out_g null: a and b alone
int launch_row_project_trimul(Ctx* c, const bf16* z, const float* mask, int R, int N, int transposed, const float* gamma,
                              const float* beta, const bf16* w_in, bf16* out_a, bf16* out_b, bf16* out_g, long long chan_stride,
                              long long row_stride, cudaStream_t st) {
  const long long M = (long long)R * N;
  CUtensorMap tmx, tmw, tmo;
  RowProjectArgs a = {};
  bool ok;
  if (!transposed) {
    ok = make_tmap_bf16_3d(&tmx, z, 128, M, 1, 128, (uint64_t)128 * M, 64, 128, 1) &&
         (!out_g || make_tmap_bf16_3d(&tmo, out_g, 128, M, 1, 128, (uint64_t)128 * M, 32, 32, 1, 64));
    a.tiles = (int)((M + 127) / 128);
  } else {  // tile rows step along the first token axis, second axis fixed: a[j][c][i]
    ok = make_tmap_bf16_3d(&tmx, z, 128, N, R, 128, (uint64_t)128 * N, 64, 1, 128) &&
         (!out_g || make_tmap_bf16_3d(&tmo, out_g, 128, N, R, 128, (uint64_t)128 * N, 32, 1, 32, 64));
    a.mode1 = 1;
    a.dim1 = N;
    a.tiles = N * ((R + 127) / 128);
  }
  ok = ok && make_tmap_bf16_3d(&tmw, w_in, 128, 640, 1, 128, 128 * 640, 64, 64, 1);
  if (!ok) return fail(c, XFOLD_ERR_ARG, "trimul: cannot encode projection tensor maps");
  a.norm = 1;
  a.gamma = gamma;
  a.beta = beta;
  a.rows = M;
  a.out_a = out_a;
  a.out_b = out_b;
  a.chan_stride = chan_stride;
  a.row_stride = row_stride;
  a.ntok = N;
  a.mask = mask;
  return out_g ? launch_row_project<RP_TRIMUL_G>(c, tmx, tmw, tmo, a, st) : launch_row_project<RP_TRIMUL>(c, tmx, tmw, tmx, a, st);
}

// norm = 0: z is normalised already, and w_bias (then null) has no output
int launch_row_project_attn(Ctx* c, const bf16* z, int R, int N, int norm, const float* gamma, const float* beta, const bf16* w_qkvg,
                            const float* scale, const float* w_bias, bf16* qkvg, bf16* bias, int pitch, long long plane,
                            cudaStream_t st) {
  const long long M = (long long)R * N;
  CUtensorMap tmx, tmw, tmo;
  RowProjectArgs a = {};
  if (!make_tmap_bf16_3d(&tmx, z, 128, M, 1, 128, (uint64_t)128 * M, 64, 128, 1) ||
      !make_tmap_bf16_3d(&tmo, qkvg, 512, M, 1, 512, (uint64_t)512 * M, 32, 32, 1, 64) ||
      !make_tmap_bf16_3d(&tmw, w_qkvg, 128, 512, 1, 128, 128 * 512, 64, 64, 1))
    return fail(c, XFOLD_ERR_ARG, "triattn: cannot encode projection tensor maps");
  a.tiles = (int)((M + 127) / 128);
  a.norm = norm;
  a.gamma = gamma;
  a.beta = beta;
  a.rows = M;
  a.scale = scale;
  a.w_bias = w_bias;
  a.bias = bias;
  a.pitch = pitch;
  a.inner = N;
  a.plane = plane;
  return launch_row_project<RP_ATTN>(c, tmx, tmw, tmo, a, st);
}

}  // namespace xf
