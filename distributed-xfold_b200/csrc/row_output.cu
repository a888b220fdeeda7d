// Output projections of the pair representation, 128 -> 128, with everything around them:
//   CM  (TriangleMultiplication): z += (LN_c(o) W^T) * sigmoid(g),  o channel-major [128][rows][tokens]
//   !CM (TriangleAttention)     : z += x W^T,                        x row-major [tokens][128]
// Bound: HBM.  CM reads o, g and z and writes z, 1024 bytes per token; !CM 768.
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
//   warps 2 - 9   : CM: token statistics from the operand tile, beside the product
//   warps 10 - 25 : epilogue, one set of four per stage and half of the columns; a set's result replaces the z half it read
//                   and leaves by TMA
#include "internal.h"
#include "stages.h"
#include "umma.cuh"

namespace xf {

constexpr uint32_t RO_TILE = 32768;
constexpr uint32_t RO_STAGE = 3 * RO_TILE;  // operand, z, g
constexpr uint32_t RO_OFF_W = 2 * RO_STAGE, RO_OFF_CS = RO_OFF_W + RO_TILE, RO_OFF_BAR = RO_OFF_CS + 1024, RO_SMEM = RO_OFF_BAR + 256 + 1024;
constexpr int RO_THREADS = 26 * 32;
static_assert(RO_SMEM <= 232448, "shared memory");

struct RowOutputArgs {
  const bf16* w;
  const float *gamma, *beta;
  long long tiles;
  int tiles_j;        // tiles per row (row mode), or 0: flat tokens
  int extent;         // tokens of a row
  int gate, resid, static_w;
  int* status;
};

template <bool CM>
__global__ void __launch_bounds__(RO_THREADS, 1)
row_output_kernel(const __grid_constant__ CUtensorMap tmx, const __grid_constant__ CUtensorMap tmz,
                  const __grid_constant__ CUtensorMap tmg, const __grid_constant__ CUtensorMap tmo, const RowOutputArgs p) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw_addr = smem_u32(smem_raw);
  uint8_t* smem = smem_raw + (((raw_addr + 1023u) & ~1023u) - raw_addr);
  float2* cs = reinterpret_cast<float2*>(smem + RO_OFF_CS);     // [128] (colsum, colbias)
  // a stage's token statistics (-mean, rstd) go over its operand tile once the product has read that
  auto rstat = [&](uint32_t s) { return reinterpret_cast<float2*>(smem + s * RO_STAGE); };
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + RO_OFF_BAR);  // [2]
  uint64_t* empty = full + 2;    // [2] the result has left shared memory (8 warps)
  uint64_t* t_full = empty + 2;  // [2] product complete
  uint64_t* t_empty = t_full + 2;  // [2] accumulator read (8 warps)
  uint64_t* st_full = t_empty + 2;  // [2] statistics written (8 warps)
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(st_full + 2);
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
    *cta_abort = 0;
    fence_barrier_init();
    tma_prefetch_desc(&tmx);
    tma_prefetch_desc(&tmz);
    tma_prefetch_desc(&tmg);
    tma_prefetch_desc(&tmo);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 256);
    tmem_relinquish();
  }
  if (!p.static_w) pdl_wait();
  // weights (times gamma) as a K-major swizzled operand; one row per half-warp, eight channels per lane
  for (int n = threadIdx.x >> 4; n < 128; n += RO_THREADS / 16) {
    const int l16 = lane & 15;
    const uint4 u = *reinterpret_cast<const uint4*>(p.w + n * 128 + l16 * 8);
    const uint32_t w4[4] = {u.x, u.y, u.z, u.w};
    uint32_t o[4];
    float s = 0.f, b = 0.f;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int c = l16 * 8 + 2 * e;
      const float w0 = bf16_lo(w4[e]), w1 = bf16_hi(w4[e]);
      o[e] = CM && p.gamma ? pack_bf16x2(w0 * p.gamma[c], w1 * p.gamma[c + 1]) : w4[e];
      s += bf16_lo(o[e]) + bf16_hi(o[e]);
      if (CM && p.beta) b += w0 * p.beta[c] + w1 * p.beta[c + 1];
    }
#pragma unroll
    for (int x = 8; x > 0; x >>= 1) {
      s += __shfl_xor_sync(0xffffffffu, s, x);
      b += __shfl_xor_sync(0xffffffffu, b, x);
    }
    *reinterpret_cast<uint4*>(smem + RO_OFF_W + (l16 >> 3) * 16384 + n * 128 + ((uint32_t(l16 & 7) ^ uint32_t(n & 7)) << 4)) =
        make_uint4(o[0], o[1], o[2], o[3]);
    if (l16 == 0) cs[n] = make_float2(s, b);
  }
  fence_proxy_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = __reduce_max_sync(0xffffffffu, *tmem_slot);
  const uint32_t base = smem_u32(smem);
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
      mbar_arrive_expect_tx_if(go, &full[s], RO_TILE * (1 + (p.resid ? 1 : 0) + (p.gate ? 1 : 0)));
      uint8_t* sx = smem + s * RO_STAGE;
      if constexpr (CM) {
#pragma unroll
        for (int kb = 0; kb < 2; ++kb)
#pragma unroll
          for (int x = 0; x < 2; ++x) tma_load_3d_if(go, sx + kb * 16384 + x * 8192, &tmx, &full[s], j + x * 64, kb * 64, i);
      } else {
        tma_load_3d_if(go, sx, &tmx, &full[s], 0, j, i);
        tma_load_3d_if(go, sx + 16384, &tmx, &full[s], 64, j, i);
      }
      if (p.gate) {
        tma_load_3d_if(go, sx + 2 * RO_TILE, &tmg, &full[s], 0, j, i);
        tma_load_3d_if(go, sx + 2 * RO_TILE + 16384, &tmg, &full[s], 64, j, i);
      }
      if (p.resid) {
        tma_load_3d_if(go, sx + RO_TILE, &tmz, &full[s], 0, j, i);
        tma_load_3d_if(go, sx + RO_TILE + 16384, &tmz, &full[s], 64, j, i);
      }
    }
  } else if (warp == 1) {
    const uint32_t leader = elect_one() ? 1u : 0u;
    constexpr uint32_t idesc = CM ? make_idesc(128, 128, 1, 0) : make_idesc(128, 128);
    const uint64_t wd = make_sdesc(base + RO_OFF_W, 16, 1024);
    for (int it = 0; it < mine; ++it) {
      const uint32_t s = it & 1, ph = (uint32_t(it) >> 1) & 1u;
      if (!mbar_wait_warp(&t_empty[s], ph ^ 1u, ab, XF_ERR_WAIT_TMEM_EMPTY)) break;
      if (!mbar_wait_warp(&full[s], ph, ab, XF_ERR_WAIT_FULL)) break;
      tc_fence_after();
      // CM: K rows of 128 bytes (64 tokens); 64-token chunks 8 KB apart, 16 channels = 2 KB
      const uint64_t xd = make_sdesc(base + s * RO_STAGE, CM ? 8192 : 16, 1024);
#pragma unroll
      for (int kh = 0; kh < 2; ++kh)
#pragma unroll
        for (int k = 0; k < 4; ++k)
          umma_ss_if(leader, tmem_base + s * 128, xd + uint64_t(kh * 1024 + k * (CM ? 128 : 2)), wd + uint64_t(kh * 1024 + 2 * k), idesc,
                     (kh | k) ? 1u : 0u);
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
        const uint8_t* sx = smem + s * RO_STAGE + (part >> 1) * 16384 + off + in;
        uint32_t xr[32];
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
    uint8_t* sz = smem + s * RO_STAGE + RO_TILE + half * 16384 + row * 128;
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
#pragma unroll 1
      for (int c = 0; c < 2; ++c) {
        uint32_t r[32];
        tmem_ld32(laddr + c * 32, r);
        tmem_ld_wait();
        if (c == 1) {
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&t_empty[s]);
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const uint32_t at = (uint32_t(c * 4 + q) ^ rsw) << 4;
          const uint4 zu = p.resid ? *reinterpret_cast<const uint4*>(sz + at) : make_uint4(0, 0, 0, 0);
          const uint32_t zw[4] = {zu.x, zu.y, zu.z, zu.w};
          uint4 gu = make_uint4(0, 0, 0, 0);
          if (CM && p.gate) gu = *reinterpret_cast<const uint4*>(sg + at);
          const uint32_t gw[4] = {gu.x, gu.y, gu.z, gu.w};
          uint32_t o[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            float v0 = __uint_as_float(r[q * 8 + 2 * e]), v1 = __uint_as_float(r[q * 8 + 2 * e + 1]);
            if constexpr (CM) {
              const float4 k = *reinterpret_cast<const float4*>(&cs[half * 64 + c * 32 + q * 8 + 2 * e]);
              v0 = fmaf(rstd, fmaf(nmean, k.x, v0), k.y) * sigmoidf_fast(bf16_lo(gw[e]));
              v1 = fmaf(rstd, fmaf(nmean, k.z, v1), k.w) * sigmoidf_fast(bf16_hi(gw[e]));
            }
            o[e] = pack_bf16x2(v0 + bf16_lo(zw[e]), v1 + bf16_hi(zw[e]));
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
      tma_store_3d_if(j < p.extent ? go : 0u, &tmo, smem + s * RO_STAGE + RO_TILE + half * 16384 + quarter * 4096, half * 64, j, i);
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
    tmem_dealloc(tmem_base, 256);
  }
}

template <bool CM>
static int launch_ro(Ctx* c, const CUtensorMap& tmx, const CUtensorMap& tmz, const CUtensorMap& tmg, const CUtensorMap& tmo,
                     RowOutputArgs& a, cudaStream_t st) {
  static bool attr_done[8] = {false};
  if (!attr_done[c->device & 7]) {
    cudaError_t e = cudaFuncSetAttribute(row_output_kernel<CM>, cudaFuncAttributeMaxDynamicSharedMemorySize, RO_SMEM);
    if (e != cudaSuccess) return fail(c, XFOLD_ERR_LAUNCH, "row output smem attribute: %s", cudaGetErrorString(e));
    attr_done[c->device & 7] = true;
  }
  if (reinterpret_cast<uintptr_t>(a.w) & 15) return fail(c, XFOLD_ERR_ARG, "row output: the weights must be 16-byte aligned");
  const int sms = c->gemm_sms > 0 && c->gemm_sms < c->sm_count ? c->gemm_sms : c->sm_count;
  a.static_w = c->static_weights;
  a.status = c->d_status;
  ProfScope ps(c, XFOLD_K_LINEAR_GATE_RESID, st);
  launch_pdl(row_output_kernel<CM>, (int)(a.tiles < sms ? a.tiles : sms), RO_THREADS, RO_SMEM, st, tmx, tmz, tmg, tmo, a);
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
  return launch_ro<false>(c, tmx, tmz, tmz, tmo, a, st);
}

// out = (resid or 0) + (LN(o) w^T) * sigmoid(g); o element (i, c, j) at i * o_rs + c * o_cs + j; g, resid, out: [R * N][128]
int launch_row_output_cm(Ctx* c, const bf16* o, long long o_cs, long long o_rs, int R, int N, const float* gamma, const float* beta,
                         const bf16* w, const bf16* g, const bf16* resid, bf16* out, cudaStream_t st) {
  if (R <= 0 || N <= 0) return XFOLD_OK;
  if ((o_cs | o_rs) & 7) return fail(c, XFOLD_ERR_ARG, "channel LayerNorm: strides must be multiples of 8");
  // rows that follow one another without padding are one long row of tokens: no partial tiles at each row's end
  const bool flat = o_rs == N && (long long)R * N < (1ll << 31);
  const uint64_t J = flat ? (uint64_t)R * N : N, I = flat ? 1 : R;
  CUtensorMap tmx, tmz, tmg, tmo;
  if (!make_tmap_bf16_3d(&tmx, o, J, 128, I, o_cs, flat ? (uint64_t)o_cs * 128 : (uint64_t)o_rs, 64, 64, 1) ||
      !make_tmap_bf16_3d(&tmz, resid ? resid : out, 128, J, I, 128, 128 * J, 64, 128, 1) ||
      !make_tmap_bf16_3d(&tmg, g, 128, J, I, 128, 128 * J, 64, 128, 1) || !make_tmap_bf16_3d(&tmo, out, 128, J, I, 128, 128 * J, 64, 32, 1))
    return fail(c, XFOLD_ERR_ARG, "row output: cannot encode tensor maps");
  RowOutputArgs a = {};
  a.w = w;
  a.gamma = gamma;
  a.beta = beta;
  a.tiles_j = flat ? 0 : (N + 127) / 128;
  a.tiles = flat ? (long long)(J + 127) / 128 : (long long)a.tiles_j * R;
  a.extent = (int)J;
  a.gate = 1;
  a.resid = resid != nullptr;
  return launch_ro<true>(c, tmx, tmz, tmg, tmo, a, st);
}

}  // namespace xf
