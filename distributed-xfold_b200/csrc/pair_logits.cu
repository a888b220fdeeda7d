// LayerNorm of the pair representation followed by a projection to H heads, written as the attention kernel's pair-bias
// operand (FP16 values times log2 e, [head][query][key], pitch pad8(N)): all pair logits of the diffusion transformer
// (24 blocks x 16 heads) in one launch.
//
// 128 x 2 bytes come in and 2 H leave per token; nothing else has to move: 157 us of HBM at N = 1000, H = 384, and the products
// (1500 clocks per tile of 128 keys and 128 heads) are 0.13 ms.  Neither is the bound: without its stores the kernel takes 237
// us, 2800 clocks per tile, the chain of a set of warps (statistics, barrier, wait for the product, conversion), and the stores
// come on top.  301 us at 1965 MHz, the first hundred calls from a cool GPU, and 353 at the 1500 MHz that calls in a row settle at
// under the power limit.  (One fp32 plane set per super-block, computed on the CUDA cores, and a conversion pass over it took
// 8.5 ms.)
//
// The product runs on the RAW rows, which are bf16 and therefore exact tensor-core operands, and keeps float32's precision
// in the weights by splitting them:
//     w'[h][c] = w[h][c] * gamma[c] - their mean over c = w0 + w1 + w2      (three bf16 numbers: 24 significant bits)
//     D[h][tok] = sum_c w'[h][c] * x[tok][c]                                (three products into one accumulator)
//     logit = rstd * D + colbias[h],  colbias[h] = sum_c beta[c] w[h][c]
// (w' adds up to zero over c, so the mean of the row falls out of the product.)
//
// The accumulator has heads as its rows and keys as its columns: a thread holds keys of one head as they follow one another
// in memory, so a pair of logits is one packed FMA with the keys' scales (broadcast from shared memory), one conversion and
// the clamp, and eight leave as one 16-byte piece for TMA.  (With keys as rows, neighbouring lanes had to trade halves for
// 4-byte stores, and every pair of logits read two pairs of column sums: the shared-memory pipe was 61 % busy, the issue
// slots 50 %; 350 us at N = 1000, H = 384, cool, now 301.)
//
// A CTA keeps the split weights of up to 128 heads in shared memory (96 KB) and walks over tiles of 128 keys of one query
// row; with more heads the CTAs divide into groups that read the same tiles at about the same time, so that all but the
// first read come from L2.  Warp 0 fetches tiles (two in flight), warp 1 issues the products into two accumulators, and two
// sets of eight warps take the tiles in turn: row statistics from the shared-memory tile while the product runs (two threads
// per row), then 32 heads x 64 keys per warp, staged and stored by itself.
//
// FEW: up to 96 heads in all.  The tensor core has no narrower rows than 128, so that form makes, converts and stages 128
// heads whatever their number; here keys are the rows and the product is as wide as the heads, stores are 4 bytes from traded
// halves, and in place of the staging tiles a third tile of x is in flight.  The same operands and sums, the same bits.
// N = 1000: 16 heads 54 us (heads as rows: 87), 64 heads 78 (93), 96 heads 98 (102), 112 heads 107 (106); N = 300: 96 heads
// 18.5 (20.7), 112 heads 19.8 (21.2); N = 40: 16 heads 4.6 (8.9).
#include <cuda_fp16.h>

#include "internal.h"
#include "stages.h"
#include "umma.cuh"

namespace xf {

constexpr int PL_G = 128;      // heads per CTA at most
constexpr int PL_FEW = 96;     // up to so many heads in all: keys as the accumulator's rows (at 112 and 1000 tokens the other form is ahead)
constexpr int PL_XS = 2;       // tiles of x in flight
constexpr uint32_t PL_TILE = 32768;
constexpr uint32_t PL_STG = 4096;                                // a warp's [32 heads][64 keys], swizzled
constexpr uint32_t PL_OFF_W = 0;                                 // [3 pieces][2 halves][128 heads][128 B], swizzled
constexpr uint32_t PL_OFF_X = 3 * 2 * PL_G * 128;
constexpr uint32_t PL_OFF_STG = PL_OFF_X + PL_XS * PL_TILE;      // [16 warps]
constexpr uint32_t PL_OFF_RL = PL_OFF_STG + 16 * PL_STG;         // [2 sets][2 tiles] float[128]: scales of the keys
constexpr uint32_t PL_OFF_CB = PL_OFF_RL + 2 * 2 * 512;          // float[128] colbias * log2 e
constexpr uint32_t PL_OFF_BAR = PL_OFF_CB + PL_G * 4;
constexpr uint32_t PL_SMEM = PL_OFF_BAR + 128;
constexpr int PL_THREADS = 64 + 512;
static_assert(PL_SMEM <= 232448, "shared memory");

struct PairLogitsArgs {
  const float *gamma, *beta, *w;
  __half* out;
  int N, H, tiles_k, groups;
  int* status;
};

template <bool FEW>
__global__ void __launch_bounds__(PL_THREADS, 1)
pair_logits_kernel(const __grid_constant__ CUtensorMap tmx, const __grid_constant__ CUtensorMap tmo, const PairLogitsArgs p) {
  constexpr float LOG2E = 1.4426950408889634f;
  constexpr int XS = FEW ? 3 : PL_XS;  // FEW: no staging, its third tile is there
  extern __shared__ __align__(1024) uint8_t smem[];  // (no room to round up)
  uint8_t* sW = smem + PL_OFF_W;
  float* cb = reinterpret_cast<float*>(smem + PL_OFF_CB);
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + PL_OFF_BAR);
  uint64_t* empty = full + XS;
  uint64_t* tfull = empty + XS;
  uint64_t* tempty = tfull + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tempty + 2);
  volatile int* cta_abort = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int warp = int(__reduce_max_sync(0xffffffffu, threadIdx.x >> 5)), lane = threadIdx.x & 31;
  const AbortCtx ab{cta_abort, p.status};

  if (threadIdx.x == 0) {
    for (int s = 0; s < XS; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 9);  // the products' commit and the eight statistics warps
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(&tfull[s], 1);
      mbar_init(&tempty[s], 8);
    }
    *cta_abort = 0;
    fence_barrier_init();
    tma_prefetch_desc(&tmx);
    if (!FEW) tma_prefetch_desc(&tmo);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 256);
    tmem_relinquish();
  }
  pdl_wait();
  const int group = blockIdx.x % p.groups, h0 = group * PL_G;
  const int ng = p.H - h0 < PL_G ? p.H - h0 : PL_G;  // heads of this CTA (a multiple of 16)
  // split weights, one head per half-warp pass; 16 lanes x 8 channels
  {
    const int half = lane >> 4, l16 = lane & 15;
    for (int h = warp * 2 + half; h < (FEW ? ng : PL_G); h += 2 * (PL_THREADS / 32)) {
      float s = 0.f, b = 0.f, r[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const int c = l16 * 8 + e;
        const float w = h < ng ? p.w[(long long)(h0 + h) * 128 + c] : 0.f;
        r[e] = w * (p.gamma ? p.gamma[c] : 1.f);
        s += r[e];
        b += (p.beta ? p.beta[c] : 0.f) * w;
      }
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) {
        s += __shfl_xor_sync(0xffffffffu, s, o);
        b += __shfl_xor_sync(0xffffffffu, b, o);
      }
      uint32_t pk[3][4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        float r0 = r[2 * e] - s * (1.f / 128), r1 = r[2 * e + 1] - s * (1.f / 128);
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          pk[k][e] = pack_bf16x2(r0, r1);
          r0 -= bf16_lo(pk[k][e]);
          r1 -= bf16_hi(pk[k][e]);
        }
      }
#pragma unroll
      for (int k = 0; k < 3; ++k)
        *reinterpret_cast<uint4*>(sW + (k * 2 + (l16 >> 3)) * (PL_G * 128) + h * 128 + ((uint32_t(l16 & 7) ^ uint32_t(h & 7)) << 4)) =
            make_uint4(pk[k][0], pk[k][1], pk[k][2], pk[k][3]);
      if (l16 == 0) cb[h] = b * LOG2E;
    }
  }
  fence_proxy_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  pdl_launch();
  const uint32_t tmem_base = __reduce_max_sync(0xffffffffu, *tmem_slot), base = smem_u32(smem);
  const long long total = (long long)p.N * p.tiles_k;  // tiles: query row x 128-key block
  const long long t0 = blockIdx.x / p.groups, step = gridDim.x / p.groups;

  if (warp == 0) {
    const uint32_t go = elect_one();  // warp-uniform, like the issuer
    uint32_t stage = 0, phase = 0;
    for (long long t = t0; t < total; t += step) {
      const int q = int(t / p.tiles_k), k0 = int(t % p.tiles_k) * 128;
      if (!mbar_wait_warp(&empty[stage], phase ^ 1u, ab, XF_ERR_WAIT_EMPTY)) break;
      mbar_arrive_expect_tx_if(go, &full[stage], PL_TILE);
      uint8_t* sx = smem + PL_OFF_X + stage * PL_TILE;
      tma_load_3d_if(go, sx, &tmx, &full[stage], 0, k0, q);
      tma_load_3d_if(go, sx + 16384, &tmx, &full[stage], 64, k0, q);
      if (++stage == XS) { stage = 0; phase ^= 1u; }
    }
  } else if (warp == 1) {
    const uint32_t go = elect_one();
    const uint32_t idesc = make_idesc(128, FEW ? ng : 128);
    const uint64_t wd = make_sdesc(base + PL_OFF_W, 16, 1024);
    uint32_t stage = 0, phase = 0, it = 0;
    for (long long t = t0; t < total; t += step, ++it) {
      const uint32_t buf = it & 1u;
      if (!mbar_wait_warp(&tempty[buf], ((it >> 1) & 1u) ^ 1u, ab, XF_ERR_WAIT_TMEM_EMPTY)) break;
      if (!mbar_wait_warp(&full[stage], phase, ab, XF_ERR_WAIT_FULL)) break;
      tc_fence_after();
      const uint32_t d = tmem_base + buf * 128;
      const uint64_t xd = make_sdesc(base + PL_OFF_X + stage * PL_TILE, 16, 1024);
#pragma unroll
      for (int k = 0; k < 3; ++k)
#pragma unroll
        for (int hf = 0; hf < 2; ++hf)
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const uint64_t wt = wd + uint64_t((k * 2 + hf) * (PL_G * 8) + 2 * j), xt = xd + uint64_t(hf * 1024 + 2 * j);
            umma_ss_if(go, d, FEW ? xt : wt, FEW ? wt : xt, idesc, (k | hf | j) ? 1u : 0u);
          }
      umma_commit_if(go, &empty[stage]);
      umma_commit_if(go, &tfull[buf]);
      if (++stage == XS) { stage = 0; phase ^= 1u; }
    }
  } else {
    // two sets of eight warps take the tiles in turn, so that one set's barriers and loads pass behind the other's work
    const uint32_t set = uint32_t(warp - 2) >> 3;
    const int w8 = (warp - 2) & 7, quarter = warp & 3, ch = w8 >> 2;
    const int srow = w8 * 16 + (lane & 15), half = lane >> 4;  // statistics: 16 rows per warp, two threads per row
    const int ldq = (p.N + 7) & ~7;
    const uint32_t go = elect_one();
    uint8_t* stg = smem + PL_OFF_STG + (warp - 2) * PL_STG;
    const float bias = FEW ? 0.f : cb[quarter * 32 + lane];
    const float2 b2 = make_float2(bias, bias);
    const __half2 lim = __float2half2_rn(60000.f);
    uint32_t it = set;
    for (long long t = t0 + set * step; t < total; t += 2 * step, it += 2) {
      const uint32_t stage = it % XS, phase = (it / XS) & 1u;
      const int q = int(t / p.tiles_k), k0 = int(t % p.tiles_k) * 128;
      // (a failed wait does not leave the loop: these warps meet at a named barrier; further waits return at once)
      mbar_wait(&full[stage], phase, ab, XF_ERR_WAIT_FULL);
      uint32_t xr[32];
      load_half_row(smem + PL_OFF_X + stage * PL_TILE, srow, half, xr);
      float nmean, rstd;
      half_row_stats(xr, nmean, rstd);
      // (by tile parity: a warp may be one tile ahead of the readers, not two -- the barrier is in between)
      float* rl = reinterpret_cast<float*>(smem + PL_OFF_RL) + (set * 2 + ((it >> 1) & 1u)) * 128;
      if (half == 0) rl[srow] = rstd * LOG2E;
      // (only now: right behind the loads, not yet used, the arrival could pass them, and the next tile would be read)
      __syncwarp();
      if (lane == 0) mbar_arrive(&empty[stage]);
      named_bar_sync(1 + set, 256);
      mbar_wait(&tfull[set], (it >> 1) & 1u, ab, XF_ERR_WAIT_TMEM_FULL);
      tc_fence_after();
      if constexpr (FEW) {
        // thread = key, 32 heads at a time; neighbouring lanes trade halves, so that the even lane holds two keys of head e and the
        // odd lane two of head e + 1
        const int row = quarter * 32 + lane, k = k0 + (row & ~1);
        const float2 rl2 = make_float2(rl[row], rl[row]);
        const bool kstore = k < ldq;
        const long long plane2 = 2ll * p.N * ldq;
        const uint32_t keep = (k < p.N ? 0xffffu : 0u) | (k + 1 < p.N ? 0xffff0000u : 0u);
        const uint32_t sel = (lane & 1) ? 0x3276u : 0x5410u;  // odd: (other.hi, own.hi), even: (own.lo, other.lo)
#pragma unroll 1
        for (int hb = ch * 32; hb < ng; hb += 64) {
          uint32_t r[32];
          tmem_ld32(tmem_base + set * 128 + hb + (uint32_t(quarter * 32) << 16), r);
          tmem_ld_wait();
          __half* d = p.out + ((long long)(hb + (lane & 1)) * p.N + q) * ldq + k;
#pragma unroll
          for (int e = 0; e < 32; e += 2) {
            if (e == 16 && hb + 16 >= ng) break;  // heads in sixteens
            const float2 v = ffma2(make_float2(__uint_as_float(r[e]), __uint_as_float(r[e + 1])), rl2, *reinterpret_cast<const float2*>(&cb[hb + e]));
            const __half2 h2 = __hmin2(__hmax2(__floats2half2_rn(v.x, v.y), __hneg2(lim)), lim);  // (NaN: -60000)
            const uint32_t own = *reinterpret_cast<const uint32_t*>(&h2), other = __shfl_xor_sync(0xffffffffu, own, 1);
            if (kstore) *reinterpret_cast<uint32_t*>(d) = __byte_perm(own, other, sel) & keep;
            d += plane2;
          }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&tempty[set]);
        continue;
      }
      const int kw = k0 + ch * 64;  // this warp's first key
      const bool edge = kw + 64 > p.N;
      tma_store_wait_read<0>();  // the tile before has left the staging buffer
      __syncwarp();
#pragma unroll 1
      for (int c = 0; c < 2; ++c) {
        uint32_t r[32];
        tmem_ld32(tmem_base + set * 128 + ch * 64 + c * 32 + (uint32_t(quarter * 32) << 16), r);
        tmem_ld_wait();
        if (c == 1) {
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&tempty[set]);
        }
#pragma unroll
        for (int g = 0; g < 4; ++g) {
          const float4 s0 = *reinterpret_cast<const float4*>(rl + ch * 64 + c * 32 + g * 8);
          const float4 s1 = *reinterpret_cast<const float4*>(rl + ch * 64 + c * 32 + g * 8 + 4);
          const float2 sc[4] = {make_float2(s0.x, s0.y), make_float2(s0.z, s0.w), make_float2(s1.x, s1.y), make_float2(s1.z, s1.w)};
          uint32_t o[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const float2 v = ffma2(make_float2(__uint_as_float(r[g * 8 + 2 * e]), __uint_as_float(r[g * 8 + 2 * e + 1])), sc[e], b2);
            const __half2 h2 = __hmin2(__hmax2(__floats2half2_rn(v.x, v.y), __hneg2(lim)), lim);  // (NaN: -60000)
            o[e] = *reinterpret_cast<const uint32_t*>(&h2);
          }
          if (edge) {  // padding of the pitch: zeros
            const int k = kw + c * 32 + g * 8;
#pragma unroll
            for (int e = 0; e < 4; ++e)
              o[e] &= (k + 2 * e < p.N ? 0xffffu : 0u) | (k + 2 * e + 1 < p.N ? 0xffff0000u : 0u);
          }
          *reinterpret_cast<uint4*>(stg + lane * 128 + ((uint32_t(c * 4 + g) ^ uint32_t(lane & 7)) << 4)) = make_uint4(o[0], o[1], o[2], o[3]);
        }
      }
      fence_proxy_async_smem();
      __syncwarp();
      tma_store_3d_if(kw < ldq && quarter * 32 < ng ? go : 0u, &tmo, stg, kw, q, h0 + quarter * 32);
      tma_store_commit();
    }
    if (!FEW) tma_store_wait_all();
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

template <bool FEW>
static int launch_pl(Ctx* c, const CUtensorMap& tmx, const CUtensorMap& tmo, const PairLogitsArgs& a, cudaStream_t st) {
  static bool attr_done[8] = {false};
  if (!attr_done[c->device & 7]) {
    cudaError_t e = cudaFuncSetAttribute(pair_logits_kernel<FEW>, cudaFuncAttributeMaxDynamicSharedMemorySize, PL_SMEM);
    if (e != cudaSuccess) return fail(c, XFOLD_ERR_LAUNCH, "pair logits smem attribute: %s", cudaGetErrorString(e));
    if (!only_dynamic_smem(pair_logits_kernel<FEW>)) return fail(c, XFOLD_ERR_LAUNCH, "pair logits: shared memory does not start at 1 KB");
    attr_done[c->device & 7] = true;
  }
  long long per_group = c->sm_count / a.groups;
  if (per_group < 1) per_group = 1;
  const long long total = (long long)a.N * a.tiles_k;
  if (per_group > total) per_group = total;
  ProfScope ps(c, XFOLD_K_LAYERNORM, st);
  launch_pdl(pair_logits_kernel<FEW>, (int)per_group * a.groups, PL_THREADS, PL_SMEM, st, tmx, tmo, a);
  return check_launch(c, "pair_logits_kernel");
}

static int launch_pair_logits(Ctx* c, const bf16* pair, int N, const float* gamma, const float* beta, const float* w, int H,
                              void* out, cudaStream_t st) {
  if (N <= 0 || H <= 0) return XFOLD_OK;
  if (H & 15) return fail(c, XFOLD_ERR_ARG, "pair logits: the number of heads must be a multiple of 16, got %d", H);
  if (reinterpret_cast<uintptr_t>(out) & 15) return fail(c, XFOLD_ERR_ARG, "pair logits: the result must be 16-byte aligned");
  CUtensorMap tmx, tmo;
  if (!make_tmap_bf16_3d(&tmx, pair, 128, N, N, 128, (uint64_t)128 * N, 64, 128, 1))
    return fail(c, XFOLD_ERR_ARG, "pair logits: cannot encode the tensor map");
  PairLogitsArgs a{gamma, beta, w, reinterpret_cast<__half*>(out), N, H, (N + 127) / 128, (H + PL_G - 1) / PL_G, c->d_status};
  if (H <= PL_FEW) return launch_pl<true>(c, tmx, tmx, a, st);
  // (fp16 as far as the stores go: 16-bit elements)
  const uint64_t ldq = (uint64_t)((N + 7) & ~7);
  if (!make_tmap_bf16_3d(&tmo, out, ldq, N, H, ldq, ldq * N, 64, 1, 32)) return fail(c, XFOLD_ERR_ARG, "pair logits: cannot encode the result's tensor map");
  return launch_pl<false>(c, tmx, tmo, a, st);
}

}  // namespace xf

using namespace xf;

extern "C" int xfold_pair_logits_prepared_fwd(xfold_ctx* cx, const void* pair, int N, const float* ln_gamma, const float* ln_beta,
                                              const float* w, int H, void* prepared, void* stream) {
  Ctx* c = reinterpret_cast<Ctx*>(cx);
  if (!c || !pair || !w || !prepared) return XFOLD_ERR_ARG;
  CallLock call(c);
  return launch_pair_logits(c, (const bf16*)pair, N, ln_gamma, ln_beta, w, H, prepared, (cudaStream_t)stream);
}
