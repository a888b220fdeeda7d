// LayerNorm of the pair representation followed by a projection to H heads, written as the attention kernel's pair-bias
// operand (FP16 values times log2 e, [head][query][key], pitch pad8(N)): all pair logits of the diffusion transformer
// (24 blocks x 16 heads) in one launch.
//
// Bound: HBM.  128 x 2 bytes come in and 2 H leave per token; nothing else has to move.  (One fp32 plane set per
// super-block, computed on the CUDA cores, and a conversion pass over it took 8.5 ms at N = 1000, H = 384; this kernel
// takes 0.40 ms, 2.5 TB/s.)
//
// The product runs on the RAW rows, which are bf16 and therefore exact tensor-core operands, and keeps float32's precision
// in the weights by splitting them:
//     w'[h][c] = w[h][c] * gamma[c] = w0 + w1 + w2      (three bf16 numbers: 24 significant bits)
//     D[tok][h] = sum_c x[tok][c] * w'[h][c]            (three products into one accumulator)
//     logit = rstd * (D - mean * colsum[h]) + colbias[h],  colsum[h] = sum_c w'[h][c],  colbias[h] = sum_c beta[c] w[h][c]
//
// A CTA keeps the split weights of up to 128 heads in shared memory (96 KB) and walks over tiles of 128 keys of one query
// row; with more heads the CTAs divide into groups that read the same tiles at about the same time, so that all but the
// first read come from L2.  Warp 0 fetches tiles (three in flight), warp 1 issues the products into two accumulators, and two
// sets of eight warps take the tiles in turn: row statistics from the shared-memory tile while the product runs, then the
// accumulator (thread = key, so a warp's store of one head is 64 contiguous bytes).  With one set and staged TMA stores the
// kernel took 0.52 ms at N = 1000, H = 384: a tile cost 6100 cycles, nearly all of it waiting.
#include <cuda_fp16.h>

#include "internal.h"
#include "stages.h"
#include "umma.cuh"

namespace xf {

constexpr int PL_G = 128;      // heads per CTA at most
constexpr int PL_XS = 3;       // tiles of x in flight
constexpr uint32_t PL_TILE = 32768;
constexpr uint32_t PL_OFF_W = 0;                                 // [3 pieces][2 halves][128 heads][128 B], swizzled
constexpr uint32_t PL_OFF_X = 3 * 2 * PL_G * 128;
constexpr uint32_t PL_OFF_CS = PL_OFF_X + PL_XS * PL_TILE;       // float[128] colsum, float[128] colbias * log2 e
constexpr uint32_t PL_OFF_PART = PL_OFF_CS + PL_G * 8;           // [2 sets] float[2][2][128]
constexpr uint32_t PL_OFF_BAR = PL_OFF_PART + 2 * 2 * 2 * 128 * 4;
constexpr uint32_t PL_SMEM = PL_OFF_BAR + 256 + 1024;
constexpr int PL_THREADS = 64 + 512;

struct PairLogitsArgs {
  const float *gamma, *beta, *w;
  __half* out;
  int N, H, tiles_k, groups;
  int* status;
};

__global__ void __launch_bounds__(PL_THREADS, 1)
pair_logits_kernel(const __grid_constant__ CUtensorMap tmx, const PairLogitsArgs p) {
  constexpr float LOG2E = 1.4426950408889634f;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw_addr = smem_u32(smem_raw);
  uint8_t* smem = smem_raw + (((raw_addr + 1023u) & ~1023u) - raw_addr);
  uint8_t* sW = smem + PL_OFF_W;
  float* cs = reinterpret_cast<float*>(smem + PL_OFF_CS);
  float* cb = cs + PL_G;
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + PL_OFF_BAR);
  uint64_t* empty = full + PL_XS;
  uint64_t* tfull = empty + PL_XS;
  uint64_t* tempty = tfull + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tempty + 2);
  volatile int* cta_abort = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const AbortCtx ab{cta_abort, p.status};

  if (threadIdx.x == 0) {
    for (int s = 0; s < PL_XS; ++s) {
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
    for (int h = warp * 2 + half; h < PL_G; h += 2 * (PL_THREADS / 32)) {
      float s = 0.f, b = 0.f;
      uint32_t pk[3][4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        float piece[3][2];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const int c = l16 * 8 + e * 2 + u;
          const float w = h < ng ? p.w[(long long)(h0 + h) * 128 + c] : 0.f;
          float r = w * (p.gamma ? p.gamma[c] : 1.f);
          s += r;
          b += (p.beta ? p.beta[c] : 0.f) * w;
#pragma unroll
          for (int k = 0; k < 3; ++k) {
            piece[k][u] = __bfloat162float(__float2bfloat16(r));
            r -= piece[k][u];
          }
        }
#pragma unroll
        for (int k = 0; k < 3; ++k) pk[k][e] = pack_bf16x2(piece[k][0], piece[k][1]);
      }
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) {
        s += __shfl_xor_sync(0xffffffffu, s, o);
        b += __shfl_xor_sync(0xffffffffu, b, o);
      }
#pragma unroll
      for (int k = 0; k < 3; ++k)
        *reinterpret_cast<uint4*>(sW + (k * 2 + (l16 >> 3)) * (PL_G * 128) + h * 128 + ((uint32_t(l16 & 7) ^ uint32_t(h & 7)) << 4)) =
            make_uint4(pk[k][0], pk[k][1], pk[k][2], pk[k][3]);
      if (l16 == 0) {
        cs[h] = s;
        cb[h] = b * LOG2E;
      }
    }
  }
  fence_proxy_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  pdl_launch();
  const uint32_t tmem_base = *tmem_slot;
  const long long total = (long long)p.N * p.tiles_k;  // tiles: query row x 128-key block
  const long long t0 = blockIdx.x / p.groups, step = gridDim.x / p.groups;

  if (warp == 0) {
    if (lane == 0) {
      uint32_t stage = 0, phase = 0;
      for (long long t = t0; t < total; t += step) {
        const int q = int(t / p.tiles_k), k0 = int(t % p.tiles_k) * 128;
        if (!mbar_wait(&empty[stage], phase ^ 1u, ab, XF_ERR_WAIT_EMPTY)) break;
        mbar_arrive_expect_tx(&full[stage], PL_TILE);
        uint8_t* sx = smem + PL_OFF_X + stage * PL_TILE;
        tma_load_3d(sx, &tmx, &full[stage], 0, k0, q);
        tma_load_3d(sx + 16384, &tmx, &full[stage], 64, k0, q);
        if (++stage == PL_XS) { stage = 0; phase ^= 1u; }
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      const uint32_t idesc = make_idesc(128, ng);
      uint32_t stage = 0, phase = 0, it = 0;
      for (long long t = t0; t < total; t += step, ++it) {
        const uint32_t buf = it & 1u;
        if (!mbar_wait(&tempty[buf], ((it >> 1) & 1u) ^ 1u, ab, XF_ERR_WAIT_TMEM_EMPTY)) break;
        if (!mbar_wait(&full[stage], phase, ab, XF_ERR_WAIT_FULL)) break;
        tc_fence_after();
        const uint32_t sx = smem_u32(smem + PL_OFF_X + stage * PL_TILE), d = tmem_base + buf * 128;
#pragma unroll
        for (int k = 0; k < 3; ++k)
#pragma unroll
          for (int hf = 0; hf < 2; ++hf) {
            const uint64_t ad = make_sdesc(sx + hf * 16384, 16, 1024);
            const uint64_t bd = make_sdesc(smem_u32(sW) + (k * 2 + hf) * (PL_G * 128), 16, 1024);
#pragma unroll
            for (int j = 0; j < 4; ++j) umma_ss(d, ad + 2 * j, bd + 2 * j, idesc, (k | hf | j) ? 1u : 0u);
          }
        umma_commit(&empty[stage]);
        umma_commit(&tfull[buf]);
        if (++stage == PL_XS) { stage = 0; phase ^= 1u; }
      }
    }
  } else {
    // two sets of eight warps take the tiles in turn, so that one set's barriers and loads pass behind the other's work
    const int quarter = warp & 3, ch = ((warp - 2) >> 2) & 1;
    const uint32_t set = uint32_t(warp - 2) >> 3;
    const int row = quarter * 32 + lane;
    const uint32_t rsw = uint32_t(row & 7);
    float(*psum)[128] = reinterpret_cast<float(*)[128]>(smem + PL_OFF_PART + set * 2048);
    float(*psq)[128] = psum + 2;
    const int ldq = (p.N + 7) & ~7;
    uint32_t it = set;
    for (long long t = t0 + set * step; t < total; t += 2 * step, it += 2) {
      const uint32_t stage = it % PL_XS, phase = (it / PL_XS) & 1u;
      const int q = int(t / p.tiles_k), k0 = int(t % p.tiles_k) * 128;
      // (a failed wait does not leave the loop: these warps meet at named barriers; further waits return at once)
      mbar_wait(&full[stage], phase, ab, XF_ERR_WAIT_FULL);
      // row statistics: this thread's 64 channels of its row; the partner of the other half adds its own
      uint32_t xr[32];
      const uint8_t* sx = smem + PL_OFF_X + stage * PL_TILE + ch * 16384 + row * 128;
      float s0 = 0.f, s1 = 0.f;
#pragma unroll
      for (int g = 0; g < 8; ++g) {
        const uint4 u = *reinterpret_cast<const uint4*>(sx + ((uint32_t(g) ^ rsw) << 4));
        xr[g * 4] = u.x; xr[g * 4 + 1] = u.y; xr[g * 4 + 2] = u.z; xr[g * 4 + 3] = u.w;
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&empty[stage]);
#pragma unroll
      for (int e = 0; e < 32; ++e)
        asm("{\n\t.reg .b16 lo, hi;\n\tmov.b32 {lo, hi}, %2;\n\tadd.rn.f32.bf16 %0, lo, %0;\n\tadd.rn.f32.bf16 %1, hi, %1;\n\t}"
            : "+f"(s0), "+f"(s1) : "r"(xr[e]));
      psum[ch][row] = s0 + s1;
      named_bar_sync(1 + set, 256);
      const float mean = (psum[0][row] + psum[1][row]) * (1.f / 128), nmean = -mean;
      float q0 = 0.f, q1 = 0.f;
#pragma unroll
      for (int e = 0; e < 32; ++e) {
        float a, b;
        asm("{\n\t.reg .b16 lo, hi;\n\tmov.b32 {lo, hi}, %2;\n\tadd.rn.f32.bf16 %0, lo, %3;\n\tadd.rn.f32.bf16 %1, hi, %3;\n\t}"
            : "=f"(a), "=f"(b) : "r"(xr[e]), "f"(nmean));
        q0 = fmaf(a, a, q0);
        q1 = fmaf(b, b, q1);
      }
      psq[ch][row] = q0 + q1;
      named_bar_sync(1 + set, 256);
      const float rl = rsqrtf((psq[0][row] + psq[1][row]) * (1.f / 128) + 1e-5f) * LOG2E;
      const float nm = -rl * mean;

      mbar_wait(&tfull[set], (it >> 1) & 1u, ab, XF_ERR_WAIT_TMEM_FULL);
      tc_fence_after();
      // Per pair of heads: this lane's key as half2 (head e, head e + 1), then neighbouring lanes trade so that the even lane
      // holds two keys of head e and the odd lane two of head e + 1.  The kernel is bound by instruction issue, hence the
      // packed FMAs and the clamp and the zeroing of padding keys on packed halves.
      const int k = k0 + (row & ~1);
      const bool kstore = k < ldq;
      __half* d = p.out + ((long long)(h0 + ch * 32 + (lane & 1)) * p.N + q) * ldq + k;
      const long long plane2 = 2ll * p.N * ldq;
      const uint32_t keep = (k < p.N ? 0xffffu : 0u) | (k + 1 < p.N ? 0xffff0000u : 0u);
      const uint32_t sel = (lane & 1) ? 0x3276u : 0x5410u;  // odd: (other.hi, own.hi), even: (own.lo, other.lo)
      const __half2 lim = __float2half2_rn(60000.f);
      const float2 rl2 = make_float2(rl, rl), nm2 = make_float2(nm, nm);
#pragma unroll 1
      for (int hb = ch * 32; hb < ng; hb += 64, d += 16 * plane2) {  // (the chunk itself advances d by 16 pairs of heads)
        uint32_t r[32];
        tmem_ld32(tmem_base + set * 128 + hb + (uint32_t(quarter * 32) << 16), r);
        tmem_ld_wait();
#pragma unroll
        for (int e = 0; e < 32; e += 2) {
          if (e == 16 && hb + 16 >= ng) {  // 16 heads in the last chunk
            d += 8 * plane2;
            break;
          }
          const float2 a = *reinterpret_cast<const float2*>(&cs[hb + e]), b = *reinterpret_cast<const float2*>(&cb[hb + e]);
          const float2 v = ffma2(rl2, make_float2(__uint_as_float(r[e]), __uint_as_float(r[e + 1])), ffma2(nm2, a, b));
          const __half2 own2 = __hmin2(__hmax2(__floats2half2_rn(v.x, v.y), __hneg2(lim)), lim);  // (NaN: -60000)
          const uint32_t own = *reinterpret_cast<const uint32_t*>(&own2);
          const uint32_t other = __shfl_xor_sync(0xffffffffu, own, 1);
          if (kstore) *reinterpret_cast<uint32_t*>(d) = __byte_perm(own, other, sel) & keep;
          d += plane2;
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&tempty[set]);
    }
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

static int launch_pair_logits(Ctx* c, const bf16* pair, int N, const float* gamma, const float* beta, const float* w, int H,
                              void* out, cudaStream_t st) {
  if (N <= 0 || H <= 0) return XFOLD_OK;
  if (H & 15) return fail(c, XFOLD_ERR_ARG, "pair logits: the number of heads must be a multiple of 16, got %d", H);
  if (reinterpret_cast<uintptr_t>(out) & 15) return fail(c, XFOLD_ERR_ARG, "pair logits: the result must be 16-byte aligned");
  CUtensorMap tmx;
  if (!make_tmap_bf16_3d(&tmx, pair, 128, N, N, 128, (uint64_t)128 * N, 64, 128, 1))
    return fail(c, XFOLD_ERR_ARG, "pair logits: cannot encode the tensor map");
  PairLogitsArgs a{gamma, beta, w, reinterpret_cast<__half*>(out), N, H, (N + 127) / 128, (H + PL_G - 1) / PL_G, c->d_status};
  static bool attr_done[8] = {false};
  if (!attr_done[c->device & 7]) {
    cudaError_t e = cudaFuncSetAttribute(pair_logits_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, PL_SMEM);
    if (e != cudaSuccess) return fail(c, XFOLD_ERR_LAUNCH, "pair logits smem attribute: %s", cudaGetErrorString(e));
    attr_done[c->device & 7] = true;
  }
  long long per_group = c->sm_count / a.groups;
  if (per_group < 1) per_group = 1;
  const long long total = (long long)N * a.tiles_k;
  if (per_group > total) per_group = total;
  ProfScope ps(c, XFOLD_K_LAYERNORM, st);
  launch_pdl(pair_logits_kernel, (int)per_group * a.groups, PL_THREADS, PL_SMEM, st, tmx, a);
  return check_launch(c, "pair_logits_kernel");
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
