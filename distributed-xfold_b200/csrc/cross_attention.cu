// Gated cross attention with a per-batch-entry bias: the core of the atom cross-attention encoder / decoder
// (`_alpha_attention::batch_diffusion_cross_attention_forward`, csrc/Alpha_Attention.cpp:127-146, 201-204; spec class
// kernel_test/batch_diffusion_cross_attention.py:23-87).  Queries come from one token set (S per batch entry, 32 atoms
// in the model), keys and values from another (K, 128 atoms), and every batch entry has its own [H][S][K] bias.
//
// The four projections run on the tcgen05 GEMM (query bias and D^-0.5 in its epilogue).  What is left is bandwidth: per
// batch entry [H][S][K] float32 biases are read once (at model size 64 KB, next to 80 KB of projections) for 2 MFLOP.
// One CTA takes 32 queries x 4 heads of a batch entry: eight warps, one per head and 16 queries.  Keys and values of the
// entry come through shared memory, 128 at a time; the products are warp-level mma.sync tiles (16 queries are too few rows
// for a tcgen05 tile), the bias is loaded straight into the accumulator fragments, and the softmax stays in registers.
// The probabilities keep float32's precision in P V: three bf16 pieces, three products.
// (One warp per query with lanes over keys, every key row read again for every query: 180 us for 257 windows; this: 15 us.)
#include "internal.h"
#include "stages.h"
#include "umma.cuh"

namespace xf {

struct XAttnArgs {
  const bf16* qg;   // [B][S][2*H*D]: scaled queries | gate pre-activations
  const bf16* kv;   // [B][K][2*H*D]: keys | values
  const float* bias;  // [B][H][S][K]
  bf16* out;        // [B][S][H*D]
  int B, S, K, H;
};

__device__ __forceinline__ void ldsm4(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldsm4_t(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
// c[16 x 8] += a[16 x 16] * b[16 x 8], bf16 operands, float32 accumulator
__device__ __forceinline__ void mma16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

constexpr int XA_KC = 128;  // keys per pass

// Shared memory: [K | V][4 heads][128 keys][D], 16-byte chunks of a row swizzled so that ldmatrix's eight rows hit
// eight different 16-byte bank groups.
// PAIRS: an even number of keys, a bias whose rows therefore start at multiples of 8 bytes and a result at a multiple of 4:
// two elements at a time.  Anything else goes one by one.  (As a branch inside: 27.8 us for 257 windows instead of 27.5.)
template <int D, bool PAIRS>
__global__ void __launch_bounds__(256, D == 64 ? 1 : 2) xattn_kernel(XAttnArgs p) {
  constexpr int CPR = D / 8;                      // 16-byte chunks per row
  constexpr int RPL = 8 / CPR;                    // rows per 128 bytes
  constexpr uint32_t HEAD_BYTES = XA_KC * D * 2;
  constexpr float LOG2E = 1.4426950408889634f;
  extern __shared__ __align__(128) uint8_t xa_smem[];
  const uint32_t sk = smem_u32(xa_smem), sv = sk + 4 * HEAD_BYTES;
  auto swz = [](int row, int chunk) { return uint32_t(row * D * 2 + ((chunk ^ ((row / RPL) & (CPR - 1))) << 4)); };
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int W = p.H * D, HG = (p.H + 3) / 4, QG = (p.S + 31) / 32;
  const long long total = (long long)p.B * HG * QG;
  pdl_wait();
  pdl_launch();
  for (long long wi = blockIdx.x; wi < total; wi += gridDim.x) {
    const int qg = int(wi % QG), hg = int((wi / QG) % HG), b = int(wi / ((long long)QG * HG));
    const int h = hg * 4 + (warp & 3), q0 = qg * 32 + (warp >> 2) * 16;
    const bool active = h < p.H && q0 < p.S;
    const int r0 = q0 + (lane >> 2), r1 = r0 + 8, cl = (lane & 3) * 2;
    // queries as A fragments (rows beyond S read row 0 and are not stored)
    uint32_t qa[D / 16][4];
    const bf16* q_r0 = p.qg + ((long long)b * p.S + (r0 < p.S ? r0 : 0)) * 2 * W + h * D;
    const bf16* q_r1 = p.qg + ((long long)b * p.S + (r1 < p.S ? r1 : 0)) * 2 * W + h * D;
    if (active) {
#pragma unroll
      for (int k = 0; k < D / 16; ++k) {
        qa[k][0] = *reinterpret_cast<const uint32_t*>(q_r0 + k * 16 + cl);
        qa[k][1] = *reinterpret_cast<const uint32_t*>(q_r1 + k * 16 + cl);
        qa[k][2] = *reinterpret_cast<const uint32_t*>(q_r0 + k * 16 + cl + 8);
        qa[k][3] = *reinterpret_cast<const uint32_t*>(q_r1 + k * 16 + cl + 8);
      }
    }
    const float* b_r0 = p.bias + (((long long)b * p.H + h) * p.S + (r0 < p.S ? r0 : 0)) * p.K;
    const float* b_r1 = p.bias + (((long long)b * p.H + h) * p.S + (r1 < p.S ? r1 : 0)) * p.K;
    float m0 = -INFINITY, m1 = -INFINITY, l0 = 0.f, l1 = 0.f, o[D / 8][4];
#pragma unroll
    for (int d = 0; d < D / 8; ++d)
#pragma unroll
      for (int e = 0; e < 4; ++e) o[d][e] = 0.f;
    for (int k0 = 0; k0 < p.K; k0 += XA_KC) {
      // this pass's keys and values on their way to shared memory
      if (k0 || wi != blockIdx.x) __syncthreads();  // everybody is done with the previous pass's
      for (int i = threadIdx.x; i < XA_KC * 4 * CPR * 2; i += 256) {
        const int chunk = i % CPR, hh = (i / CPR) & 3, isv = (i / (CPR * 4)) & 1, key = i / (CPR * 8);
        const uint32_t dst = (isv ? sv : sk) + hh * HEAD_BYTES + swz(key, chunk);
        if (k0 + key < p.K && hg * 4 + hh < p.H)
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst),
                       "l"(p.kv + ((long long)b * p.K + k0 + key) * 2 * W + isv * W + (hg * 4 + hh) * D + chunk * 8) : "memory");
        else
          asm volatile("st.shared.v4.b32 [%0], {%1, %1, %1, %1};" ::"r"(dst), "r"(0) : "memory");
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
      // meanwhile the bias, into the accumulators of the logits
      float s[16][4];
      if (active) {
#pragma unroll
        for (int t = 0; t < 16; ++t) {
          const int k = k0 + t * 8 + cl;
          if constexpr (PAIRS) {
            const float2 none = make_float2(-INFINITY, -INFINITY);
            const float2 u = k < p.K ? *reinterpret_cast<const float2*>(b_r0 + k) : none;
            const float2 v = k < p.K ? *reinterpret_cast<const float2*>(b_r1 + k) : none;
            s[t][0] = u.x; s[t][1] = u.y; s[t][2] = v.x; s[t][3] = v.y;
          } else {
            s[t][0] = k < p.K ? b_r0[k] : -INFINITY;
            s[t][1] = k + 1 < p.K ? b_r0[k + 1] : -INFINITY;
            s[t][2] = k < p.K ? b_r1[k] : -INFINITY;
            s[t][3] = k + 1 < p.K ? b_r1[k + 1] : -INFINITY;
          }
        }
      }
      asm volatile("cp.async.wait_group 0;" ::: "memory");
      __syncthreads();
      if (!active) continue;
      const uint32_t kh = sk + (warp & 3) * HEAD_BYTES, vh = sv + (warp & 3) * HEAD_BYTES;
      // logits: 16 key tiles of 8; one ldmatrix.x4 brings two key tiles x 16 head-dimension columns
#pragma unroll
      for (int t = 0; t < 16; t += 2)
#pragma unroll
        for (int k = 0; k < D / 16; ++k) {
          uint32_t bk[4];
          ldsm4(kh + swz(t * 8 + (lane & 7) + ((lane >> 4) << 3), k * 2 + ((lane >> 3) & 1)), bk);
          mma16816(s[t], qa[k], bk[0], bk[1]);
          mma16816(s[t + 1], qa[k], bk[2], bk[3]);
        }
      float c0 = m0, c1 = m1;
#pragma unroll
      for (int t = 0; t < 16; ++t) {
        c0 = fmaxf(c0, fmaxf(s[t][0], s[t][1]));
        c1 = fmaxf(c1, fmaxf(s[t][2], s[t][3]));
      }
#pragma unroll
      for (int x = 1; x < 4; x <<= 1) {
        c0 = fmaxf(c0, __shfl_xor_sync(0xffffffffu, c0, x));
        c1 = fmaxf(c1, __shfl_xor_sync(0xffffffffu, c1, x));
      }
      const float f0 = __expf(m0 - c0), f1 = __expf(m1 - c1);
      m0 = c0;
      m1 = c1;
      l0 *= f0;
      l1 *= f1;
#pragma unroll
      for (int d = 0; d < D / 8; ++d) {
        o[d][0] *= f0; o[d][1] *= f0; o[d][2] *= f1; o[d][3] *= f1;
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) {  // 16 keys: exponentials, three bf16 pieces, products
        uint32_t pa[3][4];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const int t = 2 * j + u;
          float e0 = exp2f((s[t][0] - m0) * LOG2E), e1 = exp2f((s[t][1] - m0) * LOG2E);
          float e2 = exp2f((s[t][2] - m1) * LOG2E), e3 = exp2f((s[t][3] - m1) * LOG2E);
          l0 += e0 + e1;
          l1 += e2 + e3;
#pragma unroll
          for (int piece = 0; piece < 3; ++piece) {
            const uint32_t x0 = pack_bf16x2(e0, e1), x1 = pack_bf16x2(e2, e3);
            pa[piece][u * 2] = x0;
            pa[piece][u * 2 + 1] = x1;
            e0 -= bf16_lo(x0); e1 -= bf16_hi(x0);
            e2 -= bf16_lo(x1); e3 -= bf16_hi(x1);
          }
        }
#pragma unroll
        for (int d = 0; d < D / 8; d += 2) {
          uint32_t bv[4];
          ldsm4_t(vh + swz(j * 16 + (lane & 15), d + (lane >> 4)), bv);
#pragma unroll
          for (int piece = 0; piece < 3; ++piece) {
            mma16816(o[d], pa[piece], bv[0], bv[1]);
            mma16816(o[d + 1], pa[piece], bv[2], bv[3]);
          }
        }
      }
    }
    if (!active) continue;
#pragma unroll
    for (int x = 1; x < 4; x <<= 1) {
      l0 += __shfl_xor_sync(0xffffffffu, l0, x);
      l1 += __shfl_xor_sync(0xffffffffu, l1, x);
    }
    const float i0 = 1.f / l0, i1 = 1.f / l1;
    bf16* o_r0 = p.out + ((long long)b * p.S + r0) * W + h * D;
    bf16* o_r1 = p.out + ((long long)b * p.S + r1) * W + h * D;
    auto store = [](bf16* dst, uint32_t v) {
      if constexpr (PAIRS) {
        *reinterpret_cast<uint32_t*>(dst) = v;
      } else {
        dst[0] = __ushort_as_bfloat16((unsigned short)(v & 0xFFFFu));
        dst[1] = __ushort_as_bfloat16((unsigned short)(v >> 16));
      }
    };
#pragma unroll
    for (int d = 0; d < D / 8; ++d) {
      const uint32_t g0 = *reinterpret_cast<const uint32_t*>(q_r0 + W + d * 8 + cl);
      const uint32_t g1 = *reinterpret_cast<const uint32_t*>(q_r1 + W + d * 8 + cl);
      if (r0 < p.S)
        store(o_r0 + d * 8 + cl,
              pack_bf16x2(o[d][0] * i0 * sigmoidf_fast(bf16_lo(g0)), o[d][1] * i0 * sigmoidf_fast(bf16_hi(g0))));
      if (r1 < p.S)
        store(o_r1 + d * 8 + cl,
              pack_bf16x2(o[d][2] * i1 * sigmoidf_fast(bf16_lo(g1)), o[d][3] * i1 * sigmoidf_fast(bf16_hi(g1))));
    }
  }
}

template <int D, bool PAIRS>
static int launch_xattn(Ctx* c, const XAttnArgs& a, cudaStream_t st) {
  constexpr size_t smem = 2 * 4 * XA_KC * D * 2;
  static bool attr_done[8] = {false};
  if (!attr_done[c->device & 7]) {
    cudaError_t e = cudaFuncSetAttribute(xattn_kernel<D, PAIRS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return fail(c, XFOLD_ERR_LAUNCH, "cross attention smem attribute: %s", cudaGetErrorString(e));
    attr_done[c->device & 7] = true;
  }
  const long long total = (long long)a.B * ((a.H + 3) / 4) * ((a.S + 31) / 32);
  const long long cap = (long long)c->sm_count * (D == 64 ? 1 : 2);
  ProfScope ps(c, XFOLD_K_APB_ATTENTION, st);
  launch_pdl(xattn_kernel<D, PAIRS>, (int)(total < cap ? total : cap), 256, smem, st, a);
  return check_launch(c, "xattn_kernel");
}

// ---------------------------------------------------------------------------------------------------------------
// The model's own windows (four heads of 32, 128 channels, up to 32 queries and 128 keys) in one kernel: projections and
// attention of a window by two CTAs, one for each pair of heads, two CTAs per SM.  No scratch.
// Bound: latency.  A window brings 104 KB (64 of them bias) for 0.013 GFLOP; what counts is the chain of trips -- as two
// projection launches and xattn_kernel, with queries, keys and values through memory, 257 windows took 27.6 us.
// The projections come out transposed (D = W x^T, lane = channel), so that the 32 queries are the tile's narrow side, the
// query bias and scale are one number per thread, and a thread's row of keys leaves in 16-byte pieces:
//   warp 4     : TMA and tcgen05.mma -- weights once, [q | gate] and [k | v] rows of the pair of heads; then per window
//                [128 x 32 queries] and [128 x 128 keys]
//   warps 0-3  : tensor memory -> bf16 [channel][token] over the window's inputs, then one head and 16 queries per warp as
//                in xattn_kernel, from the same roundings in the same order (the same bits).  The bias is on its way while
//                the rest is prepared.
// 257 windows, back to back: 13.8 us (one call at a time from an idle GPU, host included: 44 -> 32).
constexpr uint32_t XW_OFF_W = 0, XW_OFF_M = 65536, XW_OFF_Q = XW_OFF_M + 32768, XW_OFF_BAR = XW_OFF_Q + 8192,
                   XW_SMEM = XW_OFF_BAR + 64 + 1024;
constexpr int XW_THREADS = 160;

struct XWinArgs {
  const float *qg_bias, *qg_scale, *bias;
  bf16* out;
  int B, S, K;
  int* status;
};

__global__ void __launch_bounds__(XW_THREADS, 2)
xwin_kernel(const __grid_constant__ CUtensorMap tmq, const __grid_constant__ CUtensorMap tmm,
            const __grid_constant__ CUtensorMap tmwq, const __grid_constant__ CUtensorMap tmwk, const XWinArgs p) {
  constexpr float LOG2E = 1.4426950408889634f;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw_addr = smem_u32(smem_raw);
  uint8_t* smem = smem_raw + (((raw_addr + 1023u) & ~1023u) - raw_addr);
  uint64_t* w_full = reinterpret_cast<uint64_t*>(smem + XW_OFF_BAR);
  uint64_t* x_full = w_full + 1;   // the window's inputs have landed
  uint64_t* x_empty = x_full + 1;  // the attention has read what replaced them
  uint64_t* t_full = x_empty + 1;  // projections complete
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(t_full + 1);
  volatile int* cta_abort = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int warp = int(__reduce_max_sync(0xffffffffu, threadIdx.x >> 5)), lane = threadIdx.x & 31;
  const AbortCtx ab{cta_abort, p.status};
  if (threadIdx.x == 0) {
    mbar_init(w_full, 1);
    mbar_init(x_full, 1);
    mbar_init(x_empty, 4);
    mbar_init(t_full, 1);
    *cta_abort = 0;
    fence_barrier_init();
    tma_prefetch_desc(&tmq);
    tma_prefetch_desc(&tmm);
    tma_prefetch_desc(&tmwq);
    tma_prefetch_desc(&tmwk);
  }
  if (warp == 4) {
    tmem_alloc(tmem_slot, 256);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = __reduce_max_sync(0xffffffffu, *tmem_slot);  // [k | v]: 128 columns, [q | gate]: 32
  const uint32_t base = smem_u32(smem);
  const int hp = int(blockIdx.x) & 1, b0 = int(blockIdx.x) >> 1, step = int(gridDim.x) >> 1;
  pdl_wait();
  pdl_launch();

  if (warp == 4) {
    const uint32_t go = elect_one();
    auto load_x = [&](int b) {
      mbar_arrive_expect_tx_if(go, x_full, 32768 + 8192);
#pragma unroll
      for (int kh = 0; kh < 2; ++kh) {
        tma_load_3d_if(go, smem + XW_OFF_M + kh * 16384, &tmm, x_full, kh * 64, 0, b);
        tma_load_3d_if(go, smem + XW_OFF_Q + kh * 4096, &tmq, x_full, kh * 64, 0, b);
      }
    };
    if (b0 < p.B) load_x(b0);
    mbar_arrive_expect_tx_if(go, w_full, 65536);
#pragma unroll
    for (int kh = 0; kh < 2; ++kh)
#pragma unroll
      for (int part = 0; part < 2; ++part) {  // rows of the pair's q or k, then of its gate or v
        tma_load_3d_if(go, smem + XW_OFF_W + kh * 16384 + part * 8192, &tmwk, w_full, kh * 64, part * 128 + hp * 64, 0);
        tma_load_3d_if(go, smem + XW_OFF_W + 32768 + kh * 16384 + part * 8192, &tmwq, w_full, kh * 64, part * 128 + hp * 64, 0);
      }
    bool okay = mbar_wait_warp(w_full, 0, ab, XF_ERR_WAIT_FULL);
    uint32_t ph = 0;
    for (int b = b0; b < p.B && okay; b += step, ph ^= 1u) {
      if (!mbar_wait_warp(x_full, ph, ab, XF_ERR_WAIT_FULL)) break;
      tc_fence_after();
      const uint64_t md = make_sdesc(base + XW_OFF_M, 16, 1024), qd = make_sdesc(base + XW_OFF_Q, 16, 1024);
      const uint64_t wk = make_sdesc(base + XW_OFF_W, 16, 1024), wq = make_sdesc(base + XW_OFF_W + 32768, 16, 1024);
#pragma unroll
      for (int kh = 0; kh < 2; ++kh)
#pragma unroll
        for (int j = 0; j < 4; ++j)
          umma_ss_if(go, tmem_base, wk + uint64_t(kh * 1024 + 2 * j), md + uint64_t(kh * 1024 + 2 * j), make_idesc(128, 128), (kh | j) ? 1u : 0u);
#pragma unroll
      for (int kh = 0; kh < 2; ++kh)
#pragma unroll
        for (int j = 0; j < 4; ++j)
          umma_ss_if(go, tmem_base + 128, wq + uint64_t(kh * 1024 + 2 * j), qd + uint64_t(kh * 256 + 2 * j), make_idesc(128, 32), (kh | j) ? 1u : 0u);
      umma_commit_if(go, t_full);
      // (the next window overwrites what the attention reads, and its products the accumulators)
      if (!mbar_wait_warp(x_empty, ph, ab, XF_ERR_WAIT_EMPTY)) break;
      if (b + step < p.B) load_x(b + step);
    }
  } else {
    const int row = warp * 32 + lane;                       // channel: q | gate, or k | v, of the pair of heads
    const int col = (row >> 6) * 128 + hp * 64 + (row & 63);  // its row of w_qg
    const float qb = p.qg_bias ? p.qg_bias[col] : 0.f, qs = p.qg_scale ? p.qg_scale[col] : 1.f;
    const int hh = warp & 1, h = hp * 2 + hh, q0 = (warp >> 1) * 16;
    const int r0 = q0 + (lane >> 2), r1 = r0 + 8, cl = (lane & 3) * 2;
    const uint32_t laddr = tmem_base + (uint32_t(warp * 32) << 16);
    uint8_t* skv = smem + XW_OFF_M + row * 256;   // [128 channels][128 keys], 16-byte chunks swizzled over 8 rows
    uint8_t* sqg = smem + XW_OFF_Q + row * 64;    // [128 channels][32 queries]
    const uint32_t rsw = uint32_t(row & 7), rsw4 = uint32_t(row >> 1) & 3u;
    auto kv_at = [&](int ch, int chunk) { return base + XW_OFF_M + uint32_t(ch * 256 + ((chunk ^ (ch & 7)) << 4)); };
    auto qg_at = [&](int ch, int chunk) { return base + XW_OFF_Q + uint32_t(ch * 64 + ((chunk ^ ((ch >> 1) & 3)) << 4)); };
    const bool active = q0 < p.S;
    uint32_t ph = 0;
    for (int b = b0; b < p.B; b += step, ph ^= 1u) {
      const float* b_r0 = p.bias + (((long long)b * 4 + h) * p.S + (r0 < p.S ? r0 : 0)) * p.K;
      const float* b_r1 = p.bias + (((long long)b * 4 + h) * p.S + (r1 < p.S ? r1 : 0)) * p.K;
      float s[16][4];
      if (active) {
#pragma unroll
        for (int t = 0; t < 16; ++t) {
          const int k = t * 8 + cl;
          const float2 none = make_float2(-INFINITY, -INFINITY);
          const float2 u = k < p.K ? *reinterpret_cast<const float2*>(b_r0 + k) : none;
          const float2 v = k < p.K ? *reinterpret_cast<const float2*>(b_r1 + k) : none;
          s[t][0] = u.x; s[t][1] = u.y; s[t][2] = v.x; s[t][3] = v.y;
        }
      }
      mbar_wait_warp(t_full, ph, ab, XF_ERR_WAIT_TMEM_FULL);  // (a failed wait runs through: these warps meet at a barrier)
      tc_fence_after();
      {
        uint32_t r[32];
        tmem_ld32(laddr + 128, r);
        tmem_ld_wait();
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          uint32_t o[4];
#pragma unroll
          for (int e = 0; e < 4; ++e)
            o[e] = pack_bf16x2((__uint_as_float(r[c * 8 + 2 * e]) + qb) * qs, (__uint_as_float(r[c * 8 + 2 * e + 1]) + qb) * qs);
          *reinterpret_cast<uint4*>(sqg + ((uint32_t(c) ^ rsw4) << 4)) = make_uint4(o[0], o[1], o[2], o[3]);
        }
#pragma unroll 1
        for (int g = 0; g < 4; ++g) {
          tmem_ld32(laddr + g * 32, r);
          tmem_ld_wait();
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            uint32_t o[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) o[e] = pack_bf16x2(__uint_as_float(r[c * 8 + 2 * e]), __uint_as_float(r[c * 8 + 2 * e + 1]));
            *reinterpret_cast<uint4*>(skv + ((uint32_t(g * 4 + c) ^ rsw) << 4)) = make_uint4(o[0], o[1], o[2], o[3]);
          }
        }
      }
      tc_fence_before();
      named_bar_sync(1, 128);
      if (active) {
        uint32_t qa[2][4], gg[2][4];  // A fragments of the queries; gates of (r0, r1) x pairs of channels, two groups of 8 each
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          const int d = hh * 32 + k * 16 + (lane & 7);
          ldsm4_t(qg_at(d + ((lane >> 4) << 3), (q0 >> 3) + ((lane >> 3) & 1)), qa[k]);
          ldsm4_t(qg_at(64 + d + ((lane >> 4) << 3), (q0 >> 3) + ((lane >> 3) & 1)), gg[k]);
        }
#pragma unroll
        for (int t = 0; t < 16; t += 2)
#pragma unroll
          for (int k = 0; k < 2; ++k) {
            uint32_t bk[4];
            ldsm4_t(kv_at(hh * 32 + k * 16 + (((lane >> 3) & 1) << 3) + (lane & 7), t + (lane >> 4)), bk);
            mma16816(s[t], qa[k], bk[0], bk[1]);
            mma16816(s[t + 1], qa[k], bk[2], bk[3]);
          }
        float c0 = -INFINITY, c1 = -INFINITY, l0 = 0.f, l1 = 0.f, o[4][4];
#pragma unroll
        for (int d = 0; d < 4; ++d)
#pragma unroll
          for (int e = 0; e < 4; ++e) o[d][e] = 0.f;
#pragma unroll
        for (int t = 0; t < 16; ++t) {
          c0 = fmaxf(c0, fmaxf(s[t][0], s[t][1]));
          c1 = fmaxf(c1, fmaxf(s[t][2], s[t][3]));
        }
#pragma unroll
        for (int x = 1; x < 4; x <<= 1) {
          c0 = fmaxf(c0, __shfl_xor_sync(0xffffffffu, c0, x));
          c1 = fmaxf(c1, __shfl_xor_sync(0xffffffffu, c1, x));
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) {  // 16 keys: exponentials, three bf16 pieces, products
          uint32_t pa[3][4];
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            const int t = 2 * j + u;
            float e0 = exp2f((s[t][0] - c0) * LOG2E), e1 = exp2f((s[t][1] - c0) * LOG2E);
            float e2 = exp2f((s[t][2] - c1) * LOG2E), e3 = exp2f((s[t][3] - c1) * LOG2E);
            l0 += e0 + e1;
            l1 += e2 + e3;
#pragma unroll
            for (int piece = 0; piece < 3; ++piece) {
              const uint32_t x0 = pack_bf16x2(e0, e1), x1 = pack_bf16x2(e2, e3);
              pa[piece][u * 2] = x0;
              pa[piece][u * 2 + 1] = x1;
              e0 -= bf16_lo(x0); e1 -= bf16_hi(x0);
              e2 -= bf16_lo(x1); e3 -= bf16_hi(x1);
            }
          }
#pragma unroll
          for (int d = 0; d < 4; d += 2) {
            uint32_t bv[4];
            ldsm4(kv_at(64 + hh * 32 + d * 8 + ((lane >> 4) << 3) + (lane & 7), j * 2 + ((lane >> 3) & 1)), bv);
#pragma unroll
            for (int piece = 0; piece < 3; ++piece) {
              mma16816(o[d], pa[piece], bv[0], bv[1]);
              mma16816(o[d + 1], pa[piece], bv[2], bv[3]);
            }
          }
        }
#pragma unroll
        for (int x = 1; x < 4; x <<= 1) {
          l0 += __shfl_xor_sync(0xffffffffu, l0, x);
          l1 += __shfl_xor_sync(0xffffffffu, l1, x);
        }
        const float i0 = 1.f / l0, i1 = 1.f / l1;
        bf16* o_r0 = p.out + ((long long)b * p.S + r0) * 128 + h * 32 + cl;
        bf16* o_r1 = o_r0 + 8 * 128;
#pragma unroll
        for (int d = 0; d < 4; ++d) {
          const uint32_t g0 = gg[d >> 1][(d & 1) * 2], g1 = gg[d >> 1][(d & 1) * 2 + 1];
          if (r0 < p.S)
            *reinterpret_cast<uint32_t*>(o_r0 + d * 8) =
                pack_bf16x2(o[d][0] * i0 * sigmoidf_fast(bf16_lo(g0)), o[d][1] * i0 * sigmoidf_fast(bf16_hi(g0)));
          if (r1 < p.S)
            *reinterpret_cast<uint32_t*>(o_r1 + d * 8) =
                pack_bf16x2(o[d][2] * i1 * sigmoidf_fast(bf16_lo(g1)), o[d][3] * i1 * sigmoidf_fast(bf16_hi(g1)));
        }
      }
      fence_proxy_async_smem();  // read here, written by TMA next
      __syncwarp();
      if (lane == 0) mbar_arrive(x_empty);
    }
  }

  tc_fence_before();
  __syncthreads();
  if (*cta_abort && threadIdx.x == 0) {
    const long long t0 = clock64();
    while (clock64() - t0 < 2000000) {}
  }
  __syncthreads();
  if (warp == 4) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 256);
  }
}

static int launch_xwin(Ctx* c, const bf16* q, const bf16* m, const bf16* w_qg, const bf16* w_kv, const XWinArgs& a, cudaStream_t st) {
  CUtensorMap tmq, tmm, tmwq, tmwk;
  if (!make_tmap_bf16_3d(&tmq, q, 128, a.S, a.B, 128, (uint64_t)128 * a.S, 64, 32, 1) ||
      !make_tmap_bf16_3d(&tmm, m, 128, a.K, a.B, 128, (uint64_t)128 * a.K, 64, 128, 1) ||
      !make_tmap_bf16_3d(&tmwq, w_qg, 128, 256, 1, 128, 128 * 256, 64, 64, 1) ||
      !make_tmap_bf16_3d(&tmwk, w_kv, 128, 256, 1, 128, 128 * 256, 64, 64, 1))
    return fail(c, XFOLD_ERR_ARG, "cross attention: cannot encode tensor maps (16-byte aligned bases?)");
  static bool attr_done[8] = {false};
  if (!attr_done[c->device & 7]) {
    cudaError_t e = cudaFuncSetAttribute(xwin_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, XW_SMEM);
    if (e != cudaSuccess) return fail(c, XFOLD_ERR_LAUNCH, "cross attention smem attribute: %s", cudaGetErrorString(e));
    attr_done[c->device & 7] = true;
  }
  ProfScope ps(c, XFOLD_K_APB_ATTENTION, st);
  launch_pdl(xwin_kernel, 2 * (a.B < c->sm_count ? a.B : c->sm_count), XW_THREADS, XW_SMEM, st, tmq, tmm, tmwq, tmwk, a);
  return check_launch(c, "xwin_kernel");
}

}  // namespace xf

using namespace xf;

extern "C" {

size_t xfold_cross_attention_workspace_bytes(int B, int S, int K, int H, int D) {
  return align_up((size_t)B * S * 2 * H * D * 2, 1024) + align_up((size_t)B * K * 2 * H * D * 2, 1024) + 2048;
}

int xfold_cross_attention_fwd(xfold_ctx* cx, const void* q_data, const void* m_data, int B, int S, int K, int Ca, int Cm,
                              int H, int D, const void* w_qg, const float* qg_bias, const float* qg_scale, const void* w_kv,
                              const float* bias, void* out, void* ws, size_t ws_bytes, void* stream) {
  Ctx* c = reinterpret_cast<Ctx*>(cx);
  if (!c || !q_data || !m_data || !w_qg || !w_kv || !bias || !out) return XFOLD_ERR_ARG;
  CallLock call(c);
  if (D != 16 && D != 32 && D != 64) return fail(c, XFOLD_ERR_ARG, "cross attention: head dimension 16, 32 or 64");
  if (B <= 0 || S <= 0 || K <= 0) return XFOLD_OK;
  const int W = H * D;
  const bool pairs = !((K & 1) || (reinterpret_cast<uintptr_t>(bias) & 7) || (reinterpret_cast<uintptr_t>(out) & 3));
  Carver cv(ws, ws_bytes);
  bf16* qg = (bf16*)cv.take((size_t)B * S * 2 * W * 2);
  bf16* kv = (bf16*)cv.take((size_t)B * K * 2 * W * 2);
  if (!ws || !cv.ok()) return fail(c, XFOLD_ERR_ARG, "cross attention: workspace too small (%zu < %zu)", ws_bytes, cv.off);
  cudaStream_t st = (cudaStream_t)stream;
  int rc;
  // The model's window is one tile of xwin_kernel; more queries, keys, heads or channels take the general kernels, and so do
  // a bias and a result that pairs of elements cannot be read from or written to, and a result that lies over an operand: the
  // general kernels have read all of those before the first result is stored, the windows' CTAs have not.
  const auto apart = [&](const void* x, size_t bytes) {
    const uintptr_t at = reinterpret_cast<uintptr_t>(x), to = reinterpret_cast<uintptr_t>(out);
    return !x || at + bytes <= to || to + (size_t)B * S * W * 2 <= at;
  };
  // Many windows with few tokens too: a window costs xwin_kernel the same whatever it holds, and packed rows are less then
  // (16000 windows of 1 x 2: 320 us against 403, 4 x 20: 412 and 438, 16 x 16: 489 and 473, 20 x 4: 514 and 502, 1 x 40: 448
  // and 439; 4000 of 1 x 2: 88 and 105; 592 of 1 x 2: 18.9 both).
  const bool windows = B <= 4 * c->sm_count || S > 16 || S + K >= 40;
  if (H == 4 && D == 32 && Ca == 128 && Cm == 128 && S <= 32 && K <= XA_KC && windows && pairs && apart(q_data, (size_t)B * S * 256) &&
      apart(m_data, (size_t)B * K * 256) && apart(w_qg, 256 * 256) && apart(w_kv, 256 * 256) && apart(qg_bias, 1024) &&
      apart(qg_scale, 1024))
    return launch_xwin(c, (const bf16*)q_data, (const bf16*)m_data, (const bf16*)w_qg, (const bf16*)w_kv,
                       XWinArgs{qg_bias, qg_scale, bias, (bf16*)out, B, S, K, c->d_status}, st);
  if ((rc = linear_plain(c, (const bf16*)q_data, Ca, (long long)B * S, Ca, (const bf16*)w_qg, 2 * W, qg_bias, qg_scale, qg,
                             2 * W, st))) return rc;
  if ((rc = linear_plain(c, (const bf16*)m_data, Cm, (long long)B * K, Cm, (const bf16*)w_kv, 2 * W, nullptr, nullptr, kv,
                             2 * W, st))) return rc;
  XAttnArgs a{qg, kv, bias, (bf16*)out, B, S, K, H};
  if (!pairs)
    return D == 16 ? launch_xattn<16, false>(c, a, st) : D == 32 ? launch_xattn<32, false>(c, a, st) : launch_xattn<64, false>(c, a, st);
  return D == 16 ? launch_xattn<16, true>(c, a, st) : D == 32 ? launch_xattn<32, true>(c, a, st) : launch_xattn<64, true>(c, a, st);
}

}  // extern "C"
