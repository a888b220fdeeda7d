// One denoising step of the DiffusionTransformer as one call: all blocks, every sample
// (nn/d_diffusion_transformer.py:37-310).  Per block seven launches,
//     xn   = sigmoid(scale) * LN(act) + shift            (adaln_kernel)
//     qkvg = xn W + bias;  o = attention(qkvg, logits)   (GEMM, attention)
//     act += sigmoid(gate) * (o W_out)                   (GEMM, gate and residual in the epilogue)
//     xn   = sigmoid(scale') * LN(act) + shift'
//     h    = swiglu(xn W1);  act += sigmoid(gate') * (h W2)
// The conditioning (scale, shift, scale', shift', gate, gate') depends on single_cond alone, so the projections of many
// blocks are two GEMMs instead of four narrow ones per block: one batched over the blocks' normalised copies of single_cond
// (scale and shift come out of one matrix and are read in place), one wide one for the gates.  (With each LayerNorm's scale
// folded into the weights one copy would do, but bf16 weights are then rounded a second time: 5.79e-3 instead of 5.35e-3
// from float64 after four blocks.)  Blocks are grouped so that a group's conditioning stays in L2 (48 MB of 126) until its
// blocks have used it.
#include "internal.h"
#include "stages.h"
#include "umma.cuh"

namespace xf {

// y[row] = sigmoid(scale[row % mod]) * LN(x[row]) + shift[row % mod]; one warp per row of C bf16.  All loads of a row are
// issued before the first reduction: with a few hundred rows the launch is one latency chain.
template <int C>
__global__ void __launch_bounds__(128)
adaln_kernel(const bf16* x, bf16* __restrict__ y, int rows, const bf16* scale, const bf16* shift, long long ldm, int mod) {
  constexpr int V = C / 128;
  const int lane = threadIdx.x & 31;
  const int row = blockIdx.x * 4 + (threadIdx.x >> 5);
  const bool valid = row < rows;
  uint2 rx[V], ra[V], rb[V];
  // The modulation was written at least two launches ago (the gate projection or a whole sub-layer lies between) and has
  // landed when this kernel starts: a kernel lets its successor start only after its own pdl_wait().  So it is fetched
  // while the predecessor still runs.
  if (valid) {
    const long long mr = (long long)(row % mod) * ldm;
#pragma unroll
    for (int k = 0; k < V; ++k) {
      ra[k] = __ldcg(reinterpret_cast<const uint2*>(scale + mr) + lane + 32 * k);
      rb[k] = __ldcg(reinterpret_cast<const uint2*>(shift + mr) + lane + 32 * k);
    }
  }
  pdl_wait();
  pdl_launch();
  if (!valid) return;
#pragma unroll
  for (int k = 0; k < V; ++k) rx[k] = reinterpret_cast<const uint2*>(x + (long long)row * C)[lane + 32 * k];
  float v[V][4], s = 0.f;
#pragma unroll
  for (int k = 0; k < V; ++k) {
    v[k][0] = bf16_lo(rx[k].x); v[k][1] = bf16_hi(rx[k].x); v[k][2] = bf16_lo(rx[k].y); v[k][3] = bf16_hi(rx[k].y);
    s += v[k][0] + v[k][1] + v[k][2] + v[k][3];
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  const float mean = s * (1.f / C);
  float ss = 0.f;
#pragma unroll
  for (int k = 0; k < V; ++k)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      v[k][e] -= mean;
      ss += v[k][e] * v[k][e];
    }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
  const float rstd = rsqrtf(ss * (1.f / C) + 1e-5f);
#pragma unroll
  for (int k = 0; k < V; ++k) {
    const float o0 = sigmoidf_fast(bf16_lo(ra[k].x)) * (v[k][0] * rstd) + bf16_lo(rb[k].x);
    const float o1 = sigmoidf_fast(bf16_hi(ra[k].x)) * (v[k][1] * rstd) + bf16_hi(rb[k].x);
    const float o2 = sigmoidf_fast(bf16_lo(ra[k].y)) * (v[k][2] * rstd) + bf16_lo(rb[k].y);
    const float o3 = sigmoidf_fast(bf16_hi(ra[k].y)) * (v[k][3] * rstd) + bf16_hi(rb[k].y);
    reinterpret_cast<uint2*>(y + (long long)row * C)[lane + 32 * k] = make_uint2(pack_bf16x2(o0, o1), pack_bf16x2(o2, o3));
  }
}

static int launch_adaln(Ctx* c, const bf16* x, bf16* y, int rows, int C, const bf16* scale, const bf16* shift, long long ldm,
                        int mod, cudaStream_t st) {
  ProfScope ps(c, XFOLD_K_LAYERNORM, st);
  const int grid = (rows + 3) / 4;
  switch (C) {
    case 128: launch_pdl(adaln_kernel<128>, grid, 128, 0, st, x, y, rows, scale, shift, ldm, mod); break;
    case 384: launch_pdl(adaln_kernel<384>, grid, 128, 0, st, x, y, rows, scale, shift, ldm, mod); break;
    case 768: launch_pdl(adaln_kernel<768>, grid, 128, 0, st, x, y, rows, scale, shift, ldm, mod); break;
    default: return fail(c, XFOLD_ERR_ARG, "diffusion: unsupported width %d (128, 384, 768)", C);
  }
  return check_launch(c, "adaln_kernel");
}

// y[g][row] = LN(x[row]) * gamma[g] for `copies` LayerNorms that differ in their scale alone; one warp per row and two copies.
// All of it runs beside the predecessor: x and gamma are older than the call, y was last read at least two launches ago, and
// this is never the call's first kernel, so that both have landed when it starts (see adaln_kernel).  (Behind the wait, eight
// copies per warp: a step 1.3 % longer at 77 tokens.)
template <int C>
__global__ void __launch_bounds__(128)
cond_ln_kernel(const bf16* x, bf16* y, int rows, const float* gamma, int copies) {
  constexpr int V = C / 128;
  const int lane = threadIdx.x & 31, row = blockIdx.x * 4 + (threadIdx.x >> 5);
  if (row >= rows) {
    pdl_wait();
    pdl_launch();
    return;
  }
  const int g0 = blockIdx.y * 2, ng = copies - g0 < 2 ? copies - g0 : 2;
  float4 w[2][V];
#pragma unroll
  for (int g = 0; g < 2; ++g)
#pragma unroll
    for (int k = 0; k < V; ++k)
      if (g < ng) w[g][k] = __ldcg(reinterpret_cast<const float4*>(gamma + (long long)(g0 + g) * C) + lane + 32 * k);
  float v[V][4], s = 0.f;
#pragma unroll
  for (int k = 0; k < V; ++k) {
    const uint2 u = __ldcg(reinterpret_cast<const uint2*>(x + (long long)row * C) + lane + 32 * k);
    v[k][0] = bf16_lo(u.x); v[k][1] = bf16_hi(u.x); v[k][2] = bf16_lo(u.y); v[k][3] = bf16_hi(u.y);
    s += v[k][0] + v[k][1] + v[k][2] + v[k][3];
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  const float mean = s * (1.f / C);
  float ss = 0.f;
#pragma unroll
  for (int k = 0; k < V; ++k)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      v[k][e] -= mean;
      ss += v[k][e] * v[k][e];
    }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
  const float rstd = rsqrtf(ss * (1.f / C) + 1e-5f);
#pragma unroll
  for (int g = 0; g < 2; ++g) {
    if (g == ng) break;
    uint2* out = reinterpret_cast<uint2*>(y + ((long long)(g0 + g) * rows + row) * C);
#pragma unroll
    for (int k = 0; k < V; ++k)
      out[lane + 32 * k] = make_uint2(pack_bf16x2(v[k][0] * rstd * w[g][k].x, v[k][1] * rstd * w[g][k].y),
                                      pack_bf16x2(v[k][2] * rstd * w[g][k].z, v[k][3] * rstd * w[g][k].w));
  }
  pdl_wait();
  pdl_launch();
}

static int launch_cond_ln(Ctx* c, const bf16* x, bf16* y, int rows, int C, const float* gamma, int copies, cudaStream_t st) {
  ProfScope ps(c, XFOLD_K_LAYERNORM, st);
  const dim3 grid((rows + 3) / 4, (copies + 1) / 2);
  switch (C) {
    case 128: launch_pdl(cond_ln_kernel<128>, grid, 128, 0, st, x, y, rows, gamma, copies); break;
    case 384: launch_pdl(cond_ln_kernel<384>, grid, 128, 0, st, x, y, rows, gamma, copies); break;
    case 768: launch_pdl(cond_ln_kernel<768>, grid, 128, 0, st, x, y, rows, gamma, copies); break;
    default: return fail(c, XFOLD_ERR_ARG, "diffusion: unsupported conditioning width %d (128, 384, 768)", C);
  }
  return check_launch(c, "cond_ln_kernel");
}

struct DiffWs {
  bf16 *cn, *mod, *gate, *xn, *o, *h, *qkvg, *mext;
  int group;  // blocks whose conditioning is computed together
  size_t bytes;
};
static DiffWs carve_diffusion(void* ws, size_t cap, int S, int N, const xfold_diffusion_weights* w) {
  DiffWs d;
  Carver cv(ws, cap);
  const size_t M = (size_t)S * N, C = w->C, Wd = (size_t)w->H * w->Dp;
  const size_t per_block = (size_t)N * 6 * C * 2;
  long long g = (long long)((48u << 20) / per_block);
  d.group = g < 1 ? 1 : g > w->num_blocks ? w->num_blocks : (int)g;
  d.cn = (bf16*)cv.take((size_t)N * w->C_cond * 2 * d.group * 2);
  d.mod = (bf16*)cv.take((size_t)N * 4 * C * d.group * 2);
  d.gate = (bf16*)cv.take((size_t)N * 2 * C * d.group * 2);
  d.xn = (bf16*)cv.take(M * C * 2);
  d.o = (bf16*)cv.take(M * Wd * 2);
  d.h = (bf16*)cv.take(M * w->F * 2);
  d.qkvg = (bf16*)cv.take(M * 4 * Wd * 2);
  d.mext = (bf16*)cv.take((size_t)((N + 127) / 128) * 4096);
  d.bytes = cv.off;
  return d;
}

static bool sizes_ok(const xfold_diffusion_weights* w) {
  return w->C > 0 && w->C_cond > 0 && w->H > 0 && w->F > 0 && (w->Dp == 32 || w->Dp == 64) && (w->H * w->Dp) % 128 == 0;
}

static int diffusion_fwd(Ctx* c, bf16* act, int S, int N, const float* mask, const bf16* cond, const xfold_diffusion_weights* w,
                         const void* const* logits, void* ws, size_t ws_bytes, cudaStream_t st) {
  if (S <= 0 || N <= 0 || w->num_blocks <= 0) return XFOLD_OK;
  if ((long long)S * N >= (1ll << 31)) return fail(c, XFOLD_ERR_ARG, "diffusion: too many tokens");
  if (!sizes_ok(w)) return fail(c, XFOLD_ERR_ARG, "diffusion: positive widths, and H x Dp a multiple of 128 with Dp 32 or 64");
  if (((uintptr_t)act | (uintptr_t)cond | (uintptr_t)w->ln_cond) & 15)
    return fail(c, XFOLD_ERR_ARG, "diffusion: act, single_cond and ln_cond must be 16-byte aligned");
  for (int b = 0; b < w->num_blocks; ++b) {
    const xfold_diffusion_block_weights& k = w->blocks[b];
    if (!logits[b] || !k.w_qkvg || !k.w_out || !k.w1_packed || !k.w2)
      return fail(c, XFOLD_ERR_ARG, "diffusion: block %d has no pair logits or no weights", b);
  }
  const DiffWs D = carve_diffusion(ws, ws_bytes, S, N, w);
  if (!ws || D.bytes > ws_bytes) return fail(c, XFOLD_ERR_ARG, "diffusion: workspace too small (%zu < %zu)", ws_bytes, D.bytes);
  StaticWeights sw(c);  // the first kernel is not a GEMM
  const int C = w->C, Wd = w->H * w->Dp, M = S * N, ldq = pad8(N);
  int rc;
  if ((rc = launch_mext(c, mask, 0, D.mext, 1, N, st))) return rc;
  for (int b = 0; b < w->num_blocks; ++b) {
    const int gi = b % D.group, ng = w->num_blocks - (b - gi) < D.group ? w->num_blocks - (b - gi) : D.group;
    const long long ldm = 4ll * C * ng, ldg = 2ll * C * ng;
    if (gi == 0) {
      if ((rc = launch_cond_ln(c, cond, D.cn, N, w->C_cond, w->ln_cond + (long long)b * 2 * w->C_cond, 2 * ng, st))) return rc;
      if ((rc = linear_batched(c, D.cn, N, w->C_cond, 2 * ng, (const bf16*)w->w_mod + (long long)b * 4 * C * w->C_cond, 2 * C,
                               w->b_mod + (long long)b * 4 * C, D.mod, ldm, st))) return rc;
      if ((rc = linear_plain(c, cond, w->C_cond, N, w->C_cond, (const bf16*)w->w_gate + (long long)b * 2 * C * w->C_cond,
                             (int)ldg, w->b_gate ? w->b_gate + (long long)b * 2 * C : nullptr, nullptr, D.gate, ldg, st))) return rc;
    }
    const bf16 *mod = D.mod + (long long)gi * 4 * C, *gate = D.gate + (long long)gi * 2 * C;
    const xfold_diffusion_block_weights& k = w->blocks[b];
    if ((rc = launch_adaln(c, act, D.xn, M, C, mod, mod + C, ldm, N, st))) return rc;
    // the v columns leave the projection as fp16: P and V are the fp16 operands of the P V product
    if ((rc = linear_plain(c, D.xn, C, M, C, (const bf16*)k.w_qkvg, 4 * Wd, k.qkvg_bias, k.qkvg_scale, D.qkvg, 4 * Wd, st,
                           2 * Wd, 3 * Wd, Wd))) return rc;
    c->attn_tag = XFOLD_K_APB_ATTENTION;
    rc = launch_attention2(c, D.qkvg, 4 * Wd, N, S, 0, 0, Wd, 2 * Wd, 3 * Wd, w->H, (const bf16*)logits[b], ldq, D.mext, 1, D.o,
                           Wd, (long long)N * Wd, st, w->Dp);
    c->attn_tag = XFOLD_K_ATTENTION;
    if (rc) return rc;
    if ((rc = linear_gate_resid(c, D.o, Wd, M, Wd, (const bf16*)k.w_out, C, gate, ldg, N, act, C, act, C, st))) return rc;
    if ((rc = launch_adaln(c, act, D.xn, M, C, mod + 2 * C, mod + 3 * C, ldm, N, st))) return rc;
    if ((rc = linear_swiglu(c, D.xn, C, M, C, (const bf16*)k.w1_packed, w->F, D.h, w->F, st))) return rc;
    if ((rc = linear_gate_resid(c, D.h, w->F, M, w->F, (const bf16*)k.w2, C, gate + C, ldg, N, act, C, act, C, st))) return rc;
  }
  return XFOLD_OK;
}

}  // namespace xf

using namespace xf;

extern "C" {

size_t xfold_diffusion_workspace_bytes(int S, int N, const xfold_diffusion_weights* w) {
  return w && S > 0 && N > 0 && w->num_blocks > 0 && sizes_ok(w) ? carve_diffusion(nullptr, 0, S, N, w).bytes : 0;
}

int xfold_diffusion_transformer_fwd(xfold_ctx* cx, void* act, int S, int N, const float* mask, const void* single_cond,
                                    const xfold_diffusion_weights* w, const void* const* pair_logits, void* ws,
                                    size_t ws_bytes, void* stream) {
  Ctx* c = reinterpret_cast<Ctx*>(cx);
  if (!c || !act || !single_cond || !w || !w->blocks || !w->w_mod || !w->b_mod || !w->w_gate || !w->ln_cond || !pair_logits) return XFOLD_ERR_ARG;
  CallLock call(c);
  return diffusion_fwd(c, (bf16*)act, S, N, mask, (const bf16*)single_cond, w, pair_logits, ws, ws_bytes, (cudaStream_t)stream);
}

}  // extern "C"
