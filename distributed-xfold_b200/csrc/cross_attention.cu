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
  Carver cv(ws, ws_bytes);
  bf16* qg = (bf16*)cv.take((size_t)B * S * 2 * W * 2);
  bf16* kv = (bf16*)cv.take((size_t)B * K * 2 * W * 2);
  if (!ws || !cv.ok()) return fail(c, XFOLD_ERR_ARG, "cross attention: workspace too small (%zu < %zu)", ws_bytes, cv.off);
  cudaStream_t st = (cudaStream_t)stream;
  int rc;
  if ((rc = linear_plain(c, (const bf16*)q_data, Ca, (long long)B * S, Ca, (const bf16*)w_qg, 2 * W, qg_bias, qg_scale, qg,
                             2 * W, st))) return rc;
  if ((rc = linear_plain(c, (const bf16*)m_data, Cm, (long long)B * K, Cm, (const bf16*)w_kv, 2 * W, nullptr, nullptr, kv,
                             2 * W, st))) return rc;
  XAttnArgs a{qg, kv, bias, (bf16*)out, B, S, K, H};
  if ((K & 1) || (reinterpret_cast<uintptr_t>(bias) & 7) || (reinterpret_cast<uintptr_t>(out) & 3))
    return D == 16 ? launch_xattn<16, false>(c, a, st) : D == 32 ? launch_xattn<32, false>(c, a, st) : launch_xattn<64, false>(c, a, st);
  return D == 16 ? launch_xattn<16, true>(c, a, st) : D == 32 ? launch_xattn<32, true>(c, a, st) : launch_xattn<64, true>(c, a, st);
}

}  // extern "C"
