// Gated multi-head attention with an additive pair bias and a key mask (TriangleAttention: 4 heads x 32;
// AttentionPairBias: 16 heads x 24 padded to 32 in the trunk, 16 x 48 padded to 64 in the diffusion transformer).
//
// Bound: the exponential unit (16 results per clock and SM): N^2 heads rows exponentials, 0.98 ms for a TriangleAttention of
// 1024 tokens.  Everything else is arranged so that the softmax threads do little besides exponentiate and rarely wait:
//   * The logits arrive complete.  The tensor core adds the pair bias (bias tile x 16 x 16 identity blocks, fp16, exact) and
//     the key mask (ones x its three bf16 pieces) to Q K^T, and Q was scaled by log2(e) where it was projected, so a logit in tensor
//     memory is the base-2 exponent: per pair of keys one packed subtraction of the reference exponent, two exponentials,
//     one pack, one packed addition to the row sum.
//   * Per block of 64 keys and slot the softmax warps wait once (logits complete) and arrive once (P stored).  Logits and P
//     are double-buffered (P overwrites the logits it came from): while the exponentials of block j run, the logits of block
//     j + 1 are there already; when P(j) is published, the issuer appends  O += P(j) V(j)  and the logits of block j + 2,
//     which go over P(j) -- products of one issuing thread execute in order.
//   * Three slots (two when a slot's head is 64 wide) of 128 queries share the exponential unit, so that a slot's own waits
//     (about 400 clocks of 900 per block) pass behind the other slots' exponentials (512 clocks per block and slot).
// Measured at 1024 tokens, TriangleAttention: 1.95 ms with the bias added by the softmax threads, four heads per item and
// three barrier waits per 64 keys; 2.02 ms for this scheme with an elected-lane branch in the issuers (60 to 100 clocks per
// operation); 1.68 ms without the branch, single-buffered blocks of 128 keys; 1.41 ms double-buffered; 1.33 ms with Q double-
// buffered as well; 1.27 ms with an eighth of the exponentials on the FMA pipe.
//
// Work item = `ns` slots of (batch row, head, 128 queries).
//   ROWS: the slots are neighbouring batch rows of one head and query tile; they share the pair-bias tile, whose trips from
//         L2 would otherwise be the larger part of the traffic (a row reads 256 KB of bias per head and query tile at 1024
//         tokens, and 131 KB of keys and values).
//   TILES: the slots are neighbouring query tiles of one batch row and head; they share the keys and values.
// CTAs are persistent and run their items' key blocks as one continuous sequence.
//   warp 0         : TMA producer.  A ring of stages {K, bias, mask of block u, V of block u - 2}: what an issuer needs for
//                    one step, with one barrier each way.  (As two rings, an issuer waited and committed twice as often:
//                    41 -> 40 us at 255 tokens, 1-2 % at 1024.)
//   warps 1 .. NS  : one issuer of tcgen05.mma per slot (warp-uniform code, one elected lane).
//   warps 4 ..     : one softmax warpgroup per slot, one thread per query row.
// Tensor memory per slot: 128 columns of logits / probabilities, D columns of output.
//
// The reference exponent m_ref follows the running maximum lazily.  A block's sweep over 64 keys runs against the m_ref of the
// blocks before and looks at its partial sums afterwards; if one exceeds 2^12 in some row of the warp (fp16 P overflows at
// 2^16) the warp takes the exact path: maximum of the logits, which are still in registers, O and the row sum rescaled where it
// grew by more than 2^8, the sweep repeated.  The first block of an item starts with its maximum.  The exact path stands beside
// the sweep, not in a loop around it (a loop around each half, with a vote after each: 1.05 of the time at 1024 tokens).
#include <cuda_fp16.h>

#include "internal.h"
#include "stages.h"
#include "umma.cuh"

namespace xf {

struct AttnArgs {
  int S, B, heads, ns;        // sequence length, batch rows, heads, slots per item
  int q_col0, k_col0, v_col0, g_col0;
  const bf16* qkvg;
  long long seq_stride, batch_stride;
  const uint8_t* mext;          // [B or 1][ceil(S / 64)][64 keys x 16 bytes] mask-bias tiles
  long long mext_batch_stride;  // bytes; 0 when one mask row serves every batch row
  bf16* out;
  long long out_seq_stride, out_batch_stride;
  int* status;
};

// D: head dimension.  ROWS: slots are batch rows, else query tiles.
template <int D, bool ROWS>
struct AttnCfg {
  static constexpr int NS = ROWS ? 3 : 2;
  static constexpr int NK = ROWS ? 4 : 3;                      // stages of the ring, 64 keys each
  static constexpr int THREADS = (4 + 4 * NS) * 32;
  static constexpr uint32_t KT = 64 * D * 2;                   // one [64 keys][D] tile
  static constexpr uint32_t BT = 128 * 64 * 2;                 // one [128 queries][64 keys] bias tile
  static constexpr uint32_t MT = 1024;                         // one [64 keys][8] mask tile
  static constexpr uint32_t QT = 128 * D * 2;
  static constexpr uint32_t K_BYTES = (ROWS ? NS : 1) * KT, B_BYTES = (ROWS ? 1 : NS) * BT, M_BYTES = (ROWS ? NS : 1) * MT;
  static constexpr uint32_t STAGE = B_BYTES + 2 * K_BYTES + M_BYTES;
  static constexpr uint32_t OFF_V = B_BYTES + K_BYTES + M_BYTES, OFF_Q = NK * STAGE, OFF_ID = OFF_Q + 2 * NS * QT,
                            OFF_E1 = OFF_ID + 512, OFF_ZERO = OFF_E1 + 2048, OFF_BAR = OFF_ZERO + 2048,
                            SMEM = OFF_BAR + 512 + 1024;
  static constexpr uint32_t TM_O = NS * 128;                   // output columns behind the logits
  static_assert(STAGE % 1024 == 0 && K_BYTES % 1024 == 0 && QT % 1024 == 0, "swizzled tiles start at multiples of 1 KB");
  static_assert(SMEM <= 232448, "shared memory");
};

__device__ __forceinline__ float ex2f_(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float clamp_nan(float x, float lo, float hi) {  // (fminf and fmaxf would lose a NaN)
  asm("max.NaN.f32 %0, %0, %1;\n\tmin.NaN.f32 %0, %0, %2;" : "+f"(x) : "f"(lo), "f"(hi));
  return x;
}
// 2^y for a pair of float32 on the FMA pipe: y = n + f with n the nearest integer, 2^f by a degree-5 polynomial on
// [-1/2, 1/2], times 2^n.  0 from -127 down, NaN for NaN.  Coefficients: minimax in relative error with constant term 1 (a
// linear program over the interval, each coefficient rounded to float32 before the next is fitted), 9.3e-8; evaluated in
// float32 the relative error is at most 1.6e-7.
__device__ __forceinline__ float2 ex2_poly2(float2 y) {
  const float magic = 12582912.f;  // 1.5 * 2^23: adding it leaves the nearest integer in the low bits
  y.x = clamp_nan(y.x, -127.f, 127.f);
  y.y = clamp_nan(y.y, -127.f, 127.f);
  const float2 t = fadd2(y, make_float2(magic, magic));
  const float2 n = fadd2(t, make_float2(-magic, -magic));
  const float2 f = ffma2(n, make_float2(-1.f, -1.f), y);
  float2 q = ffma2(f, make_float2(0.0013269521296024323f, 0.0013269521296024323f), make_float2(0.009671291336417198f, 0.009671291336417198f));
  q = ffma2(q, f, make_float2(0.0555071085691452f, 0.0555071085691452f));
  q = ffma2(q, f, make_float2(0.24022246897220612f, 0.24022246897220612f));
  q = ffma2(q, f, make_float2(0.6931470036506653f, 0.6931470036506653f));
  q = ffma2(q, f, make_float2(1.f, 1.f));
  // 2^n from the exponent field (0 for n = -127)
  return make_float2(q.x * __uint_as_float(__float_as_uint(t.x) * 0x800000u + 0x3F800000u),
                     q.y * __uint_as_float(__float_as_uint(t.y) * 0x800000u + 0x3F800000u));
}
// Which of a sweep's 16 pairs take the polynomial: two, away from its ends.  (TriangleAttention, 1024 tokens: none 1.02 of the
// time, three 1.00 to 1.02, four more; at the ends of the sweep's halves 1.01 -- with more, the FMA pipe and the issue slots
// are the longer queue.)
__host__ __device__ constexpr bool poly_pair(int e) { return e % 6 == 4; }
// K-major or MN-major tile with rows of 64 bytes (D = 32) or 128 bytes (D = 64), swizzled over 8 rows
template <int D>
__device__ __forceinline__ uint64_t make_sdesc_d(uint32_t saddr) {
  uint64_t d = uint64_t((saddr & 0x3FFFFu) >> 4) | (uint64_t(1) << 16) | (uint64_t((8u * D * 2u) >> 4) << 32) | (uint64_t(1) << 46);
  return d | (uint64_t(D == 64 ? 2 : 4) << 61);  // SWIZZLE_128B : SWIZZLE_64B
}

template <int D, bool ROWS>
__global__ void __launch_bounds__(AttnCfg<D, ROWS>::THREADS, 1)
attn_kernel(const __grid_constant__ CUtensorMap tmq, const __grid_constant__ CUtensorMap tmkv,
            const __grid_constant__ CUtensorMap tmb, const AttnArgs p) {
  using Cfg = AttnCfg<D, ROWS>;
  constexpr int NS = Cfg::NS, NK = Cfg::NK;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw_addr = smem_u32(smem_raw);
  uint8_t* smem = smem_raw + (((raw_addr + 1023u) & ~1023u) - raw_addr);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + Cfg::OFF_BAR);
  uint64_t* full = bars;                // [NK] a stage's tiles have landed
  uint64_t* empty = full + NK;          // [NK] every slot's products that read the stage are complete
  uint64_t* q_full = empty + NK;       // [2] (Q of the next item arrives while this one's is in use)
  uint64_t* q_empty = q_full + 2;       // [2] every slot's last logits of the item are complete
  uint64_t* s_full = q_empty + 2;       // [NS][2] a block's logits are complete
  uint64_t* p_ready = s_full + 2 * NS;  // [NS][2] the block's P is in tensor memory
  uint64_t* pv_done = p_ready + 2 * NS; // [NS][2] a block's P V product is complete
  // (pairs by block parity: either side may be two blocks ahead, one more than a phase bit can tell apart)
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(pv_done + 2 * NS);
  volatile int* cta_abort = reinterpret_cast<volatile int*>(tmem_slot + 1);

  // (a reduction's result is in a uniform register)
  const int warp = int(__reduce_max_sync(0xffffffffu, threadIdx.x >> 5)), lane = threadIdx.x & 31;
  const AbortCtx ab{cta_abort, p.status};
  const int ns = p.ns;
  // items: query tiles fastest, then heads, then batch rows, so that the CTAs at work at one time share keys and values
  const int QT = (p.S + 127) / 128, QI = ROWS ? QT : (QT + ns - 1) / ns, BI = ROWS ? (p.B + ns - 1) / ns : p.B;
  const int NB = (p.S + 63) / 64;       // blocks (stages) per item
  const uint32_t n_items = uint32_t(QI) * uint32_t(p.heads) * uint32_t(BI);
  auto decode = [&](uint32_t t, int& qt, int& h, int& b) {
    qt = int(t % uint32_t(QI)) * (ROWS ? 1 : ns);
    h = int((t / uint32_t(QI)) % uint32_t(p.heads));
    b = int(t / (uint32_t(QI) * uint32_t(p.heads))) * (ROWS ? ns : 1);
  };

  if (threadIdx.x == 0) {
    for (int s = 0; s < NK; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], ns);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(&q_full[s], 1);
      mbar_init(&q_empty[s], ns);
    }
    for (int s = 0; s < NS; ++s) {
      for (int x = 0; x < 2; ++x) {
        mbar_init(&s_full[2 * s + x], 1);
        mbar_init(&p_ready[2 * s + x], 4);  // one lane per softmax warp
        mbar_init(&pv_done[2 * s + x], 1);
      }
    }
    *cta_abort = 0;
    fence_barrier_init();
    tma_prefetch_desc(&tmq);
    tma_prefetch_desc(&tmkv);
    tma_prefetch_desc(&tmb);
  }
  // Constant operands, un-swizzled 8 x 16-byte core matrices.  ID: the 16 x 16 fp16 identity.  E1: columns 0..7 of a
  // [128][16] matrix whose columns 0..2 are all ones.  ZERO: columns 8..15 of E1 and of the mask tiles.
  for (uint32_t i = threadIdx.x; i < (512 + 2048 + 2048) / 4; i += Cfg::THREADS) {
    uint32_t v = 0;
    if (i < 128) {
      const uint32_t core = i >> 5, row = (i & 31) >> 2, pr = i & 3;  // core = (row group, column group)
      if ((core == 0 || core == 3) && (row >> 1) == pr) v = (row & 1) ? 0x3C000000u : 0x00003C00u;
    } else if (i < 640) {
      v = (i & 3) == 0 ? 0x3F803F80u : (i & 3) == 1 ? 0x00003F80u : 0u;
    }
    reinterpret_cast<uint32_t*>(smem + Cfg::OFF_ID)[i] = v;
  }
  fence_proxy_async_smem();
  if (warp == 1) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = __reduce_max_sync(0xffffffffu, *tmem_slot);
  pdl_wait();
  pdl_launch();

  if (warp == 0) {
    // ------------------------------------------------------------------------------------------------ TMA producer
    // Stage u holds keys, bias and mask of block u and the values of block u - 2: what the issuers need for one step.
    const uint32_t go = elect_one();  // warp-uniform, like the issuers
    const uint64_t my_items = n_items > blockIdx.x ? (n_items - blockIdx.x + gridDim.x - 1) / gridDim.x : 0;
    const uint64_t total = my_items * uint64_t(NB);
    uint32_t st = 0, ph = 0, it = 0, item_k = blockIdx.x, item_v = blockIdx.x;
    int ks = 0, vs = 0, qt = 0, h = 0, b = 0, vqt, vh, vb;
    decode(item_v, vqt, vh, vb);
    for (uint64_t u = 0; u < (total ? total + 2 : 0); ++u) {
      if (u < total && ks == 0) {
        decode(item_k, qt, h, b);
        const uint32_t qb = it & 1u;
        if (!mbar_wait_warp(&q_empty[qb], ((it >> 1) & 1u) ^ 1u, ab, XF_ERR_WAIT_EMPTY)) break;
        mbar_arrive_expect_tx_if(go, &q_full[qb], (ROWS ? NS : ns) * Cfg::QT);
        uint8_t* sq = smem + Cfg::OFF_Q + qb * (NS * Cfg::QT);
        if constexpr (ROWS) tma_load_3d_if(go, sq, &tmq, &q_full[qb], p.q_col0 + h * D, qt * 128, b);
        else
          for (int s = 0; s < ns; ++s) tma_load_3d_if(go, sq + s * Cfg::QT, &tmq, &q_full[qb], p.q_col0 + h * D, (qt + s) * 128, b);
        ++it;
      }
      if (!mbar_wait_warp(&empty[st], ph ^ 1u, ab, XF_ERR_WAIT_EMPTY)) break;
      uint8_t* sb = smem + st * Cfg::STAGE;
      uint8_t* sk = sb + Cfg::B_BYTES;
      uint8_t* sm = sk + Cfg::K_BYTES;
      int nm = 1;  // mask tiles: one per batch row of the item
      if constexpr (ROWS) nm = p.mext_batch_stride == 0 ? 1 : (p.B - b < NS ? p.B - b : NS);
      mbar_arrive_expect_tx_if(go, &full[st], (u < total ? (ROWS ? 1 : ns) * Cfg::BT + Cfg::K_BYTES + nm * Cfg::MT : 0) + (u >= 2 ? Cfg::K_BYTES : 0));
      if (u < total) {
        tma_load_3d_if(go, sk, &tmkv, &full[st], p.k_col0 + h * D, ks * 64, b);
        if constexpr (ROWS) tma_load_3d_if(go, sb, &tmb, &full[st], ks * 64, qt * 128, h);
        else
          for (int s = 0; s < ns; ++s) tma_load_3d_if(go, sb + s * Cfg::BT, &tmb, &full[st], ks * 64, (qt + s) * 128, h);
        const uint8_t* mrow = p.mext + (long long)b * p.mext_batch_stride + (long long)ks * Cfg::MT;
        for (int s = 0; s < nm; ++s) bulk_load_if(go, sm + s * Cfg::MT, mrow + s * p.mext_batch_stride, Cfg::MT, &full[st]);
        if (++ks == NB) {
          ks = 0;
          item_k += gridDim.x;
        }
      }
      if (u >= 2) {
        tma_load_3d_if(go, sb + Cfg::OFF_V, &tmkv, &full[st], p.v_col0 + vh * D, vs * 64, vb);
        if (++vs == NB) {
          vs = 0;
          item_v += gridDim.x;
          decode(item_v, vqt, vh, vb);
        }
      }
      if (++st == NK) { st = 0; ph ^= 1u; }
    }
  } else if (warp <= ns && warp < 4) {
    // ---------------------------------------------------------------------------------------- issuer of slot s
    // Warp-uniform throughout (votes instead of per-lane branches; one elected lane is predicated inside each
    // instruction): descriptors and counters live in uniform registers.  With a branch around the elected lane an
    // operation cost 60 to 100 clocks, 2700 per block, and paced the kernel.
    const int s = warp - 1;
    const uint32_t leader = elect_one() ? 1u : 0u;
    constexpr uint32_t idesc_qk = make_idesc(128, 64);                 // bf16
    constexpr uint32_t idesc_bias = make_idesc(128, 16, 0, 0, 1);      // fp16
    constexpr uint32_t idesc_pv = make_idesc(128, D, 0, 1, 1);         // fp16 (the v columns are projected to fp16), V N-major
    const uint32_t base = smem_u32(smem);
    const uint32_t d_s = tmem_base + s * 128, d_o = tmem_base + Cfg::TM_O + s * D;
    // descriptors of stage 0 (a stage further: their low words move by the stage's size in 16-byte units), hi words constant
    const uint64_t qd0 = make_sdesc_d<D>(base + Cfg::OFF_Q + s * Cfg::QT);
    const uint64_t idd = make_sdesc_noswizzle(base + Cfg::OFF_ID, 128, 256);
    const uint64_t e1d = make_sdesc_noswizzle(base + Cfg::OFF_E1, Cfg::OFF_ZERO - Cfg::OFF_E1, 128);
    const uint32_t m_at = base + Cfg::B_BYTES + Cfg::K_BYTES + (ROWS && p.mext_batch_stride != 0 ? s * Cfg::MT : 0);
    const uint64_t kd0 = make_sdesc_d<D>(base + Cfg::B_BYTES + (ROWS ? s * Cfg::KT : 0));
    const uint64_t bd0 = make_sdesc(base + (ROWS ? 0 : s * Cfg::BT), 16, 1024);
    const uint64_t md0 = make_sdesc_noswizzle(m_at, base + Cfg::OFF_ZERO - m_at, 128);
    const uint64_t vd0 = make_sdesc_d<D>(base + Cfg::OFF_V + (ROWS ? s * Cfg::KT : 0));
    const uint32_t klo = uint32_t(kd0), khi = uint32_t(kd0 >> 32), blo = uint32_t(bd0), bhi = uint32_t(bd0 >> 32), mlo = uint32_t(md0),
                   mhi = uint32_t(md0 >> 32), vlo = uint32_t(vd0), vhi = uint32_t(vd0 >> 32);
    const uint32_t my_items = n_items > blockIdx.x ? (n_items - blockIdx.x + gridDim.x - 1) / gridDim.x : 0u;
    const uint32_t G = my_items * uint32_t(NB);  // (the launcher bounds it)
    uint32_t st = 0, ph = 0, it = 0, so = 0;
    int jb = 0, kb = 0;  // blocks of the logits and of the P V product within their items
    // One step: P V of block u - 2, then the logits of block u over that P (products of one issuer execute in order).
    for (uint32_t u = 0; u < (G ? G + 2 : 0); ++u) {
      if (u < G && jb == 0 && !mbar_wait_warp(&q_full[it & 1u], (it >> 1) & 1u, ab, XF_ERR_WAIT_FULL)) break;
      if (!mbar_wait_warp(&full[st], ph, ab, XF_ERR_WAIT_FULL)) break;
      const uint32_t x = u & 1u, d = d_s + x * 64;
      if (u >= 2) {
        if (!mbar_wait_warp(&p_ready[2 * s + x], ((u - 2) >> 1) & 1u, ab, XF_ERR_WAIT_ATTN)) break;
        tc_fence_after();
        const int keys = p.S - kb * 64;
#pragma unroll
        for (int j = 0; j < 4; ++j) {  // 16 keys = 32 D bytes of V = 8 columns of P
          if ((j & ~1) * 16 >= keys) break;  // keys beyond the sequence are left out in steps of 32, as in the sweeps
          umma_ts_lo_if(leader, d_o, d + j * 8, vlo + so + j * 2 * D, vhi, idesc_pv, (kb | j) ? 1u : 0u);
        }
        umma_commit_if(leader, &pv_done[2 * s + x]);
        if (++kb == NB) kb = 0;
      }
      if (u < G) {
        tc_fence_after();
        const uint32_t qb = it & 1u;
        const uint64_t qd = qd0 + uint64_t(qb * (NS * Cfg::QT / 16));
#pragma unroll
        for (int j = 0; j < D / 16; ++j)
          umma_ss_lo_if(leader, d, uint32_t(qd) + 2 * j, uint32_t(qd >> 32), klo + so + 2 * j, khi, idesc_qk, j ? 1u : 0u);
        umma_ss_lo_if(leader, d, uint32_t(e1d), uint32_t(e1d >> 32), mlo - so * 65535u, mhi, idesc_qk, 1u);
#pragma unroll
        for (int j = 0; j < 4; ++j)
          umma_ss_lo_if(leader, d + j * 16, blo + so + 2 * j, bhi, uint32_t(idd), uint32_t(idd >> 32), idesc_bias, 1u);
        umma_commit_if(leader, &s_full[2 * s + x]);
        if (++jb == NB) {
          jb = 0;
          ++it;
          umma_commit_if(leader, &q_empty[qb]);
        }
      }
      umma_commit_if(leader, &empty[st]);
      so += Cfg::STAGE / 16;
      if (++st == NK) { st = 0; ph ^= 1u; so = 0; }
    }
  } else if (warp >= 4 && warp < 4 + 4 * ns) {
    // ------------------------------------------------------------------------------------------------ softmax warps
    const int s = (warp - 4) >> 2;
    const int row = (warp & 3) * 32 + lane;
    const uint32_t lane_addr = uint32_t((warp & 3) * 32) << 16;
    const uint32_t s_addr = tmem_base + s * 128 + lane_addr, o_addr = tmem_base + Cfg::TM_O + s * D + lane_addr;
    const uint32_t FULL = 0xffffffffu;
    uint32_t g = 0;
    bool okay = true;
    for (uint32_t t = blockIdx.x; t < n_items && okay; t += gridDim.x) {
      int qt, h, b;
      decode(t, qt, h, b);
      if (ROWS) b += s;
      else qt += s;
      const int qi = qt * 128 + row;
      const bool valid = qi < p.S && b < p.B;
      float m_ref = -3.0e38f;
      float2 l2 = make_float2(0.f, 0.f);
      for (int kb = 0; kb < NB && okay; ++kb, ++g) {
        const uint32_t buf = s_addr + (g & 1u) * 64;
        okay = __all_sync(FULL, mbar_wait(&s_full[2 * s + (g & 1u)], (g >> 1) & 1u, ab, XF_ERR_WAIT_ATTN));
        if (!okay) break;
        tc_fence_after();
        const bool both = p.S - kb * 64 > 32;  // the block's second 32 keys exist
        uint32_t r[2][32];
        tmem_ld32(buf, r[0]);
        if (both) tmem_ld32(buf + 32, r[1]);
        tmem_ld_wait();
        float2 s2 = make_float2(0.f, 0.f);
        // 32 keys against m_ref: P over logits that have been read, and their sums
        auto sweep = [&](const uint32_t(&x)[32], uint32_t at) {
          const float2 nm = make_float2(-m_ref, -m_ref);
          uint32_t pk[16];
#pragma unroll
          for (int e = 0; e < 16; ++e) {
            const float2 y = fadd2(make_float2(__uint_as_float(x[2 * e]), __uint_as_float(x[2 * e + 1])), nm);
            const float2 pe = poly_pair(e) ? ex2_poly2(y) : make_float2(ex2f_(y.x), ex2f_(y.y));
            s2 = fadd2(s2, pe);
            const __half2 ph = __floats2half2_rn(pe.x, pe.y);
            pk[e] = *reinterpret_cast<const uint32_t*>(&ph);
          }
          tmem_st16(at, pk);
        };
        // the reference exponent follows the block's maximum where that is more than 8 above it
        auto follow = [&]() {
          float mx = __uint_as_float(r[0][0]);
#pragma unroll
          for (int e = 1; e < 32; ++e) mx = fmaxf(mx, __uint_as_float(r[0][e]));
          if (both) {
#pragma unroll
            for (int e = 0; e < 32; ++e) mx = fmaxf(mx, __uint_as_float(r[1][e]));
          }
          const bool grow = mx > m_ref + 8.f;
          const float m_new = grow ? mx : m_ref;
          const float alpha = ex2f_(m_ref - m_new);
          m_ref = m_new;
          l2.x *= alpha;
          l2.y *= alpha;
          return alpha;
        };
        if (kb == 0) follow();
        sweep(r[0], buf);
        if (both) sweep(r[1], buf + 16);
        if (kb > 0 && __any_sync(FULL, fmaxf(s2.x, s2.y) > 4096.f)) {
          // some row may have outgrown the reference: exact maximum, rescale, sweep again
          const float alpha = follow();
          if (__any_sync(FULL, alpha != 1.f)) {
            // every earlier P V product of the item must have landed before O is rescaled
            okay = __all_sync(FULL, mbar_wait(&pv_done[2 * s + ((g - 1) & 1u)], ((g - 1) >> 1) & 1u, ab, XF_ERR_WAIT_ATTN));
            if (!okay) break;
            tc_fence_after();
            uint32_t o[16];
#pragma unroll 1
            for (int oc = 0; oc < D; oc += 16) {
              tmem_ld16(o_addr + oc, o);
              tmem_ld_wait();
#pragma unroll
              for (int e = 0; e < 16; ++e) o[e] = __float_as_uint(__uint_as_float(o[e]) * alpha);
              tmem_st16(o_addr + oc, o);
            }
          }
          s2 = make_float2(0.f, 0.f);
          tmem_st_wait();
          sweep(r[0], buf);
          if (both) sweep(r[1], buf + 16);
        }
        l2 = fadd2(l2, s2);
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&p_ready[2 * s + (g & 1u)]);
      }
      if (!okay) break;
      // item epilogue: O / l, gate, store; the gate is on its way while the last product runs
      const int col = h * D;
      const bf16* grow_ = p.qkvg + (long long)b * p.batch_stride + (long long)qi * p.seq_stride + p.g_col0 + col;
      bf16* orow = p.out + (long long)b * p.out_batch_stride + (long long)qi * p.out_seq_stride + col;
      uint4 gu[4];
      if (valid) {
#pragma unroll
        for (int g8 = 0; g8 < 4; ++g8) gu[g8] = *reinterpret_cast<const uint4*>(grow_ + g8 * 8);
      }
      okay = __all_sync(FULL, mbar_wait(&pv_done[2 * s + ((g - 1) & 1u)], ((g - 1) >> 1) & 1u, ab, XF_ERR_WAIT_ATTN));
      if (!okay) break;
      tc_fence_after();
      const float inv = __fdividef(1.f, l2.x + l2.y);
#pragma unroll
      for (int oc = 0; oc < D; oc += 32) {
        uint32_t o[32];
        tmem_ld32(o_addr + oc, o);
        if (oc > 0 && valid) {
#pragma unroll
          for (int g8 = 0; g8 < 4; ++g8) gu[g8] = *reinterpret_cast<const uint4*>(grow_ + oc + g8 * 8);
        }
        tmem_ld_wait();
        if (valid) {
#pragma unroll
          for (int g8 = 0; g8 < 4; ++g8) {
            const uint32_t gw[4] = {gu[g8].x, gu[g8].y, gu[g8].z, gu[g8].w};
            uint32_t ow[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const float2 y = fmul2(fmul2(make_float2(__uint_as_float(o[g8 * 8 + 2 * e]), __uint_as_float(o[g8 * 8 + 2 * e + 1])),
                                           make_float2(inv, inv)), sigmoid2(make_float2(bf16_lo(gw[e]), bf16_hi(gw[e]))));
              ow[e] = pack_bf16x2(y.x, y.y);
            }
            *reinterpret_cast<uint4*>(orow + oc + g8 * 8) = make_uint4(ow[0], ow[1], ow[2], ow[3]);
          }
        }
      }
      tc_fence_before();
    }
  }

  tc_fence_before();
  __syncthreads();
  if (*cta_abort && threadIdx.x == 0) {
    // an aborted wait may have left copies in flight: give them time to land before the CTA's memory is released
    const long long t0 = clock64();
    while (clock64() - t0 < 2000000) {}
  }
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

// Mask-bias tiles: out[b][ks] is a [64 keys][8] bf16 tile (8-key groups of 128 bytes, 16 bytes per key) whose first columns
// add up to the bias of a key k < S, -1e30 for the padding of the last tile; its other columns are zero.
// A mask: 1e9 * (mask[b][k] - 1) as in the reference, in one column, floored at -60000: any such logit still exponentiates to
// exactly 0 next to an unmasked one, while a row whose keys are ALL masked keeps fp32-resolvable logits (at 1e9 the fp32
// spacing is 64).
// additive: the bias itself.  Times log2(e) like the logits it is added to, in three columns (float32's 24 bits), kept within
// +-60000 like the pair bias.
__device__ __forceinline__ void mext_tiles(const float* mask, long long mask_ld, uint4* out, int B, int S, int KS, int additive,
                                           long long first, long long step) {
  const long long n = (long long)B * KS * 64;
  for (long long idx = first; idx < n; idx += step) {
    const long long bb = idx / (KS * 64);
    const int k = int(idx - bb * (KS * 64));
    float v = -1.0e30f;
    uint32_t p[3] = {0, 0, 0};
    if (k < S) {
      v = mask ? mask[bb * mask_ld + k] : additive ? 0.f : 1.f;
      v = fminf(fmaxf(additive ? v * 1.4426950408889634f : 1.0e9f * (v - 1.f), -60000.f), additive ? 60000.f : 3.0e38f);
    }
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      const bf16 h = __float2bfloat16(v);
      p[i] = __bfloat16_as_ushort(h);
      v = additive ? v - __bfloat162float(h) : 0.f;
    }
    out[idx] = make_uint4(p[0] | p[1] << 16, p[2], 0, 0);
  }
}
__global__ void mext_kernel(const float* mask, long long mask_ld, uint4* __restrict__ out, int B, int S, int KS, int additive) {
  pdl_wait();
  pdl_launch();
  mext_tiles(mask, mask_ld, out, B, S, KS, additive, (long long)blockIdx.x * blockDim.x + threadIdx.x, (long long)gridDim.x * blockDim.x);
}

int launch_mext(Ctx* c, const float* mask, long long mask_ld, bf16* out, int B, int S, cudaStream_t st, int additive) {
  const int KS = (S + 63) / 64;
  const long long n = (long long)B * KS * 64;
  if (n <= 0) return XFOLD_OK;
  long long blocks = (n + 255) / 256;
  if (blocks > 8192) blocks = 8192;
  ProfScope ps(c, XFOLD_K_MASK_BIAS, st);
  launch_pdl(mext_kernel, (int)blocks, 256, 0, st, mask, mask_ld, reinterpret_cast<uint4*>(out), B, S, KS, additive);
  return check_launch(c, "mext_kernel");
}

// fp32 [H][S][S] -> 16-bit [H][S][ldq] (same query-major order, padded row pitch): FP16 values times log2(e), the operand
// the kernel's pair-bias tensor map expects (the kernel works in base 2 and adds the tile as it is).
__device__ __forceinline__ void bias_convert(const float* in, __half* out, long long rows, int S, int ldq, long long first, long long step) {
  const long long n = rows * ldq;
  for (long long idx = first; idx < n; idx += step) {
    const long long r = idx / ldq;
    const int k = int(idx % ldq);
    out[idx] = __float2half_rn(k < S ? fminf(fmaxf(in[r * S + k] * 1.4426950408889634f, -60000.f), 60000.f) : 0.f);
  }
}

__global__ void bias_convert_kernel(const float* in, __half* __restrict__ out, long long rows, int S, int ldq) {
  pdl_wait();
  pdl_launch();
  bias_convert(in, out, rows, S, ldq, (long long)blockIdx.x * blockDim.x + threadIdx.x, (long long)gridDim.x * blockDim.x);
}
// Both operands of a call in one launch: the first `split` blocks convert the bias, the others make the mask tiles.
__global__ void attn_prepare_kernel(const float* bias, __half* __restrict__ bias_out, long long rows, int S, int ldq, int split,
                                    const float* mask, long long mask_ld, uint4* __restrict__ mask_out, int B, int KS, int additive) {
  pdl_wait();
  pdl_launch();
  if (int(blockIdx.x) < split)
    bias_convert(bias, bias_out, rows, S, ldq, (long long)blockIdx.x * blockDim.x + threadIdx.x, (long long)split * blockDim.x);
  else
    mext_tiles(mask, mask_ld, mask_out, B, S, KS, additive, (long long)(blockIdx.x - split) * blockDim.x + threadIdx.x,
               (long long)(gridDim.x - split) * blockDim.x);
}

int launch_bias_transpose(Ctx* c, const float* in, bf16* out, int H, int S, int ldq, cudaStream_t st) {
  if (H <= 0 || S <= 0) return XFOLD_OK;
  const long long rows = (long long)H * S;
  long long blocks = (rows * ldq + 255) / 256;
  if (blocks > 16384) blocks = 16384;
  ProfScope ps(c, XFOLD_K_MASK_BIAS, st);
  launch_pdl(bias_convert_kernel, (int)blocks, 256, 0, st, in, reinterpret_cast<__half*>(out), rows, S, ldq);
  return check_launch(c, "bias_convert_kernel");
}

int launch_attn_prepare(Ctx* c, const float* bias, bf16* bias_out, int H, int S, int ldq, const float* mask, long long mask_ld,
                        bf16* mask_out, int B, int additive, cudaStream_t st) {
  if (H <= 0 || S <= 0 || B <= 0) return XFOLD_OK;
  const int KS = (S + 63) / 64;
  const long long rows = (long long)H * S, b1 = (rows * ldq + 255) / 256, b2 = ((long long)B * KS * 64 + 255) / 256;
  const int split = (int)(b1 > 16384 ? 16384 : b1), rest = (int)(b2 > 8192 ? 8192 : b2);
  ProfScope ps(c, XFOLD_K_MASK_BIAS, st);
  launch_pdl(attn_prepare_kernel, split + rest, 256, 0, st, bias, reinterpret_cast<__half*>(bias_out), rows, S, ldq, split, mask, mask_ld,
             reinterpret_cast<uint4*>(mask_out), B, KS, additive);
  return check_launch(c, "attn_prepare_kernel");
}

template <int D, bool ROWS>
static int launch_attn(Ctx* c, const CUtensorMap& tmq, const CUtensorMap& tmkv, const CUtensorMap& tmb, const AttnArgs& a,
                       cudaStream_t st) {
  using Cfg = AttnCfg<D, ROWS>;
  static bool attr_done[8] = {false};
  if (!attr_done[c->device & 7]) {
    cudaError_t e = cudaFuncSetAttribute(attn_kernel<D, ROWS>, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::SMEM);
    if (e != cudaSuccess) return fail(c, XFOLD_ERR_LAUNCH, "attention smem attribute: %s", cudaGetErrorString(e));
    attr_done[c->device & 7] = true;
  }
  const long long qt = (a.S + 127) / 128;
  const long long items = (ROWS ? qt : (qt + a.ns - 1) / a.ns) * a.heads * (ROWS ? (a.B + a.ns - 1) / a.ns : a.B);
  if (items * ((a.S + 63) / 64) >= (1ll << 30)) return fail(c, XFOLD_ERR_ARG, "attention: batch x heads x sequence too large for one launch");
  ProfScope ps(c, c->attn_tag, st);
  launch_pdl(attn_kernel<D, ROWS>, (int)(items < c->sm_count ? items : c->sm_count), Cfg::THREADS, Cfg::SMEM, st, tmq, tmkv, tmb, a);
  return check_launch(c, "attn_kernel");
}

// qkvg: projection buffer ([B][S][width], or [S][B][width] when transposed), q columns times log2(e); biasT: 16-bit
// [heads][query][ldq] holding FP16 values times log2(e); mext: tiles from launch_mext (one row of tiles per batch row, or
// one row for all when mext_rows == 1).
int launch_attention2(Ctx* c, const bf16* qkvg, int width, int S, int B, int transposed, int q_col0, int k_col0,
                      int v_col0, int g_col0, int heads, const bf16* biasT, int ldq, const bf16* mext, int mext_rows,
                      bf16* out, long long out_seq_stride, long long out_batch_stride, cudaStream_t st, int head_dim) {
  if (head_dim != 32 && head_dim != 64) return fail(c, XFOLD_ERR_ARG, "attention: head dimension must be 32 or 64");
  if ((width & 7) || (ldq & 7) || ((q_col0 | k_col0 | v_col0 | g_col0) & 7))
    return fail(c, XFOLD_ERR_ARG, "attention: width, column offsets and bias pitch must be multiples of 8");
  if (S <= 0 || B <= 0) return XFOLD_OK;
  AttnArgs a;
  a.S = S;
  a.B = B;
  a.heads = heads;
  a.q_col0 = q_col0;
  a.k_col0 = k_col0;
  a.v_col0 = v_col0;
  a.g_col0 = g_col0;
  a.qkvg = qkvg;
  a.seq_stride = transposed ? (long long)B * width : width;
  a.batch_stride = transposed ? width : (long long)S * width;
  a.mext = reinterpret_cast<const uint8_t*>(mext);
  a.mext_batch_stride = mext_rows == 1 ? 0 : (long long)((S + 63) / 64) * 1024;
  a.out = out;
  a.out_seq_stride = out_seq_stride;
  a.out_batch_stride = out_batch_stride;
  a.status = c->d_status;
  // Slots over batch rows where there are at least as many rows as slots (the pair bias is read once for three rows).
  // Otherwise over query tiles: two per item, or one where that leaves fewer waves of CTAs (a lone slot waits for its own
  // hand-overs, a pair takes about 1.3 times as long for twice the work).
  const bool rows = head_dim == 32 && B >= 3;
  const int qt = (S + 127) / 128;
  if (rows) a.ns = 3;
  else {
    const long long u1 = (long long)qt * heads * B, u2 = (long long)((qt + 1) / 2) * heads * B;
    const double t1 = double((u1 + c->sm_count - 1) / c->sm_count), t2 = 1.3 * double((u2 + c->sm_count - 1) / c->sm_count);
    a.ns = t2 < t1 ? 2 : 1;
  }
  const uint32_t nb = rows ? 3 : 1;
  const int sw = head_dim == 64 ? 128 : 64;
  CUtensorMap tmq, tmkv, tmb;
  const bool ok = make_tmap_bf16_3d(&tmq, qkvg, width, S, B, a.seq_stride, a.batch_stride, head_dim, 128, nb, sw) &&
                  make_tmap_bf16_3d(&tmkv, qkvg, width, S, B, a.seq_stride, a.batch_stride, head_dim, 64, nb, sw) &&
                  make_tmap_bf16_3d(&tmb, biasT, S, S, heads, ldq, (uint64_t)ldq * S, 64, 128, 1);
  if (!ok) return fail(c, XFOLD_ERR_ARG, "attention: cannot encode tensor maps");
  if (rows) return launch_attn<32, true>(c, tmq, tmkv, tmb, a, st);
  return head_dim == 32 ? launch_attn<32, false>(c, tmq, tmkv, tmb, a, st) : launch_attn<64, false>(c, tmq, tmkv, tmb, a, st);
}

}  // namespace xf
