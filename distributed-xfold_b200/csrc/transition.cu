// Transition of the pair representation in one kernel:  x += W2 swiglu(W1 LN(x))  for rows of 128, F hidden units
// (csrc/Alpha_Attention.cpp:72-92, kernel_test/transition.py:22-48 state the operator).
//
// Per tile of 128 rows at F = 512: 25 M multiply-adds (6100 clocks of the tensor core), 65536 sigmoids (4096 of the
// special-function unit) and 1056 KB through shared memory (8450 clocks at 128 bytes each): operands of the products 640 KB,
// weights on arrival 192 (384 KB in all, two tiles share each block of them), x, its LayerNorm and the result 224.  The only HBM
// traffic is x itself.  1024 x 1024 rows take 412 us at 1965 MHz, 14 600 clocks per tile, and 470 to 480 at the 1710 MHz of the
// power limit: shared memory is the nearest bound, at 58 %.  As three launches (LayerNorm, SwiGLU GEMM, output GEMM) the
// normalised rows and the hidden activations made six passes over 128 and 512 columns: 0.84 ms.
//
// Persistent CTAs, a pair of tiles (A, B) of 128 rows at a time, hidden units in blocks of 64; per tile
//     D1 = LN(x) W1(block)^T   [128 x (64 SiLU | 64 linear)]      tensor memory
//     h  = silu(D1a) * D1b     bf16, tensor memory, over the D1 it comes from
//     D2 += h W2(block)^T      [128 x 128]                        tensor memory
//   warp 0         : TMA -- x tiles, weight blocks of 32 KB (W1, free after D1) and 16 KB (W2), two of each
//   warp 1         : tcgen05.mma issuer, the tiles in turn: D2 of a block and right behind it D1 of the next, which goes over
//                    the h that D2 reads (products of one issuer execute in order)
//   warps 2 - 9    : LayerNorm in place, one thread per row
//   warps 10 - 17  : one set of four per tile: D1 -> h; finally D2 + x -> a staging tile in two halves, which leave by TMA
// With h in tensor memory 256 KB fewer of a tile's 1312 go through shared memory.  (h in shared memory, D1 a block ahead of it:
// 0.54 ms in the trunk of 1024 tokens, now 0.50.  Sixteen warps for D1 -> h: no gain.)
// With no more tiles than SMs a CTA takes one tile: its blocks go through the two accumulators in turn, each with its set of
// warps, D1 two blocks ahead of D2, and a set takes one half of the result.  (One accumulator and one set: four
// blocks of the trunk at 37 tokens 392 us instead of 379, at 100 tokens 485 instead of 471.)
#include "internal.h"
#include "stages.h"
#include "umma.cuh"

namespace xf {

constexpr uint32_t TR_TILE = 32768;                       // [2 halves][128 rows][64 columns], swizzled
constexpr uint32_t TR_W1 = 32768, TR_W2 = 16384;          // a block's weights: [2 K halves][128 rows][64], [128 rows][64]
constexpr uint32_t TR_H = 16384;                          // a tile's staging, [128 rows][64 columns]
constexpr uint32_t TR_OFF_N = 0, TR_OFF_W1 = 2 * TR_TILE, TR_OFF_W2 = TR_OFF_W1 + 2 * TR_W1, TR_OFF_H = TR_OFF_W2 + 2 * TR_W2,
                   TR_OFF_GB = TR_OFF_H + 2 * TR_H, TR_OFF_BAR = TR_OFF_GB + 1024, TR_SMEM = TR_OFF_BAR + 256 + 1024;
constexpr int TR_THREADS = 18 * 32;
static_assert(TR_SMEM <= 232448, "shared memory");

struct TransitionArgs {
  const float *gamma, *beta;
  const bf16* x;
  long long rows;
  int items, pair, blocks;  // items of one tile (pair = 0) or two; hidden blocks of 64
  int static_w;             // see GemmArgs::static_b
  int update_only;          // out = the update alone (x is not added)
  int* status;
};

__global__ void __launch_bounds__(TR_THREADS, 1)
transition_kernel(const __grid_constant__ CUtensorMap tmx, const __grid_constant__ CUtensorMap tmo,
                  const __grid_constant__ CUtensorMap tmw1, const __grid_constant__ CUtensorMap tmw2, const TransitionArgs p) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw_addr = smem_u32(smem_raw);
  uint8_t* smem = smem_raw + (((raw_addr + 1023u) & ~1023u) - raw_addr);
  float* gb = reinterpret_cast<float*>(smem + TR_OFF_GB);  // gamma[128], beta[128]
  uint64_t* x_full = reinterpret_cast<uint64_t*>(smem + TR_OFF_BAR);  // [tile] x has landed
  uint64_t* n_full = x_full + 2;     // [tile] normalised in place
  uint64_t* n_empty = n_full + 2;    // [tile] the item's last D1 product is complete
  uint64_t* w1_full = n_empty + 2;   // [2]
  uint64_t* w1_empty = w1_full + 2;  // [2] the block's D1 products are complete
  uint64_t* w2_full = w1_empty + 2;  // [2]
  uint64_t* w2_empty = w2_full + 2;  // [2] the block's D2 products are complete
  uint64_t* d1_full = w2_empty + 2;  // [tile]
  uint64_t* h_full = d1_full + 2;    // [tile] h stands over D1
  uint64_t* d2_full = h_full + 2;    // [tile]
  uint64_t* d2_empty = d2_full + 2;  // [tile]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(d2_empty + 2);
  volatile int* cta_abort = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int warp = int(__reduce_max_sync(0xffffffffu, threadIdx.x >> 5)), lane = threadIdx.x & 31;
  const AbortCtx ab{cta_abort, p.status};

  if (threadIdx.x == 0) {
    for (int s = 0; s < 2; ++s) {
      mbar_init(&x_full[s], 1);
      mbar_init(&n_full[s], 4);
      mbar_init(&n_empty[s], 1);
      mbar_init(&w1_full[s], 1);
      mbar_init(&w1_empty[s], 1);
      mbar_init(&w2_full[s], 1);
      mbar_init(&w2_empty[s], 1);
      mbar_init(&d1_full[s], 1);
      mbar_init(&h_full[s], 4);
      mbar_init(&d2_full[s], 1);
      mbar_init(&d2_empty[s], 4);
    }
    *cta_abort = 0;
    fence_barrier_init();
    tma_prefetch_desc(&tmx);
    tma_prefetch_desc(&tmo);
    tma_prefetch_desc(&tmw1);
    tma_prefetch_desc(&tmw2);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  if (!p.static_w) pdl_wait();  // the parameters read below may come from the kernel before
  if (threadIdx.x >= 64 && threadIdx.x < 192) {
    gb[threadIdx.x - 64] = p.gamma ? p.gamma[threadIdx.x - 64] : 1.f;
    gb[threadIdx.x + 64] = p.beta ? p.beta[threadIdx.x - 64] : 0.f;
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = __reduce_max_sync(0xffffffffu, *tmem_slot);  // D1 of A, B; D2 of A, B: 128 columns each
  const uint32_t base = smem_u32(smem);
  const int NBK = p.blocks, NT = p.pair ? 2 : 1;
  const int mine = (p.items - int(blockIdx.x) + int(gridDim.x) - 1) / int(gridDim.x);

  if (warp == 0) {
    const uint32_t go = elect_one();  // warp-uniform, like the issuers
    const long long nblk = (long long)mine * NBK;
    int hb1 = 0, hb2 = 0, t = blockIdx.x, xt = 0;
    bool okay = true;
    auto load_w1 = [&](long long i) {
      const uint32_t st = uint32_t(i) & 1u;
      if (!mbar_wait_warp(&w1_empty[st], ((uint32_t(i) >> 1) & 1u) ^ 1u, ab, XF_ERR_WAIT_EMPTY)) { okay = false; return; }
      mbar_arrive_expect_tx_if(go, &w1_full[st], TR_W1);
      uint8_t* sw = smem + TR_OFF_W1 + st * TR_W1;
      const int r0 = (hb1 >> 1) * 256 + (hb1 & 1) * 64;  // 64 SiLU units and their 64 linear partners
#pragma unroll
      for (int kh = 0; kh < 2; ++kh) {
        tma_load_3d_if(go, sw + kh * 16384, &tmw1, &w1_full[st], kh * 64, r0, 0);
        tma_load_3d_if(go, sw + kh * 16384 + 8192, &tmw1, &w1_full[st], kh * 64, r0 + 128, 0);
      }
      if (++hb1 == NBK) hb1 = 0;
    };
    auto load_w2 = [&](long long i) {
      const uint32_t st = uint32_t(i) & 1u;
      if (!mbar_wait_warp(&w2_empty[st], ((uint32_t(i) >> 1) & 1u) ^ 1u, ab, XF_ERR_WAIT_EMPTY)) { okay = false; return; }
      mbar_arrive_expect_tx_if(go, &w2_full[st], TR_W2);
      tma_load_3d_if(go, smem + TR_OFF_W2 + st * TR_W2, &tmw2, &w2_full[st], hb2 * 64, 0, 0);
      if (++hb2 == NBK) hb2 = 0;
    };
    load_w1(0);  // (weights that no kernel of the call writes: on their way before the wait for the previous kernel)
    pdl_wait();
    pdl_launch();
    // W2 runs one block behind W1, and the next item's x goes out with the item's last blocks: no load waits for a
    // buffer that is freed later than the one after it needs
    for (long long i = 0; i <= nblk && okay; ++i) {
      if (xt < mine && (long long)xt * NBK <= i) {  // i == first block of item xt: its W1 is on its way
        for (int s = 0; s < NT && okay; ++s) {
          if (!mbar_wait_warp(&n_empty[s], (uint32_t(xt) & 1u) ^ 1u, ab, XF_ERR_WAIT_EMPTY)) { okay = false; break; }
          mbar_arrive_expect_tx_if(go, &x_full[s], TR_TILE);
          uint8_t* sx = smem + TR_OFF_N + s * TR_TILE;
          const int r = (t * NT + s) * 128;
          tma_load_3d_if(go, sx, &tmx, &x_full[s], 0, r, 0);
          tma_load_3d_if(go, sx + 16384, &tmx, &x_full[s], 64, r, 0);
        }
        t += gridDim.x;
        ++xt;
      }
      if (okay && i > 0) load_w2(i - 1);
      if (okay && i + 1 < nblk) load_w1(i + 1);
    }
  } else if (warp == 1) {
    pdl_wait();
    pdl_launch();
    const uint32_t leader = elect_one() ? 1u : 0u;
    constexpr uint32_t idesc = make_idesc(128, 128);
    uint32_t g1 = 0, g2 = 0;  // blocks whose D1 / D2 have been issued
    // D1 of the next block, of tile `tile` into accumulator s (the products that read the h it goes over were issued before: in
    // order)
    auto d1 = [&](int s, int tile) {
      const uint64_t wd = make_sdesc(base + TR_OFF_W1 + (g1 & 1u) * TR_W1, 16, 1024);
      const uint64_t nd = make_sdesc(base + TR_OFF_N + tile * TR_TILE, 16, 1024);
#pragma unroll
      for (int kh = 0; kh < 2; ++kh)
#pragma unroll
        for (int j = 0; j < 4; ++j)
          umma_ss_if(leader, tmem_base + s * 128, nd + uint64_t(kh * 1024 + 2 * j), wd + uint64_t(kh * 1024 + 2 * j), idesc,
                     (kh | j) ? 1u : 0u);
      umma_commit_if(leader, &d1_full[s]);
    };
    auto w1_ready = [&]() { return mbar_wait_warp(&w1_full[g1 & 1u], (g1 >> 1) & 1u, ab, XF_ERR_WAIT_FULL); };
    bool okay = true;
    if (!p.pair && mine > 0) {
      // one tile: its blocks take the two accumulators in turn, D1 two blocks ahead of D2
      okay = mbar_wait_warp(&n_full[0], 0, ab, XF_ERR_WAIT_FULL);
      for (int hb = 0; hb < NBK + 2 && okay; ++hb) {
        const int s = hb & 1;
        if (hb >= 2) {
          const uint32_t b = g2 & 1u;
          if (!mbar_wait_warp(&w2_full[b], (g2 >> 1) & 1u, ab, XF_ERR_WAIT_FULL)) break;
          if (!mbar_wait_warp(&h_full[s], (g2 >> 1) & 1u, ab, XF_ERR_WAIT_FULL)) break;
          tc_fence_after();
          const uint64_t wd = make_sdesc(base + TR_OFF_W2 + b * TR_W2, 16, 1024);
#pragma unroll
          for (int j = 0; j < 4; ++j)
            umma_ts_if(leader, tmem_base + 256, tmem_base + s * 128 + j * 8, wd + uint64_t(2 * j), idesc, (g2 | uint32_t(j)) ? 1u : 0u);
          umma_commit_if(leader, &w2_empty[b]);
          ++g2;
        }
        if (hb < NBK) {
          if (!w1_ready()) break;
          tc_fence_after();
          d1(s, 0);
          umma_commit_if(leader, &w1_empty[g1 & 1u]);
          ++g1;
        }
      }
      umma_commit_if(leader, &d2_full[0]);
    }
    for (int it = 0; it < (p.pair ? mine : 0) && okay; ++it) {
      if (!w1_ready()) break;
      for (int s = 0; s < NT && okay; ++s) {
        okay = mbar_wait_warp(&n_full[s], uint32_t(it) & 1u, ab, XF_ERR_WAIT_FULL);
        if (!okay) break;
        tc_fence_after();
        d1(s, s);
      }
      if (!okay) break;
      umma_commit_if(leader, &w1_empty[g1 & 1u]);
      ++g1;
      for (int hb = 0; hb < NBK && okay; ++hb) {
        const uint32_t b = g2 & 1u;
        const bool more = hb + 1 < NBK;
        if (more && !w1_ready()) { okay = false; break; }
        if (!mbar_wait_warp(&w2_full[b], (g2 >> 1) & 1u, ab, XF_ERR_WAIT_FULL)) { okay = false; break; }
        const uint64_t wd = make_sdesc(base + TR_OFF_W2 + b * TR_W2, 16, 1024);
        for (int s = 0; s < NT && okay; ++s) {
          if (hb == 0 && !mbar_wait_warp(&d2_empty[s], (uint32_t(it) & 1u) ^ 1u, ab, XF_ERR_WAIT_TMEM_EMPTY)) { okay = false; break; }
          if (!mbar_wait_warp(&h_full[s], g2 & 1u, ab, XF_ERR_WAIT_FULL)) { okay = false; break; }
          tc_fence_after();
#pragma unroll
          for (int j = 0; j < 4; ++j)  // 16 hidden units = 8 columns of h
            umma_ts_if(leader, tmem_base + 256 + s * 128, tmem_base + s * 128 + j * 8, wd + uint64_t(2 * j), idesc, (hb | j) ? 1u : 0u);
          if (!more) umma_commit_if(leader, &d2_full[s]);
          else {
            d1(s, s);
            if (hb + 2 == NBK) umma_commit_if(leader, &n_empty[s]);
          }
        }
        umma_commit_if(leader, &w2_empty[b]);
        ++g2;
        if (more) {
          umma_commit_if(leader, &w1_empty[g1 & 1u]);
          ++g1;
        }
      }
    }
  } else if (warp < 10) {
    pdl_wait();
    pdl_launch();
    const int s = (warp - 2) >> 2, row = ((warp - 2) & 3) * 32 + lane;
    for (int it = 0; it < mine && s < NT; ++it) {
      if (!mbar_wait(&x_full[s], uint32_t(it) & 1u, ab, XF_ERR_WAIT_FULL)) break;
      float nmean, rstd;
      row_stats(smem + TR_OFF_N + s * TR_TILE, row, nmean, rstd);
      row_normalise(smem + TR_OFF_N + s * TR_TILE, row, nmean, rstd, gb);
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(&n_full[s]);
    }
  } else {
    pdl_wait();
    pdl_launch();
    const int s = (warp - 10) >> 2, quarter = warp & 3, row = quarter * 32 + lane;
    const uint32_t rsw = uint32_t(row & 7), laddr = tmem_base + s * 128 + (uint32_t(quarter * 32) << 16);
    uint8_t* sh = smem + TR_OFF_H + s * TR_H + row * 128;
    uint32_t g = 0;  // blocks of this set
    int t = blockIdx.x;
    // one tile: a set takes every other block, and one half of the result
    const int h0 = p.pair ? 0 : s, hstep = p.pair ? 1 : 2, tile = p.pair ? s : 0;
    const uint32_t daddr = tmem_base + 256 + tile * 128 + (uint32_t(quarter * 32) << 16);
    for (int it = 0; it < mine; ++it, t += gridDim.x) {
      for (int hb = h0; hb < NBK; hb += hstep, ++g) {
        mbar_wait(&d1_full[s], g & 1u, ab, XF_ERR_WAIT_TMEM_FULL);  // (a failed wait runs through: these warps meet at a barrier)
        tc_fence_after();
#pragma unroll
        for (int c2 = 0; c2 < 2; ++c2) {
          uint32_t ra[32], rb[32];
          tmem_ld32(laddr + c2 * 32, ra);
          tmem_ld32(laddr + 64 + c2 * 32, rb);
          tmem_ld_wait();
          uint32_t o[16];
#pragma unroll
          for (int e = 0; e < 16; ++e) {
            const float2 a = make_float2(__uint_as_float(ra[2 * e]), __uint_as_float(ra[2 * e + 1]));
            const float2 h = fmul2(fmul2(a, sigmoid2(a)), make_float2(__uint_as_float(rb[2 * e]), __uint_as_float(rb[2 * e + 1])));
            o[e] = pack_bf16x2(h.x, h.y);
          }
          tmem_st16(laddr + c2 * 16, o);  // over columns that have been read
        }
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&h_full[s]);
      }
      // the tile's result: D2 + x, through the staging tile, 64 columns at a time
      const long long tile_row = (long long)(t * NT + tile) * 128;
      const bool valid = tile_row + row < p.rows && !p.update_only;
      const uint4* xg = reinterpret_cast<const uint4*>(p.x + (tile_row + row) * 128);
#pragma unroll 1
      for (int hf = h0; hf < 2; hf += hstep) {
        uint4 xv[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) xv[q] = valid ? __ldcg(xg + hf * 8 + q) : make_uint4(0, 0, 0, 0);
        if (hf == h0) {
          mbar_wait(&d2_full[tile], uint32_t(it) & 1u, ab, XF_ERR_WAIT_TMEM_FULL);
          tc_fence_after();
        } else {
          if (quarter == 0 && lane == 0) tma_store_wait_read<0>();
          named_bar_sync(1 + s, 128);
        }
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          uint32_t r[32];
          tmem_ld32(daddr + hf * 64 + c * 32, r);
          tmem_ld_wait();
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const uint4 u = xv[q];
            const uint32_t w4[4] = {u.x, u.y, u.z, u.w};
            uint32_t o[4];
#pragma unroll
            for (int e = 0; e < 4; ++e)
              o[e] = pack_bf16x2(__uint_as_float(r[q * 8 + 2 * e]) + bf16_lo(w4[e]), __uint_as_float(r[q * 8 + 2 * e + 1]) + bf16_hi(w4[e]));
            *reinterpret_cast<uint4*>(sh + ((uint32_t(c * 4 + q) ^ rsw) << 4)) = make_uint4(o[0], o[1], o[2], o[3]);
            if (c == 0) xv[q] = valid ? __ldcg(xg + hf * 8 + 4 + q) : make_uint4(0, 0, 0, 0);
          }
        }
        if (hf == 1) {
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&d2_empty[s]);
        }
        fence_proxy_async_smem();
        named_bar_sync(1 + s, 128);
        if (quarter == 0 && lane == 0 && tile_row < p.rows) {
          tma_store_3d(&tmo, smem + TR_OFF_H + s * TR_H, hf * 64, (int)tile_row, 0);
          tma_store_commit();
        }
      }
      if (quarter == 0 && lane == 0) tma_store_wait_read<0>();
      named_bar_sync(1 + s, 128);  // the staging tile is free for the next item
    }
    if (quarter == 0 && lane == 0) tma_store_wait_all();
  }

  tc_fence_before();
  __syncthreads();
  if (*cta_abort && threadIdx.x == 0) {
    const long long t0 = clock64();
    while (clock64() - t0 < 2000000) {}
  }
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

// x, out: [rows][128]; w1: [2F][128] in groups of [128 SiLU | 128 linear] rows, w2: [128][F]
int launch_transition128(Ctx* c, const bf16* x, bf16* out, long long rows, int F, const float* gamma, const float* beta,
                         const bf16* w1, const bf16* w2, int static_w, int update_only, cudaStream_t st) {
  CUtensorMap tmx, tmo, tmw1, tmw2;
  if (!make_tmap_bf16_3d(&tmx, x, 128, rows, 1, 128, (uint64_t)128 * rows, 64, 128, 1) ||
      !make_tmap_bf16_3d(&tmo, out, 128, rows, 1, 128, (uint64_t)128 * rows, 64, 128, 1) ||
      !make_tmap_bf16_3d(&tmw1, w1, 128, 2 * F, 1, 128, (uint64_t)256 * F, 64, 64, 1) ||
      !make_tmap_bf16_3d(&tmw2, w2, F, 128, 1, F, (uint64_t)128 * F, 64, 128, 1))
    return fail(c, XFOLD_ERR_ARG, "transition: cannot encode tensor maps (16-byte aligned bases?)");
  static bool attr_done[8] = {false};
  if (!attr_done[c->device & 7]) {
    cudaError_t e = cudaFuncSetAttribute(transition_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, TR_SMEM);
    if (e != cudaSuccess) return fail(c, XFOLD_ERR_LAUNCH, "transition smem attribute: %s", cudaGetErrorString(e));
    attr_done[c->device & 7] = true;
  }
  const int sms = c->gemm_sms > 0 && c->gemm_sms < c->sm_count ? c->gemm_sms : c->sm_count;
  const int tiles = (int)((rows + 127) / 128), pair = tiles > sms ? 1 : 0, items = pair ? (tiles + 1) / 2 : tiles;
  TransitionArgs a{gamma, beta, x, rows, items, pair, F / 64, static_w, update_only, c->d_status};
  ProfScope ps(c, XFOLD_K_LINEAR_SWIGLU, st);
  launch_pdl(transition_kernel, items < sms ? items : sms, TR_THREADS, TR_SMEM, st, tmx, tmo, tmw1, tmw2, a);
  return check_launch(c, "transition_kernel");
}

}  // namespace xf
