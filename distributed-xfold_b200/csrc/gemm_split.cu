// out = [sigmoid(gate) *] (A B^T) + resid for products with few output tiles and a long K: the CTAs of a cluster share one
// tile, each takes a part of K, and the parts are added through distributed shared memory.
//
// What bounds such a product is one CTA's latency, not a rate: a 64-wide step of K cost about 0.25 us when this was measured
// (0.14 since the producers lost their lane branches; the operands' trip through a ring of a few stages, four products, the
// hand-over), so that K = 1536 takes 6 us on a dozen SMs while the others idle.  With K cut into S parts a CTA has most of its
// part in flight at once.  The exchange moves each fp32 partial sum once: the 128 rows of the tile are dealt out to the S CTAs,
// every CTA stores its rows of another's share straight from tensor memory into that CTA's shared memory, and after one cluster
// barrier each CTA adds S addends in the order of their ranks (the result does not depend on timing) and runs the epilogue on
// its 128 / S rows.
// Measured on the diffusion transformer's two output projections (768 columns, K = 1024 and 1536, 24 blocks of a step):
// 77 rows 1215 -> 986 us with S = 8, 231 rows 1195 -> 1014 with 4, 384 rows 1406 -> 1230 and 512 rows 1467 -> 1314 with 2.
// The projections before them (K = 768, 24 to 64 tiles) gain nothing: what the shorter loop saves the exchange costs.
//
//   warp 0 TMA producer, warp 1 tcgen05.mma issuer (both warp-uniform, see attention.cu), warps 2..9 exchange and epilogue.
#include "internal.h"
#include "umma.cuh"

namespace xf {

namespace {

constexpr int THREADS = 320;

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }
// address of the same shared-memory location in the cluster's CTA `rank`
__device__ __forceinline__ uint32_t cluster_addr(uint32_t saddr, uint32_t rank) {
  uint32_t a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(saddr), "r"(rank));
  return a;
}
__device__ __forceinline__ void cluster_store4(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("st.shared::cluster.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}

constexpr int BN = 64;
constexpr uint32_t A_BYTES = 128 * 64 * 2;
constexpr uint32_t STAGE_BYTES = A_BYTES + BN * 64 * 2;
constexpr int MAX_STAGES = 6;
constexpr uint32_t SLOT_BYTES = 128 * BN * 4;  // [source rank][own row][BN] fp32, 16-byte pieces XORed with row % 8
constexpr uint32_t smem_bytes(int stages) { return stages * STAGE_BYTES + SLOT_BYTES + 256 + 1024; }

}  // namespace

__global__ void __launch_bounds__(THREADS, 1)
gemm_split_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const GemmArgs p,
                  const int split, const int stages) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw_addr = smem_u32(smem_raw);
  uint8_t* smem = smem_raw + (((raw_addr + 1023u) & ~1023u) - raw_addr);
  uint8_t* slots = smem + stages * STAGE_BYTES;
  uint64_t* full = reinterpret_cast<uint64_t*>(slots + SLOT_BYTES);
  uint64_t* empty = full + MAX_STAGES;
  uint64_t* tfull = empty + MAX_STAGES;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tfull + 1);
  volatile int* cta_abort = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = __reduce_max_sync(0xffffffffu, threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  const AbortCtx ab{cta_abort, p.status};
  if (threadIdx.x == 0) {
    for (int s = 0; s < stages; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    mbar_init(tfull, 1);
    *cta_abort = 0;
    fence_barrier_init();
    tma_prefetch_desc(&tmA);
    tma_prefetch_desc(&tmB);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, BN);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = __reduce_max_sync(0xffffffffu, *tmem_slot);
  cluster_arrive();  // this CTA runs: its shared memory may be written

  const int rank = (int)cluster_rank();
  const int tile = blockIdx.x / split, tn = tile % p.tiles_n, tm = tile / p.tiles_n;
  const int KB = (p.K + 63) / 64;
  const int kb0 = rank * KB / split, kb1 = (rank + 1) * KB / split;  // split <= KB: never empty

  if (warp == 0) {
    const uint32_t go = elect_one();
    auto load_b = [&](int s, int kb) {
      mbar_arrive_expect_tx_if(go, &full[s], STAGE_BYTES);
      tma_load_3d_if(go, smem + s * STAGE_BYTES + A_BYTES, &tmB, &full[s], kb * 64, tn * BN, 0);
    };
    int pre = 0;  // stages whose weights are on their way before the wait for the previous kernel
    if (p.static_b)
      for (; pre < stages && kb0 + pre < kb1; ++pre) load_b(pre, kb0 + pre);
    pdl_wait();
    pdl_launch();
    int s = 0;
    uint32_t phase = 0;
    for (int kb = kb0; kb < kb1; ++kb) {
      if (kb - kb0 >= pre) {
        if (!mbar_wait_warp(&empty[s], phase ^ 1u, ab, XF_ERR_WAIT_EMPTY)) break;
        load_b(s, kb);
      }
      tma_load_3d_if(go, smem + s * STAGE_BYTES, &tmA, &full[s], kb * 64, tm * 128, 0);
      if (++s == stages) { s = 0; phase ^= 1u; }
    }
    cluster_wait();
  } else if (warp == 1) {
    pdl_wait();
    pdl_launch();
    const uint32_t go = elect_one();
    const uint32_t idesc = make_idesc(128, BN);
    int s = 0;
    uint32_t phase = 0;
    for (int kb = kb0; kb < kb1; ++kb) {
      if (!mbar_wait_warp(&full[s], phase, ab, XF_ERR_WAIT_FULL)) break;
      tc_fence_after();
      const uint32_t sA = smem_u32(smem + s * STAGE_BYTES);
      const uint64_t ad = make_sdesc(sA, 16, 1024), bd = make_sdesc(sA + A_BYTES, 16, 1024);
#pragma unroll
      for (int k = 0; k < 4; ++k) umma_ss_if(go, tmem_base, ad + 2 * k, bd + 2 * k, idesc, kb > kb0 || k ? 1u : 0u);
      umma_commit_if(go, &empty[s]);
      if (++s == stages) { s = 0; phase ^= 1u; }
    }
    umma_commit_if(go, tfull);
    cluster_wait();
  } else {
    constexpr int G = BN / 8;            // 16-byte pieces of an output row
    constexpr int ITEMS = 64 * G / 256;  // pieces per thread with two CTAs, the most there can be
    const int rows = 128 / split;
    const int e = threadIdx.x - 64;
    pdl_wait();
    pdl_launch();
    // what the epilogue adds and multiplies with travels beside the products (through L2: the residual is also the output)
    const bf16* gate = p.row_gate ? p.row_gate : p.gate;
    uint4 res[ITEMS], gat[ITEMS];
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
      const int idx = e + i * 256, rl = idx / G, col = tn * BN + idx % G * 8;
      const long long m = (long long)tm * 128 + rank * rows + rl;
      res[i] = gat[i] = make_uint4(0, 0, 0, 0);
      if (rl < rows && m < p.M && col < p.N) {
        if (p.resid) res[i] = __ldcg(reinterpret_cast<const uint4*>(p.resid + m * p.ldr + col));
        if (gate) gat[i] = __ldcg(reinterpret_cast<const uint4*>(gate + (p.row_gate ? m % p.row_gate_mod : m) * p.ldg + col));
      }
    }
    const int q = warp & 3, ch = (warp - 2) >> 2, row = q * 32 + lane;
    const bool okay = mbar_wait_warp(tfull, 0, ab, XF_ERR_WAIT_TMEM_FULL);
    tc_fence_after();
    cluster_wait();
    if (okay) {
      const int dest = row / rows, rl = row - dest * rows;
      const uint32_t base = cluster_addr(smem_u32(slots), dest) + (uint32_t(rank * rows + rl) * BN) * 4;
      uint32_t r[32];
      tmem_ld32(tmem_base + ch * 32 + (uint32_t(q * 32) << 16), r);
      tmem_ld_wait();
      if ((long long)tm * 128 + row < p.M) {
#pragma unroll
        for (int k = 0; k < 8; ++k)
          cluster_store4(base + (uint32_t((ch * 8 + k) ^ (rl & 7)) << 4), r[4 * k], r[4 * k + 1], r[4 * k + 2], r[4 * k + 3]);
      }
    }
    __syncwarp();
    cluster_arrive();
    cluster_wait();
    if (okay) {
#pragma unroll
      for (int i = 0; i < ITEMS; ++i) {
        const int idx = e + i * 256, rl = idx / G, g = idx % G, col = tn * BN + g * 8;
        const long long m = (long long)tm * 128 + rank * rows + rl;
        if (rl >= rows || m >= p.M || col >= p.N) continue;
        float v[8] = {};
        for (int s = 0; s < split; ++s) {
          const uint8_t* src = slots + uint32_t(s * rows + rl) * BN * 4;
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const float4 f = *reinterpret_cast<const float4*>(src + (uint32_t((g * 2 + h) ^ (rl & 7)) << 4));
            v[4 * h] += f.x; v[4 * h + 1] += f.y; v[4 * h + 2] += f.z; v[4 * h + 3] += f.w;
          }
        }
        const uint32_t wg[4] = {gat[i].x, gat[i].y, gat[i].z, gat[i].w}, wr[4] = {res[i].x, res[i].y, res[i].z, res[i].w};
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          if (gate) {
            v[2 * k] *= sigmoidf_fast(bf16_lo(wg[k]));
            v[2 * k + 1] *= sigmoidf_fast(bf16_hi(wg[k]));
          }
          v[2 * k] += bf16_lo(wr[k]);
          v[2 * k + 1] += bf16_hi(wr[k]);
        }
        *reinterpret_cast<uint4*>(p.out + m * p.ldo + col) =
            make_uint4(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]), pack_bf16x2(v[4], v[5]), pack_bf16x2(v[6], v[7]));
      }
    }
  }
  if (warp < 2) {
    __syncwarp();
    cluster_arrive();
    cluster_wait();
  }
  tc_fence_before();
  __syncthreads();
  if (*cta_abort && threadIdx.x == 0) {
    // give TMA copies that were already in flight time to land before the CTA's memory is released
    const long long t0 = clock64();
    while (clock64() - t0 < 2000000) {}
  }
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, BN);
  }
}

int launch_gemm_split(Ctx* c, int split, const CUtensorMap& tmA, const CUtensorMap& tmB, const GemmArgs& a, cudaStream_t st) {
  static bool attr_done[8] = {false};
  if (!attr_done[c->device & 7]) {
    cudaError_t e = cudaFuncSetAttribute(gemm_split_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes(MAX_STAGES));
    if (e != cudaSuccess) return fail(c, XFOLD_ERR_LAUNCH, "gemm smem attribute: %s", cudaGetErrorString(e));
    attr_done[c->device & 7] = true;
  }
  const int KB = (a.K + 63) / 64, most = (KB + split - 1) / split;
  const int stages = most < MAX_STAGES ? most : MAX_STAGES;
  ProfScope ps(c, XFOLD_K_LINEAR_GATE_RESID, st);
  launch_pdl_cluster(gemm_split_kernel, a.tiles_m * a.tiles_n * split, split, THREADS, smem_bytes(stages), st, tmA, tmB, a,
                     split, stages);
  return check_launch(c, "gemm_split_kernel");
}

// The number of CTAs that share a tile (64 columns wide); 1: no split.  At least two steps of K each (below that the
// exchange costs more than the loop), and no more clusters than run at once: pairs of SMs take any grid up to the chip,
// larger clusters have to fit into the GPCs, so an eighth of the SMs is counted out.  A second wave undoes the gain: 36 tiles
// of four CTAs take 1.04x the time of the unsplit ones.
int gemm_split(const Ctx* c, long long M, int N, int K) {
  const long long tiles = (M + 127) / 128 * ((N + 63) / 64);
  const int kb = (K + 63) / 64;
  const int sms = c->gemm_sms > 0 && c->gemm_sms < c->sm_count ? c->gemm_sms : c->sm_count;
  int s = 8;
  while (s > 1 && (kb < 2 * s || tiles * s > (s > 2 ? sms - sms / 8 : sms))) s /= 2;
  return s;
}

}  // namespace xf
