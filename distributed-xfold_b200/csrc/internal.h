// Host-side declarations shared by the translation units of libxfold_b200.so.
#pragma once
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <mutex>
#include <utility>
#include <vector>

#include "../../include/xfold_b200.h"

namespace xf {

typedef __nv_bfloat16 bf16;

struct ProfRec {
  cudaEvent_t a, b;
  int tag;
};

// Everything below that changes after creation (counters, the error text, what a call sets for its launches, the second
// stream and its events) belongs to the call that holds `mu`: every entry point takes it (CallLock) while it issues its
// launches, so several host threads may use one context.  The launches of a call are then together in its stream, and calls
// of several threads on one stream may use the same scratch.
struct Ctx {
  std::mutex mu;
  int device = 0;
  int sm_count = 148;
  int* d_status = nullptr;  // one word: first in-kernel error code (0 = ok)
  char last_error[256] = {0};
  long long launch_count = 0;  // kernels launched through this context
  int prof_on = 0;             // when set, every launch is bracketed by a pair of CUDA events
  int attn_tag = XFOLD_K_ATTENTION;  // kernel class the attention launchers account their launch to
  // Set while an operator made of several kernels runs: its weights are older than its first kernel, so that the later
  // ones may fetch them before their predecessor has finished.
  int static_weights = 0;
  // While a stage's exchange kernels are meant to run beside its GEMMs (second stream), the persistent GEMMs leave some
  // SMs free and the exchange kernels are sized for them: a GEMM CTA fills its SM, so without free SMs the two serialise.
  int gemm_sms = 0;      // SMs a GEMM launch may take (0: all)
  int peer_cta_cap = 0;  // CTAs of a peer exchange kernel (0: its own default)
  std::vector<ProfRec> prof_recs, prof_pool;
  // Second stream of the one-GPU trunk: the single representation's kernels of a block run beside the next block's.  (Events
  // are captured by the waits as they are issued: the next call may use them again.)
  cudaStream_t side = nullptr;
  cudaEvent_t ev_fork = nullptr, ev_join = nullptr, ev_pl = nullptr;
};

struct CallLock {
  std::lock_guard<std::mutex> lock;
  explicit CallLock(Ctx* c) : lock(c->mu) {}
};

// Brackets one kernel launch with events on its stream while profiling is enabled, and counts it.
struct ProfScope {
  Ctx* c;
  cudaStream_t st;
  ProfRec r;
  bool on;
  ProfScope(Ctx* c_, int tag, cudaStream_t st_) : c(c_), st(st_), on(c_->prof_on != 0) {
    c->launch_count++;
    if (!on) return;
    if (!c->prof_pool.empty()) {
      r = c->prof_pool.back();
      c->prof_pool.pop_back();
    } else {
      cudaEventCreate(&r.a);
      cudaEventCreate(&r.b);
    }
    r.tag = tag;
    cudaEventRecord(r.a, st);
  }
  ~ProfScope() {
    if (!on) return;
    cudaEventRecord(r.b, st);
    c->prof_recs.push_back(r);
  }
};

struct StaticWeights {
  Ctx* c;
  int before;
  explicit StaticWeights(Ctx* c_) : c(c_), before(c_->static_weights) { c->static_weights = 1; }
  ~StaticWeights() { c->static_weights = before; }
};

// returns XFOLD_OK or sets ctx->last_error and returns a status code
int fail(Ctx* c, int code, const char* fmt, ...);
int check_launch(Ctx* c, const char* what);

// A kernel without room to round the start of its shared memory up to 1 KB, where swizzled tiles begin, counts on the dynamic
// part's own alignment: nothing static may stand in front of it.
template <typename... KArgs>
bool only_dynamic_smem(void (*kern)(KArgs...)) {
  cudaFuncAttributes at;
  return cudaFuncGetAttributes(&at, kern) == cudaSuccess && at.sharedSizeBytes == 0;
}

// Launch that may start while the previous kernel of the stream still runs (see pdl_wait in umma.cuh).
template <typename... KArgs, typename... Args>
cudaError_t launch_pdl(void (*kern)(KArgs...), dim3 grid, int block, size_t smem, cudaStream_t st, Args&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kern, std::forward<Args>(args)...);
}

// The same with clusters of `cluster` CTAs.
template <typename... KArgs, typename... Args>
cudaError_t launch_pdl_cluster(void (*kern)(KArgs...), int grid, int cluster, int block, size_t smem, cudaStream_t st,
                               Args&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  at[1].id = cudaLaunchAttributeClusterDimension;
  at[1].val.clusterDim.x = cluster;
  at[1].val.clusterDim.y = at[1].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 2;
  return cudaLaunchKernelEx(&cfg, kern, std::forward<Args>(args)...);
}

// ---- tensor maps --------------------------------------------------------------------------
// bf16 tensor of rank 3, innermost stride 1; s1/s2 are strides of dims 1/2 in ELEMENTS.
// 128-byte swizzle (64-byte for boxes whose rows are 64 bytes, 0 for none), zero fill outside the extents.
bool make_tmap_bf16_3d(CUtensorMap* m, const void* base, uint64_t d0, uint64_t d1, uint64_t d2, uint64_t s1,
                       uint64_t s2, uint32_t b0, uint32_t b1, uint32_t b2, int swizzle_bytes = 128);

// ---- GEMM ---------------------------------------------------------------------------------
// COLS: PLAIN with column vectors or columns that leave in another form.  A kernel of its own: what PLAIN does not need would
// cost it instruction fetches (contraction of 37 tokens 4.0 -> 3.5 us).
enum GemmEpi : int { EPI_PLAIN = 0, EPI_GATE_RESID = 1, EPI_SWIGLU = 2, EPI_COLS = 3 };

struct GemmArgs {
  int M = 0, N = 0, K = 0, batches = 1;
  int tiles_m = 0, tiles_n = 0;
  int b_batched = 0;
  int static_b = 0;    // B is written by no kernel that may still run: its first tiles may be fetched before pdl_wait
  int mn_major = 0;    // operands are stored [k][m] and [k][n] (tensor maps: inner dim = m / n, boxes of 64 x 64)
  // output (row-major, all epilogues)
  bf16* out = nullptr;
  long long ldo = 0, out_batch_stride = 0;
  const float* col_bias = nullptr;  // COLS: (product + col_bias) * col_scale; N of them for each entry of the batch
  const float* col_scale = nullptr;
  int f16_col0 = 0, f16_col1 = 0;  // COLS: output columns [f16_col0, f16_col1) are stored as fp16 (multiples of 32)
  int log2e_cols = 0;  // COLS: output columns [0, log2e_cols) times log2(e) (a multiple of 32): the attention works in base 2
  const bf16* resid = nullptr;
  long long ldr = 0;
  const bf16* gate = nullptr;
  long long ldg = 0;
  const bf16* row_gate = nullptr;  // GATE_RESID: gate indexed by (m % row_gate_mod), for conditioning shared by samples
  int row_gate_mod = 0;
  int* status = nullptr;
};

// A is described by tmA (box 64 x 128 rows), B by tmB (box 64 x BN rows; SWIGLU below 256: 64 x BN / 2); BN is 64, 128 or
// 256 (GATE_RESID up to 128, SWIGLU from 128).
int launch_gemm(Ctx* c, int epi, int bn, const CUtensorMap& tmA, const CUtensorMap& tmB, const GemmArgs& a,
                cudaStream_t st);
// GATE_RESID products of few tiles and a long K: `split` (2, 4, 8) CTAs share a tile 64 columns wide and add their parts of
// K (gemm_split.cu).  N a multiple of 8, pointers of the epilogue 16-byte aligned, leading dimensions multiples of 8.
int launch_gemm_split(Ctx* c, int split, const CUtensorMap& tmA, const CUtensorMap& tmB, const GemmArgs& a, cudaStream_t st);
int gemm_split(const Ctx* c, long long M, int N, int K);
// the tile width BN to use for an [M x N x K] product (see gemm.cu)
int gemm_tile_n(const Ctx* c, long long M, int N, int K, int batches, int widest, int narrowest);

}  // namespace xf
