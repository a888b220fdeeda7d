// Thin device-side wrappers over the sm_100a instructions the kernels are built from:
// mbarrier, TMA (cp.async.bulk.tensor, never with cluster multicast), tcgen05 MMA / TMEM.
// Every wait is bounded: when it runs out it raises a CTA-wide abort flag and an error
// word in global memory, after which all later waits in the CTA return at once, the
// kernel drains and frees its TMEM, and the host reports a non-zero status.
#pragma once
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace xf {

typedef __nv_bfloat16 bf16;

// error codes written to the status word (0 = ok)
enum : int {
  XF_ERR_WAIT_FULL = 101,      // consumer never saw a TMA stage arrive
  XF_ERR_WAIT_EMPTY = 102,     // producer never got a stage back
  XF_ERR_WAIT_TMEM_FULL = 103, // epilogue never saw the accumulator commit
  XF_ERR_WAIT_TMEM_EMPTY = 104,
  XF_ERR_WAIT_ATTN = 105,
  XF_ERR_WAIT_PEER = 106,      // a peer rank never published its ready flag
};

#ifndef XF_PARK_NS
#define XF_PARK_NS 20000u  // suspend-time hint of a parked barrier wait
#endif
#ifndef XF_WAIT_CYCLES
#define XF_WAIT_CYCLES (3000000000LL)  // ~1.5 s at 1.9 GHz
#endif

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// ------------------------------------------------------------------------------------
// mbarrier
// ------------------------------------------------------------------------------------
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void fence_barrier_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void fence_proxy_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}

// Non-blocking probe of a phase (a test that succeeds has acquire semantics like a wait).  A barrier round trip
// costs ~250 cycles on this part, so a consumer probes the NEXT tile's barrier before it starts on the
// current tile and only falls back to the blocking wait when the probe failed.
__device__ __forceinline__ bool mbar_test_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}

// Shared by every role of a CTA: [0] = abort flag.
struct AbortCtx {
  volatile int* cta_abort;  // shared memory
  int* status;              // global memory
};

// Blocking form with a suspend-time hint: the hardware parks the thread until the phase completes or the hint
// (nanoseconds) runs out, instead of having it poll.  A polling loop of even one thread per warp takes issue
// slots from the warps that do the arithmetic on the same scheduler.
__device__ __forceinline__ bool mbar_try_wait_parked(uint64_t* bar, uint32_t parity, uint32_t hint_ns) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity), "r"(hint_ns)
      : "memory");
  return ok != 0;
}

// Bounded wait. Returns false when the CTA is aborting.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, const AbortCtx& ab, int code) {
  if (mbar_try_wait(bar, parity)) return true;
  if (*ab.cta_abort) return false;
  const long long t0 = clock64();
  // The loop body is what a waiting warp feeds the scheduler it shares with working warps: keep it to the probe and a
  // branch, and look at the abort flag and the clock only every 16th round.
  for (uint32_t spin = 1;; ++spin) {
    if (mbar_try_wait_parked(bar, parity, XF_PARK_NS)) return true;
    if ((spin & 15u) == 0) {
      if (*ab.cta_abort) return false;
      if (clock64() - t0 > XF_WAIT_CYCLES) {
        *ab.cta_abort = 1;
        atomicCAS(ab.status, 0, code);
        return false;
      }
    }
  }
}

// The same for a converged warp that stays converged: every branch depends on a vote.
__device__ __forceinline__ bool mbar_wait_warp(uint64_t* bar, uint32_t parity, const AbortCtx& ab, int code) {
  if (__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) return true;
  const long long t0 = clock64();
  for (uint32_t spin = 1;; ++spin) {
    if (__all_sync(0xffffffffu, mbar_try_wait_parked(bar, parity, XF_PARK_NS))) return true;
    if ((spin & 15u) == 0) {
      if (__any_sync(0xffffffffu, *ab.cta_abort != 0)) return false;
      if (__any_sync(0xffffffffu, clock64() - t0 > XF_WAIT_CYCLES)) {
        *ab.cta_abort = 1;
        atomicCAS(ab.status, 0, code);
        return false;
      }
    }
  }
}

// ------------------------------------------------------------------------------------
// TMA (tensor maps are passed as __grid_constant__ kernel parameters)
// ------------------------------------------------------------------------------------
__device__ __forceinline__ void tma_prefetch_desc(const CUtensorMap* m) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(m) : "memory");
}
// Forms for a converged warp, executed by the lanes with go != 0 (one): no branch around them, so that coordinates and
// addresses stay in uniform registers.
__device__ __forceinline__ void mbar_arrive_expect_tx_if(uint32_t go, uint64_t* bar, uint32_t bytes) {
  asm volatile(
      "{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %2, 0;\n\t"
      "@q mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n\t}" ::"r"(smem_u32(bar)), "r"(bytes), "r"(go)
      : "memory");
}
__device__ __forceinline__ void tma_load_3d_if(uint32_t go, void* dst, const CUtensorMap* m, uint64_t* bar, int c0, int c1,
                                               int c2) {
  asm volatile(
      "{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %6, 0;\n\t"
      "@q cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];\n\t}"
      ::"r"(smem_u32(dst)), "l"(m), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2), "r"(go)
      : "memory");
}

// the box on its way to L2 (no completion is signalled)
__device__ __forceinline__ void tma_prefetch_3d_if(uint32_t go, const CUtensorMap* m, int c0, int c1, int c2) {
  asm volatile(
      "{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %4, 0;\n\t"
      "@q cp.async.bulk.prefetch.tensor.3d.L2.global [%0, {%1, %2, %3}];\n\t}" ::"l"(m), "r"(c0), "r"(c1), "r"(c2), "r"(go)
      : "memory");
}

// TMA store shared -> global (bulk async-group completion); rows / columns outside the tensor are clipped
__device__ __forceinline__ void tma_store_3d(const CUtensorMap* m, const void* src, int c0, int c1, int c2) {
  asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.bulk_group [%0, {%2, %3, %4}], [%1];"
               ::"l"(m), "r"(smem_u32(src)), "r"(c0), "r"(c1), "r"(c2)
               : "memory");
}
__device__ __forceinline__ void tma_store_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
__device__ __forceinline__ void tma_store_3d_if(uint32_t go, const CUtensorMap* m, const void* src, int c0, int c1, int c2) {
  asm volatile(
      "{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %5, 0;\n\t"
      "@q cp.async.bulk.tensor.3d.global.shared::cta.bulk_group [%0, {%2, %3, %4}], [%1];\n\t}"
      ::"l"(m), "r"(smem_u32(src)), "r"(c0), "r"(c1), "r"(c2), "r"(go)
      : "memory");
}
template <int N>
__device__ __forceinline__ void tma_store_wait_read() {
  asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(N) : "memory");
}
// waits until this thread's bulk stores have been written (the .read form: only read out of shared memory)
__device__ __forceinline__ void tma_store_wait_all() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }
// (bar.sync counts a warp that is not converged once for each of its parts: a warp that stored with some lanes only converges first)
__device__ __forceinline__ void named_bar_sync(int id, int nthreads) {
  __syncwarp();
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(nthreads) : "memory");
}

// plain (untiled) bulk copy global -> shared, by the lanes with go != 0; addresses and size are multiples of 16 bytes
__device__ __forceinline__ void bulk_load_if(uint32_t go, void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile(
      "{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %4, 0;\n\t"
      "@q cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n\t}"
      ::"r"(smem_u32(dst)), "l"(src), "r"(bytes), "r"(smem_u32(bar)), "r"(go)
      : "memory");
}

// ------------------------------------------------------------------------------------
// tcgen05: TMEM allocation, MMA, commit, loads
// ------------------------------------------------------------------------------------
__device__ __forceinline__ void tmem_alloc(uint32_t* smem_dst, uint32_t ncols) {  // whole warp
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_dst)), "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {  // whole warp
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// D[tmem] (+)= A[smem] * B[smem]; bf16 inputs, fp32 accumulate; issued by ONE thread.
__device__ __forceinline__ void umma_ss(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                        uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(d_tmem), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// The same, issued by the lanes with go != 0 (one, elected by the caller) of a converged warp: no branch, so that operands
// can stay in uniform registers.
__device__ __forceinline__ void umma_ss_if(uint32_t go, uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                           uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.b32 p, %4, 0;\n\tsetp.ne.b32 q, %5, 0;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(d_tmem), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(go)
      : "memory");
}
// D[tmem] (+)= A[tmem] * B[smem]: A is read from tensor memory (lane = row, each 32-bit column holds two
// consecutive 16-bit K elements), so an operand produced by the CUDA cores never passes through shared memory.
__device__ __forceinline__ void umma_ts_if(uint32_t go, uint32_t d_tmem, uint32_t a_tmem, uint64_t bdesc, uint32_t idesc,
                                           uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.b32 p, %4, 0;\n\tsetp.ne.b32 q, %5, 0;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(d_tmem), "r"(a_tmem), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(go)
      : "memory");
}
// The same with descriptors given as two words: only the low one moves between tiles.
__device__ __forceinline__ void umma_ss_lo_if(uint32_t go, uint32_t d_tmem, uint32_t alo, uint32_t ahi, uint32_t blo, uint32_t bhi,
                                              uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t.reg .b64 a, b;\n\tmov.b64 a, {%1, %2};\n\tmov.b64 b, {%3, %4};\n\t"
      "setp.ne.b32 p, %6, 0;\n\tsetp.ne.b32 q, %7, 0;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %5, p;\n\t}"
      ::"r"(d_tmem), "r"(alo), "r"(ahi), "r"(blo), "r"(bhi), "r"(idesc), "r"(accumulate), "r"(go)
      : "memory");
}
__device__ __forceinline__ void umma_ts_lo_if(uint32_t go, uint32_t d_tmem, uint32_t a_tmem, uint32_t blo, uint32_t bhi, uint32_t idesc,
                                              uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t.reg .b64 b;\n\tmov.b64 b, {%2, %3};\n\t"
      "setp.ne.b32 p, %5, 0;\n\tsetp.ne.b32 q, %6, 0;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], b, %4, p;\n\t}"
      ::"r"(d_tmem), "r"(a_tmem), "r"(blo), "r"(bhi), "r"(idesc), "r"(accumulate), "r"(go)
      : "memory");
}
__device__ __forceinline__ void umma_commit_if(uint32_t go, uint64_t* bar) {
  asm volatile(
      "{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %1, 0;\n\t"
      "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}"
      ::"r"(smem_u32(bar)), "r"(go)
      : "memory");
}
// Arrives (count 1) on the mbarrier once every MMA issued so far by this thread is done.
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
               : "memory");
}

// Instruction descriptor: bf16 x bf16 -> fp32, M x N tile; a_mn / b_mn = 1 for an MN-major operand.
// ab_f16 = 1: both operands are fp16 instead of bf16 (the two must have the same type for kind::f16).
__host__ __device__ constexpr uint32_t make_idesc(int M, int N, int a_mn = 0, int b_mn = 0, int ab_f16 = 0) {
  return (1u << 4)                          // D format fp32
         | ((ab_f16 ? 0u : 1u) << 7)        // A format: bf16 (1) or fp16 (0)
         | ((ab_f16 ? 0u : 1u) << 10)       // B format
         | (uint32_t(a_mn) << 15) | (uint32_t(b_mn) << 16)
         | (uint32_t(N >> 3) << 17) | (uint32_t(M >> 4) << 24);
}

// Shared-memory matrix descriptor, 128-byte swizzle.
//   K-major tile  [rows][64 bf16]  (one 128 B row per M/N index, 8-row groups of 1024 B):
//       lbo = 16 B (unused by the hardware for swizzled K-major), sbo = 1024 B
//   MN-major tile [k rows][64 bf16] (one 128 B row per K index):
//       lbo = byte distance between 64-element chunks along M/N, sbo = 1024 B (8 k-rows)
__device__ __forceinline__ uint64_t make_sdesc(uint32_t saddr, uint32_t lbo_bytes, uint32_t sbo_bytes) {
  uint64_t d = 0;
  d |= uint64_t((saddr & 0x3FFFFu) >> 4);
  d |= uint64_t((lbo_bytes >> 4) & 0x3FFFu) << 16;
  d |= uint64_t((sbo_bytes >> 4) & 0x3FFFu) << 32;
  d |= uint64_t(1) << 46;  // descriptor version (Blackwell)
  d |= uint64_t(2) << 61;  // SWIZZLE_128B
  return d;
}

// Un-swizzled K-major tile made of 8-row x 16-byte core matrices (128 B each, rows 16 B apart):
// lbo = byte distance between core matrices along K, sbo = between 8-row groups along M/N.
__device__ __forceinline__ uint64_t make_sdesc_noswizzle(uint32_t saddr, uint32_t lbo_bytes, uint32_t sbo_bytes) {
  uint64_t d = 0;
  d |= uint64_t((saddr & 0x3FFFFu) >> 4);
  d |= uint64_t((lbo_bytes >> 4) & 0x3FFFu) << 16;
  d |= uint64_t((sbo_bytes >> 4) & 0x3FFFu) << 32;
  d |= uint64_t(1) << 46;
  return d;
}

// 32 lanes x 32 columns of fp32: thread l of the warp receives row (lane base + l), columns c .. c+31.
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
      "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
        "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
        "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// ------------------------------------------------------------------------------------
// Programmatic dependent launch.  A kernel launched with the attribute (launch_pdl in internal.h) may start while its
// predecessor in the stream still runs; everything up to pdl_wait() -- barriers, tensor memory, weights that no kernel of
// the call writes -- overlaps the predecessor's tail.  Rules that keep it safe:
//   * every thread calls pdl_wait() before it touches anything a predecessor wrote or still reads, so that the completion
//     of a kernel implies the completion of all before it;
//     (what a kernel two or more places ahead wrote may be read, through L2, and what it read may be overwritten, before
//     pdl_wait(): the predecessor let this kernel start only after its own pdl_wait(); adaln_kernel and cond_ln_kernel do so)
//   * pdl_launch() comes after the tensor memory allocation (a successor that got the tensor memory first would wait for
//     this kernel, and this kernel for the tensor memory) and after pdl_wait(): L1 is invalidated when a kernel starts, and
//     a kernel two places ahead must not start while this kernel's predecessor still reads what this kernel overwrites;
//   * no kernel reads through L1 a buffer that it also writes, and no pointer to activations is const __restrict__: the
//     compiler treats such loads as invariant and may move them above pdl_wait().
// ------------------------------------------------------------------------------------
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// ------------------------------------------------------------------------------------
// misc math
// ------------------------------------------------------------------------------------
// sigmoid(x) = 0.5 * tanh(0.5 x) + 0.5: one MUFU op (tanh.approx, rel. error ~2^-11) instead of ex2 + rcp
__device__ __forceinline__ float sigmoidf_fast(float x) {
  float t;
  asm("tanh.approx.f32 %0, %1;" : "=f"(t) : "f"(0.5f * x));
  return fmaf(0.5f, t, 0.5f);
}
__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&v);
}
// two float32 FMAs in one instruction: d = a * b + c, element by element
__device__ __forceinline__ float2 ffma2(float2 a, float2 b, float2 c) {
  float2 d;
  asm("{\n\t.reg .b64 ra, rb, rc, rd;\n\tmov.b64 ra, {%2, %3};\n\tmov.b64 rb, {%4, %5};\n\tmov.b64 rc, {%6, %7};\n\t"
      "fma.rn.f32x2 rd, ra, rb, rc;\n\tmov.b64 {%0, %1}, rd;\n\t}"
      : "=f"(d.x), "=f"(d.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
  return d;
}
__device__ __forceinline__ float2 fadd2(float2 a, float2 b) {
  float2 d;
  asm("{\n\t.reg .b64 ra, rb, rd;\n\tmov.b64 ra, {%2, %3};\n\tmov.b64 rb, {%4, %5};\n\tadd.rn.f32x2 rd, ra, rb;\n\t"
      "mov.b64 {%0, %1}, rd;\n\t}" : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return d;
}
__device__ __forceinline__ float2 fmul2(float2 a, float2 b) {
  float2 d;
  asm("{\n\t.reg .b64 ra, rb, rd;\n\tmov.b64 ra, {%2, %3};\n\tmov.b64 rb, {%4, %5};\n\tmul.rn.f32x2 rd, ra, rb;\n\t"
      "mov.b64 {%0, %1}, rd;\n\t}" : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return d;
}
__device__ __forceinline__ float2 sigmoid2(float2 x) {  // sigmoidf_fast of a pair
  float2 t = fmul2(x, make_float2(0.5f, 0.5f));
  asm("tanh.approx.f32 %0, %0;\n\ttanh.approx.f32 %1, %1;" : "+f"(t.x), "+f"(t.y));
  return ffma2(make_float2(0.5f, 0.5f), t, make_float2(0.5f, 0.5f));
}
__device__ __forceinline__ float bf16_lo(uint32_t v) { return __uint_as_float(v << 16); }
__device__ __forceinline__ float bf16_hi(uint32_t v) { return __uint_as_float(v & 0xFFFF0000u); }

// true in exactly one lane of a converged warp
__device__ __forceinline__ bool elect_one() {
  uint32_t pred;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(pred));
  return pred != 0;
}
// Pieces of a LayerNorm over rows of bf16.  Mixed-precision adds take the packed halves as they are: once for the sum, once
// to centre.
__device__ __forceinline__ void sum2(uint32_t x, float2& s) {
  asm("{\n\t.reg .b16 l, h;\n\tmov.b32 {l, h}, %2;\n\tadd.rn.f32.bf16 %0, l, %0;\n\tadd.rn.f32.bf16 %1, h, %1;\n\t}"
      : "+f"(s.x), "+f"(s.y) : "r"(x));
}
__device__ __forceinline__ float2 centre2(uint32_t x, float nmean) {
  float2 v;
  asm("{\n\t.reg .b16 l, h;\n\tmov.b32 {l, h}, %2;\n\tadd.rn.f32.bf16 %0, l, %3;\n\tadd.rn.f32.bf16 %1, h, %3;\n\t}"
      : "=f"(v.x), "=f"(v.y) : "r"(x), "f"(nmean));
  return v;
}
// Row `row` of a [2 halves][128 rows][64 columns] 128-byte-swizzled tile of 128 bf16 columns, by one thread: statistics, then
// (x - mean) * rstd * gamma + beta in place; gb = gamma[128], beta[128].  Three passes over shared memory: holding the row
// would take 64 registers.
__device__ __forceinline__ uint4* row_piece(uint8_t* tile, int row, int g) {
  return reinterpret_cast<uint4*>(tile + (g >> 3) * 16384 + row * 128 + ((uint32_t(g & 7) ^ uint32_t(row & 7)) << 4));
}
__device__ __forceinline__ void row_stats(uint8_t* tile, int row, float& nmean, float& rstd) {
  float2 sm = make_float2(0.f, 0.f), sq = make_float2(0.f, 0.f);
#pragma unroll
  for (int g = 0; g < 16; ++g) {
    const uint4 u = *row_piece(tile, row, g);
    sum2(u.x, sm); sum2(u.y, sm); sum2(u.z, sm); sum2(u.w, sm);
  }
  nmean = -(sm.x + sm.y) * (1.f / 128);
#pragma unroll
  for (int g = 0; g < 16; ++g) {
    const uint4 u = *row_piece(tile, row, g);
    const uint32_t w4[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float2 v = centre2(w4[e], nmean);
      sq = ffma2(v, v, sq);
    }
  }
  rstd = rsqrtf((sq.x + sq.y) * (1.f / 128) + 1e-5f);
}
// The same by two threads of a warp, lanes l and l + 16, with half a row each in registers: xr = columns [64 half, 64 half + 64).
__device__ __forceinline__ void load_half_row(uint8_t* tile, int row, int half, uint32_t (&xr)[32]) {
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    const uint4 u = *row_piece(tile, row, half * 8 + q);
    xr[q * 4] = u.x; xr[q * 4 + 1] = u.y; xr[q * 4 + 2] = u.z; xr[q * 4 + 3] = u.w;
  }
}
__device__ __forceinline__ void half_row_stats(const uint32_t (&xr)[32], float& nmean, float& rstd) {
  float2 sm[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
#pragma unroll
  for (int e = 0; e < 32; ++e) sum2(xr[e], sm[e & 1]);
  float s = (sm[0].x + sm[0].y) + (sm[1].x + sm[1].y);
  s += __shfl_xor_sync(0xffffffffu, s, 16);
  nmean = -s * (1.f / 128);
  float2 sq[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
#pragma unroll
  for (int e = 0; e < 32; ++e) {
    const float2 v = centre2(xr[e], nmean);
    sq[e & 1] = ffma2(v, v, sq[e & 1]);
  }
  s = (sq[0].x + sq[0].y) + (sq[1].x + sq[1].y);
  s += __shfl_xor_sync(0xffffffffu, s, 16);
  rstd = rsqrtf(s * (1.f / 128) + 1e-5f);
}
__device__ __forceinline__ void store_half_row(uint8_t* tile, int row, int half, const uint32_t (&xr)[32], float nmean, float rstd,
                                               const float* gb) {
  const float2 r2 = make_float2(rstd, rstd);
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    uint32_t o[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int c = half * 64 + q * 8 + 2 * e;
      const float2 ga = *reinterpret_cast<const float2*>(gb + c), be = *reinterpret_cast<const float2*>(gb + 128 + c);
      const float2 v = ffma2(ffma2(centre2(xr[q * 4 + e], nmean), r2, make_float2(0.f, 0.f)), ga, be);
      o[e] = pack_bf16x2(v.x, v.y);
    }
    *row_piece(tile, row, half * 8 + q) = make_uint4(o[0], o[1], o[2], o[3]);
  }
}
__device__ __forceinline__ void row_normalise(uint8_t* tile, int row, float nmean, float rstd, const float* gb) {
  const float2 r2 = make_float2(rstd, rstd);
#pragma unroll 4
  for (int g = 0; g < 16; ++g) {
    const uint4 u = *row_piece(tile, row, g);
    const uint32_t w4[4] = {u.x, u.y, u.z, u.w};
    uint32_t o[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float2 ga = *reinterpret_cast<const float2*>(gb + g * 8 + 2 * e), be = *reinterpret_cast<const float2*>(gb + 128 + g * 8 + 2 * e);
      const float2 v = ffma2(ffma2(centre2(w4[e], nmean), r2, make_float2(0.f, 0.f)), ga, be);
      o[e] = pack_bf16x2(v.x, v.y);
    }
    *row_piece(tile, row, g) = make_uint4(o[0], o[1], o[2], o[3]);
  }
}

}  // namespace xf
