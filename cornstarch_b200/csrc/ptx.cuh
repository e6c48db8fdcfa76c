// Thin inline-PTX layer for sm_100a: mbarrier, TMA (non-multicast), tcgen05 / TMEM.
//
// Every wait in this file is bounded.  A wait that runs out returns false; the caller
// records a status word and walks to its normal teardown (TMEM free, return), so a
// missing arrival can never leave a kernel spinning on a shared GPU.
#pragma once
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace csb {

// Status words written to the per-launch status buffer (0 = ok).
enum : int {
  ST_OK = 0,
  ST_TIMEOUT_FULL = 1,     // consumer never saw a TMA stage arrive
  ST_TIMEOUT_EMPTY = 2,    // producer never got a smem slot back
  ST_TIMEOUT_TMEM_FULL = 3,
  ST_TIMEOUT_TMEM_EMPTY = 4,
  ST_TIMEOUT_PEER_FLAG = 5,
  ST_TIMEOUT_MISC = 6,
};

// Waits are bounded in wall time: after the wait limit (CSB_WAIT_NS nanoseconds unless csb_set_wait_ns changed it) a
// wait gives up.  The limit lives in a device variable of each translation unit (no relocatable device code), read only
// on the slow path of a spin; CSB_WAIT_LIMIT_SETTER(tu) defines the host function that updates this unit's copy on the
// current device, and csb_set_wait_ns (symm.cu) calls all of them.
#ifndef CSB_WAIT_NS
#define CSB_WAIT_NS 2000000000ull
#endif
#ifndef CSB_SPIN_LIMIT
#define CSB_SPIN_LIMIT (1u << 30)
#endif
static __device__ unsigned long long g_wait_ns = CSB_WAIT_NS;
__device__ __forceinline__ uint64_t wait_limit_ns() { return *reinterpret_cast<volatile unsigned long long*>(&g_wait_ns); }
#define CSB_WAIT_LIMIT_SETTER(tu)                                                  \
  extern "C" int csb_set_wait_ns_##tu(unsigned long long ns) {                     \
    return (int)cudaMemcpyToSymbol(csb::g_wait_ns, &ns, sizeof(ns));               \
  }

// Bounds-checked debug build (-DCSB_BOUNDS_CHECK, `python -m cornstarch_b200.csrc.build --bounds-check`): every index
// that a kernel takes from DATA (token ids, source rows, positions) is compared with the extent its entry point was
// given.  A violation records a code (first one wins) and the access is skipped, so a bad index never reaches memory;
// the host reads and clears the record with csb_bounds_status().  The release build compiles the checks away.
#ifdef CSB_BOUNDS_CHECK
static __device__ int g_bounds_status = 0;
#define CSB_IN_BOUNDS(idx, extent, code) \
  (((long)(idx) >= 0 && (long)(idx) < (long)(extent)) ? true : (atomicCAS(&csb::g_bounds_status, 0, (code)), false))
#define CSB_BOUNDS_STATUS_GETTER(tu)                                                        \
  extern "C" int csb_bounds_status_##tu() {                                                 \
    int v = 0, z = 0;                                                                       \
    if (cudaMemcpyFromSymbol(&v, csb::g_bounds_status, sizeof(v)) != cudaSuccess) return -1; \
    cudaMemcpyToSymbol(csb::g_bounds_status, &z, sizeof(z));                                \
    return v;                                                                               \
  }
#else
#define CSB_IN_BOUNDS(idx, extent, code) true
#define CSB_BOUNDS_STATUS_GETTER(tu) \
  extern "C" int csb_bounds_status_##tu() { return 0; }
#endif
// violation codes
enum : int { BND_EMBED_ROW = 101, BND_FEAT_ROW = 102, BND_ROPE_POS = 103, BND_MOE_SRC_ROW = 104 };

// 2^x on the special-function unit (one MUFU.EX2; -inf -> 0, flushes denormals).
__device__ __forceinline__ float fast_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// Maximum of three values in one instruction (sm_100).
__device__ __forceinline__ float max3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}
// Two fp32 values in a 64-bit register pair: one issue slot for two independent, individually rounded operations.
__device__ __forceinline__ uint64_t pack_u32x2(uint32_t lo, uint32_t hi) {
  uint64_t d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "r"(lo), "r"(hi));
  return d;
}
__device__ __forceinline__ uint64_t pack_f32x2(float lo, float hi) { return pack_u32x2(__float_as_uint(lo), __float_as_uint(hi)); }
__device__ __forceinline__ void unpack_f32x2(uint64_t v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ uint64_t fma_f32x2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ uint64_t add_f32x2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ uint64_t mul_f32x2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}

__device__ __forceinline__ uint64_t global_timer_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ uint32_t cluster_ctarank();

// ----------------------------------------------------------------------------- mbarrier
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_fence_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
               "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// Arrive on the same-offset barrier of another CTA of the cluster.
__device__ __forceinline__ void mbar_arrive_cluster(uint64_t* bar, uint32_t cta_rank) {
  uint32_t remote;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(smem_u32(bar)), "r"(cta_rank));
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(remote) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t phase) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred P;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 P, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, P;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(phase)
      : "memory");
  return ok != 0;
}
// Bounded wait; false = gave up.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t phase) {
  uint64_t t0 = 0;
  for (uint32_t i = 0; i < CSB_SPIN_LIMIT; ++i) {
    if (mbar_try_wait(bar, phase)) return true;
    if ((i & 511u) == 511u) {
      const uint64_t now = global_timer_ns();
      if (t0 == 0) t0 = now;
      else if (now - t0 > wait_limit_ns()) return false;
    }
  }
  return false;
}

// The same for a thread of a block whose threads tell one another through `abort_flag` (shared memory) that one of them gave up.
__device__ __forceinline__ bool mbar_wait_abort(uint64_t* bar, uint32_t phase, volatile int* abort_flag) {
  if (mbar_try_wait(bar, phase)) return true;  // in front of the loop and its set-up: 41 cycles for a wait that is over, 75 inside
  uint64_t t0 = 0;
  for (uint32_t i = 0; i < CSB_SPIN_LIMIT; ++i) {
    if (mbar_try_wait(bar, phase)) return true;
    if ((i & 511u) == 511u) {
      if (*abort_flag) return false;
      const uint64_t now = global_timer_ns();
      if (t0 == 0) t0 = now;
      else if (now - t0 > wait_limit_ns()) return false;
    }
  }
  return false;
}
// For whole warps, with one verdict for all lanes: what follows is warp-wide (elect.sync, tensor-memory loads, __syncwarp), and a
// lane that gave up alone would leave the others waiting there for good.  (A phase that is over for one lane stays over for all:
// the next one needs this warp's own arrivals or MMAs.)
__device__ __forceinline__ bool mbar_wait_abort_w(uint64_t* bar, uint32_t phase, volatile int* abort_flag) {
  if (__all_sync(0xffffffffu, mbar_try_wait(bar, phase))) return true;
  uint64_t t0 = 0;
  for (uint32_t i = 0; i < CSB_SPIN_LIMIT; ++i) {
    if (__all_sync(0xffffffffu, mbar_try_wait(bar, phase))) return true;
    if ((i & 511u) == 511u) {
      const uint64_t now = global_timer_ns();
      if (t0 == 0) t0 = now;
      if (__any_sync(0xffffffffu, *abort_flag != 0 || now - t0 > wait_limit_ns())) return false;
    }
  }
  return false;
}

// ----------------------------------------------------------------------------- TMA
__device__ __forceinline__ void tma_prefetch_desc(const CUtensorMap* m) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(m)) : "memory");
}
// 2-D tiled load, completion on an mbarrier of this CTA.  x is the innermost coordinate and
// must keep x * elem_size a multiple of 16 bytes.
__device__ __forceinline__ void tma_load_4d(void* smem_dst, const CUtensorMap* m, uint64_t* bar,
                                            int x, int y, int z, int w) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4, %5, %6}], [%2];"
      ::"r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(m)), "r"(smem_u32(bar)), "r"(x), "r"(y), "r"(z), "r"(w)
      : "memory");
}
// 2-D tiled load whose completion is reported to the mbarrier at `bar_addr`, a shared::cluster address.  CG == 2: the
// barrier may belong to the other thread block of a CTA pair (the data still lands in this block's shared memory).
template <int CG>
__device__ __forceinline__ void tma_load_2d_to(void* smem_dst, const CUtensorMap* m, uint32_t bar_addr, int x, int y) {
  if constexpr (CG == 2) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%3, %4}], [%2];"
        ::"r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(m)), "r"(bar_addr), "r"(x), "r"(y)
        : "memory");
  } else {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%3, %4}], [%2];"
        ::"r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(m)), "r"(bar_addr), "r"(x), "r"(y)
        : "memory");
  }
}
// 2-D tiled store smem -> global (bulk group completion).
__device__ __forceinline__ void tma_store_2d(const CUtensorMap* m, const void* smem_src, int x, int y) {
  asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];"
               ::"l"(reinterpret_cast<uint64_t>(m)), "r"(smem_u32(smem_src)), "r"(x), "r"(y)
               : "memory");
}
// 2-D tiled reduce-add smem -> global: global[tile] += smem[tile], element type taken from the tensor map.
__device__ __forceinline__ void tma_reduce_add_2d(const CUtensorMap* m, const void* smem_src, int x, int y) {
  asm volatile("cp.reduce.async.bulk.tensor.2d.global.shared::cta.add.tile.bulk_group [%0, {%2, %3}], [%1];"
               ::"l"(reinterpret_cast<uint64_t>(m)), "r"(smem_u32(smem_src)), "r"(x), "r"(y)
               : "memory");
}
// 4-D tiled reduce-add smem -> global (fp32 gradient accumulation straight from a staged tile).
__device__ __forceinline__ void tma_reduce_add_4d(const CUtensorMap* m, const void* smem_src, int c0, int c1, int c2, int c3) {
  asm volatile("cp.reduce.async.bulk.tensor.4d.global.shared::cta.add.tile.bulk_group [%0, {%2, %3, %4, %5}], [%1];"
               ::"l"(reinterpret_cast<uint64_t>(m)), "r"(smem_u32(smem_src)), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
               : "memory");
}
// Untiled bulk copies (both addresses 16-byte aligned, size a multiple of 16 bytes): global -> shared memory, completion
// counted on an mbarrier; shared memory -> global as part of a bulk group.  The source may be a peer's memory.
__device__ __forceinline__ void bulk_load_g2s(void* smem_dst, const void* gsrc, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(smem_u32(smem_dst)), "l"(gsrc), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}
__device__ __forceinline__ void bulk_store_s2g(void* gdst, const void* smem_src, uint32_t bytes) {
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(gdst), "r"(smem_u32(smem_src)), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void tma_store_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void tma_store_wait_read() {
  asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(N) : "memory");
}
template <int N>
__device__ __forceinline__ void tma_store_wait() {
  asm volatile("cp.async.bulk.wait_group %0;" ::"n"(N) : "memory");
}
// generic-proxy smem writes -> visible to the async proxy (TMA store / tcgen05.mma reads)
__device__ __forceinline__ void fence_proxy_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// ----------------------------------------------------------------------------- tcgen05 / TMEM
__device__ __forceinline__ void tmem_alloc(uint32_t* smem_result, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_result)),
               "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tmem_alloc_2cta(uint32_t* smem_result, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_result)),
               "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish_2cta() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_2cta(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// D[tmem] (+)= A[smem desc] * B[smem desc]; issued by ONE thread.
__device__ __forceinline__ void umma_f16(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                         uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// Make the mbarrier track completion of all tcgen05 ops this thread issued so far.
// Whole-warp forms: every lane of a CONVERGED warp executes the call with the same arguments and one elected lane (always
// the same one) issues the instruction.  Warp-uniform control flow lets the compiler keep descriptors and addresses in the
// uniform datapath; a lone lane inside a divergent branch needs several times as many issue slots per MMA and is starved
// by co-resident warps with dense arithmetic (measured: 104 cycles per MMA against 67 for 128 x 128 x 16, next to eight
// warps of independent FMAs).  A commit tracks the MMAs of the thread that issues it: use these forms for both.
__device__ __forceinline__ void umma_f16_w(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                           uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "elect.sync _|q, 0xffffffff;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// Runs of MMAs of one tile pair as one block of instructions: one elect.sync for all of them and 32-bit steps of the descriptors'
// address fields, where a call per MMA pays an election and 64-bit additions each time.  Short MMAs (128 x 64 or 128 x 128 x 16 take
// the pipe 48 or 64 cycles) are issued no faster than that otherwise: eight 128 x 64 x 16 next to busy warps 750 cycles one by
// one, 450 as a run.
// D (+)= A B^T over K-major 128-byte-swizzled operands: `n` steps of 16 (at most 8); a 64-wide chunk of A / B is 4 steps.
__device__ __forceinline__ void umma_f16_run_w(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t a_chunk_bytes,
                                               uint32_t b_chunk_bytes, uint32_t idesc, int n, uint32_t accumulate) {
  const uint32_t a0 = static_cast<uint32_t>(a_desc), ah = static_cast<uint32_t>(a_desc >> 32);
  const uint32_t b0 = static_cast<uint32_t>(b_desc), bh = static_cast<uint32_t>(b_desc >> 32);
  const uint32_t a1 = a0 + (a_chunk_bytes >> 4), b1 = b0 + (b_chunk_bytes >> 4);
#define CSB_UMMA_STEP(k, a, b, off)                                                                   \
  "setp.gt.and.s32 q, %9, " #k ", e;\n\tadd.u32 x, " a ", " #off ";\n\tadd.u32 y, " b ", " #off ";\n\t" \
  "mov.b64 da, {x, %2};\n\tmov.b64 db, {y, %4};\n\t"                                                \
  "@q tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %7, 1;\n\t"
  asm volatile(
      "{\n\t.reg .pred p, q, e;\n\t.reg .b64 da, db;\n\t.reg .b32 x, y;\n\t"
      "elect.sync _|e, 0xffffffff;\n\t"
      "setp.ne.b32 p, %8, 0;\n\t"
      "mov.b64 da, {%1, %2};\n\tmov.b64 db, {%3, %4};\n\t"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %7, p;\n\t"
      CSB_UMMA_STEP(1, "%1", "%3", 2) CSB_UMMA_STEP(2, "%1", "%3", 4) CSB_UMMA_STEP(3, "%1", "%3", 6)
      CSB_UMMA_STEP(4, "%5", "%6", 0) CSB_UMMA_STEP(5, "%5", "%6", 2) CSB_UMMA_STEP(6, "%5", "%6", 4) CSB_UMMA_STEP(7, "%5", "%6", 6)
      "}" ::"r"(d_tmem), "r"(a0), "r"(ah), "r"(b0), "r"(bh), "r"(a1), "r"(b1), "r"(idesc), "r"(accumulate), "r"(n)
      : "memory");
#undef CSB_UMMA_STEP
}
// The same with steps of A_STEP and B_STEP (in units of the descriptors' address fields, 16 bytes), four or eight of them.
template <int A_STEP, int B_STEP>
__device__ __forceinline__ void umma_f16_run4_w(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
#define CSB_UMMA_STEP                                                                                                  \
  "add.u32 x, x, %7;\n\tadd.u32 y, y, %8;\n\tmov.b64 da, {x, %2};\n\tmov.b64 db, {y, %4};\n\t"                      \
  "@e tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %5, 1;\n\t"
  asm volatile(
      "{\n\t.reg .pred p, e;\n\t.reg .b64 da, db;\n\t.reg .b32 x, y;\n\t"
      "elect.sync _|e, 0xffffffff;\n\t"
      "setp.ne.b32 p, %6, 0;\n\t"
      "mov.b32 x, %1;\n\tmov.b32 y, %3;\n\tmov.b64 da, {x, %2};\n\tmov.b64 db, {y, %4};\n\t"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %5, p;\n\t"
      CSB_UMMA_STEP CSB_UMMA_STEP CSB_UMMA_STEP
      "}" ::"r"(d_tmem), "r"(static_cast<uint32_t>(a_desc)), "r"(static_cast<uint32_t>(a_desc >> 32)), "r"(static_cast<uint32_t>(b_desc)),
      "r"(static_cast<uint32_t>(b_desc >> 32)), "r"(idesc), "r"(accumulate), "n"(A_STEP), "n"(B_STEP)
      : "memory");
}
template <int A_STEP, int B_STEP>
__device__ __forceinline__ void umma_f16_run8_w(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p, e;\n\t.reg .b64 da, db;\n\t.reg .b32 x, y;\n\t"
      "elect.sync _|e, 0xffffffff;\n\t"
      "setp.ne.b32 p, %6, 0;\n\t"
      "mov.b32 x, %1;\n\tmov.b32 y, %3;\n\tmov.b64 da, {x, %2};\n\tmov.b64 db, {y, %4};\n\t"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %5, p;\n\t"
      CSB_UMMA_STEP CSB_UMMA_STEP CSB_UMMA_STEP CSB_UMMA_STEP CSB_UMMA_STEP CSB_UMMA_STEP CSB_UMMA_STEP
      "}" ::"r"(d_tmem), "r"(static_cast<uint32_t>(a_desc)), "r"(static_cast<uint32_t>(a_desc >> 32)), "r"(static_cast<uint32_t>(b_desc)),
      "r"(static_cast<uint32_t>(b_desc >> 32)), "r"(idesc), "r"(accumulate), "n"(A_STEP), "n"(B_STEP)
      : "memory");
#undef CSB_UMMA_STEP
}
// D (+)= A B with A = 64 columns of bf16 pairs in tensor memory (16 of them are 8 tensor-memory columns; step 2 starts at column HALF)
// and B MN-major in shared memory (16 rows of 128 bytes a step): four steps.
template <int HALF = 16>
__device__ __forceinline__ void umma_f16_ts_run4_w(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  const uint32_t b0 = static_cast<uint32_t>(b_desc), bh = static_cast<uint32_t>(b_desc >> 32);
#define CSB_UMMA_STEP(ao, bo)                                                                    \
  "add.u32 x, %1, " #ao ";\n\tadd.u32 y, %2, " #bo ";\n\tmov.b64 db, {y, %3};\n\t"              \
  "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [x], db, %4, 1;\n\t"
  asm volatile(
      "{\n\t.reg .pred p, e;\n\t.reg .b64 db;\n\t.reg .b32 x, y;\n\t"
      "elect.sync _|e, 0xffffffff;\n\t"
      "setp.ne.b32 p, %5, 0;\n\t"
      "mov.b64 db, {%2, %3};\n\t"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], db, %4, p;\n\t"
      CSB_UMMA_STEP(8, 128) CSB_UMMA_STEP(%6, 256) CSB_UMMA_STEP(%7, 384)
      "}" ::"r"(d_tmem), "r"(a_tmem), "r"(b0), "r"(bh), "r"(idesc), "r"(accumulate), "n"(HALF), "n"(HALF + 8)
      : "memory");
#undef CSB_UMMA_STEP
}
// umma_f16_run4_w for a CTA pair (CG = 2) or one block.
template <int CG, int A_STEP, int B_STEP>
__device__ __forceinline__ void umma_f16_run4_cg_w(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  if constexpr (CG == 1) {
    umma_f16_run4_w<A_STEP, B_STEP>(d_tmem, a_desc, b_desc, idesc, accumulate);
  } else {
#define CSB_UMMA_STEP                                                                                                  \
  "add.u32 x, x, %7;\n\tadd.u32 y, y, %8;\n\tmov.b64 da, {x, %2};\n\tmov.b64 db, {y, %4};\n\t"                      \
  "@e tcgen05.mma.cta_group::2.kind::f16 [%0], da, db, %5, 1;\n\t"
    asm volatile(
        "{\n\t.reg .pred p, e;\n\t.reg .b64 da, db;\n\t.reg .b32 x, y;\n\t"
        "elect.sync _|e, 0xffffffff;\n\t"
        "setp.ne.b32 p, %6, 0;\n\t"
        "mov.b32 x, %1;\n\tmov.b32 y, %3;\n\tmov.b64 da, {x, %2};\n\tmov.b64 db, {y, %4};\n\t"
        "@e tcgen05.mma.cta_group::2.kind::f16 [%0], da, db, %5, p;\n\t"
        CSB_UMMA_STEP CSB_UMMA_STEP CSB_UMMA_STEP
        "}" ::"r"(d_tmem), "r"(static_cast<uint32_t>(a_desc)), "r"(static_cast<uint32_t>(a_desc >> 32)), "r"(static_cast<uint32_t>(b_desc)),
        "r"(static_cast<uint32_t>(b_desc >> 32)), "r"(idesc), "r"(accumulate), "n"(A_STEP), "n"(B_STEP)
        : "memory");
#undef CSB_UMMA_STEP
  }
}
__device__ __forceinline__ void umma_commit_w(uint64_t* bar) {
  asm volatile(
      "{\n\t.reg .pred q;\n\t"
      "elect.sync _|q, 0xffffffff;\n\t"
      "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(smem_u32(bar))
      : "memory");
}
// CG == 2: the MMAs were issued for a CTA pair; the barrier at this shared-memory offset is signalled in BOTH thread
// blocks of the pair by ONE commit whose arrival is multicast to the two blocks (cta mask 0b11).  This is a barrier
// signal between the two SMs of the pair - no data is copied and no load is involved.  (Two separate commits, one per
// block, cost 12 % of the MMA rate in a measurement without loads: 1.69 against 1.90 PFLOP/s.)
template <int CG>
__device__ __forceinline__ void umma_commit_cg_w(uint64_t* bar) {
  if constexpr (CG == 2) {
    asm volatile(
        "{\n\t.reg .pred q;\n\t"
        "elect.sync _|q, 0xffffffff;\n\t"
        "@q tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;\n\t}"
        ::"r"(smem_u32(bar)), "h"(static_cast<uint16_t>(3))
        : "memory");
  } else {
    umma_commit_w(bar);
  }
}
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
               : "memory");
}

// TMEM -> registers, 32 lanes x 32 consecutive fp32 columns; thread i of the warp gets lane
// (lane_base + i), register j holds column (col + j).
__device__ __forceinline__ void tmem_ld_32x32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
        "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_ld_32x16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_st_32x32(uint32_t taddr, const uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%32], "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31};"
      ::"r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
        "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]),
        "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]),
        "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31]),
        "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_st_32x16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%16], "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15};"
      ::"r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
        "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]),
        "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// ----------------------------------------------------------------------------- descriptors
// Shared-memory matrix descriptor for tcgen05.mma (sm_100 version field = 1), 128-byte swizzle.
//   K-major operand tile  [rows][64 x bf16] : 8-row groups are 1024 B apart (SBO); LBO unused (1).
//   MN-major operand tile [k rows][64 x bf16 of MN] per 64-wide MN block: 8-k groups 1024 B apart
//   (SBO), consecutive 64-wide MN blocks `mn_block_bytes` apart (LBO).
__device__ __forceinline__ uint64_t make_desc_sw128(uint32_t saddr, uint32_t lbo_bytes, uint32_t sbo_bytes) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((saddr & 0x3FFFF) >> 4);
  d |= static_cast<uint64_t>((lbo_bytes >> 4) & 0x3FFF) << 16;
  d |= static_cast<uint64_t>((sbo_bytes >> 4) & 0x3FFF) << 32;
  d |= static_cast<uint64_t>(1) << 46;  // descriptor version (Blackwell)
  d |= static_cast<uint64_t>(2) << 61;  // SWIZZLE_128B
  return d;
}
__device__ __forceinline__ uint64_t make_desc_kmajor_sw128(uint32_t saddr) {
  return make_desc_sw128(saddr, 16, 1024);
}
__device__ __forceinline__ uint64_t make_desc_mnmajor_sw128(uint32_t saddr, uint32_t mn_block_bytes) {
  return make_desc_sw128(saddr, mn_block_bytes, 1024);
}

// Instruction descriptor for kind::f16 with bf16 inputs and fp32 accumulation.
__host__ __device__ constexpr uint32_t make_idesc_bf16(int M, int N, int a_mn_major, int b_mn_major) {
  return (1u << 4)                              // D format = F32
         | (1u << 7)                            // A format = BF16
         | (1u << 10)                           // B format = BF16
         | (static_cast<uint32_t>(a_mn_major) << 15)
         | (static_cast<uint32_t>(b_mn_major) << 16)
         | (static_cast<uint32_t>(N >> 3) << 17)
         | (static_cast<uint32_t>(M >> 4) << 24);
}

// Byte offset of element (row, col16B-chunk) inside a 128B-swizzled tile whose rows are 128 bytes:
// the 16-byte chunk index is XORed with (row mod 8).  Tile base must be 1024-byte aligned.
__device__ __forceinline__ uint32_t sw128_offset(uint32_t row, uint32_t chunk16) {
  return row * 128u + ((chunk16 ^ (row & 7u)) << 4);
}

// ----------------------------------------------------------------------------- misc
__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&v);
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}

}  // namespace csb
