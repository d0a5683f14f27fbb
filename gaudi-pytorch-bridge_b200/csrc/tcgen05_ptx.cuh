// Thin inline-PTX layer for sm_100a: mbarrier, TMA (cp.async.bulk.tensor, no multicast),
// tcgen05 (TMEM allocation, UMMA issue/commit, TMEM loads) and the descriptor encodings.
// Every wait is bounded: a wait that runs out records a code and tells the caller to stop.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace b200q {
namespace ptx {

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// ---- mbarrier ----
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void fence_barrier_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void fence_proxy_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ uint32_t mbar_try_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      "selp.u32 %0, 1, 0, p;\n"
      "}\n"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok;
}

// Bounded wait.  `abort_flag` is a shared-memory word any role may set; the wait gives up
// when it is set or after kWaitLimit polls (seconds of wall time), and then sets it itself.
// `backoff_ns` > 0 makes a waiter that is not on the critical path (an epilogue warp waiting
// for the whole main loop of its tile) sleep between polls, so that it does not take issue
// slots from the warps that feed the tensor core.
constexpr uint32_t kWaitLimit = 1u << 24;
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag, int* status,
                                          int code, uint32_t backoff_ns = 0, uint32_t limit = kWaitLimit) {
  for (uint32_t i = 0; i < limit; ++i) {
    if (mbar_try_wait(bar, parity)) return true;
    if (backoff_ns) __nanosleep(backoff_ns);
    if ((i & 255u) == 255u) {
      if (*abort_flag) return false;
      if (i > 4096u) __nanosleep(64);
    }
  }
  *abort_flag = 1;
  atomicCAS(status, 0, code);
  return false;
}

// The form for roles that a whole warp runs: control flow that is the same for all 32 lanes lets the
// compiler keep addresses and descriptors in uniform registers; a single-lane role spends some 200
// cycles per wait and 60 per MMA on getting them there.  The outcome is a vote, so it is the same for
// all lanes too.  False when the wait ran out or another role's has: the role must then neither
// arrive, commit, copy nor issue anything more -- a barrier whose phase has not completed takes no
// further arrivals -- and leave its loops (or go through them for the named barriers it shares with
// other warps only), so that the CTA ends in the ordinary way with one ring of copies in flight at most.
[[nodiscard]] __device__ __forceinline__ bool mbar_wait_uniform(uint32_t bar, uint32_t parity, volatile int* abort_flag, int* status,
                                                                int code, uint32_t limit = kWaitLimit) {
  if (__all_sync(0xFFFFFFFFu, mbar_try_wait(bar, parity))) return true;
  for (uint32_t i = 0; i < limit; ++i) {
    if ((i & 63u) == 0u && __any_sync(0xFFFFFFFFu, *abort_flag)) return false;
    if (__all_sync(0xFFFFFFFFu, mbar_try_wait(bar, parity))) return true;
    if (i > 4096u) __nanosleep(64);
  }
  *abort_flag = 1;
  atomicCAS(status, 0, code);
  return false;
}
// The same for two barriers at once: the two polls are in flight together (a poll of a completed phase takes
// about a hundred cycles).
[[nodiscard]] __device__ __forceinline__ bool mbar_wait2_uniform(uint32_t bar0, uint32_t parity0, uint32_t bar1, uint32_t parity1,
                                                                 volatile int* abort_flag, int* status, int code) {
  uint32_t ok;
  asm volatile(
      "{\n"
      ".reg .pred p, q;\n"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      "mbarrier.try_wait.parity.shared::cta.b64 q, [%3], %4;\n"
      "and.pred p, p, q;\n"
      "selp.u32 %0, 1, 0, p;\n"
      "}\n"
      : "=r"(ok)
      : "r"(bar0), "r"(parity0), "r"(bar1), "r"(parity1)
      : "memory");
  if (__all_sync(0xFFFFFFFFu, ok)) return true;
  return mbar_wait_uniform(bar0, parity0, abort_flag, status, code) && mbar_wait_uniform(bar1, parity1, abort_flag, status, code);
}
// The index of the calling warp, known to be the same in all its lanes.
__device__ __forceinline__ int uniform_warp_index() { return __shfl_sync(0xFFFFFFFFu, (int)(threadIdx.x >> 5), 0); }
// True in one lane of a converged warp (always the same one).
__device__ __forceinline__ bool elect_one() {
  uint32_t e;
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "elect.sync _|p, 0xFFFFFFFF;\n"
      "selp.u32 %0, 1, 0, p;\n"
      "}\n"
      : "=r"(e));
  return e != 0;
}

// ---- TMA: 2-D tiled load global -> shared, completion on an mbarrier (never multicast) ----
__device__ __forceinline__ void tma_load_2d(uint32_t smem_dst, const CUtensorMap* map, uint32_t bar, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(smem_dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(x), "r"(y)
      : "memory");
}
__device__ __forceinline__ void tma_load_3d(uint32_t smem_dst, const CUtensorMap* map, uint32_t bar, int x, int y,
                                            int z) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
      ::"r"(smem_dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(x), "r"(y), "r"(z)
      : "memory");
}
__device__ __forceinline__ void tma_prefetch_desc(const CUtensorMap* map) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(map)) : "memory");
}

// ---- tcgen05 ----
__device__ __forceinline__ void tmem_alloc(uint32_t smem_slot, uint32_t ncols) {  // whole warp
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_slot), "r"(ncols)
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

// Four MMAs, D[tmem] (+)= A[smem] * B[smem], whose operand descriptors advance by astep / bstep (16-byte units), as one
// instruction sequence that one thread issues; only the first one may start a new accumulator.  kind::f8f6f4: K = 32
// each; kind::f16 (bf16 or fp16 operands): K = 16.  The pair forms multiply 256 rows over both CTAs' shared
// memory and TMEM.
#define B200Q_UMMA_X4(NAME, G, KIND)                                                                                        \
  __device__ __forceinline__ void NAME(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate, \
                                       uint32_t astep, uint32_t bstep) {                                                    \
    asm volatile(                                                                                                           \
        "{\n"                                                                                                               \
        ".reg .pred p, t;\n"                                                                                                \
        "setp.ne.b32 p, %4, 0;\n"                                                                                           \
        "setp.eq.b32 t, 0, 0;\n"                                                                                            \
        "tcgen05.mma.cta_group::" G ".kind::" KIND " [%0], %1, %2, %3, p;\n"                                                \
        "tcgen05.mma.cta_group::" G ".kind::" KIND " [%0], %5, %6, %3, t;\n"                                                \
        "tcgen05.mma.cta_group::" G ".kind::" KIND " [%0], %7, %8, %3, t;\n"                                                \
        "tcgen05.mma.cta_group::" G ".kind::" KIND " [%0], %9, %10, %3, t;\n"                                               \
        "}\n" ::"r"(d_tmem),                                                                                                \
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate), "l"(adesc + astep), "l"(bdesc + bstep), "l"(adesc + 2 * astep), \
        "l"(bdesc + 2 * bstep), "l"(adesc + 3 * astep), "l"(bdesc + 3 * bstep)                                              \
        : "memory");                                                                                                        \
  }
B200Q_UMMA_X4(umma_f8_x4, "1", "f8f6f4")
B200Q_UMMA_X4(umma_f16_x4, "1", "f16")
B200Q_UMMA_X4(umma_f8_pair_x4, "2", "f8f6f4")  // (over both CTAs of a pair; issued by one thread of the even CTA)
B200Q_UMMA_X4(umma_f16_pair_x4, "2", "f16")
#undef B200Q_UMMA_X4
// Four kind::f16 MMAs whose A operand is in tensor memory (128 lanes, two bf16 per 32-bit column: 8 columns per
// K = 16 step): the TMEM address advances by astep columns, the B descriptor by bstep 16-byte units.
__device__ __forceinline__ void umma_f16_ts_x4(uint32_t d_tmem, uint32_t a_tmem, uint64_t bdesc, uint32_t idesc, uint32_t accumulate,
                                               uint32_t astep, uint32_t bstep) {
  asm volatile(
      "{\n"
      ".reg .pred p, t;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "setp.eq.b32 t, 0, 0;\n"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%5], %6, %3, t;\n"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%7], %8, %3, t;\n"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%9], %10, %3, t;\n"
      "}\n" ::"r"(d_tmem),
      "r"(a_tmem), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(a_tmem + astep), "l"(bdesc + bstep), "r"(a_tmem + 2 * astep),
      "l"(bdesc + 2 * bstep), "r"(a_tmem + 3 * astep), "l"(bdesc + 3 * bstep)
      : "memory");
}
// Arrive on an mbarrier once every previously issued MMA of this thread has completed.
__device__ __forceinline__ void umma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}


// ---- CTA pairs (cta_group::2): two CTAs of a cluster drive one 256-row MMA ----
constexpr uint32_t kPeerBitMask = 0xFEFFFFFFu;  // clears the CTA-rank bit of a shared::cluster address: the even CTA

__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
// All threads of all CTAs of the cluster.
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_alloc_pair(uint32_t smem_slot, uint32_t ncols) {  // the same warp in both CTAs
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_slot), "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish_pair() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
// TMA load into this CTA's shared memory whose completion bytes are counted on the barrier of
// the pair's even CTA (`bar` must already have the rank bit cleared).  Not a multicast: each CTA
// fetches only its own tile.
__device__ __forceinline__ void tma_load_2d_pair(uint32_t smem_dst, const CUtensorMap* map, uint32_t bar, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(smem_dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(x), "r"(y)
      : "memory");
}
// Completion of the pair's MMAs signalled on the barrier at the same offset in both CTAs.
__device__ __forceinline__ void umma_commit_pair_both(uint32_t bar) {
  asm volatile(
      "{\n"
      ".reg .b16 m;\n"
      "mov.b16 m, 3;\n"
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], m;\n"
      "}\n" ::"r"(bar)
      : "memory");
}
// Arrive on a barrier addressed in the cluster window (own CTA or the peer), with the default (CTA-scope) release: no
// cluster-wide fence is executed, which on B200 costs about a thousand cycles per arrival.  Enough when what the arrival
// publishes is that tensor memory has been read, or this CTA's own shared memory, already made visible to the async proxy by
// fence.proxy.async, and read there by the tensor core of this same SM.
__device__ __forceinline__ void mbar_arrive_remote(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}

// 32 lanes x 32 consecutive 32-bit columns: thread t of the warp gets lane (base lane + t).
__device__ __forceinline__ void tmem_ld_32x32(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
        "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_ld_32x16(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
// Stores: thread t of the warp writes 16 columns of lane (base lane + t).
__device__ __forceinline__ void tmem_st_32x16(uint32_t taddr, const uint32_t* r) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%16], "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15};" ::"r"(r[0]),
      "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]),
      "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// Named barrier among a subset of the CTA's warps.
__device__ __forceinline__ void named_bar_sync(int id, int nthreads) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(nthreads) : "memory");
}

// ---- descriptors ----
// Shared-memory matrix descriptor, K-major operand, 128-byte swizzle, rows of 128 bytes:
// 8-row groups are 1024 bytes apart (SBO); LBO is unused for swizzled K-major layouts (1).
// The tile base must be 1024-byte aligned; stepping K inside the 128-byte row adds bytes
// to the start address.
__device__ __forceinline__ uint64_t smem_desc_k_sw128(uint32_t saddr) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr & 0x3FFFFu) >> 4);       // start address, bits [0,14)
  d |= (uint64_t)1 << 16;                         // leading byte offset (16 B units), bits [16,30)
  d |= (uint64_t)(1024 >> 4) << 32;               // stride byte offset, bits [32,46)
  d |= (uint64_t)1 << 46;                         // descriptor version (Blackwell), bits [46,48)
  d |= (uint64_t)2 << 61;                         // layout: SWIZZLE_128B, bits [61,64)
  return d;
}

// MN-major operand (the M or N index is contiguous in memory), 128-byte swizzle: 64 bf16 along
// MN form a 128-byte row, 8 consecutive k form a 1024-byte atom; `lbo` is the byte distance
// between 64-element MN blocks and `sbo` the distance between 8-k groups.
__device__ __forceinline__ uint64_t smem_desc_mn_sw128(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr & 0x3FFFFu) >> 4);
  d |= (uint64_t)((lbo >> 4) & 0x3FFFu) << 16;
  d |= (uint64_t)((sbo >> 4) & 0x3FFFu) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;
  return d;
}

// Instruction descriptor (dense, fp32 accumulate, both operands K-major).
// fmt for kind::f8f6f4: 0 = e4m3, 1 = e5m2; for kind::f16: 0 = f16, 1 = bf16.
__host__ __device__ constexpr uint32_t umma_idesc(uint32_t a_fmt, uint32_t b_fmt, uint32_t m, uint32_t n) {
  return (1u << 4) | (a_fmt << 7) | (b_fmt << 10) | ((n >> 3) << 17) | ((m >> 4) << 24);
}
// Same with the operands' major-ness: bit 15 = A is MN-major, bit 16 = B is MN-major.
__host__ __device__ constexpr uint32_t umma_idesc_major(uint32_t a_fmt, uint32_t b_fmt, uint32_t m, uint32_t n,
                                                        uint32_t a_mn, uint32_t b_mn) {
  return umma_idesc(a_fmt, b_fmt, m, n) | (a_mn << 15) | (b_mn << 16);
}

}  // namespace ptx
}  // namespace b200q
