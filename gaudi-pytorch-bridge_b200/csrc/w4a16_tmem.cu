// W4A16 GEMM for up to 128 tokens: out[M][N] = x[M][K] . W[K][N] with W held as packed 4-bit words.
//
// What bounds it is the expansion: 0.5 byte per weight from DRAM is 5.2 us for K = N = 8192, and
// turning a packed word into eight bf16 costs 15 - 19 instructions per lane, about as long again when
// nothing else is executed.  So the weights are the A operand of tcgen05.mma in TENSOR MEMORY: a
// thread expands the words of one output column (its TMEM lane) and stores the registers as they are
// (tcgen05.st), with no shared-memory tile in between, no MMA fragments and no MMA instructions in the
// expanding warps; the tokens are the B operand in shared memory, the accumulator is [column][token].
//
// A CTA covers TC x 128 output columns and one k-range; the CTAs of a cluster split K between them and
// add their fp32 tiles through distributed shared memory in rank order (no scratch, no second
// kernel, the same bits on every run).  A unit is one 64-deep k-block of 128 columns, a stage two units.
// Roles:
//   warp 0       raw producer: TMA of the packed words of a stage, 96 KB in flight per SM
//   warp 1       activation producer: TMA of [NT tokens][64 k] (128-byte swizzle, rows >= M read as 0)
//   warps 2, 3   MMA issuers: four tcgen05.mma.kind::f16 per unit, each issuer into an accumulator of its
//                own: stage by stage in turn with TC = 1 (the two accumulators are added at the end), one
//                column half each with TC = 2.  One issuer that waited and committed unit by unit took
//                620 cycles a unit and set the pace (23.8 us at M = 16, K = N = 8192).
//   warps 4..27  expanders, groups of four warps (one warp per TMEM lane quarter) that take the stages in
//                turn; afterwards they read the accumulators back.  There are as many groups as A slots
//                and two raw slots for each, so that a slot belongs to one group (and, with TC = 1, to one
//                issuer: an even number of groups and of activation slots).  A barrier's phase is known by
//                its parity alone, and two waiters that are a phase apart on one barrier would take each
//                other's.
//
// Weight layouts: AutoGPTQ [K/8][N] (KP = 1) has eight consecutive k of one column in a word, so a
// lane reads its own words; the operator's [K][N/8] (KP = 0) has eight columns of one k, and the four
// warps of a group first transpose the packed 8 x 8 nibble blocks in place in shared memory (a block
// per thread, four instructions per word).
// Measured, median of launches over rotating weights, us (the kernels it replaces in brackets), group 128, tokens
// 1 / 16 / 32 / 77 / 128 on [K][N/8] words: K = N = 8192 18.6 / 18.7 / 19.1 / 22.2 / 24.7 (27.1 / 22.4 / 24.4 /
// 27.8 / 30.8), K = 4096, N = 14336 18.1 / 18.2 / 18.7 / 20.8 / 23.0 (31.1 / 28.5 / 23.4 / 31.0 / 36.7),
// K = N = 2048 6.8 / 7.0 / 7.4 / 8.4 / 13.6 (8.2 / 9.4 / 9.4 / 11.6 / 13.9); AutoGPTQ words at 1 / 16 tokens
// 16.1 / 16.2 (17.5 / 20.3) for K = N = 8192.  What is left above the 5.2 us of the stream: about 5.5 us of start, first
// copies and exchange, and the expansion: LOP3, PRMT and bf16x2 instructions issue every other cycle.
#include <cuda.h>

#include "common.cuh"
#include "tcgen05_ptx.cuh"
#include "tma_host.cuh"

namespace b200q {

using namespace ptx;

namespace w4t {

constexpr int kK = 64;             // k per block: 64 bf16 = one 128-byte swizzle row
constexpr int kCols = 128;         // columns per unit = TMEM lanes
constexpr int kUnitBytes = 4096;   // packed words of a unit
constexpr int kMaxGroups = 6;      // expander groups = expanded stages in TMEM, 64 columns each
constexpr int kExpWarp0 = 4;
constexpr int kThreads = 32 * (kExpWarp0 + 4 * kMaxGroups);
constexpr int kRawSlots = 2 * kMaxGroups;
constexpr int kRawRing = kRawSlots * 2 * kUnitBytes;
constexpr int kMaxXSlots = 12;
constexpr int kXRing = 112 * 1024;
constexpr int kXOffset = kRawRing;
constexpr int kBarOffset = kXOffset + kXRing;
constexpr int kNumBars = 2 * kRawSlots + 2 * kMaxXSlots + 2 * kMaxGroups + 1;
constexpr int kSmemBytes = kBarOffset + kNumBars * 8 + 16 + 1024;
static_assert(kSmemBytes <= 227 * 1024, "shared memory budget");
static_assert(kSmemBytes > 114 * 1024, "one CTA per SM: two CTAs must never contend for TMEM");
static_assert(2 * 128 * kCols * 4 <= kXOffset + kXRing, "the fp32 tile of the reduction overlays the rings");
static_assert(kXRing / (2 * 128 * 128) >= 2, "an activation slot for each issuer");

enum { kErrRaw = 211, kErrAct = 212, kErrMma = 213, kErrExpand = 214, kErrEpilogue = 215 };

struct Params {
  const uint16_t* scale;  // bf16 [K/group][N]
  const int32_t* zp;      // [K/group][N/8] or null
  void* out;              // [M][N], row stride ldo
  int64_t ldo;
  int M, N, num_kb, kb_per_group;
  int nt;                 // tokens rounded up to 16: N of the MMA, rows of an activation tile
  int x_slots, groups, acc_cols, out_dtype;
  int* status;
};

__device__ __forceinline__ uint32_t lds32(uint32_t a) {
  uint32_t v;
  asm volatile("ld.shared.b32 %0, [%1];" : "=r"(v) : "r"(a));
  return v;
}
__device__ __forceinline__ void sts32(uint32_t a, uint32_t v) { asm volatile("st.shared.b32 [%0], %1;" ::"r"(a), "r"(v) : "memory"); }
__device__ __forceinline__ void sts128(uint32_t a, const uint32_t* v) {
  asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(a), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]) : "memory");
}
__device__ __forceinline__ uint32_t mapa(uint32_t local_addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(local_addr), "r"(rank));
  return r;
}
__device__ __forceinline__ float4 ld_cluster_f32x4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ uint32_t ld_cluster_u32(uint32_t addr) {
  uint32_t v;
  asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ uint32_t bf2_sub(uint32_t a, uint32_t b) {
  __nv_bfloat162 r = __hsub2(*reinterpret_cast<__nv_bfloat162*>(&a), *reinterpret_cast<__nv_bfloat162*>(&b));
  return *reinterpret_cast<uint32_t*>(&r);
}
__device__ __forceinline__ uint32_t bf2_mul(uint32_t a, uint32_t b) {
  __nv_bfloat162 r = __hmul2(*reinterpret_cast<__nv_bfloat162*>(&a), *reinterpret_cast<__nv_bfloat162*>(&b));
  return *reinterpret_cast<uint32_t*>(&r);
}

// Four rows (pairs of k) of four nibbles in each 16-bit half -> four words whose half h holds nibble
// (row j) at position j: c[i] of half h, position j = nibble i of x[j], half h.
__device__ __forceinline__ void transpose_nibbles(const uint32_t* x, uint32_t* c) {
  constexpr uint32_t kLo = 0x0F0F0F0Fu;
  const uint32_t y0 = __byte_perm(x[0], x[2], 0x6240), y1 = __byte_perm(x[0], x[2], 0x7351);
  const uint32_t z0 = __byte_perm(x[1], x[3], 0x6240), z1 = __byte_perm(x[1], x[3], 0x7351);
  c[0] = (y0 & kLo) | ((z0 << 4) & ~kLo);
  c[1] = ((y0 >> 4) & kLo) | (z0 & ~kLo);
  c[2] = (y1 & kLo) | ((z1 << 4) & ~kLo);
  c[3] = ((y1 >> 4) & kLo) | (z1 & ~kLo);
}

// TC = 128-column units per CTA and k-block; KP = weight layout (see the head of the file).
template <int TC, int KP>
__global__ void __launch_bounds__(kThreads, 1)
w4a16_tmem_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w, const Params p) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + kBarOffset);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + kNumBars);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const uint32_t base = smem_u32(smem);
  // raw_full / raw_empty   packed words landed / read by the expander warps
  // x_full / x_empty       activations landed / read by the MMAs (commit)
  // a_full / a_empty       stage expanded into TMEM / read by its MMAs (commit)
  const uint32_t bar_raw_full = smem_u32(bars), bar_raw_empty = bar_raw_full + 8 * kRawSlots;
  const uint32_t bar_x_full = bar_raw_empty + 8 * kRawSlots, bar_x_empty = bar_x_full + 8 * kMaxXSlots;
  const uint32_t bar_a_full = bar_x_empty + 8 * kMaxXSlots, bar_a_empty = bar_a_full + 8 * kMaxGroups;
  const uint32_t bar_d_full = bar_a_empty + 8 * kMaxGroups;
  const int warp = uniform_warp_index(), lane = threadIdx.x & 31;
  uint32_t crank, csize;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(crank));
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(csize));

  if (threadIdx.x == 0) {
    for (int i = 0; i < kRawSlots; ++i) {
      mbar_init(bar_raw_full + 8 * i, 1);
      mbar_init(bar_raw_empty + 8 * i, 4);  // the expander warps of a group
    }
    for (int i = 0; i < kMaxXSlots; ++i) {
      mbar_init(bar_x_full + 8 * i, 1);
      mbar_init(bar_x_empty + 8 * i, TC);  // the issuers that read the slot
    }
    for (int i = 0; i < kMaxGroups; ++i) {
      mbar_init(bar_a_full + 8 * i, 4);
      mbar_init(bar_a_empty + 8 * i, TC);
    }
    mbar_init(bar_d_full, 2);
    *abort_flag = 0;
    fence_barrier_init();
    fence_proxy_async_smem();
    tma_prefetch_desc(&map_x);
    tma_prefetch_desc(&map_w);
  }
  if (warp == 3) {
    tmem_alloc(smem_u32(tmem_slot), 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  pdl_enter();  // everything above may run under the tail of the kernel in front of this one

  const int n0 = (int)(blockIdx.x / csize) * (TC * kCols);
  // this CTA's share of the k-blocks: never empty (the host gives a cluster at most num_kb CTAs)
  const int kb0 = (int)((int64_t)crank * p.num_kb / csize);
  const int kbn = (int)((int64_t)(crank + 1) * p.num_kb / csize) - kb0;
  const int nt = p.nt;
  // A stage is two units: with TC = 1 two k-blocks (the second one is missing at the end of an odd number),
  // with TC = 2 the two column halves of one.
  constexpr int kStageKb = TC == 1 ? 2 : 1;
  const int stages = TC == 1 ? (kbn + 1) >> 1 : kbn;
  const uint32_t x_slot_bytes = kStageKb * nt * 128;
  // TMEM: two accumulators of at least nt columns, then the A slots
  const uint32_t acc_cols = p.acc_cols, a_col = tmem + 2 * acc_cols;
  const int groups = p.groups;

  if (warp == 0) {
    // ------------------------------------------------------------ packed words
    uint32_t slot = 0, phase = 0;
    for (int st = 0; st < stages; ++st) {
      if (!mbar_wait_uniform(bar_raw_empty + 8 * slot, phase ^ 1, abort_flag, p.status, kErrRaw)) break;
      if (elect_one()) {
        const uint32_t full = bar_raw_full + 8 * slot, dst = base + slot * 2 * kUnitBytes;
        const int kb = kb0 + st * kStageKb;
        mbar_arrive_expect_tx(full, 2 * kUnitBytes);
        if (TC == 1) {  // one box of two k-blocks (a second one past this CTA's range is not used)
          if (KP) tma_load_2d(dst, &map_w, full, n0, kb * (kK / 8));
          else tma_load_2d(dst, &map_w, full, n0 / 8, kb * kK);
        } else {
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            if (KP) tma_load_2d(dst + h * kUnitBytes, &map_w, full, n0 + h * kCols, kb * (kK / 8));
            else tma_load_2d(dst + h * kUnitBytes, &map_w, full, (n0 + h * kCols) / 8, kb * kK);
          }
        }
      }
      if (++slot == 2u * groups) { slot = 0; phase ^= 1; }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ activations
    uint32_t slot = 0, phase = 0;
    for (int st = 0; st < stages; ++st) {
      if (!mbar_wait_uniform(bar_x_empty + 8 * slot, phase ^ 1, abort_flag, p.status, kErrAct)) break;
      if (elect_one()) {
        const uint32_t full = bar_x_full + 8 * slot, dst = base + kXOffset + slot * x_slot_bytes;
        const int i = st * kStageKb;
        const bool two = TC == 1 && i + 1 < kbn;
        mbar_arrive_expect_tx(full, two ? 2 * nt * 128 : nt * 128);
        tma_load_2d(dst, &map_x, full, (kb0 + i) * kK, 0);
        if (two) tma_load_2d(dst + nt * 128, &map_x, full, (kb0 + i + 1) * kK, 0);
      }
      if (++slot == (uint32_t)p.x_slots) { slot = 0; phase ^= 1; }
    }
  } else if (warp < kExpWarp0) {
    // ------------------------------------------------------------ MMA issuers
    const uint32_t j = warp - 2;
    const uint32_t idesc = umma_idesc(1u, 1u, 128, (uint32_t)nt);
    const uint64_t xd0 = smem_desc_k_sw128(base + kXOffset);
    const uint32_t d = tmem + j * acc_cols;
    constexpr int kStep = TC == 1 ? 2 : 1;
    uint32_t xs = TC == 1 ? j : 0, xphase = 0, as = xs, aphase = 0;
    bool ok = true;
    for (int st = TC == 1 ? (int)j : 0; st < stages; st += kStep) {
      ok = mbar_wait2_uniform(bar_x_full + 8 * xs, xphase, bar_a_full + 8 * as, aphase, abort_flag, p.status, kErrMma);
      if (!ok) break;
      tc_fence_after();
      const uint64_t xd = xd0 + (uint64_t)(xs * (x_slot_bytes >> 4));
      const uint32_t a = a_col + as * 64;
      if (elect_one()) {
        if (TC == 1) {
          umma_f16_ts_x4(d, a, xd, idesc, st >= 2, 8, 2);
          if (2 * st + 1 < kbn) umma_f16_ts_x4(d, a + 32, xd + (uint32_t)(nt * 8), idesc, 1u, 8, 2);
        } else {
          umma_f16_ts_x4(d, a + j * 32, xd, idesc, st != 0, 8, 2);
        }
        umma_commit(bar_a_empty + 8 * as);
        umma_commit(bar_x_empty + 8 * xs);
      }
      xs += kStep;
      if (xs >= (uint32_t)p.x_slots) { xs -= p.x_slots; xphase ^= 1; }
      as += kStep;
      if (as >= (uint32_t)groups) { as -= groups; aphase ^= 1; }
    }
    if (ok && elect_one()) umma_commit(bar_d_full);
  } else {
    // ------------------------------------------------------------ expanders
    const int qtr = warp & 3, grp = (warp - kExpWarp0) >> 2;
    const int col = qtr * 32 + lane;
    // The columns of the two units; past the end any finite operand will do, it is never stored.
    const int na = min(n0 + col, p.N - 1), nb = TC == 1 ? na : min(n0 + kCols + col, p.N - 1);
    const uint32_t as = grp;  // this group's A slot; its raw slots are grp and grp + groups
    uint32_t slot = grp, phase = 0, aphase = 0;
    // Scales and zero points are fetched one stage ahead.  Row of the group tables and position inside the
    // group are carried along: a division per stage costs as much as a word's expansion.
    const int step_kb = groups * kStageKb, dg = step_kb / p.kb_per_group, dr = step_kb % p.kb_per_group;
    const int kb_first = kb0 + grp * kStageKb;
    int row = kb_first / p.kb_per_group, rem = kb_first % p.kb_per_group;
    uint32_t sn[2] = {0, 0}, zn[2] = {0, 0};
    const int nw = p.N >> 3;
    auto fetch = [&](int st) {
      if (st < stages) {
        const uint16_t* sp = p.scale + (int64_t)row * p.N;
        const bool next = TC == 1 && rem + 1 == p.kb_per_group;  // the second k-block begins the next group
        const bool two = TC == 2 || 2 * st + 1 < kbn;
        const uint16_t* sp2 = next ? sp + p.N : sp;
        sn[0] = __ldg(sp + na);
        if (two) sn[1] = __ldg(sp2 + nb);
        if (p.zp) {
          const int32_t* zq = p.zp + (int64_t)row * nw;
          const int32_t* zq2 = next ? zq + nw : zq;
          zn[0] = (uint32_t)__ldg(zq + (na >> 3));
          if (two) zn[1] = (uint32_t)__ldg(zq2 + (nb >> 3));
        }
        row += dg, rem += dr;
        if (rem >= p.kb_per_group) { rem -= p.kb_per_group; ++row; }
      }
    };
    if (grp < groups) fetch(grp);
    // KP = 0: the thread's 8 x 8 block of a unit is column group ng, k-octet oct.  The half-warps read
    // their eight rows in opposite order inside each pair (banks 0-15 and 16-31) and the lanes of
    // every other four column groups store their halves in opposite order.  An octet's eight rows
    // are the 512 bytes that its transposed words go to, and only one half-warp touches them.
    const int ng = lane & 15, oct = 2 * qtr + (lane >> 4), swap = lane >> 4, hfirst = (ng >> 2) & 1;
    const uint32_t sel_lo = swap ? 0x1054u : 0x5410u, sel_hi = swap ? 0x3276u : 0x7632u;
    const uint32_t sel0 = hfirst ? sel_hi : sel_lo, sel1 = hfirst ? sel_lo : sel_hi;
    const uint32_t blk_ld = oct * 512 + ng * 4 + swap * 64, blk_st = oct * 512 + ng * 32;
    const int pair_step = swap ? -64 : 64;
    // (after a wait that ran out the warps of a group still meet at their barrier, which no limit ends)
    bool ok = true;
    for (int st = grp < groups ? grp : stages; st < stages; st += groups) {
      const bool two = TC == 2 || 2 * st + 1 < kbn;
      uint32_t s2[2], z2[2];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        s2[h] = sn[h] * 0x00010001u;
        z2[h] = (((zn[h] >> (4 * ((h ? nb : na) & 7))) & 15u) * 0x00010001u) | 0x43004300u;
      }
      ok = ok && mbar_wait_uniform(bar_raw_full + 8 * slot, phase, abort_flag, p.status, kErrExpand);
      if (!ok) {
        if (!KP) named_bar_sync(1 + grp, 128);
        continue;
      }
      fetch(st + groups);
      const uint32_t raw = base + slot * 2 * kUnitBytes;
      if (!KP) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          uint32_t v[8], x[4], c[4], c2[4];
          const uint32_t blk = raw + h * kUnitBytes + blk_ld;
#pragma unroll
          for (int r = 0; r < 8; r += 2) v[r] = lds32(blk + r * 64), v[r + 1] = lds32(blk + r * 64 + pair_step);
#pragma unroll
          for (int j = 0; j < 4; ++j) x[j] = __byte_perm(v[2 * j], v[2 * j + 1], sel0);
          transpose_nibbles(x, c);
#pragma unroll
          for (int j = 0; j < 4; ++j) x[j] = __byte_perm(v[2 * j], v[2 * j + 1], sel1);
          transpose_nibbles(x, c2);
          __syncwarp();  // the octet has been read
          sts128(raw + h * kUnitBytes + blk_st + hfirst * 16, c);
          sts128(raw + h * kUnitBytes + blk_st + (hfirst ^ 1) * 16, c2);
        }
        fence_proxy_async_smem();  // (the slot is refilled by TMA)
        named_bar_sync(1 + grp, 128);
      }
      uint32_t w[2][8];
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int o = 0; o < 8; ++o) w[h][o] = lds32(raw + h * kUnitBytes + o * 512 + col * 4);
      __syncwarp();
      if (lane == 0) mbar_arrive(bar_raw_empty + 8 * slot);
      ok = mbar_wait_uniform(bar_a_empty + 8 * as, aphase ^ 1, abort_flag, p.status, kErrExpand);
      if (!ok) continue;
      tc_fence_after();
      const uint32_t a = a_col + ((uint32_t)(qtr * 32) << 16) + as * 64;
#pragma unroll
      for (int h = 0; h < 4; ++h) {
        if (h == 2 && !two) break;
        uint32_t r[16];
#pragma unroll
        for (int o = 0; o < 4; ++o) {
          const uint32_t wo = w[h >> 1][4 * (h & 1) + o], w4 = wo >> 4;
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            // the bf16x2 {128 + q(k = 2j), 128 + q(k = 2j + 1)}: KP = 1 has them in byte j of the word,
            // KP = 0 in nibble j of its halves
            const uint32_t q = KP ? __byte_perm(wo, w4, 0x4400u + 0x1111u * j) : wo >> (4 * j);
            r[4 * o + j] = bf2_mul(bf2_sub((q & 0x000F000Fu) | 0x43004300u, z2[h >> 1]), s2[h >> 1]);
          }
        }
        tmem_st_32x16(a + 16 * h, r);
      }
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar_a_full + 8 * as);
      aphase ^= 1;
      slot += groups;
      if (slot >= 2u * groups) { slot -= 2 * groups; phase ^= 1; }
    }
    // accumulators -> fp32 tile [tc][token][128 columns] over the rings (every copy has landed and
    // been read when the last MMA retires)
    if (ok && mbar_wait_uniform(bar_d_full, 0, abort_flag, p.status, kErrEpilogue)) {
      tc_fence_after();
      for (int c = grp; c < TC * (nt >> 4); c += kMaxGroups) {
        const int ct = TC == 1 ? 0 : c & 1, t0 = (TC == 1 ? c : c >> 1) * 16;
        uint32_t d[16];
        const uint32_t addr = tmem + ((uint32_t)(qtr * 32) << 16) + ct * acc_cols + t0;
        tmem_ld_32x16(addr, d);
        if (TC == 1 && stages > 1) {  // the second issuer's stages
          uint32_t d2[16];
          tmem_ld_32x16(addr + acc_cols, d2);
          tmem_ld_wait();
#pragma unroll
          for (int t = 0; t < 16; ++t) d[t] = __float_as_uint(__uint_as_float(d[t]) + __uint_as_float(d2[t]));
        } else {
          tmem_ld_wait();
        }
#pragma unroll
        for (int t = 0; t < 16; ++t) sts32(base + ((ct * nt + t0 + t) * kCols + col) * 4, d[t]);
      }
    }
  }

  // ---------------------------------------------------------------- reduction over the cluster
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (*abort_flag) {
    for (int i = 0; i < 200; ++i) __nanosleep(1000);  // copies in flight
  }
  cluster_sync_all();
  if (warp == 3) tmem_dealloc(tmem, 512);
  uint32_t stop = 0;
  const uint32_t flag_addr = smem_u32(tmem_slot + 1);
  for (uint32_t r = 0; r < csize; ++r) stop |= ld_cluster_u32(mapa(flag_addr, r));
  if (!stop) {
    // a warp finishes one token's 128 columns; the tokens are dealt to the CTAs in turn
    for (int row = (int)crank + (int)csize * warp; row < TC * p.M; row += (int)csize * (kThreads / 32)) {
      const int ct = TC == 1 ? 0 : row & 1, tok = TC == 1 ? row : row >> 1;
      const uint32_t addr = base + ((ct * nt + tok) * kCols + 4 * lane) * 4;
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
      for (uint32_t r = 0; r < csize; ++r) {
        const float4 t = ld_cluster_f32x4(mapa(addr, r));
        v.x += t.x, v.y += t.y, v.z += t.z, v.w += t.w;
      }
      const int col = n0 + ct * kCols + 4 * lane;
      if (col < p.N) {  // (N is a multiple of 32)
        if (p.out_dtype == B200Q_BF16) {
          __nv_bfloat16* o = static_cast<__nv_bfloat16*>(p.out) + (int64_t)tok * p.ldo + col;
          if ((reinterpret_cast<uintptr_t>(o) & 7) == 0) {
            *reinterpret_cast<uint2*>(o) = make_uint2(pack_bf16x2(v.x, v.y), pack_bf16x2(v.z, v.w));
          } else {
            o[0] = __float2bfloat16_rn(v.x), o[1] = __float2bfloat16_rn(v.y);
            o[2] = __float2bfloat16_rn(v.z), o[3] = __float2bfloat16_rn(v.w);
          }
        } else {
          float* o = static_cast<float*>(p.out) + (int64_t)tok * p.ldo + col;
          if ((reinterpret_cast<uintptr_t>(o) & 15) == 0) *reinterpret_cast<float4*>(o) = v;
          else o[0] = v.x, o[1] = v.y, o[2] = v.z, o[3] = v.w;
        }
      }
    }
  }
  __syncwarp();
  cluster_sync_all();  // no CTA leaves while another may still read its tile
}

template <int TC, int KP>
static int launch(const CUtensorMap& mx, const CUtensorMap& mw, const Params& p, int tiles, int cluster, cudaStream_t st) {
  auto kern = w4a16_tmem_kernel<TC, KP>;
  static std::atomic<int> configured[kMaxDevices];
  const int dev = current_device_index();
  if (dev < 0) return B200Q_ERR_CUDA;
  if (!configured[dev].load(std::memory_order_acquire)) {
    B200Q_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes));
    configured[dev].store(1, std::memory_order_release);
  }
  launch_dependent_cluster(kern, (unsigned)cluster, dim3((unsigned)(tiles * cluster)), dim3(kThreads), kSmemBytes, st, mx, mw, p);
  B200Q_LAUNCH_CHECK();
  return B200Q_OK;
}

}  // namespace w4t

// Whether the kernel takes this problem: up to 128 tokens, whole 64-deep k-blocks that no group cuts,
// row pitches that TMA can address (N a multiple of 32).
bool w4a16_tmem_eligible(int64_t M, int64_t N, int64_t K, int64_t group) {
  return M >= 1 && M <= 128 && N >= 32 && N % 32 == 0 && N <= (1 << 30) && K >= w4t::kK && K % w4t::kK == 0 && K <= (1 << 30) &&
         group % w4t::kK == 0 && K % group == 0;
}

int w4a16_tmem_launch(const void* x, int64_t ldx, const int32_t* qweight, const void* scale, const int32_t* zp, int k_packed,
                      int64_t M, int64_t N, int64_t K, int64_t group, void* out, int out_dtype, int64_t ldo, cudaStream_t st) {
  if (!w4a16_tmem_eligible(M, N, K, group)) return B200Q_ERR_UNSUPPORTED;
  if ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(qweight) | reinterpret_cast<uintptr_t>(scale)) & 15)
    return B200Q_ERR_UNSUPPORTED;
  if (ldx % 8) return B200Q_ERR_UNSUPPORTED;
  w4t::Params p;
  p.scale = static_cast<const uint16_t*>(scale); p.zp = zp; p.out = out; p.ldo = ldo;
  p.M = (int)M; p.N = (int)N; p.num_kb = (int)(K / w4t::kK); p.kb_per_group = (int)(group / w4t::kK);
  p.nt = (int)(M + 15) / 16 * 16;
  p.out_dtype = out_dtype;
  p.status = device_status_ptr();
  if (!p.status) return B200Q_ERR_CUDA;
  // Columns per CTA and k-split, by an estimate of the longest CTA in units of 10 ns: a k-block costs
  // 9 per 128 columns of expansion or the arrival of its activation tile from L2, whichever is more, a round
  // of CTAs about 3 us of start and end, a further CTA of a cluster its share of the exchange.
  int best_tc = 1, best_s = 1;
  int64_t best = 0;
  for (int tc = 1; tc <= 2; ++tc) {
    const int64_t tiles = (N + tc * w4t::kCols - 1) / (tc * w4t::kCols);
    const int64_t per_kb = tc * 9 > p.nt / 8 ? tc * 9 : p.nt / 8;
    for (int s = 1; s <= 8 && s <= p.num_kb; s *= 2) {
      const int64_t resident = s == 8 ? 120 : s == 4 ? 140 : kNumSMs;  // CTAs of whole clusters that fit on the GPU
      const int64_t rounds = (tiles * s + resident - 1) / resident;
      const int64_t cost = rounds * ((p.num_kb + s - 1) / s * per_kb + 300) + (s > 1 ? 40 + 10 * s : 0);
      if (best == 0 || cost < best) { best = cost; best_tc = tc; best_s = s; }
    }
  }
  const int box_kb = best_tc == 1 ? 2 : 1;
  p.x_slots = w4t::kXRing / (p.nt * 128 * box_kb);
  if (p.x_slots > w4t::kMaxXSlots) p.x_slots = w4t::kMaxXSlots;
  if (best_tc == 1) p.x_slots &= ~1;  // (see the head of the file)
  // what two accumulators of nt columns leave of the 512 columns of tensor memory, 64 for a group
  p.acc_cols = p.nt <= 64 ? 64 : p.nt <= 96 && best_tc == 2 ? 96 : 128;
  p.groups = (512 - 2 * p.acc_cols) / 64;
  CUtensorMap mx, mw;
  int rc = make_tma_map_2d(&mx, x, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, K, M, ldx * 2, w4t::kK, p.nt, CU_TENSOR_MAP_SWIZZLE_128B);
  if (rc) return rc;
  if (k_packed)
    rc = make_tma_map_2d(&mw, qweight, CU_TENSOR_MAP_DATA_TYPE_INT32, 4, N, K / 8, N * 4, w4t::kCols, box_kb * w4t::kK / 8,
                         CU_TENSOR_MAP_SWIZZLE_NONE);
  else
    rc = make_tma_map_2d(&mw, qweight, CU_TENSOR_MAP_DATA_TYPE_INT32, 4, N / 8, K, N / 2, w4t::kCols / 8, box_kb * w4t::kK,
                         CU_TENSOR_MAP_SWIZZLE_NONE);
  if (rc) return rc;
  const int tiles = (int)((N + best_tc * w4t::kCols - 1) / (best_tc * w4t::kCols));
  if (best_tc == 1)
    return k_packed ? w4t::launch<1, 1>(mx, mw, p, tiles, best_s, st) : w4t::launch<1, 0>(mx, mw, p, tiles, best_s, st);
  return k_packed ? w4t::launch<2, 1>(mx, mw, p, tiles, best_s, st) : w4t::launch<2, 0>(mx, mw, p, tiles, best_s, st);
}

}  // namespace b200q
