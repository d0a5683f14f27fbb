// FP8 scaled-dot-product attention, forward: out = softmax(q k^T * scale + mask) v with q, k, v in
// e4m3 and the probabilities re-quantised to e4m3 for the second product.
//
// tcgen05 kernel (head dimension 128), persistent, one CTA per SM, 352 threads; a work item is one
// (batch x head, block of 128 queries), a step 256 keys, and group g of the softmax warps takes keys
// [128 g, 128 g + 128) of every step:
//   warp 0    TMA producer: query tiles, key tiles (twice, see below) and value tiles through
//             shared-memory rings (128-byte swizzle, no multicast)
//   warp 1    TMEM owner, issuer of S = Q K^T (kind::f8f6f4): in the first pass one product of
//             128 x 256 x 128 for both groups, in the second one per group, so that the groups need
//             not run in step
//   warps 2-9 softmax, two groups of four warps; thread = query row: tcgen05.ld of its score row,
//             scale / mask / exp2, the e4m3 probabilities written into the group's swizzled P tile
//   warp 10   issuer of O += P V, with P read from shared memory (K-major) and V through an MN-major
//             descriptor (V is stored [key][d]: no transpose)
// The roles run as one stream of steps that crosses item boundaries: the scores of the next step are
// asked for as soon as a group has its scores of this one in registers (before any of them is
// used), query tiles are double-buffered, and the next item's first scores are computed under the
// epilogue.  TMEM: columns [0, 256) = score region A (128 columns per group), [256, 512) = region B,
// the odd steps of the first pass; in the second pass its first 128 columns are the accumulator O.
//
// What bounds it: ex2 on the SFU, 16 a clock and SM: 1024 cycles per 128 x 128 scores, of which the
// tensor core is busy for 768.  Measured on the way here (causal, 16 heads x 8192 tokens): 583 us
// with one lane issuing both products of 128 keys and a CTA per item; 422 us as one stream; 326 us
// with the issuing roles run by whole warps (a lane spends 200 cycles per wait on addresses that a
// converged warp keeps in uniform registers); 274 us with 256 keys per
// step; 262 us with the two products issued by two warps and the groups out of step; 250 us with waits whose outcome
// is a vote.  What did not
// help: part of the exponentials as polynomials on the FMA pipe (the issue slots they take are as
// scarce), sixteen softmax warps with half a row each, a strict alternation of the groups' exponentials, a third group of
// warps that takes the row maxima of the next item meanwhile (16 heads x 8192 269 -> 252, but 8 x 4096 38 -> 43).
// Two passes over the keys: the first only takes the row maxima, the second recomputes the
// scores and forms exp(S - max) against the final maximum.  The probabilities are therefore
// quantised exactly where the CPU restatement quantises them (no running-maximum rescaling of
// an accumulator that already holds rounded products), the accumulator in TMEM is never read
// back and corrected, and the price is one extra Q K^T per block on a tensor pipe that the
// softmax arithmetic leaves half idle anyway.
//
// Every wait is bounded (tcgen05_ptx.cuh); a wait that runs out sets the device status word.
// Other head dimensions, and anything else the fast path does not take, run a plain CUDA kernel.
#include <cuda.h>

#include <type_traits>

#include "common.cuh"
#include "tcgen05_ptx.cuh"
#include "tma_host.cuh"

namespace b200q {

using namespace ptx;

namespace sdpa {

constexpr int kD = 128;        // head dimension of the tcgen05 path (bytes per row)
constexpr int kBM = 128;       // queries per CTA
constexpr int kBN = 128;       // keys per group and step
constexpr int kKSteps = 3;     // depth of the key ring, in steps (256 keys)
constexpr int kVTiles = 3;     // depth of the value ring, in tiles (128 keys)
constexpr int kTile = 128 * 128;  // bytes of 128 rows of any operand
constexpr int kThreads = 352;   // producer warp, two MMA warps, two softmax warpgroups
constexpr float kLog2e = 1.4426950408889634f;
constexpr float kMasked = -1.0e30f;

enum { kErrProducer = 301, kErrMma = 302, kErrSoftmax = 303 };

struct Params {
  void* out;               // bf16 or e4m3 [BH][L][D]
  int out_fp8;
  __nv_bfloat16* m_out;    // [BH][L] or null
  __nv_bfloat16* linv_out; // [BH][L] or null
  float* amax_s;           // or null; zeroed by the caller
  float* amax_o;
  const void* mask;        // additive (bf16 / f32) or boolean (1 = keep), or null
  int mask_kind;           // 0 none, 1 bf16, 2 f32, 3 bool
  int64_t mask_sb, mask_sl;  // element strides of the flattened batch x head index and of the query row
  const uint8_t* mask_end;   // behind the mask's last element
  int64_t BH, L, S;
  int kv_rep;              // query heads per key/value head: kv index = bh / kv_rep
  int causal;
  // the six scales of the operator: a device scalar when the pointer is set, else the host value
  const float* scale_dev[6];  // d_scale_q, d_scale_k, d_scale_v, q_scale_s, q_scale_o, d_scale_s
  float scale_host[6];
  int d_scale_s_given;     // 0: d_scale_s = 1 / q_scale_s
  float softmax_scale;
  int* status;
  void* zero_ptr[5];       // small buffers to clear (see b200q_sdpa_args)
  int zero_bytes[5];
  // derived in the kernel (Scales::load)
  float c_log2, q_scale_s, o_scale, q_scale_o;
};

// c_log2 = d_scale_q * d_scale_k * softmax scale * log2(e); o_scale = d_scale_s * d_scale_v
__device__ __forceinline__ void load_scales(Params& p) {
  float s[6];
#pragma unroll
  for (int i = 0; i < 6; ++i) s[i] = p.scale_dev[i] ? __ldg(p.scale_dev[i]) : p.scale_host[i];
  p.c_log2 = (s[0] * s[1]) * p.softmax_scale * kLog2e;
  p.q_scale_s = s[3];
  p.q_scale_o = s[4];
  p.o_scale = (p.d_scale_s_given ? s[5] : 1.f / s[3]) * s[2];
}

// the caller's zero-valued results: cleared by one thread of one block
__device__ __forceinline__ void clear_zero_list(const Params& p) {
  if (blockIdx.x != 0 || blockIdx.y != 0 || threadIdx.x != 0) return;
#pragma unroll
  for (int i = 0; i < 5; ++i)
    if (p.zero_ptr[i])
      for (int b = 0; b < p.zero_bytes[i]; ++b) static_cast<uint8_t*>(p.zero_ptr[i])[b] = 0;
}

// warp maximum of a non-negative float (bit patterns of non-negative floats order like the values)
__device__ __forceinline__ float ex2_approx(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float warp_max_f32_bits(float x) { return __uint_as_float(warp_max_u32(__float_as_uint(x))); }

// Term of the mask element at `a`, in the log2 domain.
template <int KIND>
__device__ __forceinline__ float mask_term(const uint8_t* a) {
  if (KIND == 1) return __bfloat162float(*reinterpret_cast<const __nv_bfloat16*>(a)) * kLog2e;
  if (KIND == 2) return *reinterpret_cast<const float*>(a) * kLog2e;
  return *a ? 0.f : kMasked;
}
__device__ __forceinline__ float mask_term(const Params& p, int64_t bh, int64_t row, int64_t key) {
  if (p.mask_kind == 0) return 0.f;
  const uint8_t* m = static_cast<const uint8_t*>(p.mask);
  const int64_t idx = bh * p.mask_sb + row * p.mask_sl + key;
  return p.mask_kind == 1 ? mask_term<1>(m + 2 * idx) : p.mask_kind == 2 ? mask_term<2>(m + 4 * idx) : mask_term<3>(m + idx);
}
template <int KIND>
constexpr int kMaskBytes = KIND == 1 ? 2 : KIND == 2 ? 4 : 1;  // of an element
// The same from element e of the words that mask_words() has read.
template <int KIND>
__device__ __forceinline__ float mask_term_at(const uint32_t* w, int e) {
  if (KIND == 1) return bf16_bits_to_float((w[e >> 1] >> (16 * (e & 1))) & 0xFFFFu) * kLog2e;
  if (KIND == 2) return __uint_as_float(w[e]) * kLog2e;
  return (w[e >> 2] >> (8 * (e & 3))) & 0xFFu ? 0.f : kMasked;
}
// The N elements of ES bytes from `a` on, of a row that ends at `row_end`, by aligned 16-byte loads and a shift: the lanes
// of a warp have different rows, so that every load takes as many L1 accesses as there are lanes, whatever its
// width, and the lines of 256 rows don't stay in what the rings leave of L1.  False, for the whole warp, when a
// piece would reach outside the mask [lo, hi); elements behind the row's end are undefined.  Against a load per
// element (64 heads x 1100 queries and keys): bool 1250 -> 163 us, fp32 1309 -> 215, bf16 1292 -> 167.
template <int ES, int N>
__device__ __forceinline__ bool mask_words(const uint8_t* a, const uint8_t* row_end, const uint8_t* lo, const uint8_t* hi, uint32_t* w) {
  constexpr int kPieces = N * ES / 16 + 1;
  const uint32_t off = (uint32_t)(reinterpret_cast<uintptr_t>(a) & 15);
  const uint8_t* g = a - off;
  const int64_t row_left = row_end - a;
  const int want = row_left >= N * ES ? N * ES : (int)row_left;  // bytes from `a` on
  const int reach = want > 0 ? (int)((off + want + 15) & ~15u) : 0;  // of the pieces, from g on
  if (__any_sync(0xFFFFFFFFu, reach > 0 && (g < lo || hi - g < reach))) return false;
  uint32_t t[4 * kPieces];
#pragma unroll
  for (int i = 0; i < kPieces; ++i) {
    uint4 v = make_uint4(0u, 0u, 0u, 0u);
    if (16 * i < reach) v = __ldg(reinterpret_cast<const uint4*>(g) + i);
    t[4 * i] = v.x, t[4 * i + 1] = v.y, t[4 * i + 2] = v.z, t[4 * i + 3] = v.w;
  }
  if (__any_sync(0xFFFFFFFFu, off)) {  // (shift by two words, by one, by bytes)
#pragma unroll
    for (int i = 0; i + 2 < 4 * kPieces; ++i) t[i] = off & 8 ? t[i + 2] : t[i];
#pragma unroll
    for (int i = 0; i + 3 < 4 * kPieces; ++i) t[i] = off & 4 ? t[i + 1] : t[i];
#pragma unroll
    for (int i = 0; i < N * ES / 4; ++i) t[i] = __funnelshift_r(t[i], t[i + 1], 8 * (off & 3));
  }
#pragma unroll
  for (int i = 0; i < N * ES / 4; ++i) w[i] = t[i];
  return true;
}

struct Smem {
  static constexpr int kQ = 0;                            // two query tiles
  static constexpr int kK = kQ + 2 * kTile;               // key ring
  static constexpr int kV = kK + kKSteps * 2 * kTile;     // value ring
  static constexpr int kP = kV + kVTiles * kTile;         // a P tile per group
  static constexpr int kStats = kP + 2 * kTile;           // [item parity][maxima | sums][2 groups][128 rows] fp32
  static constexpr int kBars = kStats + 2 * 2 * 2 * 128 * 4;
  // barriers: q_{full, empty}[2], s_{full, empty}[region][group], p_{full, empty}[group], o_{full, empty},
  // k_{full, empty}[kKSteps], v_{full, empty}[kVTiles]
  static constexpr int kNumBars = 4 + 8 + 4 + 2 + 2 * kKSteps + 2 * kVTiles;
  static constexpr int kTotal = kBars + kNumBars * 8 + 16;
};

// Work items in the order of their cost (under a causal mask the last query blocks have the most
// key blocks), dealt to the CTAs in a snake, so that the CTAs' totals differ by less than an item.
struct Item {
  int64_t bh, q0, kv;
  int nblk;   // blocks of 128 keys
  int steps;  // pairs of them; the last one may hold one block only
};
__device__ __forceinline__ bool get_item(const Params& p, int round, Item* it) {
  const int64_t g = gridDim.x, b = blockIdx.x;
  const int64_t idx = (int64_t)round * g + ((round & 1) ? g - 1 - b : b);
  const int64_t qblocks = (p.L + kBM - 1) / kBM;
  if (idx >= qblocks * p.BH) return false;
  it->bh = idx % p.BH;
  it->q0 = (qblocks - 1 - idx / p.BH) * kBM;
  it->kv = it->bh / p.kv_rep;
  int64_t keys = p.S;  // (causal: keys beyond the block's last query are all masked)
  if (p.causal && it->q0 + kBM < keys) keys = it->q0 + kBM;
  it->nblk = (int)((keys + kBN - 1) / kBN);
  it->steps = (it->nblk + 1) / 2;
  return true;
}

// The score steps of all work items of this CTA as one stream (item by item: the first pass over its
// keys, then the second), which the producer and the score issuer walk ahead of the softmax warps.
struct ScoreStream {
  Item w;
  int it = 0, t = 0;
  bool more;
  __device__ __forceinline__ explicit ScoreStream(const Params& p) { more = get_item(p, 0, &w); }
  __device__ __forceinline__ bool first() const { return t == 0; }
  __device__ __forceinline__ bool last() const { return t + 1 == 2 * w.steps; }
  __device__ __forceinline__ bool second() const { return t >= w.steps; }
  __device__ __forceinline__ int step() const { return t < w.steps ? t : t - w.steps; }
  __device__ __forceinline__ void next(const Params& p) {
    if (++t == 2 * w.steps) {
      t = 0;
      more = get_item(p, ++it, &w);
    }
  }
};
// whether step j of the item has a second block of keys
__device__ __forceinline__ bool two_blocks(const Item& w, int j) { return 2 * j + 1 < w.nblk; }

// Packed fp32 arithmetic: two results per issue slot.
__device__ __forceinline__ uint64_t pack_f32x2(float lo, float hi) {
  uint64_t d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(lo), "f"(hi));
  return d;
}
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
__device__ __forceinline__ float max3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}

// First pass over 32 scores: their maximum.
__device__ __forceinline__ float chunk_max(const uint32_t* r, float m) {
  float m0 = m, m1 = kMasked;
#pragma unroll
  for (int e = 0; e < 32; e += 4) {
    m0 = max3(m0, __uint_as_float(r[e]), __uint_as_float(r[e + 1]));
    m1 = max3(m1, __uint_as_float(r[e + 2]), __uint_as_float(r[e + 3]));
  }
  return fmaxf(m0, m1);
}
// Second pass over 32 scores (keys 32 c ... of the block): exp2(score * mul + off) = probability * q_scale_s,
// added to the row sums and written as e4m3 into the thread's row of the P tile (two 16-byte
// pieces, XOR-swizzled by the row).
__device__ __forceinline__ void chunk_exp(const uint32_t* r, int c, uint64_t mul2, uint64_t off2, uint64_t* ls, uint8_t* prow, int row) {
  uint32_t w[8];
#pragma unroll
  for (int e = 0; e < 32; e += 4) {
    float x[4];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const uint64_t y2 = fma_f32x2(pack_f32x2(__uint_as_float(r[e + 2 * h]), __uint_as_float(r[e + 2 * h + 1])), mul2, off2);
      unpack_f32x2(y2, x[2 * h], x[2 * h + 1]);
      x[2 * h] = ex2_approx(x[2 * h]);
      x[2 * h + 1] = ex2_approx(x[2 * h + 1]);
      ls[h] = add_f32x2(ls[h], pack_f32x2(x[2 * h], x[2 * h + 1]));
    }
    // (the conversion saturates at 448: a probability scale beyond that cannot overflow)
    w[e >> 2] = cvt_fp8x2<B200Q_E4M3>(x[0], x[1]) | (cvt_fp8x2<B200Q_E4M3>(x[2], x[3]) << 16);
  }
  *reinterpret_cast<uint4*>(prow + (((2 * c) ^ (row & 7)) << 4)) = make_uint4(w[0], w[1], w[2], w[3]);
  *reinterpret_cast<uint4*>(prow + (((2 * c + 1) ^ (row & 7)) << 4)) = make_uint4(w[4], w[5], w[6], w[7]);
}

// MASK = Params::mask_kind
template <int MASK>
__global__ void __launch_bounds__(kThreads, 1)
sdpa_fp8_tcgen05_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                        const __grid_constant__ CUtensorMap map_v, const Params p_in) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + Smem::kBars);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + Smem::kNumBars);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const uint32_t sbase = smem_u32(smem);
  const uint32_t b0 = smem_u32(bars);
  // s_full / s_empty of region r and group g: + 8 * (2 r + g)
  const uint32_t bar_qf = b0, bar_qe = b0 + 16, bar_sf = b0 + 32, bar_se = b0 + 64, bar_pf = b0 + 96, bar_pe = b0 + 112,
                 bar_of = b0 + 128, bar_oe = b0 + 136, bar_kf = b0 + 144, bar_ke = bar_kf + 8 * kKSteps,
                 bar_vf = bar_ke + 8 * kKSteps, bar_ve = bar_vf + 8 * kVTiles;
  const int warp = uniform_warp_index(), lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int i = 0; i < kKSteps; ++i) { mbar_init(bar_kf + 8 * i, 1); mbar_init(bar_ke + 8 * i, 1); }
    for (int i = 0; i < kVTiles; ++i) { mbar_init(bar_vf + 8 * i, 1); mbar_init(bar_ve + 8 * i, 1); }
    for (int i = 0; i < 4; ++i) { mbar_init(bar_sf + 8 * i, 1); mbar_init(bar_se + 8 * i, 4); }  // one arrival per warp of the group
    for (int i = 0; i < 2; ++i) {
      mbar_init(bar_qf + 8 * i, 1); mbar_init(bar_qe + 8 * i, 1);
      mbar_init(bar_pf + 8 * i, 4); mbar_init(bar_pe + 8 * i, 1);
    }
    mbar_init(bar_of, 1); mbar_init(bar_oe, 8);
    *abort_flag = 0;
    fence_barrier_init();
    fence_proxy_async_smem();
    tma_prefetch_desc(&map_q); tma_prefetch_desc(&map_k); tma_prefetch_desc(&map_v);
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(tmem_slot), 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;  // score regions A, B; O is the first half of B
  pdl_enter();  // everything above may run under the tail of the kernel in front of this one
  Params p = p_in;
  load_scales(p);
  clear_zero_list(p);

  if (warp == 0) {
    // ------------------------------------------------------------ producer
    uint32_t ks = 0, kph = 0, vs = 0, vph = 0;
    ScoreStream ss(p);
    bool ok = true;
    auto load_k = [&]() {
      if (ss.first()) {
        const uint32_t qb = ss.it & 1;
        ok = mbar_wait_uniform(bar_qe + 8 * qb, ((ss.it >> 1) & 1) ^ 1, abort_flag, p.status, kErrProducer);
        if (!ok) return;
        if (elect_one()) {
          mbar_arrive_expect_tx(bar_qf + 8 * qb, kTile);
          tma_load_3d(sbase + Smem::kQ + qb * kTile, &map_q, bar_qf + 8 * qb, 0, (int)ss.w.q0, (int)ss.w.bh);
        }
      }
      ok = mbar_wait_uniform(bar_ke + 8 * ks, kph ^ 1, abort_flag, p.status, kErrProducer);
      if (!ok) return;
      if (elect_one()) {
        const uint32_t dst = sbase + Smem::kK + ks * (2 * kTile), full = bar_kf + 8 * ks;
        const bool two = two_blocks(ss.w, ss.step());
        mbar_arrive_expect_tx(full, two ? 2 * kTile : kTile);
        tma_load_3d(dst, &map_k, full, 0, ss.step() * (2 * kBN), (int)ss.w.kv);
        if (two) tma_load_3d(dst + kTile, &map_k, full, 0, ss.step() * (2 * kBN) + kBN, (int)ss.w.kv);
      }
      if (++ks == kKSteps) { ks = 0; kph ^= 1; }
      ss.next(p);
    };
    // (keys run two steps ahead of values: a key tile is wanted when its group still works on the step before)
    for (int a = 0; a < 2 && ss.more && ok; ++a) load_k();
    Item w;
    for (int it = 0; ok && get_item(p, it, &w); ++it)
      for (int t = 0; t < 2 * w.steps && ok; ++t) {
        if (ss.more) load_k();
        for (int b = 2 * (t - w.steps); ok && b >= 0 && b < 2 * (t - w.steps) + 2 && b < w.nblk; ++b) {
          ok = mbar_wait_uniform(bar_ve + 8 * vs, vph ^ 1, abort_flag, p.status, kErrProducer);
          if (!ok) break;
          if (elect_one()) {
            mbar_arrive_expect_tx(bar_vf + 8 * vs, kTile);
            tma_load_3d(sbase + Smem::kV + vs * kTile, &map_v, bar_vf + 8 * vs, 0, b * kBN, (int)w.kv);
          }
          if (++vs == kVTiles) { vs = 0; vph ^= 1; }
        }
      }
  } else if (warp == 1) {
    // ------------------------------------------------------------ issuer of the scores
    const uint32_t idesc2 = umma_idesc(0, 0, kBM, 2 * kBN), idesc1 = umma_idesc(0, 0, kBM, kBN);  // Q, K both K-major e4m3
    const uint64_t qd0 = smem_desc_k_sw128(sbase + Smem::kQ), kd0 = smem_desc_k_sw128(sbase + Smem::kK);
    constexpr uint32_t kTileStep = kTile >> 4;  // (the address field of a descriptor never carries out)
    uint32_t ks = 0, kph = 0;
    uint32_t eph = 0xFu;  // bit 2 r + g: parity of the next wait for that score buffer to be free
    for (ScoreStream ss(p); ss.more; ss.next(p)) {
      const uint32_t qb = ss.it & 1;
      const bool two = two_blocks(ss.w, ss.step());
      const uint64_t qd = qd0 + qb * kTileStep, kd = kd0 + ks * (2 * kTileStep);
      if (ss.first() && !mbar_wait_uniform(bar_qf + 8 * qb, (ss.it >> 1) & 1, abort_flag, p.status, kErrMma)) break;
      if (!mbar_wait_uniform(bar_kf + 8 * ks, kph, abort_flag, p.status, kErrMma)) break;
      if (!ss.second()) {
        const uint32_t reg = ss.step() & 1;
        // region B holds the accumulator of the item before until its epilogue has read it
        if (ss.step() == 1 && ss.it > 0 && !mbar_wait_uniform(bar_oe, (ss.it - 1) & 1, abort_flag, p.status, kErrMma)) break;
        if (!mbar_wait_uniform(bar_se + 16 * reg, (eph >> (2 * reg)) & 1, abort_flag, p.status, kErrMma)) break;
        if (two && !mbar_wait_uniform(bar_se + 16 * reg + 8, (eph >> (2 * reg + 1)) & 1, abort_flag, p.status, kErrMma)) break;
        tc_fence_after();
        if (elect_one()) {
          umma_f8_x4(tmem + reg * 256, qd, kd, two ? idesc2 : idesc1, 0u, 2, 2);
          umma_commit(bar_sf + 16 * reg);
          if (two) umma_commit(bar_sf + 16 * reg + 8);
          umma_commit(bar_ke + 8 * ks);
        }
        eph ^= (two ? 3u : 1u) << (2 * reg);
      } else {
        if (!mbar_wait_uniform(bar_se, eph & 1, abort_flag, p.status, kErrMma)) break;
        tc_fence_after();
        if (elect_one()) {
          umma_f8_x4(tmem, qd, kd, idesc1, 0u, 2, 2);
          umma_commit(bar_sf);
        }
        eph ^= 1u;
        if (two) {
          if (!mbar_wait_uniform(bar_se + 8, (eph >> 1) & 1, abort_flag, p.status, kErrMma)) break;
          tc_fence_after();
          if (elect_one()) {
            umma_f8_x4(tmem + 128, qd, kd + kTileStep, idesc1, 0u, 2, 2);
            umma_commit(bar_sf + 8);
          }
          eph ^= 2u;
        }
        if (elect_one()) {
          umma_commit(bar_ke + 8 * ks);
          if (ss.last()) umma_commit(bar_qe + 8 * qb);  // the query tile has been read for the last time
        }
      }
      if (++ks == kKSteps) { ks = 0; kph ^= 1; }
    }
  } else if (warp == 10) {
    // ------------------------------------------------------------ issuer of O += P V
    // (Its first product of an item may overwrite region B: both groups have met between the passes,
    // so the scores of the first pass are in registers and the item before has been stored.)
    const uint32_t idesc_o = umma_idesc_major(0, 0, kBM, kD, 0, 1);           // P K-major, V MN-major
    const uint64_t pd0 = smem_desc_k_sw128(sbase + Smem::kP), vd0 = smem_desc_mn_sw128(sbase + Smem::kV, 128 * 128, 1024);
    constexpr uint32_t kTileStep = kTile >> 4;
    uint32_t vs = 0, vph = 0, pph = 0;  // pph bit g: parity of group g's next P tile
    Item w;
    bool ok = true;
    for (int it = 0; ok && get_item(p, it, &w); ++it)
      for (int b = 0; b < w.nblk; ++b) {
        const uint32_t g = b & 1;
        ok = mbar_wait_uniform(bar_vf + 8 * vs, vph, abort_flag, p.status, kErrMma) &&
             mbar_wait_uniform(bar_pf + 8 * g, (pph >> g) & 1, abort_flag, p.status, kErrMma);
        if (!ok) break;
        tc_fence_after();
        if (elect_one()) {
          umma_f8_x4(tmem + 256, pd0 + g * kTileStep, vd0 + vs * kTileStep, idesc_o, b > 0 ? 1u : 0u, 2, 256);
          umma_commit(bar_pe + 8 * g);
          umma_commit(bar_ve + 8 * vs);
          if (b + 1 == w.nblk) umma_commit(bar_of);
        }
        pph ^= 1u << g;
        if (++vs == kVTiles) { vs = 0; vph ^= 1; }
      }
  } else {
    // ------------------------------------------------------------ softmax (warps 2..9)
    // A warp whose wait ran out (ok = false) hands nothing on any more -- no P tile, so that no accumulator of
    // this or a later item is completed and no warp stores one -- and goes through its items only for the two
    // barriers among the softmax warps.
    const int grp = (warp - 2) >> 2;          // 0 / 1: which 128 keys of a step
    const int qtr = warp & 3;                 // TMEM lane quarter of this warp
    const int row = qtr * 32 + lane;          // query row inside the block = TMEM lane
    const uint32_t t_lane = tmem + ((uint32_t)(qtr * 32) << 16);
    float* stats = reinterpret_cast<float*>(smem + Smem::kStats);
    const float lq = log2f(p.q_scale_s);
    uint32_t fph = 0, pph = 1;                // parities: bit r of the next score tile in region r, of the P tile to be free
    bool ok = true;
    Item w;
    for (int it = 0; get_item(p, it, &w); ++it) {
      const int64_t qi = w.q0 + row;          // query index
      float* st_max = stats + (it & 1) * 512;
      float* st_sum = st_max + 256;
      float mx = kMasked;                     // row maximum, log2 domain
      float off = 0.f;                        // log2(q_scale_s) - mx (second pass)
      uint64_t ls[2] = {0ull, 0ull};          // partial row sums of the scaled probabilities

      // This group's keys of step j: scores -> row maximum (first pass) or e4m3 probabilities and
      // row sums (second pass).
      auto do_step = [&](int j, auto second_tag) {
        constexpr bool second = decltype(second_tag)::value;
        const uint32_t reg = second ? 0u : (uint32_t)(j & 1);
        const uint32_t t_score = t_lane + 256 * reg + 128 * grp, bar = 16 * reg + 8 * grp;
        const int64_t key0 = (int64_t)(2 * j + grp) * kBN;
        uint8_t* prow = smem + Smem::kP + grp * kTile + row * 128;
        ok = mbar_wait_uniform(bar_sf + bar, (fph >> reg) & 1, abort_flag, p.status, kErrSoftmax);
        if (!ok) return;
        fph ^= 1u << reg;
        tc_fence_after();
        auto release_scores = [&]() {
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(bar_se + bar);
        };
        auto wait_p_free = [&]() {
          ok = mbar_wait_uniform(bar_pe + 8 * grp, pph, abort_flag, p.status, kErrSoftmax);
          return ok;
        };
        // keys of the block that this row may see: the first `lim` of them
        int64_t lim64 = (p.causal && qi + 1 < p.S ? qi + 1 : p.S) - key0;
        const int lim = lim64 > kBN ? kBN : (int)lim64;
        const uint64_t off2 = pack_f32x2(off, off);
        if constexpr (MASK == 0) {
          // the whole row is taken into registers and the score buffer handed back before any use
          uint32_t r[128];
#pragma unroll
          for (int c = 0; c < 4; ++c) tmem_ld_32x32(t_score + 32 * c, r + 32 * c);
          tmem_ld_wait();
          release_scores();
          float mul = p.c_log2;
          // (the test is the same for all rows of the block, so that a warp takes one path)
          const bool masked = key0 + kBN > p.S || (p.causal && key0 + kBN - 1 > w.q0);
          if (masked || mul < 0.f) {
#pragma unroll
            for (int e = 0; e < 128; ++e) r[e] = __float_as_uint(e < lim ? __uint_as_float(r[e]) * mul : kMasked);
            mul = 1.f;
          }
          if (!second) {
            float m = kMasked;
#pragma unroll
            for (int c = 0; c < 4; ++c) m = chunk_max(r + 32 * c, m);
            mx = fmaxf(mx, m * mul);
          } else {
            const uint64_t mul2 = pack_f32x2(mul, mul);
            if (!wait_p_free()) return;
#pragma unroll
            for (int c = 0; c < 4; ++c) chunk_exp(r + 32 * c, c, mul2, off2, ls, prow, row);
          }
        } else {
          const uint64_t one2 = pack_f32x2(1.f, 1.f);
          const int64_t qm = qi < p.L ? qi : p.L - 1;
          if (second && !wait_p_free()) return;
          constexpr int es = kMaskBytes<MASK>;
          const uint8_t* lo = static_cast<const uint8_t*>(p.mask);
          const uint8_t* mrow = lo + (w.bh * p.mask_sb + qm * p.mask_sl) * es;
          const uint8_t* row_end = mrow + p.S * es;
          constexpr int n = es == 4 ? 16 : 32;  // (registers)
#pragma unroll 1
          for (int c = 0; c < 4; ++c) {
            uint32_t r[32];
            tmem_ld_32x32(t_score + 32 * c, r);
#pragma unroll
            for (int e0 = 0; e0 < 32; e0 += n) {
              uint32_t mw[n * es / 4];
              const uint8_t* a = mrow + (key0 + 32 * c + e0) * es;
              const bool wide = mask_words<es, n>(a, row_end, lo, p.mask_end, mw);
              if (e0 == 0) {
                tmem_ld_wait();
                if (c == 3) release_scores();
              }
              if (wide) {
#pragma unroll
                for (int e = 0; e < n; ++e)
                  r[e0 + e] = __float_as_uint(__uint_as_float(r[e0 + e]) * p.c_log2 + mask_term_at<MASK>(mw, e));
              } else {
                const int last = (int)(p.S - 1 - (key0 + 32 * c + e0));  // (the row's last key, seen from this one)
#pragma unroll
                for (int e = 0; e < n; ++e)
                  r[e0 + e] = __float_as_uint(__uint_as_float(r[e0 + e]) * p.c_log2 + mask_term<MASK>(a + (e < last ? e : last) * es));
              }
            }
#pragma unroll
            for (int e = 0; e < 32; ++e) r[e] = c * 32 + e < lim ? r[e] : __float_as_uint(kMasked);
            if (!second) mx = chunk_max(r, mx);
            else chunk_exp(r, c, one2, off2, ls, prow, row);
          }
        }
        if (second) {
          fence_proxy_async_smem();    // the P tile is read by the tensor core (async proxy)
          __syncwarp();
          if (lane == 0) mbar_arrive(bar_pf + 8 * grp);
          pph ^= 1;
        }
      };
      for (int j = 0; ok && 2 * j + grp < w.nblk; ++j) do_step(j, std::false_type{});
      // between the passes the groups meet: the row maximum over all blocks
      st_max[grp * 128 + row] = mx;
      named_bar_sync(1, 256);
      mx = fmaxf(st_max[row], st_max[128 + row]);
      off = lq - mx;
      for (int j = 0; ok && 2 * j + grp < w.nblk; ++j) do_step(j, std::true_type{});
      // ---- output: O / l, scaled.  The row sums of both groups are added, then group 0 writes the
      // first 64 output columns of its rows and group 1 the other 64.
      float l4[4];
      unpack_f32x2(ls[0], l4[0], l4[1]);
      unpack_f32x2(ls[1], l4[2], l4[3]);
      st_sum[grp * 128 + row] = (l4[0] + l4[1]) + (l4[2] + l4[3]);
      named_bar_sync(1, 256);
      const float lsum = (st_sum[row] + st_sum[128 + row]) / p.q_scale_s;
      ok = ok && mbar_wait_uniform(bar_of, it & 1, abort_flag, p.status, kErrSoftmax);
      if (!ok) continue;
      tc_fence_after();
      const float linv = lsum > 0.f ? 1.f / lsum : 0.f;
      const float osc = p.o_scale * linv;
      float amax_o = 0.f;
      const bool in = qi < p.L;
      uint32_t r[64];
      const int c0 = 64 * grp;
      tmem_ld_32x32(t_lane + 256 + c0, r);
      tmem_ld_32x32(t_lane + 256 + c0 + 32, r + 32);
      tmem_ld_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar_oe);
      float o[64];
#pragma unroll
      for (int e = 0; e < 64; ++e) {
        o[e] = __uint_as_float(r[e]) * osc;
        amax_o = fmaxf(amax_o, fabsf(o[e]));
      }
      if (in) {
        if (p.out_fp8) {
          uint8_t* dst = static_cast<uint8_t*>(p.out) + (w.bh * p.L + qi) * kD + c0;
          uint32_t b[16];
#pragma unroll
          for (int e = 0; e < 64; e += 4)
            b[e >> 2] = cvt_fp8x2<B200Q_E4M3>(clampf<B200Q_E4M3>(o[e] * p.q_scale_o), clampf<B200Q_E4M3>(o[e + 1] * p.q_scale_o)) |
                        (cvt_fp8x2<B200Q_E4M3>(clampf<B200Q_E4M3>(o[e + 2] * p.q_scale_o), clampf<B200Q_E4M3>(o[e + 3] * p.q_scale_o)) << 16);
#pragma unroll
          for (int e = 0; e < 16; e += 4) *reinterpret_cast<uint4*>(dst + 4 * e) = make_uint4(b[e], b[e + 1], b[e + 2], b[e + 3]);
        } else {
          __nv_bfloat16* dst = static_cast<__nv_bfloat16*>(p.out) + (w.bh * p.L + qi) * kD + c0;
#pragma unroll
          for (int e = 0; e < 64; e += 8)
            *reinterpret_cast<uint4*>(dst + e) = make_uint4(pack_bf16x2(o[e], o[e + 1]), pack_bf16x2(o[e + 2], o[e + 3]),
                                                          pack_bf16x2(o[e + 4], o[e + 5]), pack_bf16x2(o[e + 6], o[e + 7]));
        }
        if (grp == 0) {
          if (p.m_out) p.m_out[w.bh * p.L + qi] = __float2bfloat16_rn(mx / kLog2e);
          if (p.linv_out) p.linv_out[w.bh * p.L + qi] = __float2bfloat16_rn(linv);
        }
      }
      // amax of the probabilities (1 / l of a row is its largest probability) and of the output
      if (p.amax_s && grp == 0) {
        const float a = warp_max_f32_bits(in ? linv : 0.f);
        if (lane == 0 && a > 0.f) atomicMax(reinterpret_cast<unsigned int*>(p.amax_s), __float_as_uint(a));
      }
      if (p.amax_o) {
        const float a = warp_max_f32_bits(in ? amax_o : 0.f);
        if (lane == 0 && a > 0.f) atomicMax(reinterpret_cast<unsigned int*>(p.amax_o), __float_as_uint(a));
      }
    }
  }

  // ---------------------------------------------------------------- teardown
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (*abort_flag) {
    for (int i = 0; i < 200; ++i) __nanosleep(1000);
    __syncthreads();
  }
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

// ------------------------------------------------------------------------ plain kernel
// Any head dimensions up to 256: one block of 128 threads per (batch x head, query).  Same two
// passes, same quantisation points; scores of a block of 128 keys go through shared memory.
__global__ void __launch_bounds__(128) sdpa_fp8_plain_kernel(const uint8_t* __restrict__ q, const uint8_t* __restrict__ k,
                                                             const uint8_t* __restrict__ v, int dqk, int dv, const Params p_in) {
  Params p = p_in;
  load_scales(p);
  clear_zero_list(p);
  __shared__ float s_q[256];
  __shared__ float s_p[128];
  __shared__ float s_red[4];
  const int64_t bh = blockIdx.y, qi = blockIdx.x, kvh = bh / p.kv_rep;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  for (int d = tid; d < dqk; d += 128) s_q[d] = fp8_to_float<B200Q_E4M3>(q[(bh * p.L + qi) * dqk + d]);
  __syncthreads();
  int64_t keys = p.S;
  if (p.causal && qi + 1 < keys) keys = qi + 1;
  auto score = [&](int64_t key) {
    float acc = 0.f;
    const uint8_t* kr = k + (kvh * p.S + key) * dqk;
    for (int d = 0; d < dqk; ++d) acc += s_q[d] * fp8_to_float<B200Q_E4M3>(kr[d]);
    float x = acc * p.c_log2;
    if (p.mask_kind) x += mask_term(p, bh, qi, key);
    return x;
  };
  auto block_max = [&](float x) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x = fmaxf(x, __shfl_xor_sync(0xFFFFFFFFu, x, o));
    __syncthreads();
    if (lane == 0) s_red[wid] = x;
    __syncthreads();
    return fmaxf(fmaxf(s_red[0], s_red[1]), fmaxf(s_red[2], s_red[3]));
  };
  float mx = kMasked;
  for (int64_t k0 = 0; k0 < keys; k0 += 128)
    if (k0 + tid < keys) mx = fmaxf(mx, score(k0 + tid));
  mx = block_max(mx);
  float lsum = 0.f;
  float acc0 = 0.f, acc1 = 0.f;  // output elements tid and tid + 128
  for (int64_t k0 = 0; k0 < keys; k0 += 128) {
    float pr = 0.f;
    if (k0 + tid < keys) pr = exp2f(score(k0 + tid) - mx);
    lsum += pr;
    const float p8 = fp8_to_float<B200Q_E4M3>(cvt_fp8x2<B200Q_E4M3>(fminf(pr * p.q_scale_s, 448.f), 0.f) & 0xFFu);
    __syncthreads();
    s_p[tid] = p8;
    __syncthreads();
    const int n = (int)(keys - k0 < 128 ? keys - k0 : 128);
    for (int j = 0; j < n; ++j) {
      const uint8_t* vr = v + (kvh * p.S + k0 + j) * dv;
      if (tid < dv) acc0 += s_p[j] * fp8_to_float<B200Q_E4M3>(vr[tid]);
      if (tid + 128 < dv) acc1 += s_p[j] * fp8_to_float<B200Q_E4M3>(vr[tid + 128]);
    }
  }
  // row sum over the block
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) lsum += __shfl_xor_sync(0xFFFFFFFFu, lsum, o);
  __syncthreads();
  if (lane == 0) s_red[wid] = lsum;
  __syncthreads();
  lsum = (s_red[0] + s_red[1]) + (s_red[2] + s_red[3]);
  const float linv = lsum > 0.f ? 1.f / lsum : 0.f;
  const float osc = p.o_scale * linv;
  float amax_o = 0.f;
  for (int h = 0; h < 2; ++h) {
    const int d = tid + 128 * h;
    if (d >= dv) continue;
    const float o = (h ? acc1 : acc0) * osc;
    amax_o = fmaxf(amax_o, fabsf(o));
    const int64_t idx = (bh * p.L + qi) * dv + d;
    if (p.out_fp8) static_cast<uint8_t*>(p.out)[idx] = (uint8_t)(cvt_fp8x2<B200Q_E4M3>(clampf<B200Q_E4M3>(o * p.q_scale_o), 0.f) & 0xFFu);
    else static_cast<__nv_bfloat16*>(p.out)[idx] = __float2bfloat16_rn(o);
  }
  if (tid == 0) {
    if (p.m_out) p.m_out[bh * p.L + qi] = __float2bfloat16_rn(mx / kLog2e);
    if (p.linv_out) p.linv_out[bh * p.L + qi] = __float2bfloat16_rn(linv);
    if (p.amax_s && linv > 0.f) atomicMax(reinterpret_cast<unsigned int*>(p.amax_s), __float_as_uint(linv));
  }
  if (p.amax_o) {
    const float a = warp_max_f32_bits(amax_o);
    if (lane == 0 && a > 0.f) atomicMax(reinterpret_cast<unsigned int*>(p.amax_o), __float_as_uint(a));
  }
}

static int make_map_3d(CUtensorMap* map, const void* base, int64_t d_bytes, int64_t rows, int64_t batch) {
  EncodeTiledFn enc = get_encode_fn();
  if (!enc) return B200Q_ERR_CUDA;
  cuuint64_t dims[3] = {(cuuint64_t)d_bytes, (cuuint64_t)rows, (cuuint64_t)batch};
  cuuint64_t strides[2] = {(cuuint64_t)d_bytes, (cuuint64_t)(d_bytes * rows)};
  cuuint32_t box[3] = {128, 128, 1};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, const_cast<void*>(base), dims, strides, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? B200Q_OK : B200Q_ERR_CUDA;
}

}  // namespace sdpa

int sdpa_fp8_fwd_impl(const b200q_sdpa_args& a, cudaStream_t st) {
  const void *q = a.q, *k = a.k, *v = a.v;
  void* out = a.out;
  const int64_t BH = a.BH, L = a.L, S = a.S;
  const int dqk = a.dqk, dv = a.dv, kv_rep = a.kv_rep, force_plain = a.force_plain;
  sdpa::Params p;
  p.out = out; p.out_fp8 = a.out_dtype == B200Q_E4M3;
  p.m_out = static_cast<__nv_bfloat16*>(a.m_out); p.linv_out = static_cast<__nv_bfloat16*>(a.linv_out);
  p.amax_s = a.amax_s; p.amax_o = a.amax_o;
  p.mask = a.mask; p.mask_kind = a.mask ? a.mask_kind : 0; p.mask_sb = a.mask_sb; p.mask_sl = a.mask_sl;
  p.mask_end = p.mask_kind ? static_cast<const uint8_t*>(a.mask) +
                                 ((a.BH - 1) * a.mask_sb + (a.L - 1) * a.mask_sl + a.S) * (a.mask_kind == 1 ? 2 : a.mask_kind == 2 ? 4 : 1)
                           : nullptr;
  p.BH = BH; p.L = L; p.S = S; p.kv_rep = kv_rep; p.causal = a.causal;
  const float* devs[6] = {a.d_scale_q, a.d_scale_k, a.d_scale_v, a.q_scale_s, a.q_scale_o, a.d_scale_s};
  const float hosts[6] = {a.d_scale_q_host, a.d_scale_k_host, a.d_scale_v_host, a.q_scale_s_host, a.q_scale_o_host, a.d_scale_s_host};
  for (int i = 0; i < 6; ++i) { p.scale_dev[i] = devs[i]; p.scale_host[i] = hosts[i]; }
  p.d_scale_s_given = a.d_scale_s_given;
  p.softmax_scale = a.softmax_scale;
  for (int i = 0; i < 5; ++i) { p.zero_ptr[i] = a.zero_ptr[i]; p.zero_bytes[i] = a.zero_bytes[i]; }
  p.c_log2 = p.q_scale_s = p.o_scale = p.q_scale_o = 0.f;
  p.status = device_status_ptr();
  if (!p.status) return B200Q_ERR_CUDA;
  if (BH > 65535) return B200Q_ERR_TOO_LARGE;
  const bool aligned = ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k) | reinterpret_cast<uintptr_t>(v) |
                         reinterpret_cast<uintptr_t>(out)) & 15) == 0;
  if (!force_plain && dqk == sdpa::kD && dv == sdpa::kD && aligned && S >= 1) {
    CUtensorMap mq, mk, mv;
    int rc = sdpa::make_map_3d(&mq, q, dqk, L, BH);
    if (!rc) rc = sdpa::make_map_3d(&mk, k, dqk, S, BH / kv_rep);
    if (!rc) rc = sdpa::make_map_3d(&mv, v, dv, S, BH / kv_rep);
    if (rc) return rc;
    constexpr int smem = sdpa::Smem::kTotal + 1024;
    static_assert(smem <= 227 * 1024 && smem > 116 * 1024, "one CTA per SM");
    static decltype(&sdpa::sdpa_fp8_tcgen05_kernel<0>) const kernels[4] = {
        sdpa::sdpa_fp8_tcgen05_kernel<0>, sdpa::sdpa_fp8_tcgen05_kernel<1>, sdpa::sdpa_fp8_tcgen05_kernel<2>, sdpa::sdpa_fp8_tcgen05_kernel<3>};
    const auto kern = kernels[p.mask_kind];
    static std::atomic<int> configured[4][kMaxDevices];
    const int dev = current_device_index();
    if (dev < 0) return B200Q_ERR_CUDA;
    if (!configured[p.mask_kind][dev].load(std::memory_order_acquire)) {
      B200Q_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
      configured[p.mask_kind][dev].store(1, std::memory_order_release);
    }
    const int64_t items = ((L + sdpa::kBM - 1) / sdpa::kBM) * BH;
    const unsigned grid = (unsigned)(items < kNumSMs ? items : kNumSMs);
    launch_dependent(kern, dim3(grid), dim3(sdpa::kThreads), smem, st, mq, mk, mv, p);
    B200Q_LAUNCH_CHECK();
    return B200Q_OK;
  }
  if (dqk > 256 || dv > 256 || dqk < 1 || dv < 1) return B200Q_ERR_UNSUPPORTED;
  dim3 grid((unsigned)L, (unsigned)BH);
  sdpa::sdpa_fp8_plain_kernel<<<grid, 128, 0, st>>>(static_cast<const uint8_t*>(q), static_cast<const uint8_t*>(k),
                                                    static_cast<const uint8_t*>(v), dqk, dv, p);
  B200Q_LAUNCH_CHECK();
  return B200Q_OK;
}

}  // namespace b200q
