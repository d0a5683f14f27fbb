// FP8 scaled-dot-product attention, forward: out = softmax(q k^T * scale + mask) v with q, k, v in
// e4m3 and the probabilities re-quantised to e4m3 for the second product.
//
// tcgen05 kernel (head dimension 128), persistent, one CTA per SM, 320 threads; a work item is one
// (batch x head, block of 128 queries):
//   warp 0    TMA producer: the query tile, then the key tiles (twice, see below) and value
//             tiles through two shared-memory rings (128-byte swizzle, no multicast)
//   warp 1    TMEM owner and MMA issuer: S = Q K^T (kind::f8f6f4, 128 x 128 x 32 per instruction)
//             into one of two score buffers in TMEM, and O += P V with P read from shared memory
//             (K-major) and V through an MN-major descriptor (V is stored [key][d]: no transpose)
//   warps 2-9 softmax, two groups of four warps; a group owns one of the two score buffers (it takes
//             every other key block) and thread = query row: tcgen05.ld of its score row, scale /
//             mask / exp2, the e4m3 probabilities written into the swizzled P tile for the second
//             product.
// The three roles run as one stream of tiles that crosses item boundaries: the scores of tile t + 2
// are asked for as soon as a group has its 128 scores of tile t in registers (before any of them is
// used), query tiles and output accumulators are double-buffered, and a group has two P tiles, so
// that neither product's latency, nor the epilogue of one item, nor the first loads of the next
// one leave the softmax warps waiting.
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
constexpr int kBN = 128;       // keys per block
constexpr int kStages = 3;     // key / value ring depth
constexpr int kTile = 128 * 128;  // bytes of every tile here
constexpr int kThreads = 320;   // producer warp, MMA warp, two softmax warpgroups
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

// mask term of (row, key) in the log2 domain
__device__ __forceinline__ float mask_term(const Params& p, int64_t bh, int64_t row, int64_t key) {
  if (p.mask_kind == 0) return 0.f;
  const int64_t idx = bh * p.mask_sb + row * p.mask_sl + key;
  if (p.mask_kind == 1) return __bfloat162float(static_cast<const __nv_bfloat16*>(p.mask)[idx]) * kLog2e;
  if (p.mask_kind == 2) return static_cast<const float*>(p.mask)[idx] * kLog2e;
  return static_cast<const uint8_t*>(p.mask)[idx] ? 0.f : kMasked;
}

struct Smem {
  static constexpr int kQ = 0;                            // two query tiles
  static constexpr int kK = kQ + 2 * kTile;
  static constexpr int kV = kK + kStages * kTile;
  static constexpr int kP = kV + kStages * kTile;         // two P tiles per group
  static constexpr int kStats = kP + 4 * kTile;           // [item parity][maxima | sums][2 groups][128 rows] fp32
  static constexpr int kBars = kStats + 2 * 2 * 2 * 128 * 4;
  // barriers: {q, o, s}_{full, empty}[2], {k, v}_{full, empty}[3], p_{full, empty}[4]
  static constexpr int kNumBars = 12 + 4 * kStages + 8;
  static constexpr int kTotal = kBars + kNumBars * 8 + 16;
};

// Work items in the order of their cost (under a causal mask the last query blocks have the most
// key blocks), dealt to the CTAs in a snake, so that the CTAs' totals differ by less than an item.
struct Item {
  int64_t bh, q0, kv;
  int nblk;
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
  return true;
}

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
// pieces, XOR-swizzled by the row).  2.5 issue slots per score: packed FFMA and FADD, ex2, half a convert.
__device__ __forceinline__ void chunk_exp(const uint32_t* r, int c, uint64_t mul2, uint64_t off2, uint64_t* ls, uint8_t* prow, int row) {
  uint32_t w[8];
#pragma unroll
  for (int e = 0; e < 32; e += 4) {
    float x[4];
    unpack_f32x2(fma_f32x2(pack_f32x2(__uint_as_float(r[e]), __uint_as_float(r[e + 1])), mul2, off2), x[0], x[1]);
    unpack_f32x2(fma_f32x2(pack_f32x2(__uint_as_float(r[e + 2]), __uint_as_float(r[e + 3])), mul2, off2), x[2], x[3]);
#pragma unroll
    for (int u = 0; u < 4; ++u) x[u] = ex2_approx(x[u]);
    ls[0] = add_f32x2(ls[0], pack_f32x2(x[0], x[1]));
    ls[1] = add_f32x2(ls[1], pack_f32x2(x[2], x[3]));
    // (the conversion saturates at 448: a probability scale beyond that cannot overflow)
    w[e >> 2] = cvt_fp8x2<B200Q_E4M3>(x[0], x[1]) | (cvt_fp8x2<B200Q_E4M3>(x[2], x[3]) << 16);
  }
  *reinterpret_cast<uint4*>(prow + (((2 * c) ^ (row & 7)) << 4)) = make_uint4(w[0], w[1], w[2], w[3]);
  *reinterpret_cast<uint4*>(prow + (((2 * c + 1) ^ (row & 7)) << 4)) = make_uint4(w[4], w[5], w[6], w[7]);
}

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
  const uint32_t bar_qf = b0, bar_qe = b0 + 16, bar_of = b0 + 32, bar_oe = b0 + 48, bar_sf = b0 + 64, bar_se = b0 + 80,
                 bar_kf = b0 + 96, bar_ke = bar_kf + 8 * kStages, bar_vf = bar_ke + 8 * kStages, bar_ve = bar_vf + 8 * kStages,
                 bar_pf = bar_ve + 8 * kStages, bar_pe = bar_pf + 32;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(bar_kf + 8 * s, 1); mbar_init(bar_ke + 8 * s, 1);
      mbar_init(bar_vf + 8 * s, 1); mbar_init(bar_ve + 8 * s, 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(bar_qf + 8 * a, 1); mbar_init(bar_qe + 8 * a, 1);
      mbar_init(bar_of + 8 * a, 1); mbar_init(bar_oe + 8 * a, 8);  // one arrival per softmax warp
      mbar_init(bar_sf + 8 * a, 1); mbar_init(bar_se + 8 * a, 4);  // one per warp of the group
    }
    for (int a = 0; a < 4; ++a) { mbar_init(bar_pf + 8 * a, 4); mbar_init(bar_pe + 8 * a, 1); }
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
  const uint32_t tmem = *tmem_slot;  // columns [0,128) S0, [128,256) S1, [256,384) O0, [384,512) O1
  pdl_enter();  // everything above may run under the tail of the kernel in front of this one
  Params p = p_in;
  load_scales(p);
  clear_zero_list(p);

  if (warp == 0) {
    // ------------------------------------------------------------ producer
    if (lane == 0) {
      uint32_t ks = 0, kph = 0, vs = 0, vph = 0;
      Item w;
      bool ok = true;
      for (int it = 0; ok && get_item(p, it, &w); ++it) {
        const uint32_t qb = it & 1;
        if (!mbar_wait(bar_qe + 8 * qb, ((it >> 1) & 1) ^ 1, abort_flag, p.status, kErrProducer)) break;
        mbar_arrive_expect_tx(bar_qf + 8 * qb, kTile);
        tma_load_3d(sbase + Smem::kQ + qb * kTile, &map_q, bar_qf + 8 * qb, 0, (int)w.q0, (int)w.bh);
        for (int t = 0; t < 2 * w.nblk; ++t) {
          const int j = t < w.nblk ? t : t - w.nblk;
          if (!mbar_wait(bar_ke + 8 * ks, kph ^ 1, abort_flag, p.status, kErrProducer)) { ok = false; break; }
          mbar_arrive_expect_tx(bar_kf + 8 * ks, kTile);
          tma_load_3d(sbase + Smem::kK + ks * kTile, &map_k, bar_kf + 8 * ks, 0, j * kBN, (int)w.kv);
          if (++ks == kStages) { ks = 0; kph ^= 1; }
          if (t >= w.nblk) {
            if (!mbar_wait(bar_ve + 8 * vs, vph ^ 1, abort_flag, p.status, kErrProducer)) { ok = false; break; }
            mbar_arrive_expect_tx(bar_vf + 8 * vs, kTile);
            tma_load_3d(sbase + Smem::kV + vs * kTile, &map_v, bar_vf + 8 * vs, 0, j * kBN, (int)w.kv);
            if (++vs == kStages) { vs = 0; vph ^= 1; }
          }
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer
    if (lane == 0) {
      const uint32_t idesc_s = umma_idesc(0, 0, kBM, kBN);                      // Q, K both K-major e4m3
      const uint32_t idesc_o = umma_idesc_major(0, 0, kBM, kD, 0, 1);           // P K-major, V MN-major
      // The score stream runs two tiles ahead of the P V stream; st / sit / sw = its next tile.
      uint32_t ks = 0, kph = 0, vs = 0, vph = 0, sn = 0;   // sn: tiles issued; tile n goes to buffer n & 1
      int st = 0, sit = 0;
      Item sw;
      bool more = get_item(p, 0, &sw), ok = true;
      auto issue_s = [&]() {  // S of the next tile of the stream
        const uint32_t sb = sn & 1, qb = sit & 1;
        if (st == 0 && !mbar_wait(bar_qf + 8 * qb, (sit >> 1) & 1, abort_flag, p.status, kErrMma)) return false;
        if (!mbar_wait(bar_kf + 8 * ks, kph, abort_flag, p.status, kErrMma)) return false;
        if (!mbar_wait(bar_se + 8 * sb, ((sn >> 1) & 1) ^ 1, abort_flag, p.status, kErrMma)) return false;
        tc_fence_after();
        const uint64_t qd = smem_desc_k_sw128(sbase + Smem::kQ + qb * kTile);
        const uint64_t kd = smem_desc_k_sw128(sbase + Smem::kK + ks * kTile);
#pragma unroll
        for (int k = 0; k < 4; ++k) umma_f8(tmem + sb * 128, qd + 2 * k, kd + 2 * k, idesc_s, k > 0 ? 1u : 0u);
        umma_commit(bar_ke + 8 * ks);
        umma_commit(bar_sf + 8 * sb);
        if (++ks == kStages) { ks = 0; kph ^= 1; }
        ++sn;
        if (++st == 2 * sw.nblk) {
          umma_commit(bar_qe + 8 * qb);  // the query tile has been read for the last time
          st = 0;
          more = get_item(p, ++sit, &sw);
        }
        return true;
      };
      for (int a = 0; a < 2 && more && ok; ++a) ok = issue_s();
      uint32_t pc[2] = {0, 0};  // P tiles consumed so far, per group
      Item w;
      for (int it = 0; ok && get_item(p, it, &w); ++it) {
        const uint32_t ob = it & 1, o_tmem = tmem + 256 + 128 * ob;
        for (int t = 0; t < 2 * w.nblk && ok; ++t) {
          if (more) ok = issue_s();
          if (!ok || t < w.nblk) continue;
          // O += P_j V_j
          const int j = t - w.nblk, grp = t & 1;
          const uint32_t pb = 2 * grp + (pc[grp] & 1), pph = (pc[grp] >> 1) & 1;
          if (j == 0) ok = mbar_wait(bar_oe + 8 * ob, ((it >> 1) & 1) ^ 1, abort_flag, p.status, kErrMma);
          ok = ok && mbar_wait(bar_vf + 8 * vs, vph, abort_flag, p.status, kErrMma) &&
               mbar_wait(bar_pf + 8 * pb, pph, abort_flag, p.status, kErrMma);
          if (!ok) break;
          tc_fence_after();
          const uint64_t pd = smem_desc_k_sw128(sbase + Smem::kP + pb * kTile);
          const uint64_t vd = smem_desc_mn_sw128(sbase + Smem::kV + vs * kTile, 128 * 128, 1024);
#pragma unroll
          for (int k = 0; k < 4; ++k) umma_f8(o_tmem, pd + 2 * k, vd + 256 * k, idesc_o, (j > 0 || k > 0) ? 1u : 0u);
          umma_commit(bar_ve + 8 * vs);
          umma_commit(bar_pe + 8 * pb);
          if (++vs == kStages) { vs = 0; vph ^= 1; }
          ++pc[grp];
        }
        if (ok) umma_commit(bar_of + 8 * ob);
      }
    }
  } else {
    // ------------------------------------------------------------ softmax (warps 2..9)
    // A wait that runs out sets the abort flag, on which every later wait gives up at once: the
    // loops below then run to their end on whatever is there, with all barriers among the softmax
    // warps in place, and nothing is stored.
    const int grp = (warp - 2) >> 2;          // 0 / 1: the score buffer (and tiles t = grp mod 2) of this group
    const int qtr = warp & 3;                 // TMEM lane quarter of this warp
    const int row = qtr * 32 + lane;          // query row inside the block = TMEM lane
    const uint32_t t_lane = tmem + ((uint32_t)(qtr * 32) << 16);
    const uint32_t t_score = t_lane + grp * 128;
    float* stats = reinterpret_cast<float*>(smem + Smem::kStats);
    const float lq = log2f(p.q_scale_s);
    uint32_t sc = 0, pc = 0;                  // tiles of this group so far; P tiles so far
    Item w;
    for (int it = 0; get_item(p, it, &w); ++it) {
      const int64_t qi = w.q0 + row;          // query index
      float* st_max = stats + (it & 1) * 512;
      float* st_sum = st_max + 256;
      float mx = kMasked;                     // row maximum, log2 domain
      float off = 0.f;                        // log2(q_scale_s) - mx (second pass)
      uint64_t ls[2] = {0ull, 0ull};          // partial row sums of the scaled probabilities

      // One key block of this group: scores -> row maximum (first pass) or e4m3 probabilities and
      // row sums (second pass).
      auto do_tile = [&](int j, auto second_tag) {
        constexpr bool second = decltype(second_tag)::value;
        const uint32_t pb = 2 * grp + (pc & 1);
        const int64_t key0 = (int64_t)j * kBN;
        uint8_t* prow = smem + Smem::kP + pb * kTile + row * 128;
        mbar_wait(bar_sf + 8 * grp, sc & 1, abort_flag, p.status, kErrSoftmax);
        ++sc;
        if (second) mbar_wait(bar_pe + 8 * pb, ((pc >> 1) & 1) ^ 1, abort_flag, p.status, kErrSoftmax);
        tc_fence_after();
        auto release_scores = [&]() {
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(bar_se + 8 * grp);
        };
        // keys of the block that this row may see: the first `lim` of them
        int64_t lim64 = (p.causal && qi + 1 < p.S ? qi + 1 : p.S) - key0;
        const int lim = lim64 > kBN ? kBN : (int)lim64;
        const uint64_t off2 = pack_f32x2(off, off);
        if (p.mask_kind == 0) {
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
#pragma unroll
            for (int c = 0; c < 4; ++c) chunk_exp(r + 32 * c, c, mul2, off2, ls, prow, row);
          }
        } else {
          const uint64_t one2 = pack_f32x2(1.f, 1.f);
          const int64_t qm = qi < p.L ? qi : p.L - 1;
#pragma unroll 1
          for (int c = 0; c < 4; ++c) {
            uint32_t r[32];
            tmem_ld_32x32(t_score + 32 * c, r);
            tmem_ld_wait();
            if (c == 3) release_scores();
#pragma unroll
            for (int e = 0; e < 32; ++e) {
              const int64_t key = key0 + c * 32 + e;
              float v = __uint_as_float(r[e]) * p.c_log2 + mask_term(p, w.bh, qm, key < p.S ? key : p.S - 1);
              r[e] = __float_as_uint(c * 32 + e < lim ? v : kMasked);
            }
            if (!second) mx = chunk_max(r, mx);
            else chunk_exp(r, c, one2, off2, ls, prow, row);
          }
        }
        if (second) {
          fence_proxy_async_smem();    // the P tile is read by the tensor core (async proxy)
          __syncwarp();
          if (lane == 0) mbar_arrive(bar_pf + 8 * pb);
          ++pc;
        }
      };
      // first pass: this group's tiles t = grp, grp + 2, ... < nblk
      for (int t = grp; t < w.nblk; t += 2) do_tile(t, std::false_type{});
      // between the passes the groups meet: the row maximum over all blocks
      st_max[grp * 128 + row] = mx;
      named_bar_sync(1, 256);
      mx = fmaxf(st_max[row], st_max[128 + row]);
      off = lq - mx;
      // second pass: tiles t = nblk ... 2 nblk - 1 with t = grp (mod 2)
      for (int j = (w.nblk & 1) == grp ? 0 : 1; j < w.nblk; j += 2) do_tile(j, std::true_type{});
      // ---- output: O / l, scaled.  The row sums of both groups are added, then group 0 writes the
      // first 64 output columns of its rows and group 1 the other 64.
      float l4[4];
      unpack_f32x2(ls[0], l4[0], l4[1]);
      unpack_f32x2(ls[1], l4[2], l4[3]);
      st_sum[grp * 128 + row] = (l4[0] + l4[1]) + (l4[2] + l4[3]);
      named_bar_sync(1, 256);
      const float lsum = (st_sum[row] + st_sum[128 + row]) / p.q_scale_s;
      mbar_wait(bar_of + 8 * (it & 1), (it >> 1) & 1, abort_flag, p.status, kErrSoftmax);
      tc_fence_after();
      const float linv = lsum > 0.f ? 1.f / lsum : 0.f;
      const float osc = p.o_scale * linv;
      float amax_o = 0.f;
      const bool in = qi < p.L && !*abort_flag;
      uint32_t r[64];
      const int c0 = 64 * grp;
      tmem_ld_32x32(t_lane + 256 + 128 * (it & 1) + c0, r);
      tmem_ld_32x32(t_lane + 256 + 128 * (it & 1) + c0 + 32, r + 32);
      tmem_ld_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar_oe + 8 * (it & 1));
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
    static std::atomic<int> configured[kMaxDevices];
    const int dev = current_device_index();
    if (dev < 0) return B200Q_ERR_CUDA;
    if (!configured[dev].load(std::memory_order_acquire)) {
      B200Q_CUDA_OK(cudaFuncSetAttribute(sdpa::sdpa_fp8_tcgen05_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
      configured[dev].store(1, std::memory_order_release);
    }
    const int64_t items = ((L + sdpa::kBM - 1) / sdpa::kBM) * BH;
    const unsigned grid = (unsigned)(items < kNumSMs ? items : kNumSMs);
    launch_dependent(sdpa::sdpa_fp8_tcgen05_kernel, dim3(grid), dim3(sdpa::kThreads), smem, st, mq, mk, mv, p);
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
