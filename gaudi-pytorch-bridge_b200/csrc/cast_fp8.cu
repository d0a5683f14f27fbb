// cast_to_fp8 / cast_from_fp8 / swiglu_cast_fp8: single-pass, HBM-bound kernels.
//
// Each thread moves 16 elements per step with 128-bit loads and stores; the amax of
// the unscaled input is folded into the same pass (integer max on the |x| bit pattern,
// warp shuffle, shared memory, one atomicMax per block).
#include "common.cuh"

#include <atomic>

namespace b200q {

enum ScaleClass { SC_ONE = 0, SC_COL = 1, SC_ROW = 2, SC_FULL = 3 };

struct CastParams {
  const void* in;
  void* out;
  const float* scale;  // device scale (SCALAR_DEV / PER_COL / PER_ROW / FULL) or null
  float scale_host;
  int has_scale;       // 0: no multiply at all
  int scale_from_dev;  // SC_ONE only: read scale[0]
  int64_t n, cols;
  float* amax;
  uint64_t seed, offset, first_index;
  int mul_fp32;
  int start;  // StartMode
};

// How a cast is ordered after the kernel in front of it, and where its amax goes.
enum StartMode {
  kStartAfter = 0,       // waits for that kernel (or for the memset of the amax word) before its first access
  kStartBehindClear = 1, // that kernel cleared the amax word and has itself waited: only the atomicMax waits for it
  kStartCluster = 2,     // waits; the grid is one cluster, which reduces its amax by itself
};
__device__ __forceinline__ void cast_begin(int start) {
  if (start == kStartBehindClear) {
    pdl_release();
  } else {
    pdl_enter_spread();
    if (start == kStartCluster) cluster_amax_begin();
  }
}
__device__ __forceinline__ void cast_publish_amax(uint32_t amax_bits, float* amax, int start) {
  if (start == kStartCluster) cluster_amax_store(amax_bits, amax);
  else if (amax) block_amax_to_global(amax_bits, amax);
}

template <typename T>
struct InTraits;
template <>
struct InTraits<float> {
  static constexpr bool kIsBf16 = false;
};
template <>
struct InTraits<__nv_bfloat16> {
  static constexpr bool kIsBf16 = true;
};

// Product in the input dtype (bf16: scale and product both rounded to bf16) or in fp32.
template <bool BF16>
__device__ __forceinline__ float scaled(float x, float s, float s_in_dtype, int mul_fp32) {
  if (BF16 && !mul_fp32) return round_to_bf16(x * s_in_dtype);
  return x * s;
}


// Every NaN becomes the canonical byte 0x7F in both formats (the sign of a NaN that went
// through a multiply differs between CPUs and GPUs, so it is not carried).
template <int FMT>
__device__ __forceinline__ uint32_t nan_byte(float) {
  return 0x7Fu;
}

// Blocks per SM that the registers must leave room for (0: whatever the compiler takes; a stated 1 makes it take
// more).  Stochastic: four (64 registers), without which two of the fp32 forms take 68: row scales, 2^26 elements, 100 -> 92 us,
// element by element 565 -> 456.  bf16 with column scales: five (48), without which it takes 54: 60 -> 55 us.
template <typename InT, bool SR, int SC>
constexpr int cast_blocks_per_sm() { return SR ? 4 : InTraits<InT>::kIsBf16 && SC == SC_COL ? 5 : 0; }

template <typename InT, int FMT, bool SR, int SC>
__global__ void __launch_bounds__(256, cast_blocks_per_sm<InT, SR, SC>()) cast_to_fp8_kernel(CastParams p) {
  cast_begin(p.start);
  constexpr bool BF16 = InTraits<InT>::kIsBf16;
  const InT* __restrict__ in = static_cast<const InT*>(p.in);
  uint8_t* __restrict__ out = static_cast<uint8_t*>(p.out);
  const int64_t tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t nthreads = (int64_t)gridDim.x * blockDim.x;

  float s_one = 1.f;
  if (SC == SC_ONE && p.has_scale) s_one = p.scale_from_dev ? __ldg(p.scale) : p.scale_host;
  const float s_one_in = BF16 ? round_to_bf16(s_one) : s_one;
  const bool aligned = ((reinterpret_cast<uintptr_t>(in) | reinterpret_cast<uintptr_t>(out)) & 15) == 0 &&
                       ((SC != SC_FULL && SC != SC_COL) || (reinterpret_cast<uintptr_t>(p.scale) & 15) == 0);
  const bool col_vec = (SC != SC_COL && SC != SC_ROW) || (p.cols % 16 == 0);
  const int64_t nvec = (aligned && col_vec) ? p.n / 16 : 0;
  uint32_t amax_bits = 0;

  for (int64_t v = tid; v < nvec; v += nthreads) {
    const int64_t base = v * 16;
    float x[16];
    if (BF16) {
      const uint4* src = reinterpret_cast<const uint4*>(in + base);
      uint4 a = __ldcs(src), b = __ldcs(src + 1);
      uint32_t w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        x[2 * i] = __uint_as_float(w[i] << 16);
        x[2 * i + 1] = __uint_as_float(w[i] & 0xFFFF0000u);
      }
    } else {
      const float4* src = reinterpret_cast<const float4*>(in + base);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        float4 f = __ldcs(src + i);
        x[4 * i] = f.x; x[4 * i + 1] = f.y; x[4 * i + 2] = f.z; x[4 * i + 3] = f.w;
      }
    }
    if (p.amax) {
#pragma unroll
      for (int i = 0; i < 16; ++i) amax_bits = max(amax_bits, __float_as_uint(x[i]) & 0x7FFFFFFFu);
    }
    float s[16];
    if (SC == SC_COL) {
      const float4* sp = reinterpret_cast<const float4*>(p.scale + (base % p.cols));
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        float4 f = __ldg(sp + i);
        s[4 * i] = f.x; s[4 * i + 1] = f.y; s[4 * i + 2] = f.z; s[4 * i + 3] = f.w;
      }
    } else if (SC == SC_FULL) {
      const float4* sp = reinterpret_cast<const float4*>(p.scale + base);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        float4 f = __ldcs(sp + i);
        s[4 * i] = f.x; s[4 * i + 1] = f.y; s[4 * i + 2] = f.z; s[4 * i + 3] = f.w;
      }
    } else {
      float sv = (SC == SC_ROW) ? __ldg(p.scale + base / p.cols) : s_one;
#pragma unroll
      for (int i = 0; i < 16; ++i) s[i] = sv;
    }
    float y[16];
    bool any_nan = false;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      float si = (SC == SC_ONE) ? s_one_in : (BF16 ? round_to_bf16(s[i]) : s[i]);
      y[i] = p.has_scale ? scaled<BF16>(x[i], s[i], si, p.mul_fp32) : x[i];
      any_nan |= (y[i] != y[i]);
    }
    uint32_t o[4];
    if (SR) {
      // bf16 product: 8 random bits per element (one Philox block per 16 elements); otherwise 16
      const uint64_t g = p.first_index + (uint64_t)base;
      float z[16];
      const bool rb8 = BF16 && !p.mul_fp32;
      if ((p.first_index & 15) == 0) {
        if (rb8) {
          const uint4 r = philox4x32_10(g >> 4, p.seed, p.offset);
          const uint32_t rw[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
          for (int i = 0; i < 16; ++i) z[i] = sr_round<FMT, 8>(y[i], (rw[i >> 2] >> ((i & 3) * 8)) & 0xFFu);
        } else {
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const uint4 r = philox4x32_10((g >> 3) + h, p.seed, p.offset);
            const uint32_t rw[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
            for (int i = 0; i < 8; ++i) z[8 * h + i] = sr_round<FMT, 16>(y[8 * h + i], (rw[i >> 1] >> ((i & 1) * 16)) & 0xFFFFu);
          }
        }
      } else {
#pragma unroll 1
        for (int i = 0; i < 16; ++i)
          z[i] = rb8 ? sr_round<FMT, 8>(y[i], sr_random_bits<8>(g + i, p.seed, p.offset))
                     : sr_round<FMT, 16>(y[i], sr_random_bits<16>(g + i, p.seed, p.offset));
      }
#pragma unroll
      for (int i = 0; i < 4; ++i)
        o[i] = cvt_fp8x2<FMT>(z[4 * i], z[4 * i + 1]) | (cvt_fp8x2<FMT>(z[4 * i + 2], z[4 * i + 3]) << 16);
    } else {
#pragma unroll
      for (int i = 0; i < 4; ++i)
        o[i] = cvt_fp8x2<FMT>(clampf<FMT>(y[4 * i]), clampf<FMT>(y[4 * i + 1])) |
               (cvt_fp8x2<FMT>(clampf<FMT>(y[4 * i + 2]), clampf<FMT>(y[4 * i + 3])) << 16);
    }
    if (any_nan) {
#pragma unroll
      for (int i = 0; i < 16; ++i)
        if (y[i] != y[i]) {
          uint32_t sh = (i & 3) * 8;
          o[i >> 2] = (o[i >> 2] & ~(0xFFu << sh)) | (nan_byte<FMT>(y[i]) << sh);
        }
    }
    __stcs(reinterpret_cast<uint4*>(out + base), make_uint4(o[0], o[1], o[2], o[3]));
  }

  // scalar path: the tail, or everything when the fast path's alignment rules do not hold
  for (int64_t i = nvec * 16 + tid; i < p.n; i += nthreads) {
    float x = BF16 ? __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(in)[i])
                   : reinterpret_cast<const float*>(in)[i];
    if (p.amax) amax_bits = max(amax_bits, __float_as_uint(x) & 0x7FFFFFFFu);
    float y = x;
    if (p.has_scale) {
      float s = SC == SC_ONE ? s_one : SC == SC_COL ? p.scale[i % p.cols] : SC == SC_ROW ? p.scale[i / p.cols]
                                                                                       : p.scale[i];
      y = scaled<BF16>(x, s, BF16 ? round_to_bf16(s) : s, p.mul_fp32);
    }
    float z = clampf<FMT>(y);
    if (SR) {
      const uint64_t gi = p.first_index + (uint64_t)i;
      z = (BF16 && !p.mul_fp32) ? sr_round<FMT, 8>(y, sr_random_bits<8>(gi, p.seed, p.offset))
                                : sr_round<FMT, 16>(y, sr_random_bits<16>(gi, p.seed, p.offset));
    }
    uint32_t b = cvt_fp8x2<FMT>(z, 0.f) & 0xFFu;
    if (y != y) b = nan_byte<FMT>(y);
    out[i] = (uint8_t)b;
  }

  cast_publish_amax(amax_bits, p.amax, p.start);
}


// ------------------------------------------------------------------ bf16 -> fp8, RNE, fast path
// One scale for the whole chunk (per tensor or per row) and the product formed in bf16: the
// multiply is one packed bf16x2 instruction per two elements (exact product, one rounding to
// bf16 -- the same value as an fp32 multiply followed by a rounding to bf16), amax is a packed
// NaN-propagating max, and the saturating conversion instruction takes care of +-inf and of
// values beyond the format's maximum.  NaN bytes are made canonical on the packed output.
__device__ __forceinline__ uint32_t bf16x2_mul(uint32_t a, uint32_t b) {
  __nv_bfloat162 r = __hmul2(*reinterpret_cast<__nv_bfloat162*>(&a), *reinterpret_cast<__nv_bfloat162*>(&b));
  return *reinterpret_cast<uint32_t*>(&r);
}
// unsigned 16-bit minimum / maximum of both halves, one instruction each
__device__ __forceinline__ uint32_t min_u16x2(uint32_t a, uint32_t b) {
  uint32_t d;
  asm("min.u16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}
__device__ __forceinline__ uint32_t max_u16x2(uint32_t a, uint32_t b) {
  uint32_t d;
  asm("max.u16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}
__device__ __forceinline__ uint32_t bf16x2_max_nan(uint32_t a, uint32_t b) {
  __nv_bfloat162 r = __hmax2_nan(*reinterpret_cast<__nv_bfloat162*>(&a), *reinterpret_cast<__nv_bfloat162*>(&b));
  return *reinterpret_cast<uint32_t*>(&r);
}

// Replace every NaN code in four packed fp8 bytes by 0x7F.
template <int FMT>
__device__ __forceinline__ uint32_t canonical_nan_bytes(uint32_t w) {
  const uint32_t t = w & 0x7F7F7F7Fu;
  // e4m3: NaN is 0x7F; e5m2: NaN is 0x7D..0x7F (0x7C, inf, cannot come out of a saturating convert)
  const uint32_t hit = (t + (FMT == B200Q_E4M3 ? 0x01010101u : 0x03030303u)) & 0x80808080u;
  if (hit == 0u) return w;
  const uint32_t bytes = (hit >> 7) * 0xFFu;  // 0xFF in every NaN byte
  return (w & ~bytes) | (bytes & 0x7F7F7F7Fu);
}

template <int FMT>
__device__ __forceinline__ uint4 cast16_bf16_rne(const uint4 a, const uint4 b, uint32_t s2, bool has_scale,
                                                 uint32_t& amax2) {
  uint32_t w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
  uint32_t o[4];
#pragma unroll
  for (int i = 0; i < 8; ++i) amax2 = bf16x2_max_nan(amax2, w[i] & 0x7FFF7FFFu);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    uint32_t y0 = has_scale ? bf16x2_mul(w[2 * i], s2) : w[2 * i];
    uint32_t y1 = has_scale ? bf16x2_mul(w[2 * i + 1], s2) : w[2 * i + 1];
    uint32_t lo = cvt_fp8x2<FMT>(__uint_as_float(y0 << 16), __uint_as_float(y0 & 0xFFFF0000u));
    uint32_t hi = cvt_fp8x2<FMT>(__uint_as_float(y1 << 16), __uint_as_float(y1 & 0xFFFF0000u));
    o[i] = canonical_nan_bytes<FMT>(lo | (hi << 16));
  }
  return make_uint4(o[0], o[1], o[2], o[3]);
}

template <int FMT, bool PER_ROW>
__global__ void __launch_bounds__(256) cast_bf16_rne_fast_kernel(CastParams p) {
  cast_begin(p.start);
  const __nv_bfloat16* __restrict__ in = static_cast<const __nv_bfloat16*>(p.in);
  uint8_t* __restrict__ out = static_cast<uint8_t*>(p.out);
  const int64_t tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t nthreads = (int64_t)gridDim.x * blockDim.x;
  const int64_t nvec = p.n / 16;
  uint32_t s2 = 0;
  if (!PER_ROW && p.has_scale) {
    float s = p.scale_from_dev ? __ldg(p.scale) : p.scale_host;
    s2 = pack_bf16x2(s, s);
  }
  uint32_t amax2 = 0;
  int64_t v = tid;
  for (; v + nthreads < nvec; v += 2 * nthreads) {  // two independent chunks in flight per thread
    const int64_t b0 = v * 16, b1 = (v + nthreads) * 16;
    const uint4* s0 = reinterpret_cast<const uint4*>(in + b0);
    const uint4* s1 = reinterpret_cast<const uint4*>(in + b1);
    uint4 a0 = __ldcs(s0), a1 = __ldcs(s0 + 1), c0 = __ldcs(s1), c1 = __ldcs(s1 + 1);
    uint32_t sa = s2, sc = s2;
    if (PER_ROW) {
      float f0 = __ldg(p.scale + b0 / p.cols), f1 = __ldg(p.scale + b1 / p.cols);
      sa = pack_bf16x2(f0, f0);
      sc = pack_bf16x2(f1, f1);
    }
    __stcs(reinterpret_cast<uint4*>(out + b0), cast16_bf16_rne<FMT>(a0, a1, sa, p.has_scale, amax2));
    __stcs(reinterpret_cast<uint4*>(out + b1), cast16_bf16_rne<FMT>(c0, c1, sc, p.has_scale, amax2));
  }
  for (; v < nvec; v += nthreads) {
    const int64_t b0 = v * 16;
    const uint4* s0 = reinterpret_cast<const uint4*>(in + b0);
    uint4 a0 = __ldcs(s0), a1 = __ldcs(s0 + 1);
    uint32_t sa = s2;
    if (PER_ROW) {
      float f0 = __ldg(p.scale + b0 / p.cols);
      sa = pack_bf16x2(f0, f0);
    }
    __stcs(reinterpret_cast<uint4*>(out + b0), cast16_bf16_rne<FMT>(a0, a1, sa, p.has_scale, amax2));
  }
  // tail (fewer than 16 elements)
  uint32_t amax_bits = max(amax2 << 16, amax2 & 0xFFFF0000u);
  for (int64_t i = nvec * 16 + tid; i < p.n; i += nthreads) {
    float x = __bfloat162float(in[i]);
    amax_bits = max(amax_bits, __float_as_uint(x) & 0x7FFFFFFFu);
    float y = x;
    if (p.has_scale) {
      float s = PER_ROW ? p.scale[i / p.cols] : (p.scale_from_dev ? __ldg(p.scale) : p.scale_host);
      y = round_to_bf16(x * round_to_bf16(s));
    }
    uint32_t b = cvt_fp8x2<FMT>(y, 0.f) & 0xFFu;
    if (y != y) b = 0x7Fu;
    out[i] = (uint8_t)b;
  }
  cast_publish_amax(amax_bits, p.amax, p.start);
}

// ------------------------------------------------------------------ bf16 -> fp8, stochastic, fast path
// Same frame as the RNE fast path.  In the normal range a bf16 product needs only its low
// g = 4 (e4m3) or 5 (e5m2) mantissa bits resolved, so stochastic rounding is a packed integer
// add of g random bits to both halves of a bf16x2 word; one Philox block (16 random bytes) serves a
// 16-element chunk (2^26 elements to e5m2 45.4 -> 42.2 us against masks, shifts and conversions).  What bounds it
// are the integer multiplications of Philox as much as latency at three blocks per SM (80 registers; row scales
// without the bound 94 and two blocks: 109 -> 103 us to e4m3); five, with 48, spill: 53 us.  Chunks that hold a value below the smallest
// normal, an infinity or a NaN take the general per-element routine instead (same definition).
template <int FMT>
__device__ __forceinline__ uint4 cast16_bf16_sr(const uint4 a, const uint4 b, uint32_t s2, bool has_scale,
                                                uint32_t& amax2, uint64_t gi, uint64_t seed, uint64_t offset) {
  constexpr int g = (23 - Fp8Fmt<FMT>::kMant) - 16;
  constexpr uint32_t kMinNormalBf16 = (uint32_t)Fp8Fmt<FMT>::kEmin << 7;  // bf16 bits of 2^Emin
  uint32_t w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
  uint32_t y[8];
  uint32_t lo2 = 0xFFFFFFFFu, hi2 = 0;  // packed running min / max of the 15-bit magnitudes (both halves)
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    amax2 = bf16x2_max_nan(amax2, w[i] & 0x7FFF7FFFu);
    y[i] = has_scale ? bf16x2_mul(w[i], s2) : w[i];
    const uint32_t m = y[i] & 0x7FFF7FFFu;
    lo2 = min_u16x2(lo2, m);
    hi2 = max_u16x2(hi2, m);
  }
  const uint32_t lo_mag = min(lo2 & 0xFFFFu, lo2 >> 16), hi_mag = max(hi2 & 0xFFFFu, hi2 >> 16);
  const uint4 r = philox4x32_10(gi >> 4, seed, offset);
  const uint32_t rw[4] = {r.x, r.y, r.z, r.w};
  uint32_t o[4];
  if (lo_mag >= kMinNormalBf16 && hi_mag < 0x7F80u) {
    // The magnitude above the code of the smallest exponent, moved up so that the fp8 code is the high byte
    // of each half and the dropped g bits meet the top g bits of a whole random byte (the byte's other bits add
    // less than one unit of the value and cannot carry): no masks, no shifts and no conversions.  Values
    // past the largest code are cut to it first, as the saturating conversion would.  The product is taken
    // modulo 2^32 over both halves; each half of the difference is below 2^(16 - (8 - g)).
    constexpr uint32_t kBias = (uint32_t)(Fp8Fmt<FMT>::kEmin - 1) << 7;
    constexpr uint32_t kTop = kBias + ((FMT == B200Q_E4M3 ? 0x7Eu : 0x7Bu) << g);
    constexpr uint32_t kMul = 1u << (8 - g), kBoth = 0x00010001u;
    uint32_t t[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      // bytes 2*(i%2), 2*(i%2)+1 of word i/2 -> low bytes of the two halves
      const uint32_t rr = __byte_perm(rw[i >> 1], 0u, (i & 1) ? 0x4342 : 0x4140);
      const uint32_t m = min_u16x2(y[i] & 0x7FFF7FFFu, kTop * kBoth);
      t[i] = (m * kMul - (kBias * kBoth) * kMul) + rr;
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
      o[i] = __byte_perm(t[2 * i], t[2 * i + 1], 0x7531) | (__byte_perm(y[2 * i], y[2 * i + 1], 0x7531) & 0x80808080u);
  } else {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      uint32_t word = 0;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int e = 4 * i + j;
        const float v = __uint_as_float((e & 1) ? (y[e >> 1] & 0xFFFF0000u) : (y[e >> 1] << 16));
        const float z = sr_round<FMT, 8>(v, (rw[e >> 2] >> ((e & 3) * 8)) & 0xFFu);
        uint32_t byte = cvt_fp8x2<FMT>(z, 0.f) & 0xFFu;
        if (v != v) byte = 0x7Fu;
        word |= byte << (8 * j);
      }
      o[i] = word;
    }
  }
  return make_uint4(o[0], o[1], o[2], o[3]);
}

template <int FMT, bool PER_ROW>
__global__ void __launch_bounds__(256, 3) cast_bf16_sr_fast_kernel(CastParams p) {
  cast_begin(p.start);
  const __nv_bfloat16* __restrict__ in = static_cast<const __nv_bfloat16*>(p.in);
  uint8_t* __restrict__ out = static_cast<uint8_t*>(p.out);
  const int64_t tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t nthreads = (int64_t)gridDim.x * blockDim.x;
  const int64_t nvec = p.n / 16;
  uint32_t s2 = 0;
  if (!PER_ROW && p.has_scale) {
    float s = p.scale_from_dev ? __ldg(p.scale) : p.scale_host;
    s2 = pack_bf16x2(s, s);
  }
  uint32_t amax2 = 0;
  int64_t v = tid;
  for (; v + nthreads < nvec; v += 2 * nthreads) {
    const int64_t b0 = v * 16, b1 = (v + nthreads) * 16;
    const uint4* s0 = reinterpret_cast<const uint4*>(in + b0);
    const uint4* s1 = reinterpret_cast<const uint4*>(in + b1);
    uint4 a0 = __ldcs(s0), a1 = __ldcs(s0 + 1), c0 = __ldcs(s1), c1 = __ldcs(s1 + 1);
    uint32_t sa = s2, sc = s2;
    if (PER_ROW) {
      float f0 = __ldg(p.scale + b0 / p.cols), f1 = __ldg(p.scale + b1 / p.cols);
      sa = pack_bf16x2(f0, f0);
      sc = pack_bf16x2(f1, f1);
    }
    __stcs(reinterpret_cast<uint4*>(out + b0),
           cast16_bf16_sr<FMT>(a0, a1, sa, p.has_scale, amax2, p.first_index + (uint64_t)b0, p.seed, p.offset));
    __stcs(reinterpret_cast<uint4*>(out + b1),
           cast16_bf16_sr<FMT>(c0, c1, sc, p.has_scale, amax2, p.first_index + (uint64_t)b1, p.seed, p.offset));
  }
  for (; v < nvec; v += nthreads) {
    const int64_t b0 = v * 16;
    const uint4* s0 = reinterpret_cast<const uint4*>(in + b0);
    uint4 a0 = __ldcs(s0), a1 = __ldcs(s0 + 1);
    uint32_t sa = s2;
    if (PER_ROW) {
      float f0 = __ldg(p.scale + b0 / p.cols);
      sa = pack_bf16x2(f0, f0);
    }
    __stcs(reinterpret_cast<uint4*>(out + b0),
           cast16_bf16_sr<FMT>(a0, a1, sa, p.has_scale, amax2, p.first_index + (uint64_t)b0, p.seed, p.offset));
  }
  uint32_t amax_bits = max(amax2 << 16, amax2 & 0xFFFF0000u);
  for (int64_t i = nvec * 16 + tid; i < p.n; i += nthreads) {
    float x = __bfloat162float(in[i]);
    amax_bits = max(amax_bits, __float_as_uint(x) & 0x7FFFFFFFu);
    float y = x;
    if (p.has_scale) {
      float s = PER_ROW ? p.scale[i / p.cols] : (p.scale_from_dev ? __ldg(p.scale) : p.scale_host);
      y = round_to_bf16(x * round_to_bf16(s));
    }
    const float z = sr_round<FMT, 8>(y, sr_random_bits<8>(p.first_index + (uint64_t)i, p.seed, p.offset));
    uint32_t b = cvt_fp8x2<FMT>(z, 0.f) & 0xFFu;
    if (y != y) b = 0x7Fu;
    out[i] = (uint8_t)b;
  }
  cast_publish_amax(amax_bits, p.amax, p.start);
}

// ------------------------------------------------------------------ hybrid cast (e5m2 + e4m3 in one pass)
struct HybridParams {
  const void* in;
  uint8_t* out152;
  uint8_t* out143;
  const float* s152;
  const float* s143;
  float s152_host, s143_host;
  int has152, has143, dev152, dev143;
  int64_t n;
  float* amax;
  uint64_t seed, offset, first_index;
  int mul_fp32;
  int start;  // StartMode
};

// One read of the input, two fp8 outputs: e5m2 (RNE or stochastic) with its own per-tensor scale
// and e4m3 (always RNE) with its own.  4 bytes per bf16 element instead of 6 for two casts.
template <typename InT, bool SR>
__global__ void __launch_bounds__(256, SR ? 3 : 0) cast_hybrid_kernel(HybridParams p) {
  cast_begin(p.start);
  constexpr bool BF16 = InTraits<InT>::kIsBf16;
  const InT* __restrict__ in = static_cast<const InT*>(p.in);
  const int64_t tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t nthreads = (int64_t)gridDim.x * blockDim.x;
  float s5 = 1.f, s4 = 1.f;
  if (p.has152) s5 = p.dev152 ? __ldg(p.s152) : p.s152_host;
  if (p.has143) s4 = p.dev143 ? __ldg(p.s143) : p.s143_host;
  const float s5i = BF16 ? round_to_bf16(s5) : s5, s4i = BF16 ? round_to_bf16(s4) : s4;
  const bool aligned = ((reinterpret_cast<uintptr_t>(in) | reinterpret_cast<uintptr_t>(p.out152) |
                         reinterpret_cast<uintptr_t>(p.out143)) & 15) == 0 && (p.first_index & 15) == 0;
  const int64_t nvec = aligned ? p.n / 16 : 0;
  const bool rb8 = BF16 && !p.mul_fp32;
  uint32_t amax_bits = 0;
  for (int64_t v = tid; v < nvec; v += nthreads) {
    const int64_t base = v * 16;
    float x[16];
    if (BF16) {
      const uint4* src = reinterpret_cast<const uint4*>(in + base);
      uint4 a = __ldcs(src), b = __ldcs(src + 1);
      uint32_t w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        x[2 * i] = __uint_as_float(w[i] << 16);
        x[2 * i + 1] = __uint_as_float(w[i] & 0xFFFF0000u);
      }
    } else {
      const float4* src = reinterpret_cast<const float4*>(in + base);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        float4 f = __ldcs(src + i);
        x[4 * i] = f.x; x[4 * i + 1] = f.y; x[4 * i + 2] = f.z; x[4 * i + 3] = f.w;
      }
    }
    float y5[16], y4[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      amax_bits = max(amax_bits, __float_as_uint(x[i]) & 0x7FFFFFFFu);
      y5[i] = p.has152 ? scaled<BF16>(x[i], s5, s5i, p.mul_fp32) : x[i];
      y4[i] = p.has143 ? scaled<BF16>(x[i], s4, s4i, p.mul_fp32) : x[i];
    }
    if (SR) {
      const uint64_t g = p.first_index + (uint64_t)base;
      if (rb8) {
        const uint4 r = philox4x32_10(g >> 4, p.seed, p.offset);
        const uint32_t rw[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          const float z = sr_round<B200Q_E5M2, 8>(y5[i], (rw[i >> 2] >> ((i & 3) * 8)) & 0xFFu);
          y5[i] = z;
        }
      } else {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const uint4 r = philox4x32_10((g >> 3) + h, p.seed, p.offset);
          const uint32_t rw[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
          for (int i = 0; i < 8; ++i)
            y5[8 * h + i] = sr_round<B200Q_E5M2, 16>(y5[8 * h + i], (rw[i >> 1] >> ((i & 1) * 16)) & 0xFFFFu);
        }
      }
    }
    uint32_t o5[4], o4[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      o5[i] = canonical_nan_bytes<B200Q_E5M2>(cvt_fp8x2<B200Q_E5M2>(y5[4 * i], y5[4 * i + 1]) |
                                              (cvt_fp8x2<B200Q_E5M2>(y5[4 * i + 2], y5[4 * i + 3]) << 16));
      o4[i] = canonical_nan_bytes<B200Q_E4M3>(cvt_fp8x2<B200Q_E4M3>(y4[4 * i], y4[4 * i + 1]) |
                                              (cvt_fp8x2<B200Q_E4M3>(y4[4 * i + 2], y4[4 * i + 3]) << 16));
    }
    __stcs(reinterpret_cast<uint4*>(p.out152 + base), make_uint4(o5[0], o5[1], o5[2], o5[3]));
    __stcs(reinterpret_cast<uint4*>(p.out143 + base), make_uint4(o4[0], o4[1], o4[2], o4[3]));
  }
  for (int64_t i = nvec * 16 + tid; i < p.n; i += nthreads) {
    float x = BF16 ? __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(in)[i]) : reinterpret_cast<const float*>(in)[i];
    amax_bits = max(amax_bits, __float_as_uint(x) & 0x7FFFFFFFu);
    float y5 = p.has152 ? scaled<BF16>(x, s5, s5i, p.mul_fp32) : x;
    float y4 = p.has143 ? scaled<BF16>(x, s4, s4i, p.mul_fp32) : x;
    float z5 = y5;
    if (SR) {
      const uint64_t gi = p.first_index + (uint64_t)i;
      z5 = rb8 ? sr_round<B200Q_E5M2, 8>(y5, sr_random_bits<8>(gi, p.seed, p.offset))
               : sr_round<B200Q_E5M2, 16>(y5, sr_random_bits<16>(gi, p.seed, p.offset));
    }
    uint32_t b5 = cvt_fp8x2<B200Q_E5M2>(z5, 0.f) & 0xFFu, b4 = cvt_fp8x2<B200Q_E4M3>(y4, 0.f) & 0xFFu;
    if (y5 != y5) b5 = 0x7Fu;
    if (y4 != y4) b4 = 0x7Fu;
    p.out152[i] = (uint8_t)b5;
    p.out143[i] = (uint8_t)b4;
  }
  cast_publish_amax(amax_bits, p.amax, p.start);
}

// ------------------------------------------------------------------ cast_from_fp8
struct UncastParams {
  const uint8_t* in;
  void* out;
  const float* scale;
  float scale_host;
  int has_scale, scale_from_dev;
  int64_t n, cols;
};

// 8 fp8 bytes -> 8 values of OutT, scaled.  A thread loads 8 bytes and stores 16 (bf16) or 32
// (fp32) bytes, so that both the loads and the stores of a warp are contiguous.
template <typename OutT, int FMT, int SC>
__device__ __forceinline__ void uncast8(const UncastParams& p, OutT* __restrict__ out, int64_t base, uint2 raw,
                                        float s_one) {
  constexpr bool BF16 = InTraits<OutT>::kIsBf16;
  uint32_t w[2] = {raw.x, raw.y};
  float y[8];
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    // two bytes -> f16x2 in one conversion, then widen
    __half2_raw h0 = __nv_cvt_fp8x2_to_halfraw2((__nv_fp8x2_storage_t)(w[i] & 0xFFFFu), Fp8Fmt<FMT>::kInterp);
    __half2_raw h1 = __nv_cvt_fp8x2_to_halfraw2((__nv_fp8x2_storage_t)(w[i] >> 16), Fp8Fmt<FMT>::kInterp);
    float2 f0 = __half22float2(*reinterpret_cast<__half2*>(&h0));
    float2 f1 = __half22float2(*reinterpret_cast<__half2*>(&h1));
    y[4 * i] = f0.x; y[4 * i + 1] = f0.y; y[4 * i + 2] = f1.x; y[4 * i + 3] = f1.y;
  }
  if (p.has_scale) {
    if (SC == SC_COL || SC == SC_FULL) {
      const float4* sp = reinterpret_cast<const float4*>(p.scale + (SC == SC_COL ? base % p.cols : base));
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        float4 f = __ldg(sp + i);
        float s4[4] = {f.x, f.y, f.z, f.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) y[4 * i + j] *= BF16 ? round_to_bf16(s4[j]) : s4[j];
      }
    } else {
      float sv = s_one;
      if (SC == SC_ROW) {
        sv = __ldg(p.scale + base / p.cols);
        if (BF16) sv = round_to_bf16(sv);
      }
#pragma unroll
      for (int i = 0; i < 8; ++i) y[i] *= sv;
    }
  }
  if (BF16) {
    __stcs(reinterpret_cast<uint4*>(out + base), make_uint4(pack_bf16x2(y[0], y[1]), pack_bf16x2(y[2], y[3]),
                                                             pack_bf16x2(y[4], y[5]), pack_bf16x2(y[6], y[7])));
  } else {
    float4* dst = reinterpret_cast<float4*>(out + base);
    __stcs(dst, make_float4(y[0], y[1], y[2], y[3]));
    __stcs(dst + 1, make_float4(y[4], y[5], y[6], y[7]));
  }
}

constexpr int kUncastUnroll = 8;

template <typename OutT, int FMT, int SC>
__global__ void __launch_bounds__(256) cast_from_fp8_kernel(UncastParams p) {
  pdl_enter_spread();
  constexpr bool BF16 = InTraits<OutT>::kIsBf16;
  const int64_t tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t nthreads = (int64_t)gridDim.x * blockDim.x;
  OutT* __restrict__ out = static_cast<OutT*>(p.out);
  float s_one = 1.f;
  if (SC == SC_ONE && p.has_scale) s_one = p.scale_from_dev ? __ldg(p.scale) : p.scale_host;
  if (BF16) s_one = round_to_bf16(s_one);
  const bool aligned = ((reinterpret_cast<uintptr_t>(p.in) | reinterpret_cast<uintptr_t>(out)) & 15) == 0 &&
                       ((SC != SC_FULL && SC != SC_COL) || (reinterpret_cast<uintptr_t>(p.scale) & 15) == 0);
  const bool col_vec = (SC != SC_COL && SC != SC_ROW) || (p.cols % 8 == 0);
  const int64_t nvec = (aligned && col_vec) ? p.n / 8 : 0;

  // a block owns kUncastUnroll consecutive runs of 256 x 8 bytes; all loads are issued first
  const int64_t per_block = (int64_t)blockDim.x * kUncastUnroll;
  for (int64_t b0 = (int64_t)blockIdx.x * per_block; b0 < nvec; b0 += (int64_t)gridDim.x * per_block) {
    uint2 r[kUncastUnroll];
#pragma unroll
    for (int u = 0; u < kUncastUnroll; ++u) {
      const int64_t v = b0 + (int64_t)u * blockDim.x + threadIdx.x;
      r[u] = v < nvec ? __ldcs(reinterpret_cast<const uint2*>(p.in + v * 8)) : make_uint2(0u, 0u);
    }
#pragma unroll
    for (int u = 0; u < kUncastUnroll; ++u) {
      const int64_t v = b0 + (int64_t)u * blockDim.x + threadIdx.x;
      if (v < nvec) uncast8<OutT, FMT, SC>(p, out, v * 8, r[u], s_one);
    }
  }
  for (int64_t i = nvec * 8 + tid; i < p.n; i += nthreads) {
    float y = fp8_to_float<FMT>(p.in[i]);
    if (p.has_scale) {
      float s = SC == SC_ONE ? s_one : SC == SC_COL ? p.scale[i % p.cols] : SC == SC_ROW ? p.scale[i / p.cols]
                                                                                       : p.scale[i];
      if (BF16 && SC != SC_ONE) s = round_to_bf16(s);
      y *= s;
    }
    if (BF16) reinterpret_cast<__nv_bfloat16*>(out)[i] = __float2bfloat16_rn(y);
    else reinterpret_cast<float*>(out)[i] = y;
  }
}

// ------------------------------------------------------------------ swiglu + cast
struct SwigluParams {
  const __nv_bfloat16* gate;
  const __nv_bfloat16* up;
  uint8_t* out;
  int64_t ld_gate, ld_up, rows, cols;
  float scale;
  float* amax;
};


__global__ void __launch_bounds__(256) swiglu_cast_kernel(SwigluParams p) {
  pdl_enter();
  const int64_t vec_per_row = p.cols / 16;
  const int64_t nvec = p.rows * vec_per_row;
  const int64_t tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t nthreads = (int64_t)gridDim.x * blockDim.x;
  const float s_in = round_to_bf16(p.scale);
  uint32_t amax_bits = 0;
  for (int64_t v = tid; v < nvec; v += nthreads) {
    const int64_t r = v / vec_per_row, c = (v % vec_per_row) * 16;
    const uint4* gp = reinterpret_cast<const uint4*>(p.gate + r * p.ld_gate + c);
    const uint4* upp = reinterpret_cast<const uint4*>(p.up + r * p.ld_up + c);
    uint4 g0 = __ldcs(gp), g1 = __ldcs(gp + 1), u0 = __ldcs(upp), u1 = __ldcs(upp + 1);
    uint32_t gw[8] = {g0.x, g0.y, g0.z, g0.w, g1.x, g1.y, g1.z, g1.w};
    uint32_t uw[8] = {u0.x, u0.y, u0.z, u0.w, u1.x, u1.y, u1.z, u1.w};
    float y[16];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      float h0 = silu_mul_bf16(__uint_as_float(gw[i] << 16), __uint_as_float(uw[i] << 16));
      float h1 = silu_mul_bf16(__uint_as_float(gw[i] & 0xFFFF0000u), __uint_as_float(uw[i] & 0xFFFF0000u));
      amax_bits = max(amax_bits, max(__float_as_uint(h0) & 0x7FFFFFFFu, __float_as_uint(h1) & 0x7FFFFFFFu));
      y[2 * i] = round_to_bf16(h0 * s_in);
      y[2 * i + 1] = round_to_bf16(h1 * s_in);
    }
    uint32_t o[4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
      o[i] = cvt_fp8x2<B200Q_E4M3>(clampf<B200Q_E4M3>(y[4 * i]), clampf<B200Q_E4M3>(y[4 * i + 1])) |
             (cvt_fp8x2<B200Q_E4M3>(clampf<B200Q_E4M3>(y[4 * i + 2]), clampf<B200Q_E4M3>(y[4 * i + 3])) << 16);
    __stcs(reinterpret_cast<uint4*>(p.out + r * p.cols + c), make_uint4(o[0], o[1], o[2], o[3]));
  }
  if (p.amax) block_amax_to_global(amax_bits, p.amax);
}

// ------------------------------------------------------------------ host launchers
// Grid for the grid-stride kernels, two shapes (measured on 2^24 and 2^26 elements):
//  * one block per 256 items, capped at 16 waves of resident blocks -- the kernels with a few
//    instructions per byte (RNE casts, cast_from_fp8, SwiGLU) run at the HBM rate this way;
//  * ONE resident wave, balanced -- the kernels that are bound by instruction issue (stochastic
//    rounding, the two-output hybrid cast) gain 7-10 %: with W = threads resident at once,
//    every thread takes r = ceil(items / W) items and the grid is the number of 256-thread
//    blocks that r items per thread need, ceil(items / (256 r)) <= the resident blocks; no block
//    waits for another to retire and no thread has more than one item more than any other.
// Resident 256-thread blocks per SM of a kernel, looked up once per kernel FUNCTION (kernels that
// share a signature share a C++ type, so a cache per template instantiation would hand one
// kernel's occupancy to another); the same on every B200 of a process.
static int blocks_per_sm(const void* kernel) {
  constexpr int kSlots = 64;
  static std::atomic<const void*> keys[kSlots];
  static std::atomic<int> vals[kSlots];
  for (int i = 0; i < kSlots; ++i) {
    const void* k = keys[i].load(std::memory_order_acquire);
    if (k == kernel) {
      const int v = vals[i].load(std::memory_order_acquire);
      if (v > 0) return v;
      break;  // another thread is filling the slot: compute it here too
    }
    if (k == nullptr) break;
  }
  int per_sm = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, 256, 0) != cudaSuccess || per_sm < 1) per_sm = 4;
  for (int i = 0; i < kSlots; ++i) {
    const void* expected = nullptr;
    if (keys[i].compare_exchange_strong(expected, kernel, std::memory_order_acq_rel) || expected == kernel) {
      vals[i].store(per_sm, std::memory_order_release);
      break;
    }
  }
  return per_sm;
}

template <typename Kernel>
static int grid_for(Kernel kernel, int64_t n_items, bool one_wave = false) {
  const int per_sm = blocks_per_sm(reinterpret_cast<const void*>(kernel));
  int64_t blocks = (n_items + 255) / 256;
  const int64_t resident = (int64_t)kNumSMs * per_sm;
  if (one_wave) {
    if (blocks > resident) {
      const int64_t r = (n_items + resident * 256 - 1) / (resident * 256);
      blocks = (n_items + 256 * r - 1) / (256 * r);
    }
  } else if (blocks > resident * 16) {
    blocks = resident * 16;
  }
  if (blocks < 1) blocks = 1;
  return (int)blocks;
}

// The amax word is cleared by a one-thread kernel, not by a memset, so that both it and the cast
// can be launched with programmatic stream serialization:
//   * the clearing kernel is set up under the tail of the kernel in front of it, waits for that
//     kernel (and through it for everything earlier in the stream), lets the cast start and
//     clears the word;
//   * the cast's blocks start at that point, let the kernel behind them be set up at once
//     (pdl_release) and wait for the clearing kernel's completion only before their atomicMax
//     (block_amax_to_global).
// Of the three launch gaps of [kernel in front] [clear] [cast] [kernel behind] two are gone
// (1.5-2 us each on casts of 10-30 us).
__global__ void clear_amax_kernel(float* amax) {
  pdl_enter();
  *amax = 0.f;
}

int clear_amax(float* amax, cudaStream_t st) {
  launch_dependent(clear_amax_kernel, dim3(1), dim3(1), 0, st, amax);
  B200Q_LAUNCH_CHECK();
  return B200Q_OK;
}

static int scale_class(int mode) {
  switch (mode) {
    case B200Q_BCAST_PER_COL: return SC_COL;
    case B200Q_BCAST_PER_ROW: return SC_ROW;
    case B200Q_BCAST_FULL: return SC_FULL;
    default: return SC_ONE;
  }
}

// A cast with amax takes one of three forms, by its number of elements:
//   one cluster of up to eight blocks, which reduces its amax by itself: one launch, but eight SMs only;
//   behind a memset of the amax word: 1.4 us less of host time than a clearing kernel, but 3.5 us of
//     idle device, since nothing is set up across a memset;
//   behind clear_amax_kernel.
// So the first two end where eight SMs, or the idle time, last longer than the host takes to issue
// the call, which comes the sooner the more a cast does per element.  us per call of the forms, launched back to
// back (in brackets: in a graph, where the host costs nothing and the memset is never the best):
//                                     2^15 elements          2^17                        2^18                   2^21
//   vectors, to nearest               7.0 / 8.2 / 9.9        7.2 / 8.3 (2.7 / 6.0 / 2.6) 7.3 / 8.2 / 9.8        8.2 / 9.8
//   the same, scale per column        8.0 / 9.2 / 10.9       8.0 / 9.1 (5.9 / 6.2 / 3.3) 10.5 / 9.2 / 10.8      9.2 / 10.6
//   vectors, stochastic, bf16 -> e5m2 7.0 / 8.3 / 10.1       7.2 / 8.2                   7.3 / 8.3 / 9.8        8.2 / 9.6
//   the same to e4m3                  7.0 / 8.2 / 9.7        7.3 / 8.3 (6.7 / 8.1 / 4.7) 12.1 / 8.2 / 9.8       9.9 / 9.7
//   vectors, stochastic, otherwise    7.0 / 8.2 / 9.8        8.7 / 8.2 (8.0 / 6.2 / 3.6) 14.6 / 8.3 / 9.8       9.9 / 9.7
//   element by element, to nearest    7.0 / 8.2 / 10.0       14.7 / 8.4 (14.1 / 8.2 / 5.3) 27 / 8.4 / 9.9       9.4 / 9.7
//   the same, scale per row           8.6 / 11.5 / 10.7      28 / 12.4 (27 / 12.3 / 9.5) 52 / 12.4 / 10.4       14.4 / 11.0
//   the same, stochastic              12.8 / 15.6 / 13.0     45 / 16.5 (44 / 16.4 / 13.7) 87 / 16.6 / 14.3      24 / 21
// (packed: the kernels that round pairs of bf16 as they are.  To e4m3 a stochastic cast meets more values below the
// smallest normal, which it rounds one by one.  Element by element: as the kernels go where pointers or row lengths rule vectors out; up to 2^15
// elements the other forms have no more than eight blocks either).
struct AmaxForms {
  int64_t cluster, memset;  // up to how many elements
};
static AmaxForms amax_forms(bool vectors, bool stochastic, bool packed, int out_dtype, int sc) {
  if (!vectors) return {1 << 15, stochastic || sc != SC_ONE ? 0 : 1 << 21};
  if (stochastic && packed) return out_dtype == B200Q_E5M2 ? AmaxForms{1 << 18, 1 << 21} : AmaxForms{1 << 17, 1 << 20};
  if (stochastic) return {1 << 16, 1 << 20};
  if (sc == SC_COL || sc == SC_FULL) return {1 << 17, 1 << 21};
  return {1 << 18, 1 << 22};
}

// Decides how a cast starts and clears its amax word where that is needed.
static int cast_start(float* amax, int64_t n, AmaxForms forms, cudaStream_t st, int* start) {
  *start = kStartAfter;
  if (!amax) return B200Q_OK;
  const AmaxForms captured = {forms.cluster / 4, 0};
  if (n > captured.cluster && (n <= forms.cluster || n <= forms.memset)) {  // (asking costs the host 0.1 us)
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(st, &capture) != cudaSuccess) (void)cudaGetLastError();  // (capture is not set then)
    else if (capture != cudaStreamCaptureStatusNone) forms = captured;
  }
  if (n > 0 && n <= forms.cluster) {
    *start = kStartCluster;
  } else if (n <= forms.memset || n == 0) {
    B200Q_CUDA_OK(cudaMemsetAsync(amax, 0, sizeof(float), st));
  } else {
    *start = kStartBehindClear;
    return clear_amax(amax, st);
  }
  return B200Q_OK;
}
template <typename Params>
static auto start_of(const Params& p, int) -> decltype(p.start) { return p.start; }
template <typename Params>
static int start_of(const Params&, long) { return kStartAfter; }

// Every kernel launched here may be set up before its predecessor in the stream has finished (it
// waits as its StartMode says).
template <typename Kernel, typename Params>
static void launch_persistent(Kernel kernel, int64_t items, cudaStream_t st, const Params& p, bool one_wave = false) {
  if (start_of(p, 0) == kStartCluster) {
    const int64_t blocks = (items + 255) / 256;
    const unsigned size = blocks >= 8 ? 8u : blocks >= 4 ? 4u : blocks >= 2 ? 2u : 1u;
    launch_dependent_cluster(kernel, size, dim3(size), dim3(256), 0, st, p);
    return;
  }
  launch_dependent(kernel, dim3((unsigned)grid_for(kernel, items, one_wave)), dim3(256), 0, st, p);
}

template <typename InT, int FMT, bool SR>
static void launch_cast_sc(int sc, int64_t items, cudaStream_t st, const CastParams& p) {
  switch (sc) {
    case SC_ONE: launch_persistent(cast_to_fp8_kernel<InT, FMT, SR, SC_ONE>, items, st, p); break;
    case SC_COL: launch_persistent(cast_to_fp8_kernel<InT, FMT, SR, SC_COL>, items, st, p); break;
    case SC_ROW: launch_persistent(cast_to_fp8_kernel<InT, FMT, SR, SC_ROW>, items, st, p); break;
    default: launch_persistent(cast_to_fp8_kernel<InT, FMT, SR, SC_FULL>, items, st, p); break;
  }
}

template <typename InT, int FMT>
static void launch_cast_sr(bool sr, int sc, int64_t items, cudaStream_t st, const CastParams& p) {
  if (sr) launch_cast_sc<InT, FMT, true>(sc, items, st, p);
  else launch_cast_sc<InT, FMT, false>(sc, items, st, p);
}

int cast_to_fp8_impl(const void* in, int in_dtype, void* out, int out_dtype, const float* scale,
                     float scale_host, int scale_mode, int64_t rows, int64_t cols, float* amax, int rounding,
                     uint64_t seed, uint64_t offset, uint64_t first_index, int flags, cudaStream_t st) {
  const int64_t n = rows * cols;
  if (in_dtype == B200Q_E4M3 || in_dtype == B200Q_E5M2) {
    if (out_dtype != in_dtype || amax) return B200Q_ERR_BAD_ARGUMENT;
    if (n) B200Q_CUDA_OK(cudaMemcpyAsync(out, in, (size_t)n, cudaMemcpyDeviceToDevice, st));
    return B200Q_OK;
  }
  const int sc = scale_class(scale_mode);
  const bool sr = rounding == B200Q_ROUND_STOCHASTIC;
  const bool aligned = ((reinterpret_cast<uintptr_t>(in) | reinterpret_cast<uintptr_t>(out)) & 15) == 0;
  // (as the kernels decide it)
  const bool vectors = aligned && ((sc != SC_FULL && sc != SC_COL) || (reinterpret_cast<uintptr_t>(scale) & 15) == 0) &&
                       ((sc != SC_COL && sc != SC_ROW) || cols % 16 == 0) && (!sr || (first_index & 15) == 0);
  // fast path: bf16 input, product in bf16, one scale per 16-element chunk, aligned pointers
  const bool fast = in_dtype == B200Q_BF16 && !(flags & B200Q_CAST_MUL_IN_FP32) && aligned &&
                    (sc == SC_ONE || (sc == SC_ROW && cols % 16 == 0)) && (!sr || (first_index & 15) == 0);
  int start;
  if (int rc = cast_start(amax, n, amax_forms(vectors, sr, fast, out_dtype, sc), st, &start)) return rc;
  if (n == 0) return B200Q_OK;
  CastParams p;
  p.start = start;
  p.in = in; p.out = out; p.scale = scale; p.scale_host = scale_host;
  p.has_scale = scale_mode != B200Q_BCAST_NONE;
  p.scale_from_dev = scale_mode == B200Q_BCAST_SCALAR_DEV;
  p.n = n; p.cols = cols; p.amax = amax; p.seed = seed; p.offset = offset; p.first_index = first_index;
  p.mul_fp32 = (flags & B200Q_CAST_MUL_IN_FP32) ? 1 : 0;
  const int64_t items = (n + 15) / 16;
  if (fast && sr) {
    const int64_t half = (items + 1) / 2;
    if (out_dtype == B200Q_E4M3) {
      if (sc == SC_ROW) launch_persistent(cast_bf16_sr_fast_kernel<B200Q_E4M3, true>, half, st, p, true);
      else launch_persistent(cast_bf16_sr_fast_kernel<B200Q_E4M3, false>, half, st, p, true);
    } else {
      if (sc == SC_ROW) launch_persistent(cast_bf16_sr_fast_kernel<B200Q_E5M2, true>, half, st, p, true);
      else launch_persistent(cast_bf16_sr_fast_kernel<B200Q_E5M2, false>, half, st, p, true);
    }
  } else if (fast) {
    const int64_t half = (items + 1) / 2;  // two chunks per thread and step
    if (out_dtype == B200Q_E4M3) {
      if (sc == SC_ROW) launch_persistent(cast_bf16_rne_fast_kernel<B200Q_E4M3, true>, half, st, p);
      else launch_persistent(cast_bf16_rne_fast_kernel<B200Q_E4M3, false>, half, st, p);
    } else {
      if (sc == SC_ROW) launch_persistent(cast_bf16_rne_fast_kernel<B200Q_E5M2, true>, half, st, p);
      else launch_persistent(cast_bf16_rne_fast_kernel<B200Q_E5M2, false>, half, st, p);
    }
  } else if (in_dtype == B200Q_BF16) {
    if (out_dtype == B200Q_E4M3) launch_cast_sr<__nv_bfloat16, B200Q_E4M3>(sr, sc, items, st, p);
    else launch_cast_sr<__nv_bfloat16, B200Q_E5M2>(sr, sc, items, st, p);
  } else {
    if (out_dtype == B200Q_E4M3) launch_cast_sr<float, B200Q_E4M3>(sr, sc, items, st, p);
    else launch_cast_sr<float, B200Q_E5M2>(sr, sc, items, st, p);
  }
  B200Q_LAUNCH_CHECK();
  return B200Q_OK;
}

template <typename OutT, int FMT>
static void launch_uncast_sc(int sc, int64_t items, cudaStream_t st, const UncastParams& p) {
  switch (sc) {
    case SC_ONE: launch_persistent(cast_from_fp8_kernel<OutT, FMT, SC_ONE>, items, st, p); break;
    case SC_COL: launch_persistent(cast_from_fp8_kernel<OutT, FMT, SC_COL>, items, st, p); break;
    case SC_ROW: launch_persistent(cast_from_fp8_kernel<OutT, FMT, SC_ROW>, items, st, p); break;
    default: launch_persistent(cast_from_fp8_kernel<OutT, FMT, SC_FULL>, items, st, p); break;
  }
}

int cast_from_fp8_impl(const void* in, int in_dtype, void* out, int out_dtype, const float* scale,
                       float scale_host, int scale_mode, int64_t rows, int64_t cols, cudaStream_t st) {
  const int64_t n = rows * cols;
  if (n == 0) return B200Q_OK;
  UncastParams p;
  p.in = static_cast<const uint8_t*>(in); p.out = out; p.scale = scale; p.scale_host = scale_host;
  p.has_scale = scale_mode != B200Q_BCAST_NONE;
  p.scale_from_dev = scale_mode == B200Q_BCAST_SCALAR_DEV;
  p.n = n; p.cols = cols;
  const int sc = scale_class(scale_mode);
  const int64_t items = ((n + 7) / 8 + kUncastUnroll - 1) / kUncastUnroll;  // 8-byte items, kUncastUnroll per thread and step
  if (out_dtype == B200Q_BF16) {
    if (in_dtype == B200Q_E4M3) launch_uncast_sc<__nv_bfloat16, B200Q_E4M3>(sc, items, st, p);
    else launch_uncast_sc<__nv_bfloat16, B200Q_E5M2>(sc, items, st, p);
  } else {
    if (in_dtype == B200Q_E4M3) launch_uncast_sc<float, B200Q_E4M3>(sc, items, st, p);
    else launch_uncast_sc<float, B200Q_E5M2>(sc, items, st, p);
  }
  B200Q_LAUNCH_CHECK();
  return B200Q_OK;
}

int swiglu_cast_impl(const void* gate, int64_t ld_gate, const void* up, int64_t ld_up, void* out, float scale,
                     int64_t rows, int64_t cols, float* amax, cudaStream_t st) {
  if (cols % 16 || ld_gate % 8 || ld_up % 8) return B200Q_ERR_UNSUPPORTED;
  if (((reinterpret_cast<uintptr_t>(gate) | reinterpret_cast<uintptr_t>(up) | reinterpret_cast<uintptr_t>(out)) & 15))
    return B200Q_ERR_UNSUPPORTED;
  if (amax) B200Q_CUDA_OK(cudaMemsetAsync(amax, 0, sizeof(float), st));
  if (rows * cols == 0) return B200Q_OK;
  SwigluParams p;
  p.gate = static_cast<const __nv_bfloat16*>(gate); p.up = static_cast<const __nv_bfloat16*>(up);
  p.out = static_cast<uint8_t*>(out); p.ld_gate = ld_gate; p.ld_up = ld_up; p.rows = rows; p.cols = cols;
  p.scale = scale; p.amax = amax;
  launch_dependent(swiglu_cast_kernel, dim3((unsigned)grid_for(swiglu_cast_kernel, rows * cols / 16)), dim3(256), 0, st, p);
  B200Q_LAUNCH_CHECK();
  return B200Q_OK;
}

// bf16 input, both outputs rounded to nearest even, product in bf16, everything 16-byte
// aligned: the packed path of cast_bf16_rne_fast_kernel with two scales and two stores.
__global__ void __launch_bounds__(256) cast_hybrid_bf16_rne_fast_kernel(HybridParams p) {
  cast_begin(p.start);
  const __nv_bfloat16* __restrict__ in = static_cast<const __nv_bfloat16*>(p.in);
  const int64_t tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t nthreads = (int64_t)gridDim.x * blockDim.x;
  const int64_t nvec = p.n / 16;
  float s5 = 1.f, s4 = 1.f;
  if (p.has152) s5 = p.dev152 ? __ldg(p.s152) : p.s152_host;
  if (p.has143) s4 = p.dev143 ? __ldg(p.s143) : p.s143_host;
  const uint32_t s5_2 = pack_bf16x2(s5, s5), s4_2 = pack_bf16x2(s4, s4);
  uint32_t amax2 = 0, unused = 0;
  int64_t v = tid;
  for (; v + nthreads < nvec; v += 2 * nthreads) {  // two independent chunks in flight per thread
    const int64_t b0 = v * 16, b1 = (v + nthreads) * 16;
    const uint4* q0 = reinterpret_cast<const uint4*>(in + b0);
    const uint4* q1 = reinterpret_cast<const uint4*>(in + b1);
    const uint4 a0 = __ldcs(q0), a1 = __ldcs(q0 + 1), c0 = __ldcs(q1), c1 = __ldcs(q1 + 1);
    __stcs(reinterpret_cast<uint4*>(p.out152 + b0), cast16_bf16_rne<B200Q_E5M2>(a0, a1, s5_2, p.has152, amax2));
    __stcs(reinterpret_cast<uint4*>(p.out143 + b0), cast16_bf16_rne<B200Q_E4M3>(a0, a1, s4_2, p.has143, unused));
    __stcs(reinterpret_cast<uint4*>(p.out152 + b1), cast16_bf16_rne<B200Q_E5M2>(c0, c1, s5_2, p.has152, amax2));
    __stcs(reinterpret_cast<uint4*>(p.out143 + b1), cast16_bf16_rne<B200Q_E4M3>(c0, c1, s4_2, p.has143, unused));
  }
  for (; v < nvec; v += nthreads) {
    const int64_t b0 = v * 16;
    const uint4* q0 = reinterpret_cast<const uint4*>(in + b0);
    const uint4 a0 = __ldcs(q0), a1 = __ldcs(q0 + 1);
    __stcs(reinterpret_cast<uint4*>(p.out152 + b0), cast16_bf16_rne<B200Q_E5M2>(a0, a1, s5_2, p.has152, amax2));
    __stcs(reinterpret_cast<uint4*>(p.out143 + b0), cast16_bf16_rne<B200Q_E4M3>(a0, a1, s4_2, p.has143, unused));
  }
  uint32_t amax_bits = max(amax2 << 16, amax2 & 0xFFFF0000u);
  for (int64_t i = nvec * 16 + tid; i < p.n; i += nthreads) {  // fewer than 16 elements
    const float x = __bfloat162float(in[i]);
    amax_bits = max(amax_bits, __float_as_uint(x) & 0x7FFFFFFFu);
    const float y5 = p.has152 ? round_to_bf16(x * round_to_bf16(s5)) : x;
    const float y4 = p.has143 ? round_to_bf16(x * round_to_bf16(s4)) : x;
    uint32_t b5 = cvt_fp8x2<B200Q_E5M2>(y5, 0.f) & 0xFFu, b4 = cvt_fp8x2<B200Q_E4M3>(y4, 0.f) & 0xFFu;
    if (y5 != y5) b5 = 0x7Fu;
    if (y4 != y4) b4 = 0x7Fu;
    p.out152[i] = (uint8_t)b5;
    p.out143[i] = (uint8_t)b4;
  }
  cast_publish_amax(amax_bits, p.amax, p.start);
}

int cast_hybrid_impl(const void* in, int in_dtype, void* out152, void* out143, const float* s152, float s152_host,
                     int mode152, const float* s143, float s143_host, int mode143, int64_t n, float* amax, int rounding,
                     uint64_t seed, uint64_t offset, uint64_t first_index, int flags, cudaStream_t st) {
  const bool sr = rounding == B200Q_ROUND_STOCHASTIC;
  const bool all_aligned = ((reinterpret_cast<uintptr_t>(in) | reinterpret_cast<uintptr_t>(out152) |
                             reinterpret_cast<uintptr_t>(out143)) & 15) == 0;
  int start;
  if (int rc = cast_start(amax, n, amax_forms(all_aligned && (first_index & 15) == 0, sr, false, 0, SC_ONE), st, &start)) return rc;
  if (n == 0) return B200Q_OK;
  HybridParams p;
  p.start = start;
  p.in = in; p.out152 = static_cast<uint8_t*>(out152); p.out143 = static_cast<uint8_t*>(out143);
  p.s152 = s152; p.s143 = s143; p.s152_host = s152_host; p.s143_host = s143_host;
  p.has152 = mode152 != B200Q_BCAST_NONE; p.has143 = mode143 != B200Q_BCAST_NONE;
  p.dev152 = mode152 == B200Q_BCAST_SCALAR_DEV; p.dev143 = mode143 == B200Q_BCAST_SCALAR_DEV;
  p.n = n; p.amax = amax; p.seed = seed; p.offset = offset; p.first_index = first_index;
  p.mul_fp32 = (flags & B200Q_CAST_MUL_IN_FP32) ? 1 : 0;
  const int64_t items = (n + 15) / 16;
  if (in_dtype == B200Q_BF16 && !sr && !p.mul_fp32 && all_aligned) {
    launch_persistent(cast_hybrid_bf16_rne_fast_kernel, items, st, p, true);
  } else if (in_dtype == B200Q_BF16) {
    if (sr) launch_persistent(cast_hybrid_kernel<__nv_bfloat16, true>, items, st, p, true);
    else launch_persistent(cast_hybrid_kernel<__nv_bfloat16, false>, items, st, p, true);
  } else {
    if (sr) launch_persistent(cast_hybrid_kernel<float, true>, items, st, p, true);
    else launch_persistent(cast_hybrid_kernel<float, false>, items, st, p, true);
  }
  B200Q_LAUNCH_CHECK();
  return B200Q_OK;
}

}  // namespace b200q
