// KV-cache writer: the producer of the cache format the decode kernel reads.
//
// Per token: amax over the 512 latent values -> scale = amax / 6 (1 for an all-zero token, or a
// caller-provided scale) -> x / scale rounded to the nearest E2M1 magnitude {0,.5,1,1.5,2,3,4,6}
// with a tie going to the smaller one -> 256 packed bytes (low nibble = even element, bit 3 = sign);
// the 64 RoPE values are cast to E4M3 (as torch casts: beyond 464 the byte is NaN); row and scale are scattered to the token's slot
// (page * page_size + offset) of the paged cache.  Same arithmetic, in the same order and with IEEE
// division, as the reference's fixture builder (tests/test_cute_dsl_mla_fp4.py:56-93), so the bytes
// are identical to it; the reference leaves cache writes to the caller (README.md:81-83).
//
// Two forms.  cache_write_kernel: one warp per token.  A lane owns the 16-byte chunks lane, lane + 32, ... of the latent row, so
// every load of a warp is 512 contiguous bytes, and two RoPE values.  The next token's loads are issued before the current one
// is quantised.  cache_write_many_kernel: four tokens per warp, for many tokens of a 16-bit type (see there).
// Bound by HBM (576 input elements read and 324 bytes written per token, nothing twice) once the arithmetic is out of the way:
// with 391 instructions per token and warp 262144 BF16 tokens took 125 us (3.1 TB/s, integer pipe 70 % busy).
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_fp8.h>

#include "common.cuh"
#include "launch.h"

namespace mla {

namespace {

constexpr int kWriterWarps = 8;

template <typename T> __device__ __forceinline__ float to_f32(T v);
template <> __device__ __forceinline__ float to_f32<float>(float v) { return v; }
template <> __device__ __forceinline__ float to_f32<__half>(__half v) { return __half2float(v); }
template <> __device__ __forceinline__ float to_f32<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }

// A lane's share of a row as loaded: chunk k holds elements [kPer * (lane + 32 k), + kPer).
template <typename T> struct Raw16 {
  static constexpr int kPer = 16 / sizeof(T);  // elements per 16-byte load
  static constexpr int kChunks = 16 / kPer;
  uint4 r[kChunks];
  T rope0, rope1;
  int64_t slot;
};
// Largest magnitude among a lane's 16 elements as f32 bits; NaN if there is one.
template <typename T> __device__ __forceinline__ uint32_t amax_bits(const Raw16<T>& raw) {
  float m = 0.f;
#pragma unroll
  for (int q = 0; q < Raw16<T>::kChunks; ++q) {
    const float* e = reinterpret_cast<const float*>(&raw.r[q]);
#pragma unroll
    for (int i = 0; i < 4; ++i) asm("max.NaN.f32 %0, %0, %1;" : "+f"(m) : "f"(fabsf(e[i])));
  }
  return __float_as_uint(m) & 0x7fffffffu;
}
template <typename T2, typename T> __device__ __forceinline__ uint32_t amax_bits16(const Raw16<T>& raw) {
  T2 m = __habs2(reinterpret_cast<const T2*>(&raw.r[0])[0]);
#pragma unroll
  for (int i = 1; i < 8; ++i) m = __hmax2_nan(m, __habs2(reinterpret_cast<const T2*>(&raw.r[i >> 2])[i & 3]));
  return max(__float_as_uint(__low2float(m)) & 0x7fffffffu, __float_as_uint(__high2float(m)) & 0x7fffffffu);
}
template <> __device__ __forceinline__ uint32_t amax_bits<__nv_bfloat16>(const Raw16<__nv_bfloat16>& raw) { return amax_bits16<__nv_bfloat162>(raw); }
template <> __device__ __forceinline__ uint32_t amax_bits<__half>(const Raw16<__half>& raw) { return amax_bits16<__half2>(raw); }
constexpr uint32_t kInfBits = 0x7f800000u;
// elements 2i and 2i + 1 of a chunk
template <typename T> __device__ __forceinline__ float2 pair_of(const uint4& chunk, int i) {
  const T* e = reinterpret_cast<const T*>(&chunk);
  return make_float2(to_f32<T>(e[2 * i]), to_f32<T>(e[2 * i + 1]));
}

// E2M1 code of x / scale: magnitude = number of thresholds strictly below |n| (a tie stays on the
// smaller magnitude), bit 3 = n < 0.
__device__ __noinline__ uint32_t e2m1_code(float x, float scale) {
  const float n = __fdiv_rn(x, scale);
  const float a = fabsf(n);
  uint32_t m = 0;
  m += a > 0.25f;
  m += a > 0.75f;
  m += a > 1.25f;
  m += a > 1.75f;
  m += a > 2.5f;
  m += a > 3.5f;
  m += a > 5.0f;
  return m | (n < 0.f ? 8u : 0u);
}

// float -> E4M3 byte as the reference's writer (a torch cast) does it: round to nearest even; up to
// 464 (the midpoint above the largest finite value) rounds to 448, anything larger and NaN become NaN.
__device__ __forceinline__ uint32_t rope_e4m3(float x) {
  if (!(fabsf(x) <= 464.f)) return 0x7fu | ((__float_as_uint(x) >> 24) & 0x80u);
  return __nv_cvt_float_to_fp8(x, __NV_SATFINITE, __NV_E4M3);
}

// The same codes without the division.  x * (1/scale) is within 3 units in the last place of the correctly rounded quotient n,
// so n lies between q_lo and q_hi, the products with 1/scale taken 2^-20 down and up.  The hardware conversion
// cvt.rn.satfinite.e2m1x2.f32 is monotone, saturates at 6 and keeps the sign of values that round to magnitude zero, as the
// rule above does.  (The products are fused with an addition of +0, which takes the sign off a zero.)  Where q_lo and q_hi
// give the same code, that is the code.  Where they do not, a threshold t lies between them, and the code is that of q_hi if
// n > t and that of q_lo if not (a tie goes to the smaller magnitude).  n > t without the division: |x| / scale must lie above
// t by more than half of t's last place (at exactly half the quotient rounds to t, whose mantissa is even), and
// |x| - t * scale is exact, being the small difference of a 24-bit and a 27-bit number.
//
// 16-bit values with scale = amax / 6 need q_lo alone, for all but one token in fifteen.  With x and amax integers of at most 11
// bits (times powers of two) and t a multiple of 1/4, 6 x - t amax is zero or at least 2^-16 of either side, so the only
// values with a threshold that near are x = t amax / 6 (amax / 8 is one: every other BF16 token has some).  Their quotient is
// above t only if the rounding of amax / 6 made the scale too small by more than half of t's last place:
// amax - 6 scale > 6 scale 2^-24 / (mantissa of t), and 1.75 is the largest mantissa.  Otherwise all of them are ties.
//
// What this does not cover takes the exact division for the whole token: a NaN, a scale outside [2^-100, 2^14]
// (with which products of BF16 values could overflow or vanish), and an FP32 value below 2^-100 in magnitude, zero excepted.
constexpr float kScaleLo = 7.8886090522101181e-31f, kScaleHi = 16384.f;
// four values -> four packed codes (value 0 in the low nibble)
__device__ __forceinline__ uint32_t e2m1x4(float a, float b, float c, float d) {
  uint16_t out;
  asm("{\n\t.reg .b8 b0, b1;\n\t"
      "cvt.rn.satfinite.e2m1x2.f32 b0, %2, %1;\n\t"
      "cvt.rn.satfinite.e2m1x2.f32 b1, %4, %3;\n\t"
      "mov.b16 %0, {b0, b1};\n\t}"
      : "=h"(out)
      : "f"(a), "f"(b), "f"(c), "f"(d));
  return out;
}
// a * b + 0
__device__ __forceinline__ float2 scaled(uint64_t a, uint64_t b) {
  float2 d;
  asm("{\n\t.reg .b64 r;\n\tfma.rn.f32x2 r, %2, %3, %4;\n\tmov.b64 {%0, %1}, r;\n\t}" : "=f"(d.x), "=f"(d.y) : "l"(a), "l"(b), "l"(0ull));
  return d;
}
__device__ __forceinline__ uint64_t pack2(float a, float b) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
// What a token with a NaN gets as its largest magnitude: that of its other values.
template <typename T> __device__ __noinline__ float amax_without_nan(const T* row, int lane) {
  float m = 0.f;
#pragma unroll 1
  for (int i = lane; i < kLatent; i += 32) m = fmaxf(m, fabsf(to_f32<T>(row[i])));
  return __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(m)));
}
// Whether the quotient |x| / scale, rounded, is above the threshold between code magnitudes m and m + 1.
__device__ __forceinline__ bool above(float x, float scale, uint32_t m) {
  const uint32_t t = m < 2 ? __float_as_uint(0.25f + 0.5f * float(m)) : (m << 22) + (126u << 23) + (1u << 21);
  const float half_ulp = __uint_as_float((t & 0x7f800000u) - (24u << 23));
  return fmaf(-__uint_as_float(t), scale, fabsf(x)) > scale * half_ulp;
}

// Both values of a lane's RoPE pair as E4M3 bytes.
__device__ __forceinline__ uint32_t rope_pair(float a, float b) {
  if (fabsf(a) <= 464.f && fabsf(b) <= 464.f) return __nv_cvt_float2_to_fp8x2(make_float2(a, b), __NV_SATFINITE, __NV_E4M3);
  return rope_e4m3(a) | (rope_e4m3(b) << 8);
}

// CTAs per SM: what the registers of a prefetched token leave room for
template <typename T> constexpr int kResident = sizeof(T) == 4 ? 4 : 5;

template <typename T>
__global__ void __launch_bounds__(kWriterWarps * 32, kResident<T>)
cache_write_kernel(const T* __restrict__ latent, int64_t latent_stride, const T* __restrict__ rope, int64_t rope_stride,
                   const float* __restrict__ scale_in, const int64_t* __restrict__ slot_mapping, int64_t num_tokens,
                   uint8_t* __restrict__ cache, float* __restrict__ cache_sf, int64_t num_slots) {
  constexpr int kPer = Raw16<T>::kPer, kChunks = Raw16<T>::kChunks;
  const int lane = threadIdx.x & 31;
  const int64_t warps = int64_t(gridDim.x) * kWriterWarps;
  // A dependent launch: its CTAs are in place when the kernel before it ends, and so are those of the kernel after it.
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  auto fetch = [&](int64_t t, Raw16<T>& raw) {
    raw.slot = slot_mapping ? slot_mapping[t] : t;
    const uint4* p = reinterpret_cast<const uint4*>(latent + t * latent_stride) + lane;
#pragma unroll
    for (int q = 0; q < kChunks; ++q) raw.r[q] = p[32 * q];
    const T* rp = rope + t * rope_stride + 2 * lane;
    raw.rope0 = rp[0];
    raw.rope1 = rp[1];
  };
  int64_t t = int64_t(blockIdx.x) * kWriterWarps + (threadIdx.x >> 5);
  Raw16<T> nxt;
  if (t < num_tokens) fetch(t, nxt);
  for (; t < num_tokens; t += warps) {
    const Raw16<T> raw = nxt;
    if (t + warps < num_tokens) fetch(t + warps, nxt);  // in flight while this token is quantised
    const int64_t slot = raw.slot;
    if (slot < 0 || slot >= num_slots) continue;  // padding token (negative) or out of the pool: nothing is written
    const T* src = latent + t * latent_stride;
    const uint32_t top = __reduce_max_sync(0xffffffffu, amax_bits<T>(raw));  // non-negative floats compare as integers
    float scale;
    if (scale_in) {
      scale = scale_in[t];
    } else {
      scale = __fdiv_rn(top <= kInfBits ? __uint_as_float(top) : amax_without_nan<T>(src, lane), 6.0f);
      if (!(scale > 0.f)) scale = 1.0f;
    }
    const bool odd_token = !(scale >= kScaleLo && scale <= kScaleHi && top <= kInfBits);
    const bool lo_alone = sizeof(T) == 2 && !scale_in && fmaf(-6.f, scale, __uint_as_float(top)) <= scale * (6.f * 0x1p-24f / 1.76f);
    const float inv = __frcp_rn(scale), inv_lo = inv * (1.f - 0x1p-20f), inv_hi = inv * (1.f + 0x1p-20f);
    bool odd = odd_token;
    auto codes = [&](float f, bool look, uint32_t (&out)[2]) {  // eight codes each, in the order of the lane's elements
      const uint64_t f2 = pack2(f, f);
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        uint32_t c[2];
#pragma unroll
        for (int g = 0; g < 2; ++g) {
          const int e = 8 * k + 4 * g;
          const uint4& chunk = raw.r[e / kPer];
          const float2 a = pair_of<T>(chunk, (e % kPer) / 2), b = pair_of<T>(chunk, (e % kPer) / 2 + 1);
          const float2 qa = scaled(pack2(a.x, a.y), f2), qb = scaled(pack2(b.x, b.y), f2);
          c[g] = e2m1x4(qa.x, qa.y, qb.x, qb.y);
          if (sizeof(T) == 4 && look) {  // (2 * bits - 1: a zero becomes the largest word)
            const uint32_t least = min(min(__float_as_uint(a.x) * 2u - 1u, __float_as_uint(a.y) * 2u - 1u), min(__float_as_uint(b.x) * 2u - 1u, __float_as_uint(b.y) * 2u - 1u));
            odd |= least < 2u * __float_as_uint(kScaleLo);
          }
        }
        out[k] = c[0] | (c[1] << 16);
      }
    };
    uint32_t w[2], hi[2];
    codes(inv_lo, true, w);
    if (lo_alone) {
      hi[0] = w[0];
      hi[1] = w[1];
    } else {
      codes(inv_hi, false, hi);
    }
    uint8_t* row = cache + slot * kRowBytes;
    if (odd || ((w[0] ^ hi[0]) | (w[1] ^ hi[1]))) {
#pragma unroll 1
      for (int k = 0; k < 2; ++k) {
        uint32_t word = k ? w[1] : w[0];
        const uint32_t up = k ? hi[1] : hi[0];
        uint32_t todo = odd ? 0xffffffffu : word ^ up;
#pragma unroll 1
        while (todo) {
          const int i = (__ffs(todo) - 1) >> 2;
          const uint32_t nibble = 0xfu << (4 * i);
          todo &= ~nibble;
          const float x = to_f32<T>(src[kPer == 8 ? 256 * k + 8 * lane + i : 256 * k + 128 * (i >> 2) + 4 * lane + (i & 3)]);
          if (odd) word = (word & ~nibble) | (e2m1_code(x, scale) << (4 * i));
          else if (above(x, scale, (word >> (4 * i)) & 7u)) word = (word & ~nibble) | (up & nibble);
        }
        if (k) w[1] = word;
        else w[0] = word;
      }
    }
    if (kPer == 8) {
#pragma unroll
      for (int q = 0; q < 2; ++q) *reinterpret_cast<uint32_t*>(row + 4 * lane + 128 * q) = w[q];
    } else {
#pragma unroll
      for (int q = 0; q < 4; ++q) *reinterpret_cast<uint16_t*>(row + 2 * lane + 64 * q) = uint16_t(w[q >> 1] >> (16 * (q & 1)));
    }
    *reinterpret_cast<uint16_t*>(row + kLatent / 2 + 2 * lane) = uint16_t(rope_pair(to_f32<T>(raw.rope0), to_f32<T>(raw.rope1)));
    if (lane == 0) cache_sf[slot] = scale;
  }
}

// ------------------------------------------------------------------------------------------ many tokens of a 16-bit type
// Four tokens per warp.  Eight lanes work on a token: a lane owns the 16-byte chunks lane, lane + 8, ... of its row (128
// contiguous bytes of four rows to a load) and eight consecutive RoPE values.  What is done once per token (the slot, the division, the
// reciprocal, the tests: a third of the 241 instructions a token cost a warp) is shared by four tokens, and a warp has 4.5 KiB of loads
// in flight before it waits, so that the next token's need not be kept in registers beside this one's.  CTAs of two warps and
// no loop over the tokens (but for the largest grids): the hardware fills the place of a CTA as soon as it is done.
// 262144 BF16 tokens 75.3 -> 58.7 us, 6.63 TB/s, the rate of a plain copy (with a loop: 24 warps a SM 63.2; the next tokens in registers 74.9;
// staged with cp.async 64.8).  Fewer tokens take longer this way, a lane having four times the work one after the other:
// see launch_t.  FP32 rows gain nothing: a warp per token runs at 6.58 TB/s.
constexpr int kManyWarps = 2;
constexpr int kManyResident = 14;  // CTAs per SM, which leave 72 registers a thread: they hold a token's share without spills (BF16 70, FP16 66)
constexpr int kManyLanes = 8, kManyChunks = kLatent / (8 * kManyLanes), kManyRope = kRope / kManyLanes;
template <typename T> struct ManyShare {
  static_assert(sizeof(T) == 2, "a 16-byte chunk is eight elements");
  uint4 r[kManyChunks];
  uint4 rope;
};
// Largest magnitude among a lane's elements as f32 bits; NaN if there is one.
template <typename T2, typename T> __device__ __forceinline__ uint32_t amax_bits_many(const ManyShare<T>& raw) {
  T2 m = __habs2(reinterpret_cast<const T2*>(&raw.r[0])[0]);
#pragma unroll
  for (int i = 1; i < 4 * kManyChunks; ++i) m = __hmax2_nan(m, __habs2(reinterpret_cast<const T2*>(&raw.r[i >> 2])[i & 3]));
  return max(__float_as_uint(__low2float(m)) & 0x7fffffffu, __float_as_uint(__high2float(m)) & 0x7fffffffu);
}
template <typename T> struct PairOf;
template <> struct PairOf<__half> { using type = __half2; };
template <> struct PairOf<__nv_bfloat16> { using type = __nv_bfloat162; };
// The codes of a chunk in which q_lo and q_hi (word and up) differ.  e: the chunk's first element.
template <typename T> __device__ __noinline__ uint32_t settle(const T* e, float scale, uint32_t word, uint32_t up) {
  uint32_t todo = word ^ up;
#pragma unroll 1
  while (todo) {
    const int i = (__ffs(todo) - 1) >> 2;
    const uint32_t nibble = 0xfu << (4 * i);
    todo &= ~nibble;
    if (above(to_f32<T>(e[i]), scale, (word >> (4 * i)) & 7u)) word = (word & ~nibble) | (up & nibble);
  }
  return word;
}
// A token that takes the exact division for all its codes, by the whole warp: 16 of them a lane, as in cache_write_kernel.
template <typename T> __device__ __noinline__ void write_exactly(const T* src, float scale, uint8_t* row, int lane) {
#pragma unroll 1
  for (int q = 0; q < 2; ++q) {
    const T* e = src + 256 * q + 8 * lane;
    uint32_t word = 0;
#pragma unroll 1
    for (int i = 0; i < 8; ++i) word |= e2m1_code(to_f32<T>(e[i]), scale) << (4 * i);
    *reinterpret_cast<uint32_t*>(row + 4 * lane + 128 * q) = word;
  }
}

// another lane's pointer
template <typename P> __device__ __forceinline__ P* of_lane(P* p, int lane) {
  return reinterpret_cast<P*>(__shfl_sync(0xffffffffu, reinterpret_cast<unsigned long long>(p), lane));
}

template <typename T>
__global__ void __launch_bounds__(kManyWarps * 32, kManyResident)
cache_write_many_kernel(const T* __restrict__ latent, int64_t latent_stride, const T* __restrict__ rope, int64_t rope_stride,
                        const float* __restrict__ scale_in, const int64_t* __restrict__ slot_mapping, int64_t num_tokens,
                        uint8_t* __restrict__ cache, float* __restrict__ cache_sf, int64_t num_slots, bool rope_16) {
  const int lane = threadIdx.x & (kManyLanes - 1), group = (threadIdx.x & 31) / kManyLanes;
  constexpr int kPerCta = kManyWarps * 32 / kManyLanes;
  const int64_t step = int64_t(gridDim.x) * kPerCta;
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  // (a warp's groups stay together: those past the end go over the last token again and write nothing)
  int64_t t = int64_t(blockIdx.x) * kPerCta + threadIdx.x / kManyLanes;
  int64_t t0 = t - group;
#pragma unroll 1
  for (; t0 < num_tokens; t += step, t0 += step) {
    const int64_t at = t < num_tokens ? t : num_tokens - 1;
    const T* src = latent + at * latent_stride + 8 * lane;
    ManyShare<T> raw;
#pragma unroll
    for (int q = 0; q < kManyChunks; ++q) raw.r[q] = *reinterpret_cast<const uint4*>(src + 8 * kManyLanes * q);
    const T* rp = rope + at * rope_stride + kManyRope * lane;
    if (rope_16) {
      raw.rope = *reinterpret_cast<const uint4*>(rp);
    } else {  // rows aligned to two elements
      uint32_t* e = reinterpret_cast<uint32_t*>(&raw.rope);
#pragma unroll
      for (int i = 0; i < kManyRope / 2; ++i) e[i] = reinterpret_cast<const uint32_t*>(rp)[i];
    }
    const int64_t slot = slot_mapping ? slot_mapping[at] : at;
    const bool live = t < num_tokens && slot >= 0 && slot < num_slots;  // padding token (negative) or out of the pool: nothing is written
    uint32_t top = amax_bits_many<typename PairOf<T>::type, T>(raw);    // non-negative floats compare as integers
#pragma unroll
    for (int o = kManyLanes / 2; o > 0; o >>= 1) top = max(top, __shfl_xor_sync(0xffffffffu, top, o));
    if (!__any_sync(0xffffffffu, live)) continue;
    float scale;
    if (scale_in) {
      scale = scale_in[at];
    } else {
      float amax = __uint_as_float(top);
#pragma unroll 1
      for (uint32_t nans = __ballot_sync(0xffffffffu, top > kInfBits && live); nans;) {  // one token after the other, by the whole warp
        const int g = (__ffs(nans) - 1) / kManyLanes;
        nans &= ~(((1u << kManyLanes) - 1u) << (kManyLanes * g));
        const float m = amax_without_nan<T>(of_lane(src, kManyLanes * g), threadIdx.x & 31);
        if (g == group) amax = m;
      }
      scale = __fdiv_rn(amax, 6.0f);
      if (!(scale > 0.f)) scale = 1.0f;
    }
    const bool odd = !(scale >= kScaleLo && scale <= kScaleHi && top <= kInfBits);
    const bool lo_alone = !scale_in && fmaf(-6.f, scale, __uint_as_float(top)) <= scale * (6.f * 0x1p-24f / 1.76f);
    const bool both = !__all_sync(0xffffffffu, lo_alone);
    const float inv = __frcp_rn(scale), inv_lo = inv * (1.f - 0x1p-20f), inv_hi = inv * (1.f + 0x1p-20f);
    const uint64_t lo2 = pack2(inv_lo, inv_lo), hi2 = pack2(inv_hi, inv_hi);
    uint8_t* row = cache + slot * kRowBytes;
#pragma unroll
    for (int q = 0; q < kManyChunks; ++q) {
      auto codes = [&](uint64_t f2) {
        uint32_t c[2];
#pragma unroll
        for (int g = 0; g < 2; ++g) {
          const float2 a = pair_of<T>(raw.r[q], 2 * g), b = pair_of<T>(raw.r[q], 2 * g + 1);
          const float2 qa = scaled(pack2(a.x, a.y), f2), qb = scaled(pack2(b.x, b.y), f2);
          c[g] = e2m1x4(qa.x, qa.y, qb.x, qb.y);
        }
        return c[0] | (c[1] << 16);
      };
      uint32_t w = codes(lo2), up = w;
      if (both && !lo_alone) up = codes(hi2);
      if (w != up && !odd) w = settle<T>(src + 8 * kManyLanes * q, scale, w, up);
      if (live && !odd) *reinterpret_cast<uint32_t*>(row + 4 * (lane + kManyLanes * q)) = w;
    }
    uint32_t r8[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const float2 a = pair_of<T>(raw.rope, 2 * i), b = pair_of<T>(raw.rope, 2 * i + 1);
      r8[i] = rope_pair(a.x, a.y) | (rope_pair(b.x, b.y) << 16);
    }
    if (live) {
      *reinterpret_cast<uint2*>(row + kLatent / 2 + kManyRope * lane) = make_uint2(r8[0], r8[1]);
      if (lane == 0) cache_sf[slot] = scale;
    }
#pragma unroll 1
    for (uint32_t rest = __ballot_sync(0xffffffffu, odd && live); rest;) {
      const int from = __ffs(rest) - 1;  // (lane 0 of a token's group)
      rest &= ~(((1u << kManyLanes) - 1u) << from);
      write_exactly<T>(of_lane(src, from), __shfl_sync(0xffffffffu, scale, from), of_lane(row, from), threadIdx.x & 31);
    }
  }
}

// From how many tokens of a 16-bit type on four go to a warp: one a warp -> four, inputs that are not in L2: 8191 tokens 5.17 -> 5.04 us,
// 16384 7.94 -> 8.58, 24576 9.6 -> 9.2 (FP16 9.0 -> 8.2), 30000 11.2 -> 10.3, 60000 19.2 -> 16.2, 262144 75.3 -> 58.7; 61 tokens 1.68 -> 2.33.
// With the scales given every token is converted twice (see lo_alone), which weighs more where a lane has four times the work: 24576 10.6 ->
// 12.3, 40000 15.3 -> 16.4, 57344 20.2 -> 20.35 (FP16 18.35 -> 18.55), 200000 62.8 -> 55.2 (57.0 -> 51.1).
// Strided rows 24576 9.95 -> 9.65; nine of ten tokens padding 6.9 -> 7.5, 200000 39.1 -> 37.1; all of them 6.05 -> 5.55; a NaN in every token 46.0 -> 44.9.
constexpr int64_t kManyTokens = 24576, kManyTokensScaled = 65536;
}  // namespace
int cache_write_tokens_per_warp(bool half, int64_t n, bool scales_given) {
  return half && n >= (scales_given ? kManyTokensScaled : kManyTokens) ? 4 : 1;
}
namespace {
template <typename T>
cudaError_t launch_t(const void* latent, int64_t ls, const void* rope, int64_t rs, const float* scale_in,
                     const int64_t* slots, int64_t n, void* cache, float* sf, int64_t num_slots, cudaStream_t stream) {
  int dev = 0, sms = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg = {};
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if constexpr (sizeof(T) == 2) {
    if (cache_write_tokens_per_warp(true, n, scale_in != nullptr) > 1) {
      constexpr int64_t per = kManyWarps * 32 / kManyLanes;
      const int64_t want = (n + per - 1) / per;
      cfg.gridDim = dim3(unsigned(want < 0x7fffffff ? want : 0x7fffffff));
      cfg.blockDim = dim3(kManyWarps * 32);
      return cudaLaunchKernelEx(&cfg, cache_write_many_kernel<T>, static_cast<const T*>(latent), ls, static_cast<const T*>(rope), rs, scale_in, slots, n,
                                static_cast<uint8_t*>(cache), sf, num_slots, reinterpret_cast<uintptr_t>(rope) % 16 == 0 && rs % 8 == 0);
    }
  }
  // one wave of resident CTAs, fewer when the token count is small
  const int64_t want = (n + kWriterWarps - 1) / kWriterWarps;
  const int grid = int(want < int64_t(sms) * kResident<T> ? want : int64_t(sms) * kResident<T>);
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(kWriterWarps * 32);
  return cudaLaunchKernelEx(&cfg, cache_write_kernel<T>, static_cast<const T*>(latent), ls, static_cast<const T*>(rope), rs, scale_in, slots, n,
                            static_cast<uint8_t*>(cache), sf, num_slots);
}

}  // namespace

cudaError_t launch_cache_write(const void* latent, int64_t latent_stride, const void* rope, int64_t rope_stride, int in_dtype,
                               const float* scale_in, const int64_t* slot_mapping, int64_t num_tokens, void* cache,
                               float* cache_sf, int64_t num_slots, cudaStream_t stream) {
  if (num_tokens == 0) return cudaSuccess;
  switch (in_dtype) {
    case MLA_FP4_IN_BF16:
      return launch_t<__nv_bfloat16>(latent, latent_stride, rope, rope_stride, scale_in, slot_mapping, num_tokens, cache, cache_sf, num_slots, stream);
    case MLA_FP4_IN_F16:
      return launch_t<__half>(latent, latent_stride, rope, rope_stride, scale_in, slot_mapping, num_tokens, cache, cache_sf, num_slots, stream);
    default:
      return launch_t<float>(latent, latent_stride, rope, rope_stride, scale_in, slot_mapping, num_tokens, cache, cache_sf, num_slots, stream);
  }
}

}  // namespace mla
