// Products over rows of the quantised pool on mma.sync: what decode and prompt attention share.
#pragma once
#include <cuda_fp8.h>

#include "warp_mma.cuh"

namespace kanso {

__device__ __forceinline__ void mma_s8(int (&c)[4], const uint32_t (&a)[4], uint32_t b0,
                                       uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};"
      : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void mma_f16(float (&c)[4], const uint32_t (&a)[4], uint32_t b0,
                                        uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t h2_bits(__half2 h) { return *reinterpret_cast<uint32_t*>(&h); }
// x = hi + lo, two values at a time
__device__ __forceinline__ void split_f16(float x0, float x1, uint32_t& hi, uint32_t& lo) {
  const __half2 h = __floats2half2_rn(x0, x1);
  const float2 f = __half22float2(h);
  hi = h2_bits(h);
  lo = h2_bits(__floats2half2_rn(x0 - f.x, x1 - f.y));
}
// Four bytes of the pool as two f16 pairs, exactly.
template <bool FP8>
__device__ __forceinline__ uint2 bytes_to_f16(uint32_t w) {
  uint2 r;
  if (FP8) {
    __half2_raw a = __nv_cvt_fp8x2_to_halfraw2((__nv_fp8x2_storage_t)(w & 0xFFFFu), __NV_E4M3);
    __half2_raw b = __nv_cvt_fp8x2_to_halfraw2((__nv_fp8x2_storage_t)(w >> 16), __NV_E4M3);
    r.x = h2_bits(__half2(a));
    r.y = h2_bits(__half2(b));
  } else {
    // value + 128 in the low byte of 1024's f16 pattern, minus 1152
    w ^= 0x80808080u;
    const __half2 off = __float2half2_rn(1152.f);
    uint32_t a = __byte_perm(w, 0x64646464u, 0x4140), b = __byte_perm(w, 0x64646464u, 0x4342);
    r.x = h2_bits(__hsub2(*reinterpret_cast<__half2*>(&a), off));
    r.y = h2_bits(__hsub2(*reinterpret_cast<__half2*>(&b), off));
  }
  return r;
}

// A power of two that brings |x| <= top under one, from the exponent's bits (a row beyond the normal
// numbers keeps its values).
__device__ __forceinline__ void pow2_scale(float top, float& up, float& down) {
  const int e = (int)(__float_as_uint(top) >> 23);
  const bool ok = e >= 2 && e <= 252;
  down = ok ? __uint_as_float((uint32_t)(253 - e) << 23) : 1.f;
  up = ok ? __uint_as_float((uint32_t)(e + 1) << 23) : 1.f;
}
// u * log2(e) + lv, the constant in two parts: its own rounding would be the largest error of a score
// whose other factors are powers of two (fp8)
__device__ __forceinline__ float log2_score(float u, float lv) {
  return fmaf(u, 1.44269502f, fmaf(u, 1.92596303e-8f, lv));
}
// u * log2(e) alone.
__device__ __forceinline__ float log2_units(float u) {
  return fmaf(u, 1.44269502f, u * 1.92596303e-8f);
}

// ---- V scales ----
// The V scale cannot leave the sum over tokens. The kernels take it into the weight, w = 2^(s + log2 vs - max),
// so that the largest contribution is the reference of the two f16 values (22 bits, down to 2^-38 of it),
// and add w / vs to the denominator. That is exact enough if scales are far from the ends of f32 and the
// reference does contribute; a row of zeros, stored with the scale 1, does not, and may outweigh rows
// that are far smaller. Both show at the end of a pass: some scale was outside of 2^-32 to 2^32, or no
// element of the sums reaches 2^14, the reference's weight (its largest value is 32 or more). Then the
// pass is made once more in the careful form: exponentials of the score alone, which the denominator adds;
// scales relative to the tile's largest; weights brought up tile by tile (lift_weights), sums in units
// of the largest weight so far.
constexpr float REFERENCE_WEIGHT = 16384.f;
// Bits above 28 in the union of these over all scales: one was unusual. Tests of every scale and row as they
// pass took 4 % of both kernels' time; this and the look at the sums 3 % of the prompt kernel's (2048
// query tokens, 15 / 5 heads of 64: 100 -> 103 us) and nothing of the decode kernel's at head size 64.
__device__ __forceinline__ uint32_t scale_bits(float v) { return __float_as_uint(v) - (95u << 23); }
__device__ __forceinline__ bool unusual_scales(uint32_t bits) { return bits >> 29; }
// Whether the 16 N bytes at p hold any value but zero (E4M3 has a second one).
template <bool FP8, int N>
__device__ __forceinline__ bool any_value(const uint8_t* p) {
  uint32_t o = 0;
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const uint4 v = *reinterpret_cast<const uint4*>(p + 16 * i);
    o |= v.x | v.y | v.z | v.w;
  }
  return (o & (FP8 ? 0x7F7F7F7Fu : ~0u)) != 0;
}
// Careful form, all lanes of a warp: the power of two that brings the lanes' scales (0 for no row or a
// row of zeros) under 2^14, and its inverse, which is a normal number.
struct TileUnit {
  float up, down;
};
__device__ __forceinline__ TileUnit tile_unit(float v0, float v1) {
  const uint32_t top =
      __reduce_max_sync(0xFFFFFFFFu, max(__float_as_uint(v0), __float_as_uint(v1))) >> 23;
  const uint32_t e = min(max(top, 14u), 254u);
  return {__uint_as_float((267u - e) << 23), __uint_as_float((e - 13u) << 23)};
}
__device__ __forceinline__ float exp2i(int e) { return __uint_as_float((uint32_t)(127 + e) << 23); }
// The logarithm of the power of two that brings weights up whose largest is `top`, in units of `down`: to
// under 2^14, or to the unit of the earlier sums if those are the larger ones. f: what the earlier sums
// are worth under the new maximum, made their factor; unit: theirs, made the new one.
__device__ __forceinline__ int lift_weights(float top, float down, float& f, float& unit) {
  const int d = (int)(__float_as_uint(down) >> 23);
  const int by = max(min(140 - max((int)(__float_as_uint(top) >> 23), 40), d - 1), 0);
  const float least = __uint_as_float((uint32_t)(d - by) << 23), before = unit * f;
  const int b = (int)(__float_as_uint(before) >> 23) + 1;
  unit = before > least ? __uint_as_float((uint32_t)b << 23) : least;
  f = before / unit;
  return before > least ? max(d - b, -100) : by;
}
// x as two f16 values, side by side
__device__ __forceinline__ uint32_t split_pair(float x) {
  const __half h = __float2half_rn(x);
  return h2_bits(__halves2half2(h, __float2half_rn(x - __half2float(h))));
}
// 8 x 8 matrix of 16-bit values, lane (g, t) holding columns 2t, 2t + 1 of row g
__device__ __forceinline__ uint32_t transpose_pairs(uint32_t v) {
  uint32_t r;
  asm("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(r) : "r"(v));
  return r;
}
// Four bytes of one token and the same of another: (first, second) as f16, per byte.
template <bool FP8>
__device__ __forceinline__ void token_pairs(uint32_t first, uint32_t second, uint32_t (&r)[4]) {
  const uint2 a = bytes_to_f16<FP8>(__byte_perm(first, second, 0x5140));
  const uint2 b = bytes_to_f16<FP8>(__byte_perm(first, second, 0x7362));
  r[0] = a.x;
  r[1] = a.y;
  r[2] = b.x;
  r[3] = b.y;
}

}  // namespace kanso
