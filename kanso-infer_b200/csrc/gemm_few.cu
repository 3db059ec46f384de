// Quantised products of a few activation rows: LinearWeight::forward (src/weights.rs:43-45) for
// decoding batches and short portions of prompts.
//
//   y[M,N] = x[M,K] @ W[N,K]^T,  W in GGUF Q8_0 / Q4_K blocks, x and y f32.
//
// At these row counts the operand goes from the raw bytes in shared memory through registers
// straight into mma.sync fragments: no dequantised tile is written back, fenced and issued from
// another thread, which is what the tcgen05 form (gemm_tma.cu) spends its time on below about a
// hundred rows. mma.sync reaches 1024 (f16) and 2048 (int8) multiply-adds per clock and SM here,
// which is enough up to about 64 rows.
//
//   * A unit is 128 weight rows (int8 form: 128 or 112) x 256 k: one tensor-map copy of 272 (Q8_0) or 144
//     (Q4_K) bytes a row, whole blocks, in rows whose stride is 16 bytes past a multiple of 128, so that
//     8 rows x 4 lanes of 4-byte reads meet 32 different banks without a swizzle.
//   * Units are numbered tile by tile and dealt out in equal contiguous runs; the runs ignore tile
//     borders, so there is no last wave. A run that ends inside a tile adds its sums to y with
//     atomics; the pack kernel has cleared y.
//   * The order of k inside a block is free as long as both operands agree: lane t of a fragment's
//     four takes bytes 4t..4t+3 and 16+4t..16+4t+3 of each 32, and the pack kernel lays the
//     activations out so that the matching values are 16 (f16) or 8 (int8) bytes of one lane.
//   * F16 form: weights become f16 (Q8_0: exact integer, one rounding in d*q; Q4_K:
//     d*sc*(q-8) + (8*d*sc - dmin*m), both factors rounded once), activations are rounded once to
//     f16, sums are f32. 8 warps: 4 groups of 32 rows x 2 halves of the unit's k.
//   * INT8 form (KANSO_ACT_Q8): activations quantised as quantize_row_q8_0 does; one
//     mma.m16n8k32.s8 gives the exact int32 block sums of 16 x 8 results. Scaling and addition are
//     separately rounded and in block order, so that a row whose K is not split equals
//     scalar_gemv_q8_0 (src/quant/q8_0.rs:60-92) bit for bit. The last addition is a scalar one:
//     a packed multiplication followed by a packed addition came back as one rounding.
//
// What bounds it (counters at 14336 x 4096, Q8_0): at one to eight rows the weights' bytes and the
// about 100 instructions that turn 1024 of them into fragments (issue slots 45 % used), at 64 rows
// mma.sync (half its rate); the int8 form the latency of the chain product, subtraction, scaling, addition
// (29 clocks a product and scheduler at 100 rows; the f32 pipe alone would take 16, mma.sync 8).
#include "ctx.h"
#include "tc05.cuh"
#include "tensor_map.h"

namespace kanso {

enum FewForm { FEW_Q8_F16, FEW_Q4_F16, FEW_Q8_INT8 };

constexpr int FEW_K = 256;     // k of a unit
constexpr int FEW_MAX_STAGES = 6;

template <int FORM>
__host__ __device__ constexpr int few_row_bytes() {  // of one weight row in a unit
  return FORM == FEW_Q4_F16 ? Q4K_BYTES : FEW_K / 32 * Q8_BYTES;
}
template <int FORM>
__host__ __device__ constexpr int few_x_bytes() {  // of one activation row in a unit
  return FORM == FEW_Q8_INT8 ? FEW_K + FEW_K / 32 * 4 : FEW_K * 2;
}

struct FewArgs {
  float* y;
  const uint8_t* xp;  // packed activations, one unit's rows after another
  int64_t N;
  int M;
  int chunks;  // units of a tile: K / 256
  int units;
  int stages;
  bool add;  // results are added to a cleared y
  int* status;
};

struct FewZero {
  float* p;
  int64_t n;
};

// ---- activations ----

// One thread: the 8 values of lane t in block b of row m, as 16 bytes. Blocks of odd rows change
// places in pairs, so that a fragment read's 16-byte pieces of two rows fall on different banks.
template <bool VEC>
__global__ void few_pack_f16_kernel(const float* __restrict__ x, uint8_t* __restrict__ xp, int M,
                                    int Mp, int K, const FewZero zero) {
  pdl_launch_dependents();
  pdl_wait();
  const int64_t gtid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t nthreads = (int64_t)gridDim.x * blockDim.x;
  for (int64_t j = gtid; j < zero.n; j += nthreads) zero.p[j] = 0.f;
  const int64_t total = (int64_t)(K / FEW_K) * Mp * 32;
  for (int64_t i = gtid; i < total; i += nthreads) {
    const int t = (int)i & 3, b = (int)(i >> 2) & 7;
    const int64_t cm = i >> 5;  // unit of the row * Mp + row
    const int m = (int)(cm % Mp);
    const int64_t c = cm / Mp;
    float v[8] = {};
    if (m < M) {
      const float* src = x + (int64_t)m * K + c * FEW_K + b * 32 + 4 * t;
      if (VEC) {
        *reinterpret_cast<float4*>(v) = *reinterpret_cast<const float4*>(src);
        *reinterpret_cast<float4*>(v + 4) = *reinterpret_cast<const float4*>(src + 16);
      } else {
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = src[(j & 3) + (j >> 2) * 16];
      }
    }
    uint32_t o[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const __half2 h = __floats2half2_rn(v[2 * j], v[2 * j + 1]);
      o[j] = *reinterpret_cast<const uint32_t*>(&h);
    }
    *reinterpret_cast<uint4*>(xp + cm * (FEW_K * 2) + ((b ^ (m & 1)) * 64) + t * 16) =
        make_uint4(o[0], o[1], o[2], o[3]);
  }
}

// quantize_row_q8_0 (src/quant/q8_0.rs:13-32,43-48), eight threads to a (row, block), four values
// each. A unit: Mp rows of 256 int8, then 8 x Mp scales.
template <bool VEC>
__global__ void few_pack_int8_kernel(const float* __restrict__ x, uint8_t* __restrict__ xp, int M,
                                     int Mp, int K, const FewZero zero) {
  pdl_launch_dependents();
  pdl_wait();
  const int64_t gtid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t nthreads = (int64_t)gridDim.x * blockDim.x;
  for (int64_t j = gtid; j < zero.n; j += nthreads) zero.p[j] = 0.f;
  // total is a multiple of 64: the lanes of a warp stay together
  const int64_t total = (int64_t)(K / FEW_K) * Mp * 64;
  for (int64_t i = gtid; i < total; i += nthreads) {
    const int e = (int)i & 7, b = (int)(i >> 3) & 7;
    const int64_t cm = i >> 6;
    const int m = (int)(cm % Mp);
    const int64_t c = cm / Mp;
    float v[4] = {};
    if (m < M) {
      const float* src = x + (int64_t)m * K + c * FEW_K + b * 32 + 4 * e;
      if (VEC) {
        *reinterpret_cast<float4*>(v) = *reinterpret_cast<const float4*>(src);
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j) v[j] = src[j];
      }
    }
    float amax = fmaxf(fmaxf(fabsf(v[0]), fabsf(v[1])), fmaxf(fabsf(v[2]), fabsf(v[3])));
#pragma unroll
    for (int o = 4; o; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xFFFFFFFFu, amax, o));
    const float d = __fdiv_rn(amax, 127.0f);
    const float id = d != 0.0f ? __fdiv_rn(1.0f, d) : 0.0f;
    uint32_t q = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float r = roundf(__fmul_rn(v[j], id));  // half away from zero, as f32::round
      r = fminf(fmaxf(r, -128.0f), 127.0f);
      q |= ((uint32_t)(uint8_t)(int8_t)r) << (8 * j);
    }
    uint8_t* unit = xp + c * (int64_t)Mp * few_x_bytes<FEW_Q8_INT8>();
    // values 4e..4e+3 belong to lane e % 4, its first or its second four
    *reinterpret_cast<uint32_t*>(unit + m * FEW_K + ((b ^ (m & 3)) * 32) + (e & 3) * 8 +
                                 (e >> 2) * 4) = q;
    if (e == 0) reinterpret_cast<float*>(unit + Mp * FEW_K)[b * Mp + m] = d;
  }
}

// ---- the product ----

__device__ __forceinline__ void few_mma_f16(float (&c)[4], const uint32_t (&a)[4], uint32_t b0,
                                            uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// BIASED: sums that start from the bits of 1.5 * 2^23: below 2^22 in magnitude (here 2^19 at most) the result, read
// as a float, is that value plus the sum. A subtraction, exact, takes the place of a conversion, of which
// an SM does 16 per clock: 32 of the 35 clocks that a product and its roundings took at 100 rows. It is one more
// operation of the pipe that scales and adds, though, and only the forms of 8 or 14 warps above 64 rows, which are
// bound by latency, gain by it (few_launch_int8): with it 17 to 64 rows took 3.5 % longer.
constexpr uint32_t FEW_BIAS = 0x4B400000u;
template <bool BIASED>
__device__ __forceinline__ void few_mma_i8(uint32_t (&d)[4], const uint32_t (&a)[4], uint32_t b0,
                                           uint32_t b1) {
  asm("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%10,%10,%10,%10};"
      : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "r"(BIASED ? FEW_BIAS : 0u));
}
template <typename T>
__device__ __forceinline__ T lds(const uint8_t* p) {
  return *reinterpret_cast<const T*>(p);
}
__device__ __forceinline__ uint64_t f32x2(uint32_t lo, uint32_t hi) {
  return (uint64_t)hi << 32 | lo;
}
__device__ __forceinline__ uint64_t f32x2_mul(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ uint64_t f32x2_add(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ uint32_t h2_bits(__half2 h) { return *reinterpret_cast<uint32_t*>(&h); }
__device__ __forceinline__ __half2 h2_of(uint32_t v) { return *reinterpret_cast<__half2*>(&v); }

// Four bytes of a Q8_0 row's unit, which starts on a word: in even blocks (34 bytes each, two of
// scale) they lie across two words.
template <bool ODD>
__device__ __forceinline__ uint32_t q8_word(const uint8_t* addr) {
  if (ODD) return lds<uint32_t>(addr);
  return __byte_perm(lds<uint32_t>(addr - 2), lds<uint32_t>(addr + 2), 0x5432);
}

// F16 form: one block (32 k) of the warp's 32 rows against NT groups of 8 activation rows.
template <int NT>
__device__ __forceinline__ void few_block_f16(float (&acc)[2][NT][4],
                                              const uint32_t (&a)[2][2][4], const uint8_t* x) {
#pragma unroll
  for (int n = 0; n < NT; ++n) {
    const uint4 b = lds<uint4>(x + n * 8 * FEW_K * 2);
    few_mma_f16(acc[0][n], a[0][0], b.x, b.y);
    few_mma_f16(acc[1][n], a[1][0], b.x, b.y);
    few_mma_f16(acc[0][n], a[0][1], b.z, b.w);
    few_mma_f16(acc[1][n], a[1][1], b.z, b.w);
  }
}

// Four int8 -> d * value as two f16 pairs: the biased byte in the mantissa of 1024 gives the exact
// integer after one subtraction.
__device__ __forceinline__ void q8_pairs(uint32_t w, __half2 d, uint32_t& lo, uint32_t& hi) {
  const __half2 bias = __half2half2(__float2half(1152.f));
  w ^= 0x80808080u;
  lo = h2_bits(__hmul2(__hsub2(h2_of(__byte_perm(w, 0x64646464u, 0x4140)), bias), d));
  hi = h2_bits(__hmul2(__hsub2(h2_of(__byte_perm(w, 0x64646464u, 0x4342)), bias), d));
}

template <int NT, bool ODD>
__device__ __forceinline__ void few_q8_block(float (&acc)[2][NT][4], const uint8_t* w,
                                             const uint8_t* x) {
  uint32_t a[2][2][4];
#pragma unroll
  for (int r = 0; r < 4; ++r) {  // rows g + 8r
    const uint8_t* row = w + r * 8 * few_row_bytes<FEW_Q8_F16>();
    const int t4 = 4 * (threadIdx.x & 3);
    const __half2 d = __half2half2(__ushort_as_half(lds<uint16_t>(row)));
#pragma unroll
    for (int s = 0; s < 2; ++s)
      q8_pairs(q8_word<ODD>(row + 2 + t4 + 16 * s), d, a[r >> 1][s][r & 1],
               a[r >> 1][s][2 + (r & 1)]);
  }
  few_block_f16<NT>(acc, a, x);
}

// Blocks 4 * half .. +3 of a unit.
template <int NT>
__device__ __forceinline__ void few_unit_q8_f16(float (&acc)[2][NT][4], const uint8_t* w,
                                                const uint8_t* x, int half, int g, int t) {
  w += g * few_row_bytes<FEW_Q8_F16>() + half * 4 * Q8_BYTES;
  x += g * FEW_K * 2 + t * 16;
#pragma unroll
  for (int b = 0; b < 4; b += 2) {
    few_q8_block<NT, false>(acc, w + b * Q8_BYTES, x + ((half * 4 + b) ^ (g & 1)) * 64);
    few_q8_block<NT, true>(acc, w + (b + 1) * Q8_BYTES, x + ((half * 4 + b + 1) ^ (g & 1)) * 64);
  }
}

// Four nibbles (one a byte) -> s * (nibble - 8) + c as two f16 pairs.
__device__ __forceinline__ void q4_pairs(uint32_t w, __half2 s, __half2 c, uint32_t& lo,
                                         uint32_t& hi) {
  const __half2 bias = __half2half2(__float2half(1032.f));
  lo = h2_bits(__hfma2(__hsub2(h2_of(__byte_perm(w, 0x64646464u, 0x4140)), bias), s, c));
  hi = h2_bits(__hfma2(__hsub2(h2_of(__byte_perm(w, 0x64646464u, 0x4342)), bias), s, c));
}

template <int NT>
__device__ __forceinline__ void few_unit_q4_f16(float (&acc)[2][NT][4], const uint8_t* w,
                                                const uint8_t* x, int half, int g, int t) {
  w += g * Q4K_BYTES;
  x += g * FEW_K * 2 + t * 16;
  // lane t unpacks the header of row g + 8t: (scale, offset) of the half's four sub-blocks
  uint32_t sc[4];
  {
    const uint4 h = lds<uint4>(w + t * 8 * Q4K_BYTES);
    uint32_t sl, sh, ml, mh;
    unpack_scales_k4(h.y, h.z, h.w, sl, sh, ml, mh);
    const float d = f16_bits_to_f32(h.x), dmin = f16_bits_to_f32(h.x >> 16);
    const uint32_t s4 = half ? sh : sl, m4 = half ? mh : ml;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float s = d * (float)(s4 >> (8 * i) & 63u);
      const float c = 8.f * s - dmin * (float)(m4 >> (8 * i) & 63u);
      sc[i] = h2_bits(__floats2half2_rn(s, c));
    }
  }
#pragma unroll
  for (int p = 0; p < 2; ++p) {  // 32 bytes: the low nibbles are one sub-block, the high the next
    uint32_t raw[4][2];
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int s = 0; s < 2; ++s)
        raw[r][s] =
            lds<uint32_t>(w + r * 8 * Q4K_BYTES + 16 + (half * 2 + p) * 32 + t * 4 + s * 16);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      uint32_t a[2][2][4];
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const uint32_t v = __shfl_sync(0xFFFFFFFFu, sc[2 * p + h], (4 * g) | r);
        const __half2 s2 = __low2half2(h2_of(v)), c2 = __high2half2(h2_of(v));
#pragma unroll
        for (int s = 0; s < 2; ++s)
          q4_pairs((h ? raw[r][s] >> 4 : raw[r][s]) & 0x0F0F0F0Fu, s2, c2, a[r >> 1][s][r & 1],
                   a[r >> 1][s][2 + (r & 1)]);
      }
      few_block_f16<NT>(acc, a, x + ((half * 4 + 2 * p + h) ^ (g & 1)) * 64);
    }
  }
}

// INT8 form: one block of the warp's RT x 16 rows against NT groups of 8 activation rows.
template <int RT, int NT, bool ODD>
__device__ __forceinline__ void few_int8_block(float (&acc)[RT][NT][4], const uint8_t* w,
                                               const uint8_t* x, const uint8_t* dx, int t) {
  uint32_t a[RT][4];
  uint64_t dw[RT][2];
#pragma unroll
  for (int r = 0; r < 2 * RT; ++r) {
    const uint8_t* row = w + r * 8 * few_row_bytes<FEW_Q8_INT8>();
    a[r >> 1][r & 1] = q8_word<ODD>(row + 2 + 4 * t);
    a[r >> 1][2 + (r & 1)] = q8_word<ODD>(row + 18 + 4 * t);
    const uint32_t d = __float_as_uint(f16_bits_to_f32(lds<uint16_t>(row)));
    dw[r >> 1][r & 1] = f32x2(d, d);
  }
#pragma unroll
  for (int n = 0; n < NT; ++n) {
    const uint2 b = lds<uint2>(x + n * 8 * FEW_K);
    const uint2 d2 = lds<uint2>(dx + n * 32);
    const uint64_t dxp = f32x2(d2.x, d2.y);
#pragma unroll
    for (int r = 0; r < RT; ++r) {
      constexpr bool BIASED = NT >= 6;
      uint32_t s[4];
      few_mma_i8<BIASED>(s, a[r], b.x, b.y);
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const uint64_t sum =
            BIASED ? f32x2_add(f32x2(s[2 * j], s[2 * j + 1]),
                               f32x2(FEW_BIAS | 1u << 31, FEW_BIAS | 1u << 31))
                   : f32x2(__float_as_uint((float)(int)s[2 * j]),
                           __float_as_uint((float)(int)s[2 * j + 1]));
        const uint64_t term = f32x2_mul(f32x2_mul(dw[r][j], dxp), sum);
        acc[r][n][2 * j] = __fadd_rn(acc[r][n][2 * j], __uint_as_float((uint32_t)term));
        acc[r][n][2 * j + 1] =
            __fadd_rn(acc[r][n][2 * j + 1], __uint_as_float((uint32_t)(term >> 32)));
      }
    }
  }
}

template <int RT, int NT>
__device__ __forceinline__ void few_unit_int8(float (&acc)[RT][NT][4], const uint8_t* w,
                                              const uint8_t* x, const uint8_t* dx, int Mp, int g,
                                              int t) {
  w += g * few_row_bytes<FEW_Q8_INT8>();
  x += g * FEW_K + t * 8;
  dx += t * 8;
#pragma unroll
  for (int b = 0; b < 8; b += 2) {
    few_int8_block<RT, NT, false>(acc, w + b * Q8_BYTES, x + (b ^ (g & 3)) * 32, dx + b * Mp * 4, t);
    few_int8_block<RT, NT, true>(acc, w + (b + 1) * Q8_BYTES, x + ((b + 1) ^ (g & 3)) * 32,
                                 dx + (b + 1) * Mp * 4, t);
  }
}

// WR groups of RT x 16 rows; the OTHER warps of a row group share out either the unit's k (F16;
// their sums meet in shared memory before they leave the CTA) or the activation rows (INT8: groups
// of NT x 8). No wait is unbounded: after one that ran out a warp skips its work but still takes
// part in the barriers of its row group.
template <int FORM, int TILE, int RT, int NT, int OTHER, int CTAS>
__global__ void __launch_bounds__(TILE / (16 * RT) * OTHER * 32 + 32, CTAS)
    gemm_few_kernel(const __grid_constant__ CUtensorMap tmap, const FewArgs a) {
  constexpr int WR = TILE / (16 * RT), WARPS = WR * OTHER;
  constexpr int Mp = NT * 8 * (FORM == FEW_Q8_INT8 ? OTHER : 1);
  constexpr uint32_t W_BYTES = TILE * few_row_bytes<FORM>();
  constexpr uint32_t X_BYTES = Mp * few_x_bytes<FORM>();
  constexpr uint32_t STAGE = W_BYTES + X_BYTES;
  extern __shared__ __align__(128) uint8_t smem[];
  __shared__ uint64_t full[FEW_MAX_STAGES], empty[FEW_MAX_STAGES];
  __shared__ int abort_flag;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int u0 = (int)((int64_t)a.units * blockIdx.x / gridDim.x);
  const int u1 = (int)((int64_t)a.units * (blockIdx.x + 1) / gridDim.x);

  if (threadIdx.x == 0) {
    for (int i = 0; i < a.stages; ++i) {
      mbar_init(&full[i], 1);
      mbar_init(&empty[i], WARPS);
    }
    abort_flag = 0;
    mbar_fence_init();
  }
  __syncthreads();
  pdl_launch_dependents();

  if (warp == WARPS) {
    if (elect_one()) {
      auto weights = [&](int u, int slot) {
        mbar_arrive_expect_tx(&full[slot], STAGE);
        tma_load_2d(smem + slot * STAGE, &tmap, u % a.chunks * (few_row_bytes<FORM>() / 4),
                    u / a.chunks * TILE, &full[slot]);
      };
      auto rows = [&](int u, int slot) {
        bulk_g2s(smem + slot * STAGE + W_BYTES, a.xp + (int64_t)(u % a.chunks) * X_BYTES, X_BYTES,
                 &full[slot]);
      };
      // the weights do not depend on the kernel before this one
      const int ahead = min(a.stages, u1 - u0);
      for (int i = 0; i < ahead; ++i) weights(u0 + i, i);
      pdl_wait();
      for (int i = 0; i < ahead; ++i) rows(u0 + i, i);
      int issued = ahead;
      for (int i = ahead; i < u1 - u0; ++i) {
        const int slot = i % a.stages;
        if (!mbar_wait_abort(&empty[slot], ((uint32_t)(i / a.stages) & 1u) ^ 1u, &abort_flag))
          break;
        weights(u0 + i, slot);
        rows(u0 + i, slot);
        issued = i + 1;
      }
      // this CTA's copies have landed before it may end
      for (int i = max(0, issued - a.stages); i < issued; ++i)
        mbar_wait_bounded(&full[i % a.stages], (uint32_t)(i / a.stages) & 1u);
    }
    return;
  }

  const int g = lane >> 2, t = lane & 3, wr = warp % WR, other = warp / WR;
  float acc[RT][NT][4] = {};
  bool ok = true;
  for (int i = 0, u = u0; u < u1; ++i, ++u) {
    const int slot = i % a.stages;
    if (ok)
      ok = __all_sync(0xFFFFFFFFu,
                      mbar_wait_abort(&full[slot], (uint32_t)(i / a.stages) & 1u, &abort_flag));
    if (ok) {
      const uint8_t* w = smem + slot * STAGE + wr * (16 * RT) * few_row_bytes<FORM>();
      const uint8_t* x = smem + slot * STAGE + W_BYTES;
      if constexpr (FORM == FEW_Q8_F16)
        few_unit_q8_f16<NT>(acc, w, x, other, g, t);
      else if constexpr (FORM == FEW_Q4_F16)
        few_unit_q4_f16<NT>(acc, w, x, other, g, t);
      else
        few_unit_int8<RT, NT>(acc, w, x + other * NT * 8 * FEW_K,
                              x + Mp * FEW_K + other * NT * 32, Mp, g, t);
      __syncwarp();
      if (lane == 0) mbar_arrive(&empty[slot]);
    }
    if (u + 1 < u1 && (u + 1) % a.chunks) continue;
    // the run leaves this tile
    pdl_wait();
    if constexpr (FORM != FEW_Q8_INT8 && OTHER > 1) {
      float* slab = reinterpret_cast<float*>(smem + a.stages * STAGE) + lane;
      constexpr int STEP = NT < 2 ? NT : 2, PER = RT * STEP * 4 * 32;
#pragma unroll
      for (int n0 = 0; n0 < NT; n0 += STEP) {
        if (other) {
          float* mine = slab + ((other - 1) * WR + wr) * PER;
#pragma unroll
          for (int e = 0; e < RT * STEP * 4; ++e)
            if (n0 + e / 4 % STEP < NT) mine[e * 32] = acc[e / 4 / STEP][n0 + e / 4 % STEP][e & 3];
        }
        asm volatile("bar.sync %0, %1;" ::"r"(1 + wr), "n"(OTHER * 32) : "memory");
        if (!other)
#pragma unroll
          for (int o = 0; o < OTHER - 1; ++o)
#pragma unroll
            for (int e = 0; e < RT * STEP * 4; ++e)
              if (n0 + e / 4 % STEP < NT)
                acc[e / 4 / STEP][n0 + e / 4 % STEP][e & 3] += slab[(o * WR + wr) * PER + e * 32];
        asm volatile("bar.sync %0, %1;" ::"r"(1 + wr), "n"(OTHER * 32) : "memory");
      }
    }
    const int64_t n0 = (int64_t)(u / a.chunks) * TILE + wr * (16 * RT) + g;
    const int m0 = (FORM == FEW_Q8_INT8 ? other * NT * 8 : 0) + 2 * t;
    if (ok && (FORM == FEW_Q8_INT8 || other == 0))
#pragma unroll
      for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const int m = m0 + n * 8 + j;
          if (m < a.M)
#pragma unroll
            for (int r = 0; r < 2 * RT; ++r) {
              const int64_t row = n0 + 8 * r;
              if (row < a.N) {
                float* dst = a.y + (int64_t)m * a.N + row;
                const float v = acc[r >> 1][n][(r & 1) * 2 + j];
                if (a.add)
                  atomicAdd(dst, v);
                else
                  *dst = v;
              }
            }
        }
#pragma unroll
    for (int r = 0; r < RT; ++r)
#pragma unroll
      for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[r][n][j] = 0.f;
  }
  if (!ok && lane == 0) atomicOr(a.status, DEV_WAIT_TIMEOUT);
}

template <int FORM, int TILE, int RT, int NT, int OTHER, int CTAS>
static int32_t few_launch(kanso_cuda_ctx* ctx, const CUtensorMap& map, FewArgs a, int grid) {
  constexpr int WR = TILE / (16 * RT);
  constexpr int Mp = NT * 8 * (FORM == FEW_Q8_INT8 ? OTHER : 1);
  constexpr size_t stage = TILE * few_row_bytes<FORM>() + Mp * few_x_bytes<FORM>();
  constexpr size_t slab =
      FORM == FEW_Q8_INT8 ? 0 : (OTHER - 1) * WR * RT * (NT < 2 ? NT : 2) * 4 * 32 * 4;
  // CTAS blocks share an SM's memory, of which each needs 1 KB besides and its static part
  const size_t room = CTAS == 1 ? (size_t)ctx->smem_optin - 1024
                                : (size_t)ctx->smem_per_sm / CTAS - 2048;
  int stages = (int)((room - slab) / stage);
  if (stages > FEW_MAX_STAGES) stages = FEW_MAX_STAGES;
  if (stages < 2) return fail(ctx, KANSO_ERR_UNSUPPORTED, "gemm_few: no room for two stages");
  a.stages = stages;
  auto kern = gemm_few_kernel<FORM, TILE, RT, NT, OTHER, CTAS>;
  const int32_t st = allow_max_smem(ctx, (const void*)kern);
  if (st) return st;
  prefer_max_shared(ctx, (const void*)kern);
  if (grid == 0) grid = a.units < CTAS * ctx->sm_count ? a.units : CTAS * ctx->sm_count;
  const cudaError_t le = launch_dependent(ctx, kern, dim3((unsigned)grid),
                                          dim3(WR * OTHER * 32 + 32), stages * stage + slab, map, a);
  if (le != cudaSuccess) return cuda_fail(ctx, le, "gemm_few launch");
  return after_launch(ctx, "gemm_few");
}

// Two CTAs per SM up to 32 rows, one with more registers above.
template <int FORM>
static int32_t few_launch_f16(kanso_cuda_ctx* ctx, int nt, const CUtensorMap& map,
                              const FewArgs& a) {
  switch (nt) {
    case 1: return few_launch<FORM, 128, 2, 1, 2, 2>(ctx, map, a, 0);
    case 2: return few_launch<FORM, 128, 2, 2, 2, 2>(ctx, map, a, 0);
    case 3: return few_launch<FORM, 128, 2, 3, 2, 2>(ctx, map, a, 0);
    case 4: return few_launch<FORM, 128, 2, 4, 2, 2>(ctx, map, a, 0);
    case 6: return few_launch<FORM, 128, 2, 6, 2, 1>(ctx, map, a, 0);
    default: return few_launch<FORM, 128, 2, 8, 2, 1>(ctx, map, a, 0);
  }
}

template <int TILE>
static int32_t few_launch_int8(kanso_cuda_ctx* ctx, int nt, const CUtensorMap& map,
                               const FewArgs& a, int grid) {
  switch (nt) {
    case 2: return few_launch<FEW_Q8_INT8, TILE, 1, 2, 1, 1>(ctx, map, a, grid);
    case 3: return few_launch<FEW_Q8_INT8, TILE, 1, 3, 1, 1>(ctx, map, a, grid);
    case 4: return few_launch<FEW_Q8_INT8, TILE, 1, 4, 1, 1>(ctx, map, a, grid);
    case 6: return few_launch<FEW_Q8_INT8, TILE, 1, 3, 2, 1>(ctx, map, a, grid);
    case 8: return few_launch<FEW_Q8_INT8, TILE, 1, 4, 2, 1>(ctx, map, a, grid);
  }
  // More than 64 rows: 8 or 14 warps with registers enough. 28 warps of 16 rows x 32 kept 70 each and
  // spilled: 14336 x 4096 at 100 rows 66 us, 60 with 14 warps of 16 rows x 56. Two strips of 16 weight rows to
  // a warp read an activation once for both (61 us for 128 rows, 66 with one); 112 weight rows are not even strips,
  // and there 28 warps are the faster ones at more than 112 rows (68.1 and 70.7 us; 4096 x 14336 63.4 and 65.8), but
  // not where K is split and a CTA has no more than four units (4096 x 2048 16.5 and 16.0, 4096 x 4096 24.4 and 24.3).
  constexpr int RT = TILE == 128 ? 2 : 1;
  if (nt == 12) return few_launch<FEW_Q8_INT8, TILE, RT, 6, 2, 1>(ctx, map, a, grid);
  if (nt == 14) return few_launch<FEW_Q8_INT8, TILE, RT, 7, 2, 1>(ctx, map, a, grid);
  if constexpr (TILE == 112) {
    if (!(a.add && a.units <= 4 * grid))
      return few_launch<FEW_Q8_INT8, TILE, 1, 4, 4, 1>(ctx, map, a, grid);
  }
  return few_launch<FEW_Q8_INT8, TILE, RT, 8, 2, 1>(ctx, map, a, grid);
}

// How an int8 product is shared out: whole rows per CTA (results bit-identical to the CPU's) while the
// tiles fill the GPU; fewer tiles are split along K while the grid stays within about one wave and
// every part keeps two units (K below 1024 stays whole whatever the number of rows).
struct FewShare {
  int tile, split;
  int64_t tiles, chain;  // chain: weight rows x units that the busiest SM goes through
};
static FewShare few_share(const kanso_cuda_ctx* ctx, int tile, int64_t N, int64_t chunks) {
  FewShare s = {tile, 1, (N + tile - 1) / tile, 0};
  while (s.tiles * s.split * 2 <= ctx->sm_count + ctx->sm_count / 4 &&
         chunks / (s.split * 2) >= 2)
    s.split *= 2;
  const int64_t waves = (s.tiles * s.split + ctx->sm_count - 1) / ctx->sm_count;
  s.chain = waves * tile * ((chunks + s.split - 1) / s.split);
  return s;
}

// y[M,N] = x[M,K] @ W^T for up to 64 activation rows in f16 (act_mode F32) or 128 in exact int8
// block sums (act_mode Q8, Q8_0 weights). Sets *handled = false (and launches nothing) when the
// shape is outside this kernel's range: rows of the block matrix must start on 16-byte boundaries.
int32_t few_matmul(kanso_cuda_ctx* ctx, int32_t dtype, const void* w, const float* x, float* y,
                   int64_t M, int64_t N, int64_t K, int32_t act_mode, bool* handled) {
  *handled = false;
  const bool q4 = dtype == KANSO_DTYPE_Q4_K, int8 = act_mode == KANSO_ACT_Q8;
  if ((!q4 && dtype != KANSO_DTYPE_Q8_0) || (int8 && q4) || (!int8 && act_mode != KANSO_ACT_F32))
    return KANSO_OK;
  if (M < 1 || M > (int8 ? 128 : 64) || N < 1 || K < FEW_K || K % FEW_K != 0 || !w || !x || !y)
    return KANSO_OK;
  const int64_t row_bytes = K / FEW_K * (q4 ? Q4K_BYTES : FEW_K / 32 * Q8_BYTES);
  const int64_t chunks = K / FEW_K;
  // The int8 form is bound by the arithmetic of the SMs that have any: tiles of 112 rows where they
  // shorten the longest chain of rows on an SM. us at 100 and 128 activation rows with 112 | with 128: 14336 x 4096
  // (128 and 112 busy SMs) 62, 68 | 63, 71; 10500 x 4096 62, 68 | 66, 75; 17408 x 4096 (two waves of 112 rows,
  // one of 128) 118, 131 | 63, 72; 18944 x 3584 104, 116 | 56, 64.
  const FewShare s128 = few_share(ctx, 128, N, chunks), s112 = few_share(ctx, 112, N, chunks);
  const FewShare& share = int8 && s112.chain < s128.chain ? s112 : s128;
  const int tile = share.tile;
  const int64_t tiles = share.tiles;
  if (!aligned16(w) || row_bytes > (1 << 28) || tiles * chunks > (1 << 30) || N > (1 << 30))
    return KANSO_OK;
  TmEncodeFn encode = tm_encoder();
  if (!encode) return KANSO_OK;
  CUtensorMap map;
  const cuuint64_t gdim[2] = {(cuuint64_t)row_bytes / 4, (cuuint64_t)N};
  const cuuint64_t gstride[1] = {(cuuint64_t)row_bytes};
  const cuuint32_t box[2] = {(cuuint32_t)(q4 ? Q4K_BYTES : FEW_K / 32 * Q8_BYTES) / 4,
                             (cuuint32_t)tile};
  const cuuint32_t estr[2] = {1, 1};
  const CUresult cr = encode(&map, CU_TENSOR_MAP_DATA_TYPE_UINT32, 2, const_cast<void*>(w), gdim,
                             gstride, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                             CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (cr != CUDA_SUCCESS)
    return fail(ctx, KANSO_ERR_DEVICE, "gemm_few: cuTensorMapEncodeTiled failed (%d)", (int)cr);

  FewArgs a;
  a.y = y;
  a.N = N;
  a.M = (int)M;
  a.chunks = (int)chunks;
  a.units = (int)(tiles * chunks);
  a.status = ctx->dev_status;
  int nt = (int)(M + 7) / 8, grid = 0;
  if (int8) {
    grid = (int)tiles * share.split;
    a.add = share.split > 1;
    // groups of eight rows, shared out to one warp of a row group, two, or (112 weight rows, 16 groups) four
    // (a test per group cost 45 % at 32 rows)
    nt = M <= 16 ? 2 : M <= 24 ? 3 : M <= 32 ? 4 : M <= 48 ? 6 : M <= 64 ? 8 : M <= 96 ? 12 : M <= 112 ? 14 : 16;
  } else {
    a.add = true;
    if (nt > 4) nt = nt <= 6 ? 6 : 8;
  }
  const int Mp = nt * 8;
  const size_t xb = (size_t)chunks * Mp *
                    (int8 ? few_x_bytes<FEW_Q8_INT8>() : few_x_bytes<FEW_Q8_F16>());
  uint8_t* scratch = (uint8_t*)ctx_scratch(ctx, xb + 256);
  if (!scratch) return KANSO_ERR_DEVICE;
  *handled = true;
  a.xp = scratch;
  const FewZero zero = {a.add ? y : nullptr, a.add ? M * N : 0};
  int64_t items = chunks * Mp * (int8 ? 64 : 32);
  if (zero.n / 8 > items) items = zero.n / 8;
  int64_t blocks = (items + 255) / 256;
  if (blocks > 8 * ctx->sm_count) blocks = 8 * ctx->sm_count;
  const bool vec = aligned16(x);
  auto pack = int8 ? (vec ? few_pack_int8_kernel<true> : few_pack_int8_kernel<false>)
                   : (vec ? few_pack_f16_kernel<true> : few_pack_f16_kernel<false>);
  // the same split of an SM's memory as the product's, so that its blocks start beside this one's
  prefer_max_shared(ctx, (const void*)pack);
  const cudaError_t le = launch_dependent(ctx, pack, dim3((unsigned)blocks), dim3(256), 0, x,
                                          scratch, (int)M, Mp, (int)K, zero);
  if (le != cudaSuccess) return cuda_fail(ctx, le, "gemm_few pack launch");
  const int32_t st = after_launch(ctx, "gemm_few pack activations");
  if (st) return st;
  if (!int8)
    return q4 ? few_launch_f16<FEW_Q4_F16>(ctx, nt, map, a)
              : few_launch_f16<FEW_Q8_F16>(ctx, nt, map, a);
  return tile == 112 ? few_launch_int8<112>(ctx, nt, map, a, grid)
                     : few_launch_int8<128>(ctx, nt, map, a, grid);
}

}  // namespace kanso
