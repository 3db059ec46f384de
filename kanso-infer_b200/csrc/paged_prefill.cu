// Prompt attention over the int8 / fp8 KV pool on mma.sync tiles: many query tokens per sequence
// (forward_prefill and mixed batches, src/model.rs:1002-1099,1470-1529).
//
// The rows of a tile are (query token, head of the GQA group) pairs of one sequence and kv head, so
// that a staged K/V tile of 64 tokens serves 16 rows in each of four warps. The one-row-per-CTA form
// that decoding uses walks each row's prefix on its own: at 2048 query tokens in four sequences of
// up to 2240 tokens (15 / 5 heads of 64) that is 2.5 GB of record reads out of L2 and dp4a arithmetic,
// 838 us with the chunk's store; this form takes 103 us.
//
// Numbers, no less exact than the decode form's:
//   * int8: the query row is two int8 planes (q ~ d (hi + lo / 254)); both products with the int8
//     K rows are exact int32 sums on m16n8k32. fp8: K as f16 (every E4M3 value is one), the query
//     row over a power of two as two f16 values.
//   * V as f16 (exact for both types). The V scale cannot leave the sum over tokens, so it goes into
//     the weights: w_j = 2^(s_j + log2 vs_j - max), and the softmax's denominator takes w_j / vs_j
//     (pool_mma.cuh: unless scales are out of the ordinary). The weights, at most 2^14, go into the
//     products as the sum of two f16 values (22 bits).
//   * f32 sums, running maximum, one rescaling per tile and only where a maximum moved.
//
// Bound: the tensor pipe at mma.sync rates, 8 cycles an instruction per SM quarter (two products for
// each of Q.K and P.V: 37 us of the 103), and the issue of about 20 instructions per score and lane
// of softmax, splitting and matrix loads beside it (38 M instructions, 35 us), which overlap only
// as far as the three CTAs of an SM are in different phases.
#include <cuda_fp8.h>

#include <algorithm>
#include <type_traits>

#include "kv_pool.h"
#include "paged_prefill.h"
#include "pool_mma.cuh"

namespace kanso {

constexpr int PP_TOK = 64;  // tokens of a staged tile
// Rows of a CTA. Four warps rather than eight: 15 / 5 heads of 64, 2048 query tokens in four
// sequences 98 against 126 us, since twice the CTAs even out the sequences' lengths better than a
// V tile shared by 128 rows saves conversions.
constexpr int PP_WARPS = 4, PP_ROWS = PP_WARPS * 16;
constexpr uint32_t PP_SEQS = 128;  // sequences of one launch, in its arguments

struct PpSeq {
  uint32_t ctx, q_len, row0, tile0;  // row0: first query token; tile0: first row tile
};
struct PpArgs {
  KvGeom g;
  const float* q;
  const uint32_t* tables;
  float* out;
  float* part;  // splits > 1: [split][query token][head][hd], then [split][query token][head][2]
  int* status;
  uint32_t layer, num_heads, max_blocks, group, num_seqs, num_tiles, splits, rows;
  uint32_t seq0;  // this launch's first sequence
  float scale;
  PpSeq seq[PP_SEQS];
};

__device__ __forceinline__ void cp_async4(void* dst, const void* src, bool in) {
  const int n = in ? 4 : 0;
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(n)
               : "memory");
}
// Shared memory: raw K and V rows [2][64][HD] each (16-byte chunks swizzled for the matrix loads of
// K), V as f16 [64][HD] (and K, fp8), the raw scales [2][2][64], the derived ones [3][64], the unit.
template <int HD, bool FP8>
struct PpSmem {
  static constexpr uint32_t raw = PP_TOK * HD;       // one raw tile
  static constexpr uint32_t f16 = PP_TOK * HD * 2;   // one f16 tile
  static constexpr uint32_t v16 = 4 * raw, k16 = v16 + f16;
  static constexpr uint32_t sc = FP8 ? k16 + f16 : k16;
  static constexpr uint32_t der = sc + 4 * PP_TOK * 4;
  static constexpr uint32_t bytes = der + 3 * PP_TOK * 4 + 16;
};

template <int HD, bool FP8>
__global__ void __launch_bounds__(PP_WARPS * 32, HD == 64 ? 3 : 2)
    paged_prefill_kernel(const __grid_constant__ PpArgs a) {
  extern __shared__ __align__(128) uint8_t smem[];
  using S = PpSmem<HD, FP8>;
  constexpr int NT = PP_WARPS * 32, CH = HD / 16;  // 16-byte chunks of a row
  constexpr int ITEMS = PP_TOK * CH / NT;    // K (and V) chunks a thread copies per tile
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t kvh = blockIdx.y, split = blockIdx.z, G = a.group, bs = a.g.block_size;
  pdl_launch_dependents();

  // the last tiles of a sequence see the most keys: they go first
  const uint32_t tile = a.num_tiles - 1 - blockIdx.x;
  uint32_t s = 0;
  for (uint32_t step = PP_SEQS / 2; step; step >>= 1)
    if (s + step < a.num_seqs && a.seq[s + step].tile0 <= tile) s += step;
  const PpSeq sq = a.seq[s];
  const uint32_t r0 = (tile - sq.tile0) * PP_ROWS, rows = sq.q_len * G;
  const uint32_t first_pos = sq.ctx - sq.q_len;
  const uint32_t last_row = min(r0 + PP_ROWS, rows) - 1;
  const uint32_t keys = first_pos + last_row / G + 1;  // keys that any row of the CTA sees
  const uint32_t n_all = (keys + PP_TOK - 1) / PP_TOK;
  const uint32_t i0 = n_all * split / a.splits, i1 = n_all * (split + 1) / a.splits;
  const uint32_t* table = a.tables + (size_t)(a.seq0 + s) * a.max_blocks;

  // this lane's two rows: query token, head, last visible key (-1: no such row)
  uint32_t tok[2], head[2];
  int lim[2];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const uint32_t r = r0 + warp * 16 + (lane >> 2) + 8 * h;
    const bool in = r < rows;
    tok[h] = in ? r / G : 0;
    head[h] = kvh * G + (in ? r - tok[h] * G : 0);
    lim[h] = in ? (int)(first_pos + tok[h]) : -1;
    tok[h] += sq.row0;
  }
  const bool warp_live = r0 + warp * 16 < rows;
  const uint32_t wrow = min(r0 + warp * 16, rows - 1);
  const int wmin = (int)(first_pos + wrow / G);  // every row of the warp sees keys 0 .. wmin
  const int wmax = (int)(first_pos + min(r0 + warp * 16 + 15, rows - 1) / G);

  pdl_wait();  // q, the tables and the pool may come from earlier kernels

  // One 16-byte chunk of K and of V per item; the first chunk's thread brings the row's scales. Block
  // ids are read a tile ahead of the copies that need them.
  uint32_t blk[ITEMS], off[ITEMS];
  auto find_tile = [&](uint32_t i) {
#pragma unroll
    for (int it = 0; it < ITEMS; ++it) {
      const uint32_t key = min(i * PP_TOK + (tid + it * NT) / CH, keys - 1), b = key / bs;
      off[it] = key - b * bs;
      blk[it] = __ldg(table + b);
    }
  };
  auto load_tile = [&](uint32_t i, uint32_t st) {
    uint8_t* kd = smem + st * S::raw;
    uint8_t* vd = smem + (2 + st) * S::raw;
    float* sd = reinterpret_cast<float*>(smem + S::sc) + st * 2 * PP_TOK;
#pragma unroll
    for (int it = 0; it < ITEMS; ++it) {
      const uint32_t item = tid + it * NT, t = item / CH, c = item % CH;
      const bool in = i * PP_TOK + t < keys;
      if (blk[it] >= a.g.num_blocks) {
        atomicOr(a.status, DEV_BAD_INDEX);
        blk[it] = 0;
      }
      const uint8_t* rec = a.g.pool + a.g.rec_offset(a.layer, blk[it], kvh);
      const uint32_t sw = HD == 64 ? c ^ ((t >> 1) & 3) : c ^ (t & 7);
      cp_async16(kd + t * HD + sw * 16, rec + (size_t)off[it] * HD + c * 16, in);
      cp_async16(vd + t * HD + c * 16, rec + a.g.v_off() + (size_t)off[it] * HD + c * 16, in);
      if (c == 0) {
        cp_async4(sd + t, rec + a.g.ks_off() + off[it] * 4, in);
        cp_async4(sd + PP_TOK + t, rec + a.g.vs_off() + off[it] * 4, in);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  auto start = [&] {
    if (i0 >= i1) return;
    find_tile(i0);
    load_tile(i0, 0);
    find_tile(i0 + 1);
  };
  start();

  // ---- the query rows as A fragments, two terms each ----
  constexpr int KS = FP8 ? HD / 16 : HD / 32;  // k steps of an instruction
  uint32_t qh[KS][4], ql[KS][4];
  float cr[2];  // what a product with the raw K bytes is multiplied by
  if (!FP8) {
    float x[2][KS][8];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const float* row = a.q + ((size_t)tok[h] * a.num_heads + head[h]) * HD + (lane & 3) * 4;
      float top = 0.f;
#pragma unroll
      for (int ks = 0; ks < KS; ++ks)
#pragma unroll
        for (int p = 0; p < 2; ++p) {
          const float4 v = *reinterpret_cast<const float4*>(row + ks * 32 + p * 16);
          x[h][ks][p * 4 + 0] = v.x;
          x[h][ks][p * 4 + 1] = v.y;
          x[h][ks][p * 4 + 2] = v.z;
          x[h][ks][p * 4 + 3] = v.w;
          top = fmaxf(fmaxf(top, fmaxf(fabsf(v.x), fabsf(v.y))), fmaxf(fabsf(v.z), fabsf(v.w)));
        }
      top = fmaxf(top, __shfl_xor_sync(0xFFFFFFFFu, top, 1));
      top = fmaxf(top, __shfl_xor_sync(0xFFFFFFFFu, top, 2));
      const float d = top / 127.0f, id = d != 0.f ? 1.0f / d : 0.f;
      cr[h] = d * (1.0f / 254.0f);
#pragma unroll
      for (int ks = 0; ks < KS; ++ks)
#pragma unroll
        for (int p = 0; p < 2; ++p) {
          uint32_t wh = 0, wl = 0;
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const float v = x[h][ks][p * 4 + e];
            const float hi = fminf(fmaxf(rintf(v * id), -127.f), 127.f);
            const float lo = fminf(fmaxf(rintf(fmaf(-d, hi, v) * (254.0f * id)), -127.f), 127.f);
            wh |= ((uint32_t)(int)hi & 0xFFu) << (8 * e);
            wl |= ((uint32_t)(int)lo & 0xFFu) << (8 * e);
          }
          qh[ks][p * 2 + h] = wh;
          ql[ks][p * 2 + h] = wl;
        }
    }
  } else {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const float* row = a.q + ((size_t)tok[h] * a.num_heads + head[h]) * HD + (lane & 3) * 2;
      float2 x[KS][2];
      float top = 0.f;
#pragma unroll
      for (int ks = 0; ks < KS; ++ks)
#pragma unroll
        for (int p = 0; p < 2; ++p) {
          x[ks][p] = *reinterpret_cast<const float2*>(row + ks * 16 + p * 8);
          top = fmaxf(top, fmaxf(fabsf(x[ks][p].x), fabsf(x[ks][p].y)));
        }
      top = fmaxf(top, __shfl_xor_sync(0xFFFFFFFFu, top, 1));
      top = fmaxf(top, __shfl_xor_sync(0xFFFFFFFFu, top, 2));
      float down;
      pow2_scale(top, cr[h], down);
#pragma unroll
      for (int ks = 0; ks < KS; ++ks)
#pragma unroll
        for (int p = 0; p < 2; ++p)
          split_f16(x[ks][p].x * down, x[ks][p].y * down, qh[ks][p * 2 + h], ql[ks][p * 2 + h]);
    }
  }

  float o[HD / 8][4], mt[2], l[2], unit[2];  // o counts in units, and is worth 2^mt
  const float* der = reinterpret_cast<const float*>(smem + S::der);

  // All tiles in order; false: a row or token of this thread asks for the careful form.
  auto walk = [&](auto careful) {
    constexpr bool CAREFUL = decltype(careful)::value;
    uint32_t seen = 0;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      mt[h] = -INFINITY;
      l[h] = 0.f;
      unit[h] = CAREFUL ? 0.f : 1.f;
    }
#pragma unroll
    for (int j = 0; j < HD / 8; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) o[j][e] = 0.f;
    for (uint32_t i = i0; i < i1; ++i) {
      const uint32_t st = (i - i0) & 1;
      asm volatile("cp.async.wait_group 0;" ::: "memory");
      __syncthreads();  // the tile has landed, and nothing of the one before is still read
      if (i + 1 < i1) {
        load_tile(i + 1, st ^ 1);
        find_tile(i + 2);
      }
      // ---- V (fp8: and K) to f16; scales to what the softmax wants ----
#pragma unroll
      for (int w = 0; w < (FP8 ? 2 : 1); ++w) {
#pragma unroll
        for (int it = 0; it < ITEMS; ++it) {
          const uint32_t item = tid + it * NT, t = item / CH, c = item % CH;
          const uint32_t sw = HD == 64 ? c ^ ((t >> 1) & 3) : c ^ (t & 7);
          const uint4 raw = *reinterpret_cast<const uint4*>(
              w ? smem + st * S::raw + t * HD + sw * 16 : smem + (2 + st) * S::raw + t * HD + c * 16);
          const uint2 a0 = bytes_to_f16<FP8>(raw.x), a1 = bytes_to_f16<FP8>(raw.y);
          const uint2 a2 = bytes_to_f16<FP8>(raw.z), a3 = bytes_to_f16<FP8>(raw.w);
          uint8_t* d = smem + (w ? S::k16 : S::v16) + t * (HD * 2);
          *reinterpret_cast<uint4*>(d + (((2 * c) ^ (t & 7)) * 16)) = make_uint4(a0.x, a0.y, a1.x, a1.y);
          *reinterpret_cast<uint4*>(d + (((2 * c + 1) ^ (t & 7)) * 16)) =
              make_uint4(a2.x, a2.y, a3.x, a3.y);
        }
      }
      if (tid < PP_TOK) {
        const float* sc = reinterpret_cast<const float*>(smem + S::sc) + st * 2 * PP_TOK;
        float* d = reinterpret_cast<float*>(smem + S::der);
        d[tid] = sc[tid] * a.scale;
        if (CAREFUL) {
          float vs[2];  // both warps look at the whole tile
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const uint32_t t = lane + 32 * h;
            vs[h] = any_value<FP8, CH>(smem + (2 + st) * S::raw + t * HD) ? sc[PP_TOK + t] : 0.f;
          }
          const TileUnit tu = tile_unit(vs[0], vs[1]);
          // finite: rows that do not see a token must not meet its infinite scale
          d[PP_TOK + tid] = fminf((warp ? vs[1] : vs[0]) * tu.up, 3.4028235e38f);
          if (tid == 0) d[3 * PP_TOK] = tu.down;
        } else {
          const float vs = i * PP_TOK + tid < keys ? sc[PP_TOK + tid] : 1.f;
          seen |= scale_bits(vs);
          d[PP_TOK + tid] = __log2f(vs);
          d[2 * PP_TOK + tid] = 1.0f / vs;
        }
      }
      const bool work = warp_live && (int)(i * PP_TOK) <= wmax;  // the warp has rows that see the tile
      int sc_i[PP_TOK / 8][4];
      if (!FP8 && work) {
        const uint32_t kb = smem_u32(smem + st * S::raw);
#pragma unroll
        for (int j = 0; j < PP_TOK / 8; ++j) {
          const uint32_t t = j * 8 + (lane & 7);
          uint32_t b[KS][2];
#pragma unroll
          for (int p = 0; p < KS / 2; ++p) {
            const uint32_t c = p * 4 + (lane >> 3);
            const uint32_t sw = HD == 64 ? c ^ ((t >> 1) & 3) : c ^ (t & 7);
            uint32_t r[4];
            ldm_x4(r, kb + t * HD + sw * 16);
            b[2 * p][0] = r[0];
            b[2 * p][1] = r[1];
            b[2 * p + 1][0] = r[2];
            b[2 * p + 1][1] = r[3];
          }
#pragma unroll
          for (int e = 0; e < 4; ++e) sc_i[j][e] = 0;
#pragma unroll
          for (int ks = 0; ks < KS; ++ks) mma_s8(sc_i[j], qh[ks], b[ks][0], b[ks][1]);
#pragma unroll
          for (int e = 0; e < 4; ++e) sc_i[j][e] *= 254;
#pragma unroll
          for (int ks = 0; ks < KS; ++ks) mma_s8(sc_i[j], ql[ks], b[ks][0], b[ks][1]);
        }
      }
      __syncthreads();  // the f16 tiles and the scales are complete
      if (!work) continue;
      float t_[PP_TOK / 8][4];
      if (FP8) {
        const uint32_t kb = smem_u32(smem + S::k16);
#pragma unroll
        for (int j = 0; j < PP_TOK / 8; ++j) {
          const uint32_t t = j * 8 + (lane & 7);
#pragma unroll
          for (int e = 0; e < 4; ++e) t_[j][e] = 0.f;
#pragma unroll
          for (int p = 0; p < KS / 2; ++p) {
            uint32_t r[4];
            ldm_x4(r, kb + t * (HD * 2) + (((p * 4 + (lane >> 3)) ^ (t & 7)) * 16));
            float c0[4] = {0.f, 0.f, 0.f, 0.f}, c1[4] = {0.f, 0.f, 0.f, 0.f};
            mma_f16(c0, ql[2 * p], r[0], r[1]);
            mma_f16(c1, ql[2 * p + 1], r[2], r[3]);
            mma_f16(c0, qh[2 * p], r[0], r[1]);
            mma_f16(c1, qh[2 * p + 1], r[2], r[3]);
#pragma unroll
            for (int e = 0; e < 4; ++e) t_[j][e] += c0[e] + c1[e];
          }
        }
      }
      // ---- scores in units of log2, with the V scale's logarithm ----
      float top[2] = {-INFINITY, -INFINITY};
#pragma unroll
      for (int j = 0; j < PP_TOK / 8; ++j) {
        const float2 ks2 = *reinterpret_cast<const float2*>(der + j * 8 + (lane & 3) * 2);
        const float2 lv2 = *reinterpret_cast<const float2*>(der + PP_TOK + j * 8 + (lane & 3) * 2);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float x = FP8 ? t_[j][e] : (float)sc_i[j][e];
          const float u = x * cr[e >> 1] * ((e & 1) ? ks2.y : ks2.x);
          t_[j][e] = CAREFUL ? log2_units(u) : log2_score(u, (e & 1) ? lv2.y : lv2.x);
        }
      }
      if ((int)(i * PP_TOK + PP_TOK - 1) > wmin) {  // some row of the warp does not see all of it
#pragma unroll
        for (int j = 0; j < PP_TOK / 8; ++j)
#pragma unroll
          for (int e = 0; e < 4; ++e)
            if ((int)(i * PP_TOK + j * 8 + (lane & 3) * 2 + (e & 1)) > lim[e >> 1])
              t_[j][e] = -INFINITY;
      }
#pragma unroll
      for (int j = 0; j < PP_TOK / 8; ++j) {
        top[0] = fmaxf(top[0], fmaxf(t_[j][0], t_[j][1]));
        top[1] = fmaxf(top[1], fmaxf(t_[j][2], t_[j][3]));
      }
      float base[2];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        top[h] = fmaxf(top[h], __shfl_xor_sync(0xFFFFFFFFu, top[h], 1));
        top[h] = fmaxf(top[h], __shfl_xor_sync(0xFFFFFFFFu, top[h], 2));
        // a whole number in the careful form, whose later changes to the reference are then exact
        top[h] = fmaxf(CAREFUL ? ceilf(top[h]) : top[h], mt[h]);
        base[h] = top[h] == -INFINITY ? 0.f : CAREFUL ? top[h] : top[h] - 14.f;  // weights up to 2^14
      }
      float f[2];  // what the earlier sums are worth under the new maximum
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        f[h] = mt[h] == -INFINITY ? 0.f : ex2_approx(mt[h] - top[h]);
        l[h] *= f[h];
        mt[h] = top[h];
      }
      float own[2] = {1.f, 1.f};  // careful: what the exponentials' sums are worth
      if (CAREFUL) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          float largest = 0.f;
#pragma unroll
          for (int j = 0; j < PP_TOK / 8; ++j) {
            const float* vn = der + PP_TOK + j * 8 + (lane & 3) * 2;
            largest = fmaxf(largest, ex2_approx(t_[j][2 * h] - base[h]) * vn[0]);
            largest = fmaxf(largest, ex2_approx(t_[j][2 * h + 1] - base[h]) * vn[1]);
          }
          largest = fmaxf(largest, __shfl_xor_sync(0xFFFFFFFFu, largest, 1));
          largest = fmaxf(largest, __shfl_xor_sync(0xFFFFFFFFu, largest, 2));
          const int by = lift_weights(largest, der[3 * PP_TOK], f[h], unit[h]);
          base[h] -= (float)by;
          own[h] = exp2i(-by);
        }
      }
      // ---- weights and their sums ----
      uint32_t ph[PP_TOK / 16][4], pl[PP_TOK / 16][4];
#pragma unroll
      for (int k = 0; k < PP_TOK / 16; ++k) {
#pragma unroll
        for (int p = 0; p < 2; ++p) {  // tokens 16k + 8p ..
          const int j = 2 * k + p;
          const float2 iv = *reinterpret_cast<const float2*>(
              der + (CAREFUL ? 1 : 2) * PP_TOK + j * 8 + (lane & 3) * 2);
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            float w0 = ex2_approx(t_[j][2 * h] - base[h]);
            float w1 = ex2_approx(t_[j][2 * h + 1] - base[h]);
            l[h] = fmaf(w0, CAREFUL ? own[h] : iv.x, l[h]);
            l[h] = fmaf(w1, CAREFUL ? own[h] : iv.y, l[h]);
            if (CAREFUL) {
              w0 *= iv.x;
              w1 *= iv.y;
            }
            split_f16(w0, w1, ph[k][p * 2 + h], pl[k][p * 2 + h]);
          }
        }
      }
      // ---- the tile's product with V, added to the sums outside of the tensor cores: those cut
      // off where an f32 addition rounds, which over hundreds of steps is a bias of 3e-6 ----
      const uint32_t vb = smem_u32(smem + S::v16);
#pragma unroll
      for (int d = 0; d < HD / 16; ++d) {
        float s0[4] = {0.f, 0.f, 0.f, 0.f}, s1[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int k = 0; k < PP_TOK / 16; ++k) {
          const uint32_t t = k * 16 + (lane & 15);
          uint32_t r[4];
          ldm_x4_t(r, vb + t * (HD * 2) + (((2 * d + (lane >> 4)) ^ (t & 7)) * 16));
          if (FP8) {  // sums of 16 tokens there (and of 32 dims above): 3e-7 against 4.6e-7 of 64
            float c0[4] = {0.f, 0.f, 0.f, 0.f}, c1[4] = {0.f, 0.f, 0.f, 0.f};
            mma_f16(c0, pl[k], r[0], r[1]);
            mma_f16(c1, pl[k], r[2], r[3]);
            mma_f16(c0, ph[k], r[0], r[1]);
            mma_f16(c1, ph[k], r[2], r[3]);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              s0[e] += c0[e];
              s1[e] += c1[e];
            }
          } else {
            mma_f16(s0, pl[k], r[0], r[1]);
            mma_f16(s1, pl[k], r[2], r[3]);
            mma_f16(s0, ph[k], r[0], r[1]);
            mma_f16(s1, ph[k], r[2], r[3]);
          }
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          o[2 * d][e] = fmaf(o[2 * d][e], f[e >> 1], s0[e]);
          o[2 * d + 1][e] = fmaf(o[2 * d + 1][e], f[e >> 1], s1[e]);
        }
      }
    }

    bool good = CAREFUL || !unusual_scales(seen);
#pragma unroll
    for (int h = 0; h < 2 && !CAREFUL; ++h) {
      float top = 0.f;
#pragma unroll
      for (int j = 0; j < HD / 8; ++j)
        top = fmaxf(top, fmaxf(fabsf(o[j][2 * h]), fabsf(o[j][2 * h + 1])));
      top = fmaxf(top, __shfl_xor_sync(0xFFFFFFFFu, top, 1));
      top = fmaxf(top, __shfl_xor_sync(0xFFFFFFFFu, top, 2));
      good &= top >= REFERENCE_WEIGHT || mt[h] == -INFINITY;
      mt[h] -= 14.f;
    }
    return good;
  };
  if (__syncthreads_or(!walk(std::false_type{}))) {
    start();
    walk(std::true_type{});
  }

#pragma unroll
  for (int h = 0; h < 2; ++h) {
    l[h] += __shfl_xor_sync(0xFFFFFFFFu, l[h], 1);
    l[h] += __shfl_xor_sync(0xFFFFFFFFu, l[h], 2);
    if (lim[h] < 0) continue;
    const size_t row = (size_t)tok[h] * a.num_heads + head[h];
    const size_t all = (size_t)a.rows * a.num_heads;
    float* dst = a.splits == 1 ? a.out + row * HD : a.part + (split * all + row) * HD;
    const float inv = a.splits > 1 ? 1.f : l[h] > 0.f ? 1.0f / l[h] : 0.f;
#pragma unroll
    for (int j = 0; j < HD / 8; ++j)
      *reinterpret_cast<float2*>(dst + j * 8 + (lane & 3) * 2) =
          make_float2(o[j][2 * h] * inv * unit[h], o[j][2 * h + 1] * inv * unit[h]);
    if (a.splits > 1 && (lane & 3) == 0)
      *reinterpret_cast<float2*>(a.part + a.splits * all * HD + (split * all + row) * 2) =
          make_float2(mt[h], l[h]);
  }
}

// The splits of one (query token, head): one warp.
template <int HD>
__global__ void paged_prefill_merge_kernel(const __grid_constant__ PpArgs a) {
  pdl_launch_dependents();
  pdl_wait();
  const size_t all = (size_t)a.rows * a.num_heads;
  const size_t row = (size_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (row >= all) return;
  const float2* ml = reinterpret_cast<const float2*>(a.part + a.splits * all * HD);
  float M = -INFINITY;
  for (uint32_t s = 0; s < a.splits; ++s) M = fmaxf(M, ml[s * all + row].x);
  float l = 0.f, v[HD / 32];
#pragma unroll
  for (int e = 0; e < HD / 32; ++e) v[e] = 0.f;
  for (uint32_t s = 0; s < a.splits; ++s) {
    const float2 x = ml[s * all + row];
    if (x.x == -INFINITY) continue;  // no key of this split is visible
    const float f = ex2_approx(x.x - M);
    l = fmaf(x.y, f, l);
#pragma unroll
    for (int e = 0; e < HD / 32; ++e)
      v[e] = fmaf(a.part[(s * all + row) * HD + e * 32 + lane], f, v[e]);
  }
  const float inv = l > 0.f ? 1.0f / l : 0.f;
#pragma unroll
  for (int e = 0; e < HD / 32; ++e) a.out[row * HD + e * 32 + lane] = v[e] * inv;
}

template <int HD, bool FP8>
static int32_t pp_launch(kanso_cuda_ctx* ctx, const PpArgs& a) {
  constexpr size_t smem = PpSmem<HD, FP8>::bytes;
  int32_t st = allow_max_smem(ctx, (const void*)paged_prefill_kernel<HD, FP8>);
  if (st) return st;
  launch_dependent(ctx, paged_prefill_kernel<HD, FP8>,
                   dim3(a.num_tiles, a.g.kv_heads, a.splits), dim3(PP_WARPS * 32), smem, a);
  if ((st = after_launch(ctx, "paged_attention_prefill")) || a.splits == 1) return st;
  launch_dependent(ctx, paged_prefill_merge_kernel<HD>,
                   dim3((a.rows * a.num_heads + 7) / 8), dim3(256), 0, a);
  return after_launch(ctx, "paged_attention_prefill merge");
}

int32_t launch_paged_prefill(kanso_cuda_ctx* ctx, const kanso_cuda_kv* kv, uint32_t layer,
                             const float* q, const uint32_t* tables, const uint32_t* ctx_lens,
                             const uint32_t* q_lens, float* out,
                             const kanso_paged_attention_params* p, bool* handled) {
  *handled = false;
  const uint32_t hd = p->head_dim, G = p->num_heads / p->num_kv_heads, S = p->num_seqs;
  if ((hd != 64 && hd != 128) || !aligned16(q) || !aligned16(out)) return KANSO_OK;
  uint64_t T = 0, longest = 0;
  for (uint32_t s = 0; s < S; ++s) {
    T += q_lens[s];
    longest = std::max<uint64_t>(longest, ctx_lens[s]);
  }
  // Below three query tokens per sequence the row kernel's CTAs, one per token, are as many and do
  // less: 40 sequences on 1000 cached tokens, 15 / 5 heads of 64: 1 token each 25 us there, 27 us
  // here; 2 tokens 32 and 27; 3 tokens 40 and 27 (8 / 8 heads: 24 and 33, 33 and 37, 41 and 37).
  if (T < 3ull * S) return KANSO_OK;
  *handled = true;

  PpArgs a;
  a.g = kv_geom(kv);
  a.q = q;
  a.tables = tables;
  a.out = out;
  a.part = nullptr;
  a.status = ctx->dev_status;
  a.layer = layer;
  a.num_heads = p->num_heads;
  a.max_blocks = p->max_num_blocks_per_seq;
  a.group = G;
  a.rows = (uint32_t)T;
  a.scale = p->scale;
  a.splits = 1;
  uint32_t row0 = 0;
  for (uint32_t s0 = 0; s0 < S; s0 += PP_SEQS) {
    a.seq0 = s0;
    a.num_seqs = 0;
    a.num_tiles = 0;
    const uint32_t end = std::min(S, s0 + PP_SEQS);
    for (uint32_t s = s0; s < end; ++s) {
      a.seq[a.num_seqs++] = {ctx_lens[s], q_lens[s], row0, a.num_tiles};
      a.num_tiles += (uint32_t)(((uint64_t)q_lens[s] * G + PP_ROWS - 1) / PP_ROWS);
      row0 += q_lens[s];
    }
    if (!a.num_tiles) continue;
    if (S <= PP_SEQS) {
      // Few rows: the keys are shared out too, at least four tiles of them to a CTA, until two CTAs
      // per SM have work (one sequence of 1500 tokens, 8 / 1 heads of 128: 74 us in one piece, 56 us
      // with two CTAs per SM, 58 and 64 us with four and eight).
      const uint64_t ctas = (uint64_t)a.num_tiles * p->num_kv_heads, goal = 2ull * ctx->sm_count;
      const uint64_t most = std::max<uint64_t>(1, longest / (4 * PP_TOK));
      if (ctas < goal) a.splits = (uint32_t)std::min<uint64_t>({most, (goal + ctas - 1) / ctas, 32});
      if (a.splits > 1) {
        a.part = (float*)ctx_scratch(ctx, (size_t)a.splits * T * p->num_heads * (hd + 2) * 4);
        if (!a.part) return KANSO_ERR_DEVICE;
      }
    }
    int32_t st;
    if (hd == 64)
      st = a.g.fp8 ? pp_launch<64, true>(ctx, a) : pp_launch<64, false>(ctx, a);
    else
      st = a.g.fp8 ? pp_launch<128, true>(ctx, a) : pp_launch<128, false>(ctx, a);
    if (st) return st;
  }
  return KANSO_OK;
}

}  // namespace kanso
