// Decode attention over the int8 / fp8 pool in tiles of 16 tokens on mma.sync (head sizes 64 and 128,
// blocks of whole 16 tokens); every other call is paged_attn_stage1's (paged_attention.cu), whose
// arguments, decode-step fusion and merge of partitions this kernel shares.
//
// One CTA per (context partition, kv head, sequence) serves the heads of the GQA group. Each of its 8
// warps walks tiles of its own through a small ring of shared memory (one bulk copy per 16-token
// record, a few tiles ahead), with a running maximum and sums of its own: nothing but the staging of
// the query and the end of the partition needs a barrier. Numbers as in paged_prefill.cu, and no less
// exact than one thread per token was:
//   * scores: A = K rows of 16 tokens as they lie in the record (a lane takes 16 bytes of a row), B =
//     the query heads' two planes, column 2 * head + plane, so that a lane has both of its head.
//     int8: exact sums of q ~ d (hi + lo / 254); fp8: K as f16 (every E4M3 value is one), the query
//     over a power of two as two f16 values.
//   * the tokens of a tile go through A in the order 0 5 1 4 2 7 3 6 (+ 8): a transposition of 8 x 8
//     pairs (first and second f16 value of a weight) then gives the B operand of the next product,
//     and the V words that a lane needs come from different banks.
//   * values: A = V^T from pairs of tokens' words as f16 (exact), sums of a tile in the tensor core,
//     across tiles in f32 registers. The V scale goes into the weights: w = 2^(s + log2 vs - max),
//     the denominator takes w / vs (pool_mma.cuh: unless scales are out of the ordinary).
#include <type_traits>

#include "paged_attention.cuh"
#include "pool_mma.cuh"

namespace kanso {

constexpr int PD_NT = 256, PD_WARPS = PD_NT / 32;
constexpr uint32_t PD_TILE = 16;  // tokens

template <int HD>
struct PdTile {
  static constexpr uint32_t bytes = 2 * PD_TILE * HD + 8 * PD_TILE;  // K, V, both scales
  // Tiles of a warp's ring: three CTAs to an SM at head size 64, two at 128.
  static constexpr uint32_t slots = HD == 64 ? 4 : 3;
};

template <int G, bool FP8, int HD>
__global__ void __launch_bounds__(PD_NT, HD == 64 ? 3 : 2)
    paged_decode_kernel(const __grid_constant__ PaArgs a) {
  constexpr int HT = (G + 3) / 4, NV = HD / 32;      // tiles of four heads; V words of a lane
  constexpr int QS = FP8 ? HD / 16 : HD / 32;        // steps of the score product
  constexpr int QE = HD / 32;
  constexpr uint32_t SLOTS = PdTile<HD>::slots, TB = PdTile<HD>::bytes;
  extern __shared__ __align__(128) uint8_t smem[];
  __shared__ __align__(16) uint8_t s_q[(FP8 ? 4 : 2) * G * HD];  // [plane][head][dim]
  __shared__ float s_qd[G];
  __shared__ float s_cos[HD / 2], s_sin[HD / 2];
  __shared__ float s_m[PD_WARPS][G], s_l[PD_WARPS][G];
  __shared__ uint64_t s_full[PD_WARPS][SLOTS];
  pdl_launch_dependents();
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  // every sequence's first partitions, which are the long ones, before any sequence's second
  const uint32_t kvh = blockIdx.x, seq = blockIdx.y, part = blockIdx.z, bs = a.g.block_size;

  // Inside the decode step (fused) lengths, positions, slots and the table are inputs of the whole
  // step, and the cache rows of earlier steps are older still: only q and the new K and V rows come
  // from the kernel before this one.
  const bool fused = a.k_new != nullptr;
  if (!fused) pdl_wait();
  uint32_t ctx = a.lens[seq], pos = fused ? a.positions[seq] : 0;
  ctx = pa_clamp_ctx(a, ctx, part == 0 && kvh == 0 && tid == 0);
  const uint32_t t0 = part * a.part_tokens;
  if (ctx == 0 && part == 0) {
    // the CPU statement leaves zeros (src/metal/paged_attention.rs:112-115)
    float* o = a.out + ((size_t)seq * a.num_heads + (size_t)kvh * G) * HD;
    if (fused) pdl_wait();  // readers of the buffer are earlier kernels of the stream
    for (uint32_t e = tid; e < G * HD; e += PD_NT) o[e] = 0.f;
    if (a.xp) {
      for (uint32_t e = tid; e < G * HD; e += PD_NT) pa_store_packed(a, seq, kvh * G * HD + e, 0.f);
      if (seq == 0) pa_zero_packed_rows(a, gridDim.y, kvh * G * HD, G * HD, tid, PD_NT);
    }
  }
  if (t0 >= ctx) return;
  const uint32_t n = min(a.part_tokens, ctx - t0), ntile = (n + PD_TILE - 1) / PD_TILE;

  // ---- this warp's tiles: warp, warp + 8, ... of the partition ----
  const uint32_t tseq = a.row_seq ? a.row_seq[seq] : seq;
  const uint32_t* table = a.tables + (size_t)tseq * a.max_blocks;
  const uint32_t mine = ntile > (uint32_t)warp ? (ntile - warp + PD_WARPS - 1) / PD_WARPS : 0;
  uint8_t* ring = smem + warp * SLOTS * TB;
  // lane i knows the pool blocks of the warp's tiles i, i + 32, ...; the first ones now
  auto tile_block = [&](uint32_t i) {
    if (i >= mine) return 0u;
    uint32_t phys = table[(t0 + (warp + i * PD_WARPS) * PD_TILE) / bs];
    if (phys >= a.g.num_blocks) {
      atomicOr(a.status, DEV_BAD_INDEX);
      phys = 0;
    }
    return phys;
  };
  uint32_t blocks = tile_block(lane);
  if (lane == 0) {
    for (uint32_t i = 0; i < SLOTS; ++i) mbar_init(&s_full[warp][i], 1);
    mbar_fence_init();
  }
  __syncwarp();
  // all lanes: tile i of the warp into the slot of the p-th copy, p % SLOTS
  auto load = [&](uint32_t i, uint32_t p) {
    if (i && i % 32 == 0) blocks = tile_block(i + lane);
    const uint32_t phys = __shfl_sync(0xFFFFFFFFu, blocks, i & 31);
    if (lane == 0) {
      uint64_t* bar = &s_full[warp][p % SLOTS];
      uint8_t* dst = ring + p % SLOTS * TB;
      const uint8_t* rec = a.g.pool + a.g.rec_offset(a.layer, phys, kvh);
      mbar_arrive_expect_tx(bar, TB);
      if (bs == PD_TILE) {
        bulk_g2s(dst, rec, TB, bar);
      } else {
        const uint32_t off = (t0 + (warp + i * PD_WARPS) * PD_TILE) % bs;
        bulk_g2s(dst, rec + a.g.k_off() + off * HD, PD_TILE * HD, bar);
        bulk_g2s(dst + PD_TILE * HD, rec + a.g.v_off() + off * HD, PD_TILE * HD, bar);
        bulk_g2s(dst + 2 * PD_TILE * HD, rec + a.g.ks_off() + off * 4, PD_TILE * 4, bar);
        bulk_g2s(dst + 2 * PD_TILE * HD + PD_TILE * 4, rec + a.g.vs_off() + off * 4, PD_TILE * 4,
                 bar);
      }
    }
  };
  const uint32_t ahead = min(mine, SLOTS);
  for (uint32_t i = 0; i < ahead; ++i) load(i, i);

  uint32_t new_slot = 0;
  if (fused) {
    if (pos >= (uint32_t)a.table_len) {
      if (tid == 0) atomicOr(a.status, DEV_BAD_INDEX);
      pos = 0;
    }
    if (tid < HD / 2) {
      s_cos[tid] = a.cos_t[(size_t)pos * (HD / 2) + tid];
      s_sin[tid] = a.sin_t[(size_t)pos * (HD / 2) + tid];
    }
    new_slot = a.slots[seq];
    __syncthreads();  // the RoPE factors are in shared memory
    pdl_wait();
  }
  if (a.xp && seq == 0 && part == 0)
    pa_zero_packed_rows(a, gridDim.y, kvh * G * HD, G * HD, tid, PD_NT);

  // element d of a head after rotate-half RoPE; multiplies and adds round separately, as the
  // reference's tensor ops do (the stored K bytes must equal the CPU path's)
  auto roped = [&](const float* row, uint32_t d) {
    if (!fused) return row[d];
    const uint32_t j = d < HD / 2 ? d : d - HD / 2;
    const float x0 = row[j], x1 = row[j + HD / 2], c_ = s_cos[j], s_ = s_sin[j];
    return d < HD / 2 ? __fsub_rn(__fmul_rn(x0, c_), __fmul_rn(x1, s_))
                      : __fadd_rn(__fmul_rn(x0, s_), __fmul_rn(x1, c_));
  };
  auto warp_max = [&](float v) {
#pragma unroll
    for (int o = 16; o; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xFFFFFFFFu, v, o));
    return v;
  };
  // The warp whose tile ends with the newest token quantises that token's K and V
  // (quantize_head_slice, src/kv_cache/quantized_storage.rs:452-469) and stores them in the pool, and in
  // its own copy once that has landed: the last tile of the warp, so no later copy meets the stores.
  const uint32_t i_new = ctx - 1 - t0;  // inside the partition: the context ends in it
  const bool writer =
      fused && ctx - 1 < t0 + n && (uint32_t)warp == (i_new / PD_TILE) % PD_WARPS;
  uint32_t new_q[2] = {0, 0};  // K and V: QE bytes of this lane
  float new_scale[2] = {1.f, 1.f};
  if (writer) {
#pragma unroll
    for (int kv = 0; kv < 2; ++kv) {
      const float* src = (kv ? a.v_new : a.k_new) + ((size_t)seq * a.g.kv_heads + kvh) * HD;
      float x[QE], amax = 0.f;
#pragma unroll
      for (int i = 0; i < QE; ++i) {
        x[i] = kv ? src[lane + 32 * i] : roped(src, lane + 32 * i);
        amax = fmaxf(amax, fabsf(x[i]));
      }
      new_scale[kv] = kv_scale_of(warp_max(amax), FP8);
      const float inv = __fdiv_rn(1.0f, new_scale[kv]);
#pragma unroll
      for (int i = 0; i < QE; ++i) {
        const float scaled = __fmul_rn(x[i], inv);
        const uint8_t qv = FP8 ? (uint8_t)__nv_cvt_float_to_fp8(scaled, __NV_SATFINITE, __NV_E4M3)
                               : (uint8_t)(int8_t)fminf(fmaxf(roundf(scaled), -127.f), 127.f);
        new_q[kv] |= (uint32_t)qv << (8 * i);
      }
    }
    const uint32_t block = new_slot / bs, off = new_slot % bs;
    if (block >= a.g.num_blocks) {
      if (lane == 0) atomicOr(a.status, DEV_BAD_INDEX);
    } else {
      uint8_t* rec = a.g.pool + a.g.rec_offset(a.layer, block, kvh);
#pragma unroll
      for (int kv = 0; kv < 2; ++kv) {
#pragma unroll
        for (int i = 0; i < QE; ++i)
          rec[(kv ? a.g.v_off() : a.g.k_off()) + off * HD + lane + 32 * i] =
              (uint8_t)(new_q[kv] >> (8 * i));
        if (lane == 0)
          reinterpret_cast<float*>(rec + (kv ? a.g.vs_off() : a.g.ks_off()))[off] = new_scale[kv];
      }
    }
  }
  // ---- the query heads' planes: warps from the last one down, which have the fewest tiles ----
  for (int gq = PD_WARPS - 1 - warp; gq < G; gq += PD_WARPS) {
    const float* qrow = a.q + ((size_t)seq * a.num_heads + (size_t)kvh * G + gq) * HD;
    float qe[QE], amax = 0.f;
#pragma unroll
    for (int i = 0; i < QE; ++i) {
      qe[i] = roped(qrow, lane + 32 * i);
      amax = fmaxf(amax, fabsf(qe[i]));
    }
    amax = warp_max(amax);
    if (FP8) {
      __half* qh = reinterpret_cast<__half*>(s_q);
      float up, down;
      pow2_scale(amax, up, down);
#pragma unroll
      for (int i = 0; i < QE; ++i) {
        const float x = qe[i] * down;
        const __half h = __float2half_rn(x);
        qh[gq * HD + lane + 32 * i] = h;
        qh[(G + gq) * HD + lane + 32 * i] = __float2half_rn(x - __half2float(h));
      }
      if (lane == 0) s_qd[gq] = up;
    } else {
      const float d_ = amax / 127.0f, id = d_ != 0.f ? 1.0f / d_ : 0.f;
#pragma unroll
      for (int i = 0; i < QE; ++i) {
        const float h = fminf(fmaxf(rintf(qe[i] * id), -127.f), 127.f);
        const float l = fminf(fmaxf(rintf(fmaf(-d_, h, qe[i]) * (254.0f * id)), -127.f), 127.f);
        s_q[gq * HD + lane + 32 * i] = (uint8_t)(int8_t)h;
        s_q[(G + gq) * HD + lane + 32 * i] = (uint8_t)(int8_t)l;
      }
      if (lane == 0) s_qd[gq] = d_ * (1.0f / 254.0f);
    }
  }
  __syncthreads();
  uint32_t qb[HT][QS][2];
  float cr[HT];
#pragma unroll
  for (int ht = 0; ht < HT; ++ht) {
    const int h = ht * 4 + (g >> 1);
    const uint8_t* row = s_q + ((g & 1) * G + min(h, G - 1)) * HD * (FP8 ? 2 : 1);
#pragma unroll
    for (int c = 0; c < HD / 64; ++c)  // dims 16 (t + 4c) .. + 15
#pragma unroll
      for (int k = 0; k < (FP8 ? 2 : 1); ++k) {
        uint4 v = *reinterpret_cast<const uint4*>(row + (t + 4 * c) * (FP8 ? 32 : 16) + 16 * k);
        if (h >= G) v = make_uint4(0, 0, 0, 0);
        const int s = (c * (FP8 ? 2 : 1) + k) * 2;
        qb[ht][s][0] = v.x;
        qb[ht][s][1] = v.y;
        qb[ht][s + 1][0] = v.z;
        qb[ht][s + 1][1] = v.w;
      }
    cr[ht] = ht * 4 + t < G ? s_qd[ht * 4 + t] * a.scale : 0.f;
  }

  float m[HT], l[HT], acc[HT][2 * NV][2];
  float unit[HT];  // what acc counts in
  const uint32_t ka = (g & 1) ? 4 + ((g >> 1) ^ 1) : g >> 1;  // rows g and g + 8 of A: ka, ka + 8
  // All tiles in order, as the ring's next copies; false: the careful form is asked for.
  auto walk = [&](auto careful) {
    constexpr bool CAREFUL = decltype(careful)::value;
    uint32_t seen = 0;
#pragma unroll
    for (int ht = 0; ht < HT; ++ht) {
      m[ht] = -INFINITY;
      l[ht] = 0.f;
      unit[ht] = CAREFUL ? 0.f : 1.f;
#pragma unroll
      for (int j = 0; j < 2 * NV; ++j) acc[ht][j][0] = acc[ht][j][1] = 0.f;
    }
    for (uint32_t i = 0; i < mine; ++i) {
      const uint32_t p = CAREFUL ? mine + i : i;
      uint8_t* slot = ring + p % SLOTS * TB;
      // bounded: a copy that never lands is reported, the warp carries on with what it has
      if (!mbar_wait_bounded(&s_full[warp][p % SLOTS], (p / SLOTS) & 1u) && lane == 0)
        atomicOr(a.status, DEV_WAIT_TIMEOUT);
      const uint32_t first = (warp + i * PD_WARPS) * PD_TILE;  // of the partition
      if (writer && i + 1 == mine) {
#pragma unroll
        for (int kv = 0; kv < 2; ++kv) {
#pragma unroll
          for (int e = 0; e < QE; ++e)
            slot[(kv * PD_TILE + i_new - first) * HD + lane + 32 * e] =
                (uint8_t)(new_q[kv] >> (8 * e));
          if (lane == 0)
            reinterpret_cast<float*>(slot + 2 * PD_TILE * HD)[kv * PD_TILE + i_new - first] =
                new_scale[kv];
        }
        __syncwarp();
      }
      const uint8_t* kr = slot;
      const uint8_t* vr = slot + PD_TILE * HD;
      const float* ks = reinterpret_cast<const float*>(slot + 2 * PD_TILE * HD);
      const float* vs = ks + PD_TILE;
      const bool in0 = first + ka < n, in1 = first + ka + 8 < n, whole = first + PD_TILE <= n;

      // ---- V words of tokens t, 4 + (t ^ 1) and the same + 8, by pairs ----
      uint32_t vw[4][NV];
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const uint32_t tk = ((r & 1) ? 4 + (t ^ 1) : t) + 8 * (r >> 1);
        const uint32_t* row = reinterpret_cast<const uint32_t*>(vr + tk * HD) + g;
        uint32_t raw[NV];
        if constexpr (NV == 2) {
          raw[0] = row[8 * (t >> 1)];
          raw[1] = row[8 * ((t >> 1) ^ 1)];
          vw[r][0] = (t >> 1) ? raw[1] : raw[0];
          vw[r][1] = (t >> 1) ? raw[0] : raw[1];
        } else {
          uint32_t one[NV];
#pragma unroll
          for (int j = 0; j < NV; ++j) raw[j] = row[8 * ((j + t) & 3)];
#pragma unroll
          for (int j = 0; j < NV; ++j) one[j] = (t & 1) ? raw[(j + 3) & 3] : raw[j];
#pragma unroll
          for (int j = 0; j < NV; ++j) vw[r][j] = (t & 2) ? one[(j + 2) & 3] : one[j];
        }
        if (!whole && first + tk >= n) {  // never written bytes: E4M3 has NaN patterns
#pragma unroll
          for (int j = 0; j < NV; ++j) vw[r][j] = 0;
        }
      }
      float vs0 = in0 ? vs[ka] : CAREFUL ? 0.f : 1.f, vs1 = in1 ? vs[ka + 8] : CAREFUL ? 0.f : 1.f;
      const float ks0 = ks[ka], ks1 = ks[ka + 8];
      uint4 k0[HD / 64], k1[HD / 64];
#pragma unroll
      for (int c = 0; c < HD / 64; ++c) {
        k0[c] = *reinterpret_cast<const uint4*>(kr + ka * HD + (t + 4 * c) * 16);
        k1[c] = *reinterpret_cast<const uint4*>(kr + (ka + 8) * HD + (t + 4 * c) * 16);
      }
      if (CAREFUL) {
        const uint32_t used =
            __ballot_sync(0xFFFFFFFFu, any_value<FP8, HD / 32>(vr + lane * (HD / 2)));
        if (!(used >> (2 * ka) & 3u)) vs0 = 0.f;
        if (!(used >> (2 * ka + 16) & 3u)) vs1 = 0.f;
      } else {
        seen |= scale_bits(vs0) | scale_bits(vs1);
      }
      // everything of the slot is in registers: the next copy may go there
      __syncwarp();
      if (i + SLOTS < mine) load(i + SLOTS, p + SLOTS);

      // ---- scores ----
      float x0[HT], x1[HT];
#pragma unroll
      for (int ht = 0; ht < HT; ++ht) {
        if constexpr (!FP8) {
          int c4[4] = {0, 0, 0, 0};
#pragma unroll
          for (int c = 0; c < HD / 64; ++c) {
            mma_s8(c4, {k0[c].x, k1[c].x, k0[c].y, k1[c].y}, qb[ht][2 * c][0], qb[ht][2 * c][1]);
            mma_s8(c4, {k0[c].z, k1[c].z, k0[c].w, k1[c].w}, qb[ht][2 * c + 1][0],
                   qb[ht][2 * c + 1][1]);
          }
          x0[ht] = (float)(c4[0] * 254 + c4[1]);
          x1[ht] = (float)(c4[2] * 254 + c4[3]);
        } else {
          // sums of 32 dims in the tensor core, which cuts off where an addition rounds
          float c4[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
          for (int c = 0; c < HD / 64; ++c) {
            const uint32_t w0[4] = {k0[c].x, k0[c].y, k0[c].z, k0[c].w};
            const uint32_t w1[4] = {k1[c].x, k1[c].y, k1[c].z, k1[c].w};
#pragma unroll
            for (int s = 0; s < 4; s += 2) {
              float d4[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
              for (int h = s; h < s + 2; ++h) {
                const uint2 r0 = bytes_to_f16<true>(w0[h]), r1 = bytes_to_f16<true>(w1[h]);
                mma_f16(d4, {r0.x, r1.x, r0.y, r1.y}, qb[ht][4 * c + h][0], qb[ht][4 * c + h][1]);
              }
#pragma unroll
              for (int e = 0; e < 4; ++e) c4[e] += d4[e];
            }
          }
          x0[ht] = c4[0] + c4[1];
          x1[ht] = c4[2] + c4[3];
        }
      }
      // ---- weights ----
      const TileUnit tu = CAREFUL ? tile_unit(vs0, vs1) : TileUnit{1.f, 1.f};
      const float lv0 = CAREFUL ? 0.f : __log2f(vs0), lv1 = CAREFUL ? 0.f : __log2f(vs1);
      const float iv0 = CAREFUL ? vs0 * tu.up : __fdividef(1.0f, vs0);
      const float iv1 = CAREFUL ? vs1 * tu.up : __fdividef(1.0f, vs1);
      uint32_t pb[HT][2];
      float f[HT];
#pragma unroll
      for (int ht = 0; ht < HT; ++ht) {
        const float u0 = x0[ht] * cr[ht] * ks0, u1 = x1[ht] * cr[ht] * ks1;
        const float s0 = !in0 ? -INFINITY : CAREFUL ? log2_units(u0) : log2_score(u0, lv0);
        const float s1 = !in1 ? -INFINITY : CAREFUL ? log2_units(u1) : log2_score(u1, lv1);
        float top = fmaxf(s0, s1);
#pragma unroll
        for (int o = 4; o < 32; o <<= 1) top = fmaxf(top, __shfl_xor_sync(0xFFFFFFFFu, top, o));
        top = fmaxf(top, m[ht]);
        // weights up to 2^14
        const float base = top == -INFINITY ? 0.f : CAREFUL ? top : top - 14.f;
        f[ht] = m[ht] == -INFINITY ? 0.f : ex2_approx(m[ht] - top);
        m[ht] = top;
        float w0 = ex2_approx(s0 - base), w1 = ex2_approx(s1 - base);
        if (CAREFUL) {
          l[ht] = fmaf(l[ht], f[ht], w0 + w1);
          w0 = fmaxf(w0 * iv0, 0.f);  // not a number: no weight, infinite scale
          w1 = fmaxf(w1 * iv1, 0.f);
          float largest = fmaxf(w0, w1);
#pragma unroll
          for (int o = 4; o < 32; o <<= 1)
            largest = fmaxf(largest, __shfl_xor_sync(0xFFFFFFFFu, largest, o));
          const float lift = exp2i(lift_weights(largest, tu.down, f[ht], unit[ht]));
          w0 *= lift;
          w1 *= lift;
        } else {
          l[ht] = fmaf(l[ht], f[ht], fmaf(w0, iv0, w1 * iv1));
        }
        pb[ht][0] = transpose_pairs(split_pair(w0));
        pb[ht][1] = transpose_pairs(split_pair(w1));
      }
      // ---- values ----
#pragma unroll
      for (int j = 0; j < NV; ++j) {
        uint32_t lo[4], hi[4];  // dims 32j + 4g + 0..3 of the first and of the second token pair
        token_pairs<FP8>(vw[0][j], vw[1][j], lo);
        token_pairs<FP8>(vw[2][j], vw[3][j], hi);
#pragma unroll
        for (int ht = 0; ht < HT; ++ht)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            float d4[4] = {0.f, 0.f, 0.f, 0.f};
            mma_f16(d4, {lo[2 * e], lo[2 * e + 1], hi[2 * e], hi[2 * e + 1]}, pb[ht][0], pb[ht][1]);
            float(&c)[2] = acc[ht][2 * j + e];
            c[0] = fmaf(c[0], f[ht], d4[0] + d4[1]);
            c[1] = fmaf(c[1], f[ht], d4[2] + d4[3]);
          }
      }
    }
    if (CAREFUL) return true;
    bool good = !unusual_scales(seen);
#pragma unroll
    for (int ht = 0; ht < HT; ++ht) {
      float top = 0.f;
#pragma unroll
      for (int j = 0; j < 2 * NV; ++j)
        top = fmaxf(top, fmaxf(fabsf(acc[ht][j][0]), fabsf(acc[ht][j][1])));
#pragma unroll
      for (int o = 4; o < 32; o <<= 1) top = fmaxf(top, __shfl_xor_sync(0xFFFFFFFFu, top, o));
      good &= top >= REFERENCE_WEIGHT || ht * 4 + t >= G;
      m[ht] -= 14.f;  // the sums are worth 2^m
    }
    return mine == 0 || __all_sync(0xFFFFFFFFu, good) != 0;
  };
  if (!walk(std::false_type{})) {
    blocks = tile_block(lane);
    // the newest token's bytes lie in the pool and in a slot: before the copies that read and overwrite them
    asm volatile("fence.proxy.async;" ::: "memory");
    __syncwarp();
    for (uint32_t i = 0; i < ahead; ++i) load(i, mine + i);
    walk(std::true_type{});
  }
  // ---- the warps' maxima, sums and accumulators under a common maximum ----
#pragma unroll
  for (int ht = 0; ht < HT; ++ht) {
#pragma unroll
    for (int o = 4; o < 32; o <<= 1) l[ht] += __shfl_xor_sync(0xFFFFFFFFu, l[ht], o);
    if (g == 0 && ht * 4 + t < G) {
      s_m[warp][ht * 4 + t] = m[ht];
      s_l[warp][ht * 4 + t] = l[ht];
    }
  }
  __syncthreads();  // also: every warp is done with its ring, over which `red` lies
  float* red = reinterpret_cast<float*>(smem);
  float pmax[G], psum[G];
#pragma unroll
  for (int gq = 0; gq < G; ++gq) {
    pmax[gq] = s_m[0][gq];
#pragma unroll
    for (int w = 1; w < PD_WARPS; ++w) pmax[gq] = fmaxf(pmax[gq], s_m[w][gq]);
    psum[gq] = 0.f;
#pragma unroll
    for (int w = 0; w < PD_WARPS; ++w)
      psum[gq] += s_m[w][gq] == -INFINITY ? 0.f : s_l[w][gq] * ex2_approx(s_m[w][gq] - pmax[gq]);
  }
#pragma unroll
  for (int ht = 0; ht < HT; ++ht) {
    const int h = ht * 4 + t;
    if (h >= G) continue;
    float top = m[ht];
#pragma unroll
    for (int gq = 0; gq < G; ++gq)
      if (gq == h) top = pmax[gq];
    const float up = m[ht] == -INFINITY ? 0.f : ex2_approx(m[ht] - top);
    float* dst = red + (warp * G + h) * HD + 4 * g;
#pragma unroll
    for (int j = 0; j < NV; ++j)
      *reinterpret_cast<float4*>(dst + 32 * j) = make_float4(
          acc[ht][2 * j][0] * up * unit[ht], acc[ht][2 * j][1] * up * unit[ht],
          acc[ht][2 * j + 1][0] * up * unit[ht], acc[ht][2 * j + 1][1] * up * unit[ht]);
  }
  __syncthreads();
  // warps beyond the partition's tiles have only zeros
  pa_publish<G, PD_NT, true>(a, seq, kvh, part, ctx, HD, red, min(ntile, (uint32_t)PD_WARPS), pmax,
                             psum);
}

uint32_t pa_mma_partition_tokens(const kanso_cuda_ctx* ctx, const kanso_paged_attention_params* p,
                                 const KvGeom& g, uint64_t cap) {
  if ((g.head_dim != 64 && g.head_dim != 128) || g.block_size % PD_TILE) return 0;
  // Long partitions: what a CTA does besides its tiles (lengths, table, query, ticket) costs as much as
  // 40 of them. 64 sequences of 256..4096 tokens, 15 / 5 heads of 64: 56, 48 and 44 us with up to
  // 512, 1024 and 2048 tokens. Shorter ones, down to one tile per warp, while there are fewer than two
  // CTAs per SM (24 sequences of 200..1000 tokens, 16 / 4 heads: 16.8, 15.5 and 18.3 us for one,
  // two and four per SM).
  uint32_t pt = 2048;
  while (pt > PD_WARPS * PD_TILE &&
         (uint64_t)p->num_seqs * p->num_kv_heads * ((cap + pt - 1) / pt) <
             2 * (uint64_t)ctx->sm_count)
    pt >>= 1;
  pt = (pt + g.block_size - 1) / g.block_size * g.block_size;
  // partitions lie along the grid's third dimension (a table of 134 million tokens, no host lengths)
  return (cap + pt - 1) / pt > 65535 ? 0 : pt;
}

template <int G, bool FP8, int HD>
static int32_t pd_launch(kanso_cuda_ctx* ctx, const PaArgs& a, dim3 grid) {
  constexpr size_t ring = (size_t)PD_WARPS * PdTile<HD>::slots * PdTile<HD>::bytes;
  static_assert(ring >= (size_t)PD_WARPS * G * HD * sizeof(float), "the sums lie over the ring");
  auto kern = paged_decode_kernel<G, FP8, HD>;
  const int32_t st = allow_max_smem(ctx, (const void*)kern);
  if (st) return st;
  prefer_max_shared(ctx, (const void*)kern);
  const cudaError_t le = launch_dependent(ctx, kern, grid, dim3(PD_NT), ring, a);
  if (le != cudaSuccess) return cuda_fail(ctx, le, "paged_decode launch");
  return after_launch(ctx, "paged_decode");
}
template <int G>
static int32_t pd_launch_form(kanso_cuda_ctx* ctx, const PaArgs& a, dim3 grid) {
  if (a.g.head_dim == 64)
    return a.g.fp8 ? pd_launch<G, true, 64>(ctx, a, grid) : pd_launch<G, false, 64>(ctx, a, grid);
  return a.g.fp8 ? pd_launch<G, true, 128>(ctx, a, grid) : pd_launch<G, false, 128>(ctx, a, grid);
}

int32_t launch_paged_decode(kanso_cuda_ctx* ctx, const PaArgs& a, uint32_t group, dim3 grid) {
  switch (group) {
    case 1: return pd_launch_form<1>(ctx, a, grid);
    case 2: return pd_launch_form<2>(ctx, a, grid);
    case 3: return pd_launch_form<3>(ctx, a, grid);
    case 4: return pd_launch_form<4>(ctx, a, grid);
    case 5: return pd_launch_form<5>(ctx, a, grid);
    case 6: return pd_launch_form<6>(ctx, a, grid);
    case 7: return pd_launch_form<7>(ctx, a, grid);
    default: return pd_launch_form<8>(ctx, a, grid);
  }
}

}  // namespace kanso
