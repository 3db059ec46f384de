// Prompt attention with sigmoid weights on tcgen05 (bfloat16): 128 query rows of one head against
// key tiles of 64, scores and the output accumulator in TMEM.
//
// Because the weights are not normalised over keys there is no running maximum and nothing to
// rescale: the output is one accumulator that every tile's weights x values product adds to.
//
//   the first warps, two or three groups of four, one per score buffer: a thread owns a query row, reads
//              its scores from TMEM, forms the weights and writes them as the bfloat16 A operand P
//   then       K copies: a tile's pages by tensor map, one box per page and 64 columns, into a ring of two to
//              four stages (128-byte swizzle); page numbers are looked up in the block table
//   then       S = Q K^T (M = 128, N = 64) into one score buffer after another
//   then       V copies, in a warp of their own: a V tile's place is free much later than a K tile's
//   last       O += P V (V as it lies in the pool, N-major). A thread of its own: in turns with the scores'
//              it waits for K tile i + 2 before P V of tile i.
//
// The distance term, the head's constant and the mask come from one table in shared memory,
// tab[d] = -log2(e) * (cap + pb - r1 ln(1 + r2 d)) for visible distances and +infinity for the
// others, so that a masked weight is 1 / (1 + 2^inf) = 0 without a comparison.
//
// us at 2048 rows behind 2048 cached ones, 16 heads of 128, window 2048: 137 with one copying warp, a ring
// of two and one issuing thread, where every tile took a copy's round trip; 98 with warps and rings of their own and reciprocals shared, 85 with three groups.
#include <algorithm>

#include "dense.cuh"
#include "tc05.cuh"
#include "tensor_map.h"
#include "warp_mma.cuh"

namespace kanso {

constexpr int SP_Q = 128, SP_K = 64, SP_MAX_STAGES = 4;
constexpr int SP_MAX_GROUPS = 3, SP_THREADS = (SP_MAX_GROUPS + 1) * 128;
constexpr int SP_TAB_BELOW = 192, SP_TAB_ABOVE = 208;  // masked entries at the table's two ends
constexpr uint32_t SP_MAX_WINDOW = 8192;
constexpr int SP_P_BYTES = SP_Q * SP_K * 2;

struct PrefillArgs {
  SigmoidAttn a;
  const uint32_t* tables;
  const AttnTile* tiles;
  void* out;
  int64_t out_ld;
  uint32_t max_blocks, num_blocks, block_size, kv_heads, group;
  int out_f32, v_dim, nv;        // nv: v_dim rounded up to 16
  int k_panels, v_panels, k_steps;  // 64-column panels of K and V; 16-column steps of the scores
  int tab_n, stages, groups;  // groups of four warps that form weights
  uint32_t tmem_cols;
  int* status;
};

__device__ __forceinline__ float min_nan(float a, float b) {  // a value that is none stays none
  float m;
  asm("min.NaN.f32 %0, %1, %2;" : "=f"(m) : "f"(a), "f"(b));
  return m;
}
// Reciprocals are taken of products, of four or two values at a time, and multiplied apart again: what bounds
// this kernel once its copies run ahead is the unit for 2^x and 1 / x (four uses a weight, 2.75 so).
// v[e] = c1 / (1 + 2^(v[e] * k1)) + tb[-e]. Exponents end at 30: what that leaves of the quotient, c1 * 2^-30, is
// below the last place of the sum.
__device__ __forceinline__ void sp_capped(float (&v)[8], float k1, float c1, const float* tb) {
#pragma unroll
  for (int g = 0; g < 8; g += 4) {
    float a[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) a[e] = 1.f + ex2_approx(min_nan(v[g + e] * k1, 30.f));
    const float ab = a[0] * a[1], cd = a[2] * a[3], q = c1 * rcp_approx(ab * cd);
    const float qab = q * cd, qcd = q * ab;
    v[g] = fmaf(qab, a[1], tb[-g]);
    v[g + 1] = fmaf(qab, a[0], tb[-g - 1]);
    v[g + 2] = fmaf(qcd, a[3], tb[-g - 2]);
    v[g + 3] = fmaf(qcd, a[2], tb[-g - 3]);
  }
}
// v = 1 / (1 + 2^v); alone: some exponent of the warp is above SP_SHARED (a masked key's is infinite).
constexpr float SP_SHARED = 60.f;
__device__ __forceinline__ void sp_weights(float (&v)[8], bool alone) {
#pragma unroll
  for (int e = 0; e < 8; ++e) v[e] = 1.f + ex2_approx(v[e]);
  if (alone) {
#pragma unroll
    for (int e = 0; e < 8; ++e) v[e] = rcp_approx(v[e]);
    return;
  }
#pragma unroll
  for (int e = 0; e < 8; e += 2) {
    const float q = rcp_approx(v[e] * v[e + 1]), a = v[e];
    v[e] = q * v[e + 1];
    v[e + 1] = q * a;
  }
}

__global__ void __launch_bounds__(SP_THREADS, 1)
    sigmoid_prefill_kernel(const __grid_constant__ CUtensorMap qmap,
                           const __grid_constant__ CUtensorMap kmap,
                           const __grid_constant__ CUtensorMap vmap, const PrefillArgs p) {
  extern __shared__ uint8_t raw[];
  __shared__ uint64_t q_full, k_full[SP_MAX_STAGES], k_empty[SP_MAX_STAGES], v_full[SP_MAX_STAGES],
      v_empty[SP_MAX_STAGES], s_full[SP_MAX_GROUPS], s_free[SP_MAX_GROUPS], p_full[SP_MAX_GROUPS],
      p_free[SP_MAX_GROUPS], o_full;
  __shared__ uint32_t tmem_slot;
  __shared__ volatile int abort_flag;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int role = warp - p.groups * 4;  // 0: K, 1: scores, 2: V, 3: P V
  const int h = blockIdx.y, g = h / (int)p.group;
  const uint32_t k_bytes = (uint32_t)p.k_panels * SP_K * 128u;
  const uint32_t v_bytes = (uint32_t)p.v_panels * SP_K * 128u;
  const uint32_t q_panel = SP_Q * 128u;
  uint8_t* Qs = raw + ((1024u - (smem_u32(raw) & 1023u)) & 1023u);
  uint8_t* Ks = Qs + (size_t)p.k_panels * q_panel;
  uint8_t* Vs = Ks + (size_t)p.stages * k_bytes;
  uint8_t* Ps = Vs + (size_t)p.stages * v_bytes;
  float* tab = reinterpret_cast<float*>(Ps + p.groups * SP_P_BYTES);  // [below + window + above]

  pdl_launch_dependents();
  if (tid == 0) {
    mbar_init(&q_full, 1);
    mbar_init(&o_full, 1);
    for (int i = 0; i < SP_MAX_STAGES; ++i) {
      mbar_init(&k_full[i], 1);
      mbar_init(&k_empty[i], 1);
      mbar_init(&v_full[i], 1);
      mbar_init(&v_empty[i], 1);
    }
    for (int i = 0; i < SP_MAX_GROUPS; ++i) {
      mbar_init(&s_full[i], 1);
      mbar_init(&s_free[i], 4);
      mbar_init(&p_full[i], 4);
      mbar_init(&p_free[i], 1);
    }
    mbar_fence_init();
    abort_flag = 0;
  }
  const float cap = p.a.softcap;
  const float L2E = 1.44269504088896340736f;
  for (int i = tid; i < p.tab_n; i += (int)blockDim.x) {
    const int d = i - SP_TAB_BELOW;
    tab[i] = d >= 0 && d < (int)p.a.window
                 ? -L2E * (cap + p.a.bias[(size_t)h * p.a.bias_len + d])
                 : INFINITY;
  }
  const AttnTile tile = p.tiles[blockIdx.x];
  const uint32_t q_end = tile.pos0 + tile.rows;  // exclusive
  const uint32_t lo = tile.pos0 + 1 > p.a.window ? tile.pos0 + 1 - p.a.window : 0;
  const uint32_t k_begin = lo / p.block_size * p.block_size;  // tiles start on a page
  const int n_tiles = (int)((q_end - k_begin + SP_K - 1) / SP_K);
  // TMEM only once the kernels in front have ended: they may hold or still want some of it
  pdl_wait();
  if (role == 1) tmem_alloc(&tmem_slot, p.tmem_cols);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_slot, o_tmem = tmem + (uint32_t)(p.groups * SP_K);

  if (role == 0 || role == 2) {
    // ---- copies ----
    const bool keys = role == 0;
    const int pages = SP_K / (int)p.block_size;  // at most eight
    const int panels = keys ? p.k_panels : p.v_panels;
    const uint32_t bytes = keys ? k_bytes : v_bytes;
    uint64_t *full = keys ? k_full : v_full, *empty = keys ? k_empty : v_empty;
    const uint32_t last_page = (q_end - 1) / p.block_size;
    const uint32_t* table = p.tables + (size_t)tile.seq * p.max_blocks;
    if (keys && lane == 0) {
      mbar_arrive_expect_tx(&q_full, (uint32_t)p.k_panels * q_panel);
      for (int c = 0; c < p.k_panels; ++c)
        tma_load_3d(Qs + (size_t)c * q_panel, &qmap, c * 64, h, (int)tile.row0, &q_full);
    }
    auto page_of = [&](int i) {
      // pages past the last token hold no visible key: the last one stands in for them
      const uint32_t pg =
          min(k_begin / p.block_size + (uint32_t)(i * pages + min(lane, pages - 1)), last_page);
      uint32_t b = table[pg];
      if (b >= p.num_blocks) {
        atomicOr(p.status, DEV_BAD_INDEX);
        b = 0;
      }
      return b;
    };
    uint32_t block = page_of(0);
    int issued = 0;
    for (int i = 0; i < n_tiles; ++i) {
      const int s = i % p.stages;
      const uint32_t next = i + 1 < n_tiles ? page_of(i + 1) : 0u;
      const bool ok =
          mbar_wait_abort(&empty[s], ((uint32_t)(i / p.stages) & 1u) ^ 1u, &abort_flag);
      if (!__all_sync(0xFFFFFFFFu, ok)) break;
      if (lane == 0) mbar_arrive_expect_tx(&full[s], bytes);
      __syncwarp();
      const int rec = (int)(block * p.kv_heads + (uint32_t)g);
      uint8_t* dst = (keys ? Ks : Vs) + (size_t)s * bytes + (size_t)lane * p.block_size * 128;
      if (lane < pages)
        for (int c = 0; c < panels; ++c)
          tma_load_3d(dst + (size_t)c * SP_K * 128, keys ? &kmap : &vmap, c * 64, 0, rec, &full[s]);
      issued = i + 1;
      block = next;
    }
    // leave only when every copy has landed (bounded)
    if (lane == 0) {
      if (keys) mbar_wait_bounded(&q_full, 0);
      for (int i = max(0, issued - p.stages); i < issued; ++i)
        mbar_wait_bounded(&full[i % p.stages], (uint32_t)(i / p.stages) & 1u);
    }
    __syncwarp();
  } else if (role == 1) {
    // ---- scores ----
    if (elect_one()) {
      const uint32_t idesc = tc_idesc_bf16(SP_Q, SP_K);
      const uint32_t queries = smem_u32(Qs), keys = smem_u32(Ks);
      bool ok = mbar_wait_abort(&q_full, 0, &abort_flag);
      int b = 0;
      uint32_t par = 0;
      for (int i = 0; i < n_tiles && ok; ++i) {
        const int s = i % p.stages;
        // the group has read the scores of its tile before
        ok = mbar_wait_abort(&s_free[b], par ^ 1u, &abort_flag);
        if (ok) ok = mbar_wait_abort(&k_full[s], (uint32_t)(i / p.stages) & 1u, &abort_flag);
        if (!ok) break;
        tc_fence_after();
        tc_mma_panels(tmem + (uint32_t)b * SP_K, queries, keys + (uint32_t)s * k_bytes, q_panel,
                      SP_K * 128u, p.k_steps, idesc, 0);
        tc_commit(&s_full[b]);
        tc_commit(&k_empty[s]);
        if (++b == p.groups) {
          b = 0;
          par ^= 1u;
        }
      }
      if (!ok) abort_flag = 1;
    }
    __syncwarp();
  } else if (role == 3) {
    // ---- weights x values ----
    if (elect_one()) {
      const uint32_t idesc = tc_idesc_bf16(SP_Q, p.nv) | (1u << 16);  // B is N-major
      const uint64_t weights = tc_smem_desc_sw128(smem_u32(Ps));
      const uint64_t values = tc_smem_desc_nmajor(smem_u32(Vs), SP_K * 128u);
      bool ok = true;
      int b = 0;
      uint32_t par = 0;
      for (int i = 0; i < n_tiles && ok; ++i) {
        const int s = i % p.stages;
        ok = mbar_wait_abort(&v_full[s], (uint32_t)(i / p.stages) & 1u, &abort_flag);
        if (ok) ok = mbar_wait_abort(&p_full[b], par, &abort_flag);
        if (!ok) break;
        tc_fence_after();
        const uint64_t ad = weights + (uint32_t)b * (SP_P_BYTES >> 4);
        const uint64_t bd = values + (uint32_t)s * (v_bytes >> 4);
        tc_mma_f16(o_tmem, ad, bd, idesc, i > 0);
#pragma unroll
        for (int k = 1; k < SP_K / 16; ++k) tc_mma_f16(o_tmem, ad + 2 * k, bd + 128 * k, idesc, 1);
        tc_commit(&p_free[b]);
        tc_commit(&v_empty[s]);
        if (++b == p.groups) {
          b = 0;
          par ^= 1u;
        }
      }
      if (ok)
        tc_commit(&o_full);
      else
        abort_flag = 1;
    }
    __syncwarp();
  } else {
    // ---- weights ----
    const int wg = warp >> 2, row = (warp & 3) * 32 + lane;
    const uint32_t s_lane = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)wg * SP_K;
    uint8_t* prow = Ps + (size_t)wg * SP_P_BYTES + (size_t)row * 128;
    const float k1 = cap != 0.f ? p.a.scale * 2.f * L2E / cap : 0.f;
    const float c1 = 2.f * cap * L2E, k0s = -L2E * p.a.scale;
    uint32_t par = 0;
    for (int i = wg; i < n_tiles; i += p.groups, par ^= 1u) {
      // a warp gives up as one: what follows is done by all its lanes together
      const bool got = mbar_wait_abort(&s_full[wg], par, &abort_flag) &&
                       mbar_wait_abort(&p_free[wg], par ^ 1u, &abort_flag);
      if (!__all_sync(0xFFFFFFFFu, got)) break;
      tc_fence_after();
      // tab index of the tile's first key; it falls by one per key
      const float* tb = tab + ((int)(tile.pos0 + row) - (int)(k_begin + (uint32_t)i * SP_K) +
                               SP_TAB_BELOW);
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        uint32_t r[32];
        tmem_ld32(s_lane + half * 32, r);
        if (half == 1) {
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&s_free[wg]);
        }
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          uint32_t w[4];
          float v[8], top = -INFINITY;
#pragma unroll
          for (int e = 0; e < 8; ++e) v[e] = __uint_as_float(r[c * 8 + e]);
          if (cap != 0.f) sp_capped(v, k1, c1, tb - (half * 32 + c * 8));
#pragma unroll
          for (int e = 0; e < 8; ++e) {
            if (cap == 0.f) v[e] = fmaf(v[e], k0s, tb[-(half * 32 + c * 8 + e)]);
            top = fmaxf(top, v[e]);
          }
          sp_weights(v, __any_sync(0xFFFFFFFFu, !(top <= SP_SHARED)));
#pragma unroll
          for (int e = 0; e < 4; ++e) w[e] = pack_bf16(v[2 * e], v[2 * e + 1]);
          const int chunk = (half * 4 + c) ^ (row & 7);  // the copy engine's 128-byte swizzle
          *reinterpret_cast<uint4*>(prow + chunk * 16) = make_uint4(w[0], w[1], w[2], w[3]);
        }
      }
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(&p_full[wg]);
    }
  }
  __syncthreads();
  int failed = abort_flag != 0;
  if (!failed) failed = !mbar_wait_bounded(&o_full, 0);
  failed = __syncthreads_or(failed);
  tc_fence_after();
  if (failed) {
    if (tid == 0) atomicOr(p.status, DEV_WAIT_TIMEOUT);
  } else if (role < 0) {
    const int row = (warp & 3) * 32 + lane;
    const uint32_t base = o_tmem + ((uint32_t)((warp & 3) * 32) << 16);
    const int64_t at = (int64_t)(tile.row0 + row) * p.out_ld + (int64_t)h * p.v_dim;
    for (int c = (warp >> 2) * 16; c < p.nv; c += p.groups * 16) {
      uint32_t r[16];
      tmem_ld16(base + c, r);
      if ((uint32_t)row < tile.rows) {
        if (p.out_f32) {
          float* o = static_cast<float*>(p.out) + at + c;
#pragma unroll
          for (int e = 0; e < 16; ++e)
            if (c + e < p.v_dim) o[e] = __uint_as_float(r[e]);
        } else {
          bf16* o = static_cast<bf16*>(p.out) + at + c;
          if (c + 16 <= p.v_dim && (reinterpret_cast<uintptr_t>(o) & 15u) == 0) {
            uint32_t w[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) {
              const __nv_bfloat162 pk = __floats2bfloat162_rn(__uint_as_float(r[2 * e]),
                                                              __uint_as_float(r[2 * e + 1]));
              w[e] = *reinterpret_cast<const uint32_t*>(&pk);
            }
            reinterpret_cast<uint4*>(o)[0] = make_uint4(w[0], w[1], w[2], w[3]);
            reinterpret_cast<uint4*>(o)[1] = make_uint4(w[4], w[5], w[6], w[7]);
          } else {
#pragma unroll
            for (int e = 0; e < 16; ++e)
              if (c + e < p.v_dim) o[e] = to_elem<bf16>(__uint_as_float(r[e]));
          }
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (role == 1) tmem_dealloc(tmem, p.tmem_cols);
}

int32_t launch_sigmoid_attn_prefill(kanso_cuda_ctx* ctx, const SigmoidAttn& a,
                                    const KvDenseLayer& kv, const void* q, int64_t q_rows,
                                    const RowMap& map, const AttnTile* tiles, uint32_t n_tiles,
                                    void* out, bool out_f32, int64_t out_ld, bool* handled) {
  *handled = false;
  TmEncodeFn encode = tm_encoder();
  const uint32_t bs = kv.block_size;
  if (!encode || kv.k_dim > 256 || kv.v_dim > 256 || a.heads > 65535 || !a.window ||
      a.window > std::min(a.bias_len, SP_MAX_WINDOW) || (bs != 8 && bs != 16 && bs != 32 && bs != 64))
    return KANSO_OK;
  PrefillArgs p;
  p.a = a;
  p.tables = map.tables;
  p.tiles = tiles;
  p.out = out;
  p.out_ld = out_ld;
  p.max_blocks = map.max_blocks;
  p.num_blocks = kv.num_blocks;
  p.block_size = bs;
  p.kv_heads = kv.kv_heads;
  p.group = a.heads / kv.kv_heads;
  p.out_f32 = out_f32;
  p.v_dim = (int)kv.v_dim;
  p.nv = (int)((kv.v_dim + 15u) & ~15u);
  p.k_panels = (int)((kv.k_dim + 63u) / 64u);
  p.v_panels = (int)((kv.v_dim + 63u) / 64u);
  p.k_steps = (int)((kv.k_dim + 15u) / 16u);
  p.tab_n = SP_TAB_BELOW + (int)a.window + SP_TAB_ABOVE;
  p.status = ctx->dev_status;
  // Three groups keep the unit for 2^x and 1 / x busier than two (85 us and 98 at 2048 rows, 16 heads of 128), which need one weight
  // buffer less.
  const size_t fixed = 1024 + (size_t)p.k_panels * SP_Q * 128 + (size_t)p.tab_n * 4;
  const size_t stage = (size_t)SP_K * 128 * (p.k_panels + p.v_panels), room = 225 * 1024;
  p.groups = fixed + 3 * (size_t)SP_P_BYTES + 2 * stage <= room ? 3 : 2;
  p.stages = SP_MAX_STAGES;
  while (p.stages > 2 && fixed + p.groups * (size_t)SP_P_BYTES + p.stages * stage > room) --p.stages;
  const size_t smem = fixed + p.groups * (size_t)SP_P_BYTES + p.stages * stage;
  p.tmem_cols = p.groups * SP_K + p.nv <= 256 ? 256 : 512;
  if (smem > room) return KANSO_OK;
  const uint64_t records = (uint64_t)kv.num_blocks * kv.kv_heads;
  CUtensorMap qm, km, vm;
  const bf16* pool = reinterpret_cast<const bf16*>(kv.base);
  if (!tm_map3(encode, q, kv.k_ld, a.heads, (uint64_t)q_rows, kv.k_ld, (uint64_t)a.heads * kv.k_ld, 1,
            SP_Q, &qm) ||
      !tm_map3(encode, pool, kv.k_ld, bs, records, kv.k_ld, kv.rec_elems, bs, 1, &km) ||
      !tm_map3(encode, pool + (size_t)bs * kv.k_ld, kv.v_ld, bs, records, kv.v_ld, kv.rec_elems, bs, 1,
            &vm))
    return KANSO_OK;
  int32_t st = allow_max_smem(ctx, (const void*)sigmoid_prefill_kernel);
  if (st) return st;
  *handled = true;
  const cudaError_t e = launch_dependent(ctx, sigmoid_prefill_kernel, dim3(n_tiles, a.heads),
                                         dim3((unsigned)(p.groups + 1) * 128u), smem, qm, km, vm, p);
  if (e != cudaSuccess) return cuda_fail(ctx, e, "sigmoid prefill launch");
  return after_launch(ctx, "sigmoid_prefill");
}

}  // namespace kanso
