// Tile products of unquantised weights, large ones: bfloat16, pairs of CTAs on one tile.
//
// A pair (a cluster of two, cta_group::2) computes 256 weight rows x up to 256 activation rows: each CTA
// holds 128 of the weight rows and half of the activation rows, and the tensor cores of both read both
// halves. That is 8 KB of operands per CTA and 16 columns for 128 cycles of products, where two CTAs by
// themselves (gemm_dense.cu, 256 x 128) fetch 12 KB: those were bound by what the L2 hands to an SM.
// For the experts' silu(gate) * up each CTA's 128 rows are 64 of the gate and the same 64 of the up matrix,
// in lanes that lie 64 apart: the warps that store them exchange halves through shared memory. (Two
// accumulators of 128 rows in each CTA fill TMEM, so that every tile waits for the stores of the one
// before: 104 us where this form takes 74.)
//
// One pair of CTAs per two SMs stays for the whole product and takes tiles in turn. One thread copies
// (tensor maps, 128-byte swizzle, K-major), one thread of the even CTA issues the products of both, and
// eight warps store the results of a tile while the next one is multiplied into the other half of TMEM.
// us (of the form before): 2048 x 2048 x 2048 19 (21), 2048 x 3072 x 2048 25 (37), 8192 x 2048 x 1024 34
// (73), 4096 x 4736 x 2048 65 (124), 8192 x 8192 x 8192 794 (1070; 1386 TFLOP/s).
//
// The activation rows of a tile are a multiple of 32, at most 256, the same for all tiles of a group: the
// group's rows in equal parts, so that no tile is mostly padding, as many as the waves of tiles make best
// use of (gp_cost). Where the group sizes are on the device (routed experts) a pair finds its tiles from the
// offsets. A tile that runs past its group's end computes
// rows of the next group and does not store them.
#include <algorithm>

#include "gemm_dense.cuh"
#include "tc05.cuh"

namespace kanso {
namespace {

constexpr int GP_THREADS = 384;  // copies, products, TMEM, idle, eight warps of results
constexpr int GP_ROWS = 256;     // weight rows of a pair's tile
constexpr int GP_MAX_N = 256;    // activation rows of a tile
constexpr int GP_HALF = 128 * 128;  // bytes of 128 rows x 64 columns
constexpr int GP_BOX = 32;       // activation rows per copy where the tile's rows are not known here
constexpr int GP_STAGE = 2 * GP_HALF;
constexpr int GP_STAGES = 6;
constexpr int GP_ACCS = 2;  // tiles whose results TMEM holds
constexpr uint32_t GP_POLLS = 1u << 18;  // about a second: a poll that finds nothing lasts 4 us
constexpr uint32_t GP_LAND_POLLS = 1u << 12;  // about 16 ms, for what is on its way when a CTA gives up
constexpr size_t GP_SMEM = (size_t)GP_STAGE * GP_STAGES + 1024;

// What `tiles` of n activation rows cost `pairs` pairs, in cycles per 16 columns: a wave takes the products'
// n / 2 or the 4 KB + 16 n bytes of each CTA at the 55 a cycle that the L2 gave here, and its ends.
__host__ __device__ __forceinline__ int gp_cost(int64_t tiles, int n, int pairs) {
  const int bytes = (4096 + 16 * n) / 55;
  return (int)((tiles + pairs - 1) / pairs) * ((bytes > n / 2 ? bytes : n / 2) + 16);
}

struct GpTiles {
  int col_tiles;   // of 256 weight rows (128 of the gate and of the up matrix)
  int row_tiles;   // of a group, where all are alike
  int n;           // activation rows of a tile, likewise
  int box;         // activation rows per copy
  int most;        // tiles there can be at the most, whatever the offsets say
};

struct GpTile {
  int group, col, n;  // n: a multiple of 32
  int64_t first;
  int valid;
};

// The most activation rows of a tile where the groups' sizes are on the device, by a whole warp.
__device__ __forceinline__ int gp_max_n(const GemmDenseArgs& a, const GpTiles& t, int lane, int pairs) {
  if (!a.offsets) return t.n;
  int best = 0, best_n = GP_MAX_N;
  for (int n = GP_MAX_N; n >= 128; n -= 2 * GP_BOX) {
    int tiles = 0;
    for (int g = lane; g < a.groups; g += 32) tiles += (int)(a.offsets[g + 1] - a.offsets[g] + n - 1) / n;
    tiles = __reduce_add_sync(0xFFFFFFFFu, tiles);
    const int cost = gp_cost((int64_t)tiles * t.col_tiles, n, pairs);
    if (n == GP_MAX_N || cost < best) {
      best = cost;
      best_n = n;
    }
  }
  return best_n;
}

// Tile `tile`, by a whole warp; the same answer in both CTAs. false: past the last one.
__device__ __forceinline__ bool gp_tile(const GemmDenseArgs& a, const GpTiles& t, int max_n, int tile,
                                        int lane, GpTile* out) {
  if (tile >= t.most) return false;
  const int row_tile = tile / t.col_tiles;
  out->col = tile - row_tile * t.col_tiles;
  if (!a.offsets) {
    const int g = row_tile / t.row_tiles;
    const int64_t per = (uint32_t)a.T / (uint32_t)a.groups;
    const int64_t at = (int64_t)(row_tile - g * t.row_tiles) * t.n;
    out->group = g;
    out->n = t.n;
    out->first = g * per + at;
    out->valid = (int)min((int64_t)t.n, per - at);
    return g < a.groups;
  }
  int before = 0;
  for (int g0 = 0; g0 < a.groups; g0 += 32) {
    const int g = g0 + lane;
    const uint32_t b = g < a.groups ? a.offsets[g] : 0u, e = g < a.groups ? a.offsets[g + 1] : 0u;
    const int rows = (int)(e - b), tiles = (rows + max_n - 1) / max_n;
    int incl = tiles;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xFFFFFFFFu, incl, o);
      if (lane >= o) incl += v;
    }
    const unsigned hit = __ballot_sync(0xFFFFFFFFu, before + incl > row_tile);
    if (hit) {
      const int l = __ffs(hit) - 1;
      const int in = row_tile - before - __shfl_sync(0xFFFFFFFFu, incl - tiles, l);
      const int gr = __shfl_sync(0xFFFFFFFFu, rows, l), gt = __shfl_sync(0xFFFFFFFFu, tiles, l);
      // equal parts in whole copies of both CTAs
      const int n = ((gr + gt - 1) / gt + 2 * GP_BOX - 1) / (2 * GP_BOX) * (2 * GP_BOX);
      out->group = g0 + l;
      out->n = n;
      out->first = (int64_t)__shfl_sync(0xFFFFFFFFu, b, l) + (int64_t)in * n;
      out->valid = min(n, gr - in * n);
      return true;
    }
    before += __shfl_sync(0xFFFFFFFFu, incl, 31);
  }
  return false;
}

// ---- what differs for a pair of CTAs ----
__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release;\nbarrier.cluster.wait.acquire;" ::: "memory");
}
// The even CTA's copy of a barrier at the same place of its shared memory.
__device__ __forceinline__ uint32_t even_bar(const uint64_t* bar) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(r) : "r"(smem_u32(bar)));
  return r;
}
__device__ __forceinline__ void mbar_arrive_at(uint32_t bar) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
// Waits are for arrivals of the other CTA too.
__device__ __forceinline__ bool mbar_wait_pair(uint64_t* bar, uint32_t parity,
                                               volatile int* abort_flag) {
  for (uint32_t i = 0; i < GP_POLLS; ++i) {
    uint32_t ok;
    asm volatile(
        "{\n.reg .pred p;\nmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n"
        "selp.b32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    if (ok) return true;
    if ((i & 63u) == 63u && *abort_flag) break;
  }
  *abort_flag = 1;
  return false;
}
// Until what a CTA that gives up has still on its way has landed or retired. A stage that the other CTA never
// asked for does not complete: there the limit ends the wait, long after this CTA's own copies.
__device__ __forceinline__ void mbar_wait_land(uint64_t* bar, uint32_t parity) {
  mbar_wait_bounded(bar, parity, GP_LAND_POLLS);
}
// A word of the other CTA's shared memory, at the same place.
__device__ __forceinline__ void store_other(volatile int* p, uint32_t rank, int v) {
  asm volatile(
      "{\n.reg .b32 a;\nmapa.shared::cluster.u32 a, %0, %1;\nst.shared::cluster.u32 [a], %2;\n}\n" ::"r"(
          smem_u32(const_cast<int*>(p))),
      "r"(rank ^ 1u), "r"(v)
      : "memory");
}
// Copies into this CTA's shared memory whose bytes count on the even CTA's barrier.
__device__ __forceinline__ void pair_load_3d(void* dst, const CUtensorMap* map, int x, int y, int z,
                                             uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], "
      "[%1, {%2, %3, %4}], [%5];" ::"r"(smem_u32(dst)),
      "l"(map), "r"(x), "r"(y), "r"(z), "r"(bar)
      : "memory");
}
__device__ __forceinline__ void pair_load_2d(void* dst, const CUtensorMap* map, int x, int y,
                                             uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], "
      "[%1, {%2, %3}], [%4];" ::"r"(smem_u32(dst)),
      "l"(map), "r"(x), "r"(y), "r"(bar)
      : "memory");
}
__device__ __forceinline__ void pair_mma(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc,
                                         uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(d_tmem),
      "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// Arrives at the barrier in both CTAs when the products issued so far have retired.
__device__ __forceinline__ void pair_commit(uint64_t* bar) {
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], "
      "%1;" ::"r"(smem_u32(bar)),
      "h"((uint16_t)3)
      : "memory");
}

// A barrier of two warps: does either say so?
__device__ __forceinline__ bool partners_any(int bar, bool mine) {
  uint32_t any;
  asm volatile(
      "{\n.reg .pred p, q;\nsetp.ne.u32 p, %1, 0;\nbarrier.cta.red.or.pred q, %2, 64, p;\n"
      "selp.b32 %0, 1, 0, q;\n}\n"
      : "=r"(any)
      : "r"((uint32_t)mine), "r"(bar)
      : "memory");
  return any != 0;
}

// A chunk of 16 activation rows of weight row n: bias, activation, element type, place.
template <typename O>
__device__ __forceinline__ void gp_store_ext(const GemmDenseArgs& a, const RowPlace& place, O* out,
                                             const uint32_t (&r)[16], int n, int64_t row0, int valid) {
  const float bias = a.bias_of(n);
  if (n >= a.n_end) return;
#pragma unroll
  for (int j = 0; j < 16; ++j) {
    if (j >= valid) continue;
    const float x = __uint_as_float(r[j]) + bias;
    out[place.at(row0 + j, a.out_ld) + n] = to_elem<O>(a.relu2 ? relu_squared(x) : x);
  }
}

template <bool GATE_UP, bool EXT>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(GP_THREADS, 1)
    gemm_pair_kernel(const __grid_constant__ CUtensorMap wmap,
                     const __grid_constant__ CUtensorMap wmap2,
                     const __grid_constant__ CUtensorMap xmap, const GemmDenseArgs a,
                     const GpTiles tiles) {
  extern __shared__ uint8_t raw[];
  // full, acc_empty: the even CTA's are the ones that count
  __shared__ uint64_t full[GP_STAGES], empty[GP_STAGES], acc_full[GP_ACCS], acc_empty[GP_ACCS];
  __shared__ float swap[GATE_UP ? 8 : 1][2][8][32];  // what a warp hands to its partner, two chunks
  __shared__ uint32_t tmem_slot;
  __shared__ volatile int abort_flag, other_issued;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_rank();
  const int first_tile = (int)(blockIdx.x >> 1), step = (int)(gridDim.x >> 1);
  uint8_t* ring = raw + ((1024u - (smem_u32(raw) & 1023u)) & 1023u);

  if (threadIdx.x == 0) {
    for (int i = 0; i < GP_STAGES; ++i) {
      mbar_init(&full[i], 1);
      mbar_init(&empty[i], 1);
    }
    for (int i = 0; i < GP_ACCS; ++i) {
      mbar_init(&acc_full[i], 1);
      mbar_init(&acc_empty[i], 16);  // the result warps of both CTAs
    }
    mbar_fence_init();
    abort_flag = other_issued = 0;
  }
  cluster_sync();
  pdl_launch_dependents();
  pdl_wait();
  // TMEM only once the kernels in front have ended: a CTA that waits for it waits without a limit
  if (warp == 2) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(
                     smem_u32(&tmem_slot))
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  cluster_sync();
  tc_fence_after();
  const uint32_t tmem = tmem_slot;
  const int max_n = gp_max_n(a, tiles, lane, step);
  int issued = 0;  // warp 0: the stages that it has asked for

  if (warp == 0) {
    // ---- copies: this CTA's weight rows and its half of the activation rows ----
    bool ok = true;
    GpTile t;
    for (int tile = first_tile; ok && gp_tile(a, tiles, max_n, tile, lane, &t); tile += step) {
      if (elect_one()) {
        const int n0 = (t.col * 2 + (int)rank) * (GATE_UP ? 64 : 128);
        const int half = t.n / 2, row0 = (int)t.first + (int)rank * half;
        const uint32_t bytes = 2u * (uint32_t)(GP_HALF + half * 128);
        for (int k = 0; k < a.k_steps; ++k, ++issued) {
          const int s = issued % GP_STAGES;
          if (!mbar_wait_pair(&empty[s], ((uint32_t)(issued / GP_STAGES) & 1u) ^ 1u, &abort_flag)) {
            ok = false;
            break;
          }
          uint8_t* st = ring + s * GP_STAGE;
          const uint32_t bar = even_bar(&full[s]);
          if (rank == 0) mbar_arrive_expect_tx(&full[s], bytes);
          pair_load_3d(st, &wmap, k * GD_K, n0, t.group, bar);
          if (GATE_UP) pair_load_3d(st + GP_HALF / 2, &wmap2, k * GD_K, n0, t.group, bar);
          uint8_t* xs = st + GP_HALF;
          for (int r = 0; r < half; r += tiles.box)
            pair_load_2d(xs + r * 128, &xmap, k * GD_K, row0 + r, bar);
        }
      }
      ok = __all_sync(0xFFFFFFFFu, ok);
      issued = __reduce_max_sync(0xFFFFFFFFu, issued);
    }
    // The products have read every stage, and their arrivals, some from the other CTA, have come, before
    // this CTA ends (bounded).
    if (ok)
      for (int i = max(0, issued - GP_STAGES); i < issued; ++i)
        mbar_wait_pair(&empty[i % GP_STAGES], (uint32_t)(i / GP_STAGES) & 1u, &abort_flag);
  } else if (warp == 1 && rank == 0) {
    // ---- products of both CTAs ----
    uint32_t at = 0;
    int count = 0;
    bool ok = true;
    GpTile t;
    for (int tile = first_tile; ok && gp_tile(a, tiles, max_n, tile, lane, &t); tile += step, ++count) {
      const int b = count % GP_ACCS;
      if (elect_one()) {
        const uint32_t idesc = tc_idesc_bf16(GP_ROWS, t.n);
        const uint32_t acc = tmem + (uint32_t)b * 256u;
        ok = mbar_wait_pair(&acc_empty[b], ((uint32_t)(count / GP_ACCS) & 1u) ^ 1u, &abort_flag);
        tc_fence_after();
        for (int k = 0; k < a.k_steps && ok; ++k, ++at) {
          const uint32_t s = at % GP_STAGES;
          if (!mbar_wait_pair(&full[s], (at / GP_STAGES) & 1u, &abort_flag)) {
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t base = smem_u32(ring + s * GP_STAGE);
          const uint64_t ad = tc_smem_desc_sw128(base);
          const uint64_t bd = tc_smem_desc_sw128(base + GP_HALF);
#pragma unroll
          for (int j = 0; j < GD_K / 16; ++j)
            pair_mma(acc, ad + 2 * j, bd + 2 * j, idesc, (k > 0 || j > 0) ? 1u : 0u);
          pair_commit(&empty[s]);
        }
        if (ok)
          pair_commit(&acc_full[b]);
        else if (at)  // the products issued so far still read shared memory
          mbar_wait_land(&empty[(at - 1) % GP_STAGES], ((at - 1) / GP_STAGES) & 1u);
      }
      ok = __all_sync(0xFFFFFFFFu, ok);
      at = __reduce_max_sync(0xFFFFFFFFu, at);
    }
  } else if (warp >= 4) {
    // ---- results: a warp reaches its own quarter of the TMEM lanes; two share the columns ----
    const int quarter = warp & 3, half = (warp - 4) >> 2;
    const int bar = 1 + half * 2 + (quarter & 1);  // of this warp and the one two quarters on
    int count = 0;
    GpTile t;
    for (int tile = first_tile; gp_tile(a, tiles, max_n, tile, lane, &t); tile += step, ++count) {
      const int b = count % GP_ACCS;
      const bool got = mbar_wait_pair(&acc_full[b], (uint32_t)(count / GP_ACCS) & 1u, &abort_flag);
      if (GATE_UP ? partners_any(bar, !got) : !__all_sync(0xFFFFFFFFu, got)) break;
      tc_fence_after();
      const int n = GATE_UP ? (t.col * 2 + (int)rank) * 64 + (quarter & 1) * 32 + lane
                            : (t.col * 2 + (int)rank) * 128 + quarter * 32 + lane;
      const uint32_t acc = tmem + (uint32_t)b * 256u + ((uint32_t)(quarter * 32) << 16);
      const RowPlace place(a, t.group);
      for (int c = half * 16; c < t.n && c < t.valid; c += 32) {
        uint32_t r0[16];
        tmem_ld16(acc + c, r0);
        const int64_t row0 = t.first + c;
        const int valid = t.valid - c;
        if (EXT) {
          if (a.elem)
            gp_store_ext(a, place, static_cast<bf16*>(a.out), r0, n, row0, valid);
          else
            gp_store_ext(a, place, static_cast<float*>(a.out), r0, n, row0, valid);
        } else if (GATE_UP) {
          // The gate's warp takes the first eight rows of the chunk, the up matrix's the others. Two chunks
          // in turn: the barrier of a chunk is behind the reads of the chunk before the last.
          const int which = quarter >> 1, two = (c >> 5) & 1;  // 0: gate
          float(*mine)[32] = swap[warp - 4][two], (*theirs)[32] = swap[(warp - 4) ^ 2][two];
#pragma unroll
          for (int j = 0; j < 8; ++j)
            mine[j][lane] = __uint_as_float(which ? r0[j] : r0[j + 8]);
          partners_any(bar, false);
          // the pad columns multiply weight rows that were zero-filled: they come out as zero
          bf16* o = static_cast<bf16*>(a.out) + (row0 + 8 * which) * a.out_ld + n;
          if (n < a.out_ld)
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              const float own = __uint_as_float(which ? r0[j + 8] : r0[j]), other = theirs[j][lane];
              if (8 * which + j < valid)
                o[j * a.out_ld] = to_elem<bf16>(silu(which ? other : own) * (which ? own : other));
            }
        } else if (n < a.rows) {
          float* o = static_cast<float*>(a.out) + row0 * a.out_ld + n;
#pragma unroll
          for (int j = 0; j < 16; ++j)
            if (j < valid) o[j * a.out_ld] = __uint_as_float(r0[j]);
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_at(even_bar(&acc_empty[b]));
    }
  }
  __syncthreads();
  if (abort_flag && threadIdx.x == 0) {
    atomicOr(a.status, DEV_WAIT_TIMEOUT);
    store_other(&other_issued, rank, issued);
    store_other(&abort_flag, rank, 1);
  }
  tc_fence_before();
  cluster_sync();
  if (abort_flag) {  // in both CTAs: one of them has given up
    // Copies of both that are still on their way land before either ends (bounded); they count on the
    // even CTA's barriers.
    if (warp == 0 && rank == 0) {
      const int last = max(issued, other_issued);
      for (int i = max(0, last - GP_STAGES); i < last; ++i)
        mbar_wait_land(&full[i % GP_STAGES], (uint32_t)(i / GP_STAGES) & 1u);
    }
    cluster_sync();
  }
  if (warp == 2)
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
}

template <bool GATE_UP, bool EXT>
int32_t gp_launch(kanso_cuda_ctx* ctx, int pairs, const CUtensorMap& wm, const CUtensorMap& wm2,
                  const CUtensorMap& xm, const GemmDenseArgs& a, const GpTiles& t) {
  auto kern = gemm_pair_kernel<GATE_UP, EXT>;
  const int32_t st = allow_max_smem(ctx, (const void*)kern);
  if (st) return st;
  const cudaError_t e = launch_dependent(ctx, kern, dim3((unsigned)(2 * pairs)), dim3(GP_THREADS),
                                         GP_SMEM, wm, wm2, xm, a, t);
  if (e != cudaSuccess) return cuda_fail(ctx, e, "gemm_pair launch");
  return after_launch(ctx, "gemm_pair");
}

}  // namespace

int32_t launch_gemm_pair(kanso_cuda_ctx* ctx, const DenseMat& w, const DenseMat* up, const void* x,
                         const GemmRows& r, GemmDenseArgs a, bool ext, bool* handled) {
  *handled = false;
  const int pairs = ctx->sm_count / 2;
  GpTiles t;
  const int tile_rows = up ? GP_ROWS / 2 : GP_ROWS;
  t.col_tiles = (int)((w.rows + tile_rows - 1) / tile_rows);
  const int64_t per = r.T / r.groups;
  t.row_tiles = 1;
  t.n = 0;
  t.box = GP_BOX;
  int64_t total, most;
  if (r.offsets) {
    if (per < 96) return KANSO_OK;
    total = t.col_tiles * ((r.T + GP_MAX_N - 1) / GP_MAX_N);
    most = t.col_tiles * (r.T / 128 + r.groups);  // gp_max_n: 128 and more
  } else {
    // equal parts of a group's rows: the number of them with which the last wave is fullest
    const int64_t cols = (int64_t)t.col_tiles * r.groups;
    int64_t best = 0;
    for (int64_t parts = (per + GP_MAX_N - 1) / GP_MAX_N; parts * 96 <= per; ++parts) {
      const int64_t n = ((per + parts - 1) / parts + 31) / 32 * 32;
      const int64_t cost = gp_cost(cols * parts, (int)n, pairs);
      if (!best || cost < best) {
        best = cost;
        t.row_tiles = (int)parts;
        t.n = (int)n;
      }
    }
    if (!best) return KANSO_OK;
    t.row_tiles = (int)((per + t.n - 1) / t.n);  // parts rounded to 32 may be fewer
    t.box = t.n / 2;
    most = total = cols * t.row_tiles;
  }
  if (most > (1 << 30)) return KANSO_OK;
  t.most = (int)most;
  // Where the lines lie (us of one product, gemm_dense.cu's form / this one). Rows: below 96 a tile is mostly its
  // 4 KB of weights per 16 columns, and 32768 x 2048 takes 30.5 / 33.0 at 64 rows, 34.8 / 35.8 at 90, 37.4 / 37.5 at
  // 128, 60 / 38 at 144; smaller matrices are ahead from 72 rows on. Pairs: with fewer than three quarters of them busy
  // the other form is the one that can share out the columns too (3072 x 2048 at eight rows 6 in four parts, 11 in
  // one); in one part pairs are ahead well below that (1024 x 2048 at 256 rows, 4 tiles, 15.9 / 13.2), which
  // makes this a cautious line.
  if (total * 4 < pairs * 3) return KANSO_OK;
  // Where all of the other form's tiles lie on the GPU at once, two to an SM, they are ahead if pairs need a second
  // round (6152 x 2048 at 640 rows 21.7 / 23.9, at 800, which are two rounds either way, 32.6 / 24.8) or have one
  // tile of the largest size and few columns, where it is stored with nothing behind it to multiply (4096 x 512 at 1024
  // rows 11.5 / 12.5, 8192 x 1024 at 512 14.9 / 15.3, 2048 x 2048 at 2048 21.1 / 19.9).
  if (!r.offsets && (w.rows + 127) / 128 * r.groups * ((per + 127) / 128) <= 2 * (int64_t)ctx->sm_count &&
      (total > pairs || (t.n == GP_MAX_N && w.cols <= 1024)))
    return KANSO_OK;
  CUtensorMap wm, um, xm;
  int32_t st = weight_map(ctx, w, &wm, up ? 64 : 128);
  if (!st && up) st = weight_map(ctx, *up, &um, 64);
  if (!st) st = rows_map(ctx, x, r.T, w.cols, w.ld, t.box, &xm);
  if (st) return st;
  *handled = true;
  a.k_steps = a.steps_per_split = (int)((w.cols + GD_K - 1) / GD_K);
  // where the rows' shares are on the device there may be more tiles than `total`
  const int grid = r.offsets ? pairs : (int)std::min<int64_t>(pairs, total);
  if (up) return gp_launch<true, false>(ctx, grid, wm, um, xm, a, t);
  return ext ? gp_launch<false, true>(ctx, grid, wm, wm, xm, a, t)
             : gp_launch<false, false>(ctx, grid, wm, wm, xm, a, t);
}

}  // namespace kanso
