// Decode attention over the quantised pool: the arguments of its kernels (paged_attention.cu: any head
// and block size; paged_decode.cu: tiles of 16 tokens on mma.sync) and what they share.
#pragma once
#include "glue.cuh"
#include "kv_pool.h"
#include "warp_mma.cuh"

namespace kanso {

constexpr int PA_THREADS = 128;
constexpr int PA_BIG_THREADS = 256;  // partitions of 256 tokens and more
__host__ inline uint32_t pa_threads(uint32_t pt) { return pt >= 256 ? PA_BIG_THREADS : PA_THREADS; }
constexpr int PA_MAX_GROUP = 8;      // MAX_KV_GROUP_SIZE, src/metal/paged_attention.rs:10
constexpr int PA_MAX_HEAD_DIM = 256; // MAX_HEAD_DIM, src/metal/paged_attention.rs:8

struct PaArgs {
  KvGeom g;
  uint32_t layer;
  const float* q;
  const uint32_t* tables;
  const uint32_t* lens;
  float* out;
  float* part_acc;  // [seq][head][part][hd]
  float* part_ml;   // [seq][head][part][2]
  uint32_t num_heads, max_blocks, part_tokens, num_parts;
  float scale;
  int* status;
  uint32_t* tickets;  // [seq][kv head], zero between calls; nullptr = separate stage-2 launch
  // Chunked prefill: grid row `seq` is one query token; row_seq[seq] names the sequence whose
  // block table it walks (nullptr: the row is the sequence, as in decode).
  const uint32_t* row_seq;
  // Decode-step fusion (src/model.rs:1141-1207), off when k_new is nullptr: q arrives
  // un-rotated and is rotated as it is staged; the CTA whose partition holds the newest token
  // (position context_len - 1) rotates that token's K, quantises K and V and stores them in
  // the pool slot slots[seq] before it reads the partition.
  const float* k_new;  // [seq][kv head][hd]
  const float* v_new;
  const uint32_t* positions;
  const uint32_t* slots;
  const float* cos_t;  // [table_len][hd / 2]
  const float* sin_t;
  int table_len;
  // Batched decode: the output is ALSO written as the f16 hi/lo activation tile that the
  // o-projection's tensor-core GEMM reads (stage of 64 k-values, plane, k-chunk of 8, row:
  // the layout of tc_pack_activations_kernel), which saves that GEMM its pack launch. xp_mt =
  // rows of the tile (the batch rounded up to 16; the rows past the batch are zeroed here).
  __half* xp;  // nullptr: off
  uint32_t xp_mt;
};

// One output element into the packed tile: row = sequence, kk = head * head_dim + d.
__device__ __forceinline__ void pa_store_packed(const PaArgs& a, uint32_t row, uint32_t kk,
                                                float v) {
  const __half hi = __float2half_rn(v);
  const __half lo = __float2half_rn(v - __half2float(hi));
  const uint32_t c = (kk >> 3) & 7u, e = kk & 7u;
  __half* base = a.xp + (size_t)(kk >> 6) * (128u * a.xp_mt);
  base[((size_t)c * a.xp_mt + row) * 8 + e] = hi;
  base[((size_t)(8 + c) * a.xp_mt + row) * 8 + e] = lo;
}
// The tile's rows past the batch, for the k range of one KV head's query heads.
__device__ __forceinline__ void pa_zero_packed_rows(const PaArgs& a, uint32_t rows, uint32_t k0,
                                                    uint32_t nk, uint32_t tid, uint32_t nt) {
  const uint32_t pad = a.xp_mt - rows;
  for (uint32_t i = tid; i < pad * nk; i += nt)
    pa_store_packed(a, rows + i / nk, k0 + i % nk, 0.f);
}

// The context length a launch can serve: the table's capacity (max_blocks * block_size; the
// reference rejects a longer context on the host, src/metal/paged_attention.rs:343-355) and the
// window of partitions this grid was sized for. A device length beyond either is cut off there
// (the reference's kernel clamps its partition range the same way,
// src/metal/kernels/paged_attention_v2.metal:86-87) and reported through the status word, so no
// table entry, partial or scratch cell outside the launch's own range is ever addressed.
__device__ __forceinline__ uint32_t pa_clamp_ctx(const PaArgs& a, uint32_t ctx, bool report) {
  const uint64_t cap = (uint64_t)a.max_blocks * a.g.block_size;
  const uint64_t window = (uint64_t)a.num_parts * a.part_tokens;
  const uint64_t lim = cap < window ? cap : window;
  if ((uint64_t)ctx > lim) {
    if (report) atomicOr(a.status, DEV_BAD_INDEX);
    ctx = (uint32_t)lim;
  }
  return ctx;
}

// What a CTA does with its partition's sums: red[nslice][G][hd] in shared memory, complete; maxima pmax
// and denominators psum of the G heads in every thread. LOG2: maxima in units of log2.
template <int G, int NT, bool LOG2>
__device__ __forceinline__ void pa_publish(const PaArgs& a, uint32_t seq, uint32_t kvh,
                                           uint32_t part, uint32_t ctx, uint32_t hd,
                                           const float* red, uint32_t nslice,
                                           const float (&pmax)[G], const float (&psum)[G]) {
  const int tid = threadIdx.x;
  // partitions that exist in this grid (a context longer than the host said is cut off there)
  const uint32_t np = min((ctx + a.part_tokens - 1) / a.part_tokens, a.num_parts);
  const bool single = a.tickets && np == 1;  // the only partition: normalise and finish here
  for (uint32_t e = tid; e < G * hd; e += NT) {
    float s = 0.f;
    for (uint32_t sl = 0; sl < nslice; ++sl) s += red[sl * G * hd + e];
    const uint32_t gq = e / hd, d = e % hd;
    const size_t head = (size_t)seq * a.num_heads + (size_t)kvh * G + gq;
    if (single) {
      float l = 0.f;
#pragma unroll
      for (int k = 0; k < G; ++k)
        if (k == (int)gq) l = psum[k];
      const float o = l > 0.f ? s / l : 0.f;
      a.out[head * hd + d] = o;
      if (a.xp) pa_store_packed(a, seq, (kvh * G + gq) * hd + d, o);
    } else {
      a.part_acc[(head * a.num_parts + part) * hd + d] = s;
    }
  }
  if (single) return;
  if (tid < G) {
    const size_t head = (size_t)seq * a.num_heads + (size_t)kvh * G + tid;
    float m = 0.f, l = 0.f;
#pragma unroll
    for (int gq = 0; gq < G; ++gq)
      if (gq == tid) {
        m = pmax[gq];
        l = psum[gq];
      }
    a.part_ml[(head * a.num_parts + part) * 2 + 0] = m;
    a.part_ml[(head * a.num_parts + part) * 2 + 1] = l;
  }
  if (!a.tickets) return;  // a separate stage-2 launch merges

  // --- merge, by the CTA that draws the last ticket of this (sequence, kv head)
  __shared__ uint32_t s_last;
  // This CTA's partials must be visible device-wide before its ticket is drawn. One fence by
  // the thread that draws it is enough: the block barrier orders every thread's stores before
  // that thread, and its fence is cumulative over what it has observed (256 fences per CTA
  // showed up as 0.47 membar stall cycles per issued instruction).
  __syncthreads();
  if (tid == 0) {
    __threadfence();
    uint32_t* ticket = a.tickets + (size_t)seq * a.g.kv_heads + kvh;
    const uint32_t drawn = atomicAdd(ticket, 1u);
    s_last = drawn == np - 1;
    if (s_last) *ticket = 0;  // every CTA of the group has drawn: ready for the next call
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  // Each thread merges its output elements on its own: the (max, sum) pairs and the
  // accumulators of up to 16 partitions are requested together (one trip to L2), then folded
  // in with the running-maximum form of the softmax merge.
  for (uint32_t e = tid; e < G * hd; e += NT) {
    const uint32_t gq = e / hd, d = e % hd;
    const size_t head = (size_t)seq * a.num_heads + (size_t)kvh * G + gq;
    const float* ml = a.part_ml + head * a.num_parts * 2;
    const float* pa = a.part_acc + head * a.num_parts * hd + d;
    float M = -INFINITY, s = 0.f, l = 0.f;
    for (uint32_t p0 = 0; p0 < np; p0 += 16) {
      float2 mlv[16];
      float av[16];
#pragma unroll
      for (int k = 0; k < 16; ++k) {
        const uint32_t pp = min(p0 + k, np - 1);
        mlv[k] = __ldcg(reinterpret_cast<const float2*>(ml) + pp);
        av[k] = __ldcg(pa + (size_t)pp * hd);
      }
#pragma unroll
      for (int k = 0; k < 16; ++k) {
        if (p0 + k < np) {
          const float Mn = fmaxf(M, mlv[k].x);
          const float so = LOG2 ? ex2_approx(M - Mn) : expf(M - Mn);
          const float sn = LOG2 ? ex2_approx(mlv[k].x - Mn) : expf(mlv[k].x - Mn);
          s = s * so + av[k] * sn;
          l = l * so + mlv[k].y * sn;
          M = Mn;
        }
      }
    }
    const float o = l > 0.f ? s / l : 0.f;
    a.out[head * hd + d] = o;
    if (a.xp) pa_store_packed(a, seq, (kvh * G + gq) * hd + d, o);
  }
}

// paged_decode.cu. Tokens per partition of a call that it takes, 0: it does not take the call.
uint32_t pa_mma_partition_tokens(const kanso_cuda_ctx* ctx, const kanso_paged_attention_params* p,
                                 const KvGeom& g, uint64_t cap);
int32_t launch_paged_decode(kanso_cuda_ctx* ctx, const PaArgs& a, uint32_t group, dim3 grid);

}  // namespace kanso
