// Element-wise pieces of the decode step: RMSNorm, rotate-half RoPE, SiLU*up,
// residual add, greedy argmax (src/model.rs:653-737,367-382; src/sampler.rs:7-17).
#include <cmath>

#include "ctx.h"
#include "glue.cuh"
#include "kv_pool.h"

namespace kanso {

// x / sqrt(mean(x^2) + eps) * w, one CTA per row (src/model.rs:653-659).
// VEC: rows of whole float4. KEEP: float4 of a row that a thread keeps between the passes, for rows of at most
// KEEP * 1024 columns (0: wider ones are read twice).
template <bool VEC, int KEEP>
__global__ void rmsnorm_kernel(const float* __restrict__ x, const float* __restrict__ w,
                               float* __restrict__ out, int hidden, float eps) {
  __shared__ float red[32];
  const float* xr = x + (int64_t)blockIdx.x * hidden;
  float ss = 0.f;
  if constexpr (KEEP > 0) {
    float* o = out + (int64_t)blockIdx.x * hidden;
    float4 v[KEEP], k[KEEP];
    pdl_launch_dependents();
    pdl_wait();
#pragma unroll
    for (int c = 0; c < KEEP; ++c) {
      const int i = (threadIdx.x + c * 256) * 4;
      v[c] = k[c] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (i < hidden) {
        v[c] = *reinterpret_cast<const float4*>(xr + i);
        k[c] = *reinterpret_cast<const float4*>(w + i);
      }
    }
#pragma unroll
    for (int c = 0; c < KEEP; ++c)
      ss += v[c].x * v[c].x + v[c].y * v[c].y + v[c].z * v[c].z + v[c].w * v[c].w;
    const float rms = sqrtf(block_sum(ss, red) / (float)hidden + eps);
#pragma unroll
    for (int c = 0; c < KEEP; ++c) {
      const int i = (threadIdx.x + c * 256) * 4;
      if (i < hidden)
        *reinterpret_cast<float4*>(o + i) =
            make_float4(v[c].x / rms * k[c].x, v[c].y / rms * k[c].y, v[c].z / rms * k[c].z,
                        v[c].w / rms * k[c].w);
    }
    return;
  }
  pdl_launch_dependents();
  pdl_wait();
  if constexpr (VEC) {
    float* o = out + (int64_t)blockIdx.x * hidden;
#pragma unroll 4
    for (int i = threadIdx.x * 4; i < hidden; i += 1024) {
      const float4 v = *reinterpret_cast<const float4*>(xr + i);
      ss += v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w;
    }
    const float rms = sqrtf(block_sum(ss, red) / (float)hidden + eps);
#pragma unroll 4
    for (int i = threadIdx.x * 4; i < hidden; i += 1024) {
      const float4 v = *reinterpret_cast<const float4*>(xr + i);
      const float4 k = *reinterpret_cast<const float4*>(w + i);
      *reinterpret_cast<float4*>(o + i) =
          make_float4(v.x / rms * k.x, v.y / rms * k.y, v.z / rms * k.z, v.w / rms * k.w);
    }
    return;
  }
  for (int i = threadIdx.x; i < hidden; i += blockDim.x) ss += xr[i] * xr[i];
  ss = block_sum(ss, red);
  float rms = sqrtf(ss / (float)hidden + eps);
  for (int i = threadIdx.x; i < hidden; i += blockDim.x)
    out[(int64_t)blockIdx.x * hidden + i] = xr[i] / rms * w[i];
}

// Rotate-half RoPE in place (src/model.rs:721-737). With a table: cos/sin rows of
// build_rope_table (src/model.rs:698-719); without: computed on the fly.
constexpr int ROPE_MAX_HALF = 128;  // head_dim <= 256
struct RopeFreq {
  float f[ROPE_MAX_HALF];
};
__global__ void rope_kernel(float* __restrict__ x, const uint32_t* __restrict__ positions,
                            int heads, int head_dim, const RopeFreq freq,
                            const float* __restrict__ cos_t, const float* __restrict__ sin_t,
                            int table_len, int* status) {
  int t = blockIdx.x;
  int half = head_dim / 2;
  uint32_t pos = positions[t];
  if (cos_t && pos >= (uint32_t)table_len) {
    if (threadIdx.x == 0) atomicOr(status, DEV_BAD_INDEX);
    return;
  }
  for (int i = threadIdx.x; i < heads * half; i += blockDim.x) {
    int h = i / half, j = i - h * half;
    float c, s;
    if (cos_t) {
      c = cos_t[(int64_t)pos * half + j];
      s = sin_t[(int64_t)pos * half + j];
    } else {
      float ang = __fmul_rn((float)pos, freq.f[j]);
      c = cosf(ang);
      s = sinf(ang);
    }
    float* v = x + ((int64_t)t * heads + h) * head_dim;
    float a = v[j], b = v[j + half];
    v[j] = a * c - b * s;
    v[j + half] = a * s + b * c;
  }
}

// Bound by its 12 bytes an element; launch and drain below a few MB. A thread takes two groups of four
// (VEC: all three pointers on 16 bytes; else single elements), so that four loads are in flight before
// the first result. As a programmatic dependent of the product before it its launch hides behind that
// product's drain.
constexpr int SILU_PER = 8;  // elements a thread
__device__ __forceinline__ float silu_mul_one(float g, float u) {
  return g / (1.0f + expf(-g)) * u;
}
template <bool VEC>
__global__ void __launch_bounds__(256)
    silu_mul_kernel(const float* g, const float* u, float* out, int64_t n) {
  // No early launch of the kernel behind this one: a product placed around these few CTAs gets two of its
  // CTAs on some SMs and none on others (4096 x 14336 Q4_K at one row: 45 against 33 us for the block).
  pdl_wait();
  const int64_t base = (int64_t)blockIdx.x * (256 * SILU_PER);
  if (VEC && base + 256 * SILU_PER <= n) {
    float4 a[SILU_PER / 4], b[SILU_PER / 4];
#pragma unroll
    for (int j = 0; j < SILU_PER / 4; ++j) {
      const int64_t i = base + (j * 256 + threadIdx.x) * 4;
      a[j] = *reinterpret_cast<const float4*>(g + i);
      b[j] = *reinterpret_cast<const float4*>(u + i);
    }
#pragma unroll
    for (int j = 0; j < SILU_PER / 4; ++j)
      *reinterpret_cast<float4*>(out + base + (j * 256 + threadIdx.x) * 4) =
          make_float4(silu_mul_one(a[j].x, b[j].x), silu_mul_one(a[j].y, b[j].y),
                      silu_mul_one(a[j].z, b[j].z), silu_mul_one(a[j].w, b[j].w));
    return;
  }
  float a[SILU_PER], b[SILU_PER];  // all loads in front of the stores: out may be where g or u is
#pragma unroll
  for (int j = 0; j < SILU_PER; ++j) {
    const int64_t i = base + j * 256 + threadIdx.x;
    a[j] = i < n ? g[i] : 0.f;
    b[j] = i < n ? u[i] : 0.f;
  }
#pragma unroll
  for (int j = 0; j < SILU_PER; ++j) {
    const int64_t i = base + j * 256 + threadIdx.x;
    if (i < n) out[i] = silu_mul_one(a[j], b[j]);
  }
}

// Bound as silu_mul is. A CTA takes 2048 elements: as a dependent each waits for the kernel in front, which CTAs
// of 256 elements paid in every wave (us: 2048 x 5000 elements 42, launched plainly 26, 11 so; 64 x 2048 1.8, 3.6 and
// 1.8).
template <bool VEC>
__global__ void __launch_bounds__(256) residual_add_kernel(float* h, const float* p, int64_t n) {
  pdl_launch_dependents();
  pdl_wait();
  const int64_t base = (int64_t)blockIdx.x * (256 * SILU_PER);
  if (VEC && base + 256 * SILU_PER <= n) {
    float4 a[SILU_PER / 4], b[SILU_PER / 4];
#pragma unroll
    for (int j = 0; j < SILU_PER / 4; ++j) {
      const int64_t i = base + (j * 256 + threadIdx.x) * 4;
      a[j] = *reinterpret_cast<const float4*>(h + i);
      b[j] = *reinterpret_cast<const float4*>(p + i);
    }
#pragma unroll
    for (int j = 0; j < SILU_PER / 4; ++j)
      *reinterpret_cast<float4*>(h + base + (j * 256 + threadIdx.x) * 4) =
          make_float4(a[j].x + b[j].x, a[j].y + b[j].y, a[j].z + b[j].z, a[j].w + b[j].w);
    return;
  }
  float a[SILU_PER], b[SILU_PER];  // all loads in front of the stores, which may be to where others come from
#pragma unroll
  for (int j = 0; j < SILU_PER; ++j) {
    const int64_t i = base + j * 256 + threadIdx.x;
    a[j] = i < n ? h[i] : 0.f;
    b[j] = i < n ? p[i] : 0.f;
  }
#pragma unroll
  for (int j = 0; j < SILU_PER; ++j) {
    const int64_t i = base + j * 256 + threadIdx.x;
    if (i < n) h[i] = a[j] + b[j];
  }
}

// First maximum wins (src/sampler.rs:7-17). One CTA per row.
__global__ void greedy_token_kernel(const float* __restrict__ logits, uint32_t* __restrict__ out,
                                    int64_t vocab) {
  __shared__ float bv[32];
  __shared__ int64_t bi[32];
  const float* row = logits + (int64_t)blockIdx.x * vocab;
  float best = -INFINITY;
  int64_t idx = 0x7FFFFFFFFFFFFFFFll;
  for (int64_t i = threadIdx.x; i < vocab; i += blockDim.x)
    if (row[i] > best) {
      best = row[i];
      idx = i;
    }
  auto better = [](float v1, int64_t i1, float v2, int64_t i2) {
    return v1 > v2 || (v1 == v2 && i1 < i2);
  };
  for (int o = 16; o; o >>= 1) {
    float v = __shfl_xor_sync(0xFFFFFFFFu, best, o);
    int64_t i = __shfl_xor_sync(0xFFFFFFFFu, idx, o);
    if (better(v, i, best, idx)) {
      best = v;
      idx = i;
    }
  }
  int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (lane == 0) {
    bv[warp] = best;
    bi[warp] = idx;
  }
  __syncthreads();
  if (warp == 0) {
    int nw = blockDim.x >> 5;
    best = lane < nw ? bv[lane] : -INFINITY;
    idx = lane < nw ? bi[lane] : 0x7FFFFFFFFFFFFFFFll;
    for (int o = 16; o; o >>= 1) {
      float v = __shfl_xor_sync(0xFFFFFFFFu, best, o);
      int64_t i = __shfl_xor_sync(0xFFFFFFFFu, idx, o);
      if (better(v, i, best, idx)) {
        best = v;
        idx = i;
      }
    }
    // all -inf / NaN rows keep index 0, as the reference's loop does
    if (lane == 0) out[blockIdx.x] = idx == 0x7FFFFFFFFFFFFFFFll ? 0u : (uint32_t)idx;
  }
}

int32_t launch_rmsnorm(kanso_cuda_ctx* ctx, const float* x, const float* w, float* out,
                       int64_t rows, int64_t hidden, float eps) {
  // us: two rows of 2048 6.4 a float at a time, twice over the row and launched plainly, 2.4 so; 512 of 5000
  // 13.2 and 7.1. Four kept float4 take 52 registers, four CTAs an SM: rows beyond those that need one alone keep
  // one (2048 rows of 64 5.5 us with four, 3.8 with one; 2048 of 1024 6.2 and 4.9; but 512 of 1024 2.6 and 3.0).
  const bool vec = hidden % 4 == 0 && aligned16(x) && aligned16(w) && aligned16(out);
  const cudaError_t e =
      launch_dependent(ctx,
                       !vec            ? rmsnorm_kernel<false, 0>
                       : hidden > 4096 ? rmsnorm_kernel<true, 0>
                       : hidden <= 1024 && rows > 4 * (int64_t)ctx->sm_count
                           ? rmsnorm_kernel<true, 1>
                           : rmsnorm_kernel<true, 4>,
                       dim3((unsigned)rows), dim3(256), 0, x, w, out, (int)hidden, eps);
  if (e != cudaSuccess) return cuda_fail(ctx, e, "rmsnorm launch");
  return after_launch(ctx, "rmsnorm");
}

int32_t launch_rope(kanso_cuda_ctx* ctx, float* x, const uint32_t* positions, int64_t T,
                    int64_t heads, int64_t head_dim, float theta, const float* cos_t,
                    const float* sin_t, int table_len) {
  RopeFreq freq;
  if (!cos_t)  // theta^(-2j/head_dim) with the host's powf, as build_rope_table (src/model.rs:700-707)
    for (int j = 0; j < head_dim / 2; ++j)
      freq.f[j] = std::pow(theta, -2.0f * (float)j / (float)head_dim);
  rope_kernel<<<(unsigned)T, 128, 0, ctx->stream>>>(x, positions, (int)heads, (int)head_dim, freq,
                                                    cos_t, sin_t, table_len, ctx->dev_status);
  return after_launch(ctx, "rope");
}

int32_t launch_silu_mul(kanso_cuda_ctx* ctx, const float* g, const float* u, float* out,
                        int64_t n) {
  const bool vec = aligned16(g) && aligned16(u) && aligned16(out);
  auto kern = vec ? silu_mul_kernel<true> : silu_mul_kernel<false>;
  // the same split of an SM's memory as the products': an SM does not drain to change it
  prefer_max_shared(ctx, (const void*)kern);
  const int64_t per = 256 * SILU_PER;
  const cudaError_t le = launch_dependent(ctx, kern, dim3((unsigned)((n + per - 1) / per)),
                                          dim3(256), 0, g, u, out, n);
  if (le != cudaSuccess) return cuda_fail(ctx, le, "silu_mul launch");
  return after_launch(ctx, "silu_mul");
}

int32_t launch_residual_add(kanso_cuda_ctx* ctx, float* h, const float* p, int64_t n) {
  const int64_t per = 256 * SILU_PER;
  const cudaError_t e = launch_dependent(
      ctx, aligned16(h) && aligned16(p) ? residual_add_kernel<true> : residual_add_kernel<false>,
      dim3((unsigned)((n + per - 1) / per)), dim3(256), 0, h, p, n);
  if (e != cudaSuccess) return cuda_fail(ctx, e, "residual_add launch");
  return after_launch(ctx, "residual_add");
}

}  // namespace kanso

using namespace kanso;

extern "C" {

int32_t kanso_cuda_rmsnorm(kanso_cuda_ctx* ctx, const float* x, const float* weight, float* out,
                           int64_t rows, int64_t hidden, float eps) {
  if (!ctx) return fail(nullptr, KANSO_ERR_CONFIG, "rmsnorm: ctx is NULL");
  if (rows < 0 || hidden <= 0) return fail(ctx, KANSO_ERR_SHAPE, "rmsnorm: bad shape");
  if (rows == 0) return KANSO_OK;
  return launch_rmsnorm(ctx, x, weight, out, rows, hidden, eps);
}

int32_t kanso_cuda_rope(kanso_cuda_ctx* ctx, float* x, const uint32_t* positions, int64_t T,
                        int64_t heads, int64_t head_dim, float theta) {
  if (!ctx) return fail(nullptr, KANSO_ERR_CONFIG, "rope: ctx is NULL");
  if (T < 0 || heads <= 0 || head_dim <= 0 || head_dim % 2 || head_dim > 2 * ROPE_MAX_HALF)
    return fail(ctx, KANSO_ERR_SHAPE, "rope: head_dim %lld must be even, positive and <= %d",
                (long long)head_dim, 2 * ROPE_MAX_HALF);
  if (T == 0) return KANSO_OK;
  return launch_rope(ctx, x, positions, T, heads, head_dim, theta, nullptr, nullptr, 0);
}

int32_t kanso_cuda_silu_mul(kanso_cuda_ctx* ctx, const float* gate, const float* up, float* out,
                            int64_t n) {
  if (!ctx) return fail(nullptr, KANSO_ERR_CONFIG, "silu_mul: ctx is NULL");
  if (n < 0) return fail(ctx, KANSO_ERR_SHAPE, "silu_mul: n < 0");
  if (n == 0) return KANSO_OK;
  return launch_silu_mul(ctx, gate, up, out, n);
}

int32_t kanso_cuda_residual_add(kanso_cuda_ctx* ctx, float* hidden, const float* proj, int64_t n) {
  if (!ctx) return fail(nullptr, KANSO_ERR_CONFIG, "residual_add: ctx is NULL");
  if (n < 0) return fail(ctx, KANSO_ERR_SHAPE, "residual_add: n < 0");
  if (n == 0) return KANSO_OK;
  return launch_residual_add(ctx, hidden, proj, n);
}

int32_t kanso_cuda_greedy_token(kanso_cuda_ctx* ctx, const float* logits, uint32_t* out,
                                int64_t B, int64_t vocab) {
  if (!ctx) return fail(nullptr, KANSO_ERR_CONFIG, "greedy_token: ctx is NULL");
  if (B < 0 || vocab <= 0) return fail(ctx, KANSO_ERR_SHAPE, "greedy_token: bad shape");
  if (B == 0) return KANSO_OK;
  greedy_token_kernel<<<(unsigned)B, 256, 0, ctx->stream>>>(logits, out, vocab);
  return after_launch(ctx, "greedy_token");
}

}  // extern "C"
