// Chooses the kernel behind LinearWeight::forward (src/weights.rs:43-45) by the number
// of activation rows, and exposes the pointer-level GEMM entry points.
#include "ctx.h"

namespace kanso {
int32_t stream_matmul(kanso_cuda_ctx* ctx, int32_t dtype, const void* w, const float* x, float* y,
                      int64_t M, int64_t N, int64_t K, int32_t act_mode);

int32_t tc_matmul(kanso_cuda_ctx* ctx, int32_t dtype, const void* w, const float* x, float* y,
                  int64_t M, int64_t N, int64_t K, bool* handled);
int32_t q4k_direct_matmul(kanso_cuda_ctx* ctx, const void* w, const float* x, float* y, int64_t M,
                          int64_t N, int64_t K, bool* handled);

int32_t q8_mma_matmul(kanso_cuda_ctx* ctx, int nseg, const void* const* w, float* const* y,
                      const int64_t* rows, const float* x, const float* x2, const float* norm_w,
                      float eps, const float* resid, int64_t K, int M, int32_t act_mode,
                      bool decode_chain, bool* handled);

int32_t tma_matmul(kanso_cuda_ctx* ctx, int32_t dtype, const void* w, const float* x, float* y,
                   int64_t M, int64_t N, int64_t K, bool* handled);
int32_t few_matmul(kanso_cuda_ctx* ctx, int32_t dtype, const void* w, const float* x, float* y,
                   int64_t M, int64_t N, int64_t K, int32_t act_mode, bool* handled);

int32_t matmul_dispatch(kanso_cuda_ctx* ctx, int32_t dtype, const void* w, const float* x,
                        float* y, int64_t M, int64_t N, int64_t K, int32_t act_mode) {
  // 9..48 activation rows (Q8_0: from two rows on), mostly 49..64 too, and any number above 8 with Q8
  // activations: the weight-streaming kernel, in passes of at most 64 (128) rows. us per product, all
  // in graphs of products behind one another over more than 300 MB of weights, against the kernels
  // below, which keep what it does not take. 14336 x 4096: Q8_0 at 2 / 24 / 48 / 64 rows 16 / 20 / 27 /
  // 34 against 30 / 32 / 33 / 34, Q4_K at 16 / 24 / 48 / 64 rows 17 / 20 / 28 / 33 against 31 / 33 / 34 /
  // 36; 4096 x 4096 Q8_0 at 9 / 32 / 48 rows 8 / 12 / 13 against 12 / 15 / 15. Fewer Q4_K rows keep the
  // int8 GEMV's finer activations. Q8 activations at 16 / 32 / 64 / 128 rows: 20 / 27 / 41 / 68 against
  // the 87 / 87 / 87 / 113 of a tcgen05 kind::i8 form that drained an accumulator per block.
  // 49..64 rows take one CTA per SM with all its registers: between one and nine units for it (128
  // weight rows x 256 k) they do not share out evenly, and the kernel below is the faster one: Q8_0
  // at 64 rows of 4096 x 4096 17.6 against 15.3, 8192 x 4096 23.6 and 22.4; but 2048 x 1024 7.5 and
  // 10.2, 4096 x 14336 35 and 38, 11008 x 4096 29 and 36.
  const int64_t units = (N + 127) / 128 * (K / 256);
  const bool even = !ctx || units <= ctx->sm_count || units >= 9 * (int64_t)ctx->sm_count;
  const bool few = act_mode == KANSO_ACT_Q8
                       ? M > 8 && dtype == KANSO_DTYPE_Q8_0
                       : M <= (even ? 64 : 48) && M >= (dtype == KANSO_DTYPE_Q8_0 ? 2 : 9);
  if (few && w && x && y) {
    bool all = true;
    for (int64_t m0 = 0; m0 < M && all;) {
      int64_t mc = M - m0 < 128 ? M - m0 : 128;
      if (M - m0 - mc > 0 && M - m0 - mc < 9) mc -= 16;  // no short tail
      bool handled = false;
      int32_t st = few_matmul(ctx, dtype, w, x + m0 * K, y + m0 * N, mc, N, K, act_mode, &handled);
      if (st != KANSO_OK) return st;
      if (!handled) all = false;
      m0 += mc;
    }
    if (all) return KANSO_OK;
  }
  // More rows on a matrix whose rows start on 16-byte boundaries: the TMA-staged tcgen05 GEMM, up
  // to 512 rows per pass over the weights (96 rows of 14336 x 4096: 57 against 68 us of the
  // weight-streaming kernel, whose mma.sync rate is the bound there).
  const bool tma_rows = M > 64 || (M > 48 && !even);
  if (tma_rows && act_mode == KANSO_ACT_F32 && N > 0 && K > 0 && w && x && y) {
    bool all = true;
    for (int64_t m0 = 0; m0 < M && all; m0 += 512) {
      bool handled = false;
      // a tail of fewer than 9 rows rides with the chunk before it
      int64_t mc = M - m0 < 512 ? M - m0 : 512;
      if (M - m0 - mc > 0 && M - m0 - mc < 9) mc -= 16;
      int32_t st = tma_matmul(ctx, dtype, w, x + m0 * K, y + m0 * N, mc, N, K, &handled);
      if (st != KANSO_OK) return st;
      if (!handled) all = false;
      m0 -= 512 - mc;
    }
    if (all) return KANSO_OK;
  }
  // More than 8 activation rows: the tcgen05 GEMM, at most 128 rows per pass over the weights
  // (the A/B tiles of two stages plus the raw-byte ring fill one SM's shared memory).
  if (M > 8 && act_mode == KANSO_ACT_F32 && (dtype == KANSO_DTYPE_Q8_0 || dtype == KANSO_DTYPE_Q4_K) &&
      N > 0 && K > 0 && w && x && y && aligned16(x)) {
    bool all = true;
    for (int64_t m0 = 0; m0 < M && all; m0 += 128) {
      bool handled = false;
      int32_t st = tc_matmul(ctx, dtype, w, x + m0 * K, y + m0 * N, M - m0 < 128 ? M - m0 : 128, N,
                             K, &handled);
      if (st != KANSO_OK) return st;
      if (!handled) all = false;
    }
    if (all) return KANSO_OK;
  }
  if (dtype == KANSO_DTYPE_Q4_K && act_mode == KANSO_ACT_F32 && K > 0 && K % 256 == 0 && M > 0 &&
      N > 0 && w && x && y && aligned16(w) && aligned16(x)) {
    // int8 tensor-core GEMV. Up to 6 activation rows go in one pass over the weights; from 7
    // rows on, passes of 4 are faster than the kernel's 7- and 8-row forms (which spill
    // registers): 22.6 us against 36.5 us for 8 rows of a 14336 x 4096 matrix. Fewer rows per
    // pass also when the activation planes of a long K do not fit in shared memory.
    const int64_t mp0 = M > 6 ? 4 : 8;
    for (int64_t mp = mp0; mp >= 1; mp /= 2) {
      if (mp < mp0 && M <= mp) continue;  // the same single pass as the attempt before
      bool all = true;
      for (int64_t m0 = 0; m0 < M && all; m0 += mp) {
        bool handled = false;
        int32_t st = q4k_direct_matmul(ctx, w, x + m0 * K, y + m0 * N, M - m0 < mp ? M - m0 : mp,
                                       N, K, &handled);
        if (st != KANSO_OK) return st;
        if (!handled) all = false;  // decided by the shape of the largest (first) pass
      }
      if (all) return KANSO_OK;
    }
  }
  if (dtype == KANSO_DTYPE_Q8_0 && (act_mode == KANSO_ACT_F32 || act_mode == KANSO_ACT_Q8) &&
      K > 0 && M > 0 && N > 0 && w && x && y) {
    // int8 tensor-core GEMV, at most 8 activation rows per pass over the weights
    bool all = true;
    for (int64_t m0 = 0; m0 < M && all; m0 += 8) {
      bool handled = false;
      const void* w1[1] = {w};
      float* y1[1] = {y + m0 * N};
      const int64_t r1[1] = {N};
      int32_t st = q8_mma_matmul(ctx, 1, w1, y1, r1, x + m0 * K, nullptr, nullptr, 0.f, nullptr, K,
                                 (int)(M - m0 < 8 ? M - m0 : 8), act_mode, false, &handled);
      if (st != KANSO_OK) return st;
      if (!handled) all = false;
    }
    if (all) return KANSO_OK;
  }
  return stream_matmul(ctx, dtype, w, x, y, M, N, K, act_mode);
}
}  // namespace kanso

using namespace kanso;

extern "C" {
int32_t kanso_cuda_gemm_q8_0(kanso_cuda_ctx* ctx, const void* w, const float* x, float* y,
                             int64_t M, int64_t N, int64_t K, int32_t act_mode) {
  if (!ctx) return fail(nullptr, KANSO_ERR_CONFIG, "gemm_q8_0: ctx is NULL");
  return matmul_dispatch(ctx, KANSO_DTYPE_Q8_0, w, x, y, M, N, K, act_mode);
}
int32_t kanso_cuda_gemm_q4_k(kanso_cuda_ctx* ctx, const void* w, const float* x, float* y,
                             int64_t M, int64_t N, int64_t K, int32_t act_mode) {
  if (!ctx) return fail(nullptr, KANSO_ERR_CONFIG, "gemm_q4_k: ctx is NULL");
  return matmul_dispatch(ctx, KANSO_DTYPE_Q4_K, w, x, y, M, N, K, act_mode);
}
}
