// Batched quantized GEMM with TMA-staged weight tiles (cp.async.bulk.tensor) feeding
// tcgen05 / TMEM: LinearWeight::forward for continuous-batching and chunked-prefill rows
// (src/weights.rs:43-45; callers src/model.rs:390-421,1418-1740), up to 512 activation rows in
// ONE pass over the weights.
//
//   y[M,N] = x[M,K] @ W[N,K]^T,  W in GGUF Q8_0 / Q4_K blocks, x and y f32.
//
// The contraction runs over the BYTE STREAM of a weight row, not over k. A CTA owns 128 weight
// rows; one elected thread pulls boxes of 128 rows x 128 bytes of the block matrix
// [N][row_bytes] into a ring of shared-memory slots with 2-D tensor-map copies (128-byte
// swizzle, so that 16-byte reads with one lane per row are free of bank conflicts; rows and
// bytes past the matrix are zero-filled by the copy engine). A box does not line up with the
// 34-byte (Q8_0) or 144-byte (Q4_K) blocks and it does not have to: the sum over k may be taken
// in any order as long as both operands agree, so every 16-byte chunk of the stream becomes MMA
// k-positions in the order its bytes lie in memory, and a small pack kernel lays the
// activations out in that same order (zero at the positions of scale bytes and headers):
//   * Q8_0: one chunk = 16 positions = one k-step; a position that holds a byte of a block's
//     f16 scale is multiplied by a zero on the activation side. No realignment of the 2-byte-
//     aligned int8 runs is ever done.
//   * Q4_K: one nibble chunk = 16 low nibbles + 16 high nibbles = two k-steps (sub-blocks 2g
//     and 2g+1 of the chunk's 64-weight group); header chunks produce nothing and are skipped
//     by the MMA issuer.
// 16 producer warps (thread = weight row x 32 stream bytes) read the raw chunks, dequantise with
// packed f16 arithmetic (Q8_0: exact int8 -> f16 by byte permute, one rounding in d*q; Q4_K:
// d*sc*(q-8) - (dmin*m - 8*d*sc) with both factors rounded once to f16) and store 16-byte
// core-matrix rows of the A tile (K-major, no swizzle). Where a block's scale or header falls
// inside a thread's bytes repeats with a short period (17 positions for Q8_0, 9 for Q4_K), so the
// dequantising code exists once per position, with every selection resolved at compile time, and
// a switch picks the body. One warp issues tcgen05.mma
// (kind::f16, M = 128 weight rows, N = up to 256 activation rows per instruction, f32
// accumulation in up to 512 TMEM columns); one warp streams the packed activations through a
// ring of bulk copies. All hand-offs are mbarriers with bounded waits: a wait that runs out sets
// the status word, the CTA drains its own copies, frees its TMEM and returns.
//
// Numerics: both operands are rounded once to f16 (as the f16 tensor path prescribes); the
// products are exact and accumulate in f32. The error of a K = 4096 product is about 1e-4 of
// the output scale against the 1e-3 bound. The decode step's chain of matmuls keeps the
// three-product kernel in gemm_tc.cu.
#include "gemm_tma_kernel.cuh"
#include "tensor_map.h"

namespace kanso {

// Activations into stream order. A tile is 32 rows x 256 k (K % 256 == 0 for both formats here: rows of
// blocks that start on 16 bytes), which is 17 chunks of a Q8_0 stream and 36 half k-steps of a Q4_K one:
// it is read along k, whole sectors, rounded to f16 in shared memory and written with lanes along the
// rows, 512 bytes at a time. A thread that gathered its 8 values from memory itself, its neighbours a row
// apart, took 17 us for 512 x 4096 and 31 us for 512 x 14336 (8.4 and 29 MB read, half of that written).
// Tiles behind the last k are the stream's padding: zeros.
constexpr int PACK_ROWS = 32, PACK_K = 256;
constexpr int PACK_PITCH = PACK_K + 2;  // an odd number of words: lanes along the rows, 32 banks
// PARTS: CTAs that read one tile and write a part of it each (blockIdx.z).
template <int FMT, bool VEC, int PARTS>
__global__ void __launch_bounds__(256)
    tm_pack_kernel(const float* __restrict__ x, __half* __restrict__ bp, int M, int Mt, int K,
                   int units_total, const TmZero zero) {
  // unit halves (8 positions of every row) of a tile
  constexpr int HALVES = FMT == TM_FMT_Q8_0 ? 2 * (PACK_K / 32 * Q8_BYTES / 16)
                                            : 4 * (Q4K_BYTES / 16);
  __shared__ __half tile[PACK_ROWS * PACK_PITCH];
  pdl_launch_dependents();
  pdl_wait();  // x (and the readers of the buffer cleared here) belong to earlier kernels
  const int64_t cta = (blockIdx.z * (int64_t)gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x;
  const int64_t nthreads = (int64_t)gridDim.x * gridDim.y * gridDim.z * blockDim.x;
  for (int64_t j = cta * blockDim.x + threadIdx.x; j < zero.n; j += nthreads) zero.p[j] = 0.f;
  const int k0 = blockIdx.x * PACK_K, m0 = blockIdx.y * PACK_ROWS;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (k0 < K) {
    // warp: rows warp, warp + 8, ...; lane: four values at 4 * lane and 128 further on
    float4 v[PACK_ROWS / 8][2];
#pragma unroll
    for (int i = 0; i < PACK_ROWS / 8; ++i)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int m = m0 + warp + 8 * i;
        const float* src = x + (int64_t)m * K + k0 + h * 128 + lane * 4;
        v[i][h] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (m < M) {
          if (VEC)
            v[i][h] = *reinterpret_cast<const float4*>(src);
          else
            v[i][h] = make_float4(src[0], src[1], src[2], src[3]);
        }
      }
#pragma unroll
    for (int i = 0; i < PACK_ROWS / 8; ++i)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        __half2* dst = reinterpret_cast<__half2*>(tile + (warp + 8 * i) * PACK_PITCH + h * 128 +
                                                  lane * 4);
        dst[0] = __floats2half2_rn(v[i][h].x, v[i][h].y);
        dst[1] = __floats2half2_rn(v[i][h].z, v[i][h].w);
      }
    __syncthreads();
  }
  const int m = m0 + lane;
  const int first = blockIdx.x * HALVES;
  const uint16_t* row = reinterpret_cast<const uint16_t*>(tile) + lane * PACK_PITCH;
  for (int j = warp + 8 * blockIdx.z; j < HALVES && first + j < 2 * units_total; j += 8 * PARTS) {
    uint32_t o[4] = {};
    if (k0 < K) {
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const int k = FMT == TM_FMT_Q8_0 ? tm_k_of_q8_0(j >> 1, 8 * (j & 1) + e)
                                         : tm_k_of_q4_k(j >> 2, (j >> 1) & 1, 8 * (j & 1) + e);
        if (k >= 0) o[e >> 1] |= (uint32_t)row[k] << (16 * (e & 1));
      }
    }
    if (m < Mt)
      *reinterpret_cast<uint4*>(bp + ((int64_t)(first + j) * Mt + m) * 8) =
          make_uint4(o[0], o[1], o[2], o[3]);
  }
}

template <int FMT>
static int32_t tm_pack(kanso_cuda_ctx* ctx, const float* x, void* bp, int M, int Mt, int K,
                       int units_total, const TmZero& zero) {
  constexpr int UNITS = FMT == TM_FMT_Q8_0 ? PACK_K / 32 * Q8_BYTES / 16 : 2 * (Q4K_BYTES / 16);
  dim3 grid((unsigned)((units_total + UNITS - 1) / UNITS),
            (unsigned)((Mt + PACK_ROWS - 1) / PACK_ROWS));
  // few tiles: two or four CTAs share one (2048 x 1024 at 65 rows, 15 tiles: 10.8 -> 9.9 us)
  const int64_t room = ctx->sm_count / ((int64_t)grid.x * grid.y);
  grid.z = room >= 4 ? 4 : room >= 2 ? 2 : 1;
  const bool vec = aligned16(x);
  auto kern = grid.z == 4   ? (vec ? tm_pack_kernel<FMT, true, 4> : tm_pack_kernel<FMT, false, 4>)
              : grid.z == 2 ? (vec ? tm_pack_kernel<FMT, true, 2> : tm_pack_kernel<FMT, false, 2>)
                            : (vec ? tm_pack_kernel<FMT, true, 1> : tm_pack_kernel<FMT, false, 1>);
  const cudaError_t le = launch_dependent(ctx, kern, grid, dim3(256), 0, x,
                                          reinterpret_cast<__half*>(bp), M, Mt, K, units_total,
                                          zero);
  if (le != cudaSuccess) return cuda_fail(ctx, le, "gemm_tma pack launch");
  return after_launch(ctx, "gemm_tma pack activations");
}

// y[M,N] = x[M,K] @ W^T for 9..512 activation rows (fewer than 49 are gemm_few.cu's, and come here
// only as the last rows of a larger product). Sets *handled = false (and launches nothing) when the shape
// is outside this kernel's range: rows of the block matrix must start on 16-byte boundaries (every
// Q4_K matrix; Q8_0 when K % 256 == 0).
int32_t tma_matmul(kanso_cuda_ctx* ctx, int32_t dtype, const void* w, const float* x, float* y,
                   int64_t M, int64_t N, int64_t K, bool* handled) {
  *handled = false;
  if (dtype != KANSO_DTYPE_Q8_0 && dtype != KANSO_DTYPE_Q4_K) return KANSO_OK;
  const int blk = dtype == KANSO_DTYPE_Q8_0 ? 32 : 256;
  const int bb = dtype == KANSO_DTYPE_Q8_0 ? Q8_BYTES : Q4K_BYTES;
  if (M < 9 || M > TM_MAX_M || N < 1 || K < blk || K % blk != 0 || !w || !x || !y)
    return KANSO_OK;
  const int64_t row_bytes = K / blk * bb;
  if (row_bytes % 16 != 0 || !aligned16(w) || row_bytes > (1 << 28) || N > (1 << 30))
    return KANSO_OK;
  TmEncodeFn encode = tm_encoder();
  if (!encode) return KANSO_OK;

  const int Mt = (int)((M + 15) / 16 * 16);
  const int boxes_total = (int)((row_bytes + TM_BOX_W - 1) / TM_BOX_W);
  const int upc = dtype == KANSO_DTYPE_Q8_0 ? 1 : 2;
  const int units_total = boxes_total * 8 * upc;
  const int tiles_n = (int)((N + TM_TILE_N - 1) / TM_TILE_N);
  // Split the stream while the grid stays within about one wave of CTAs (one CTA per SM) and
  // every CTA keeps at least four boxes; the partial sums of a split are added with atomics
  // onto a y that the pack kernel clears.
  int ksplit = 1;
  while (tiles_n * ksplit * 2 <= ctx->sm_count + ctx->sm_count / 4 &&
         boxes_total / (ksplit * 2) >= 4)
    ksplit *= 2;
  // activation units per ring slot: a whole stage (8 k-steps) when a slot holds that, else the
  // largest power-of-two share of it that fits
  const int b_slots = Mt <= 128 ? TM_B_SLOTS_TWO : TM_B_SLOTS_ONE;
  const int b_slot = Mt <= 128 ? TM_B_SLOT_TWO : TM_B_SLOT_ONE;
  int ub = 1;
  while (ub * 2 <= 8 && ub * 2 * 32 * Mt <= b_slot) ub *= 2;

  CUtensorMap tmap;
  const cuuint64_t gdim[2] = {(cuuint64_t)row_bytes, (cuuint64_t)N};
  const cuuint64_t gstride[1] = {(cuuint64_t)row_bytes};
  const cuuint32_t box[2] = {TM_BOX_W, TM_TILE_N};
  const cuuint32_t estr[2] = {1, 1};
  const CUresult cr = encode(&tmap, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(w), gdim,
                             gstride, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                             CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (cr != CUDA_SUCCESS)
    return fail(ctx, KANSO_ERR_DEVICE, "gemm_tma: cuTensorMapEncodeTiled failed (%d)", (int)cr);

  const size_t bp_bytes = (size_t)units_total * 32 * Mt;
  uint8_t* scratch = (uint8_t*)ctx_scratch(ctx, bp_bytes + 256);
  if (!scratch) return KANSO_ERR_DEVICE;
  *handled = true;

  TmZero zero = {nullptr, 0};
  if (ksplit > 1) {
    zero.p = y;
    zero.n = M * N;
  }
  const int32_t st =
      dtype == KANSO_DTYPE_Q8_0
          ? tm_pack<TM_FMT_Q8_0>(ctx, x, scratch, (int)M, Mt, (int)K, units_total, zero)
          : tm_pack<TM_FMT_Q4_K>(ctx, x, scratch, (int)M, Mt, (int)K, units_total, zero);
  if (st) return st;

  TmArgs a;
  a.y = y;
  a.bp = scratch;
  a.N = N;
  a.M = (int)M;
  a.Mt = Mt;
  a.row_bytes = (int)row_bytes;
  a.boxes_total = boxes_total;
  a.ksplit = ksplit;
  a.ub = ub;
  a.status = ctx->dev_status;
  size_t smem = (size_t)TM_RAW_SLOTS * TM_BOX + (size_t)TM_A_STAGES * TM_A_STAGE +
                      (size_t)b_slots * ub * 32 * Mt + 256;
  // An SM's shared memory is split in steps, of which 196 KB and 228 KB come into question. A product that leaves no
  // room for a pack's CTA (16 KB) in the 196 KB asks for a little more than those: else the next pack waits until
  // the SM has drained and changed its split (18944 x 3584 Q8_0 at 112 rows, 184 KB: 36.9 us, 31.0 with more; at 96
  // rows, 176 KB, 30.5).
  constexpr size_t STEP = 196 * 1024, PACK = PACK_ROWS * PACK_PITCH * 2 + 2048;
  if (smem + 1024 <= STEP && smem + 1024 + PACK > STEP) smem = STEP;
  if (smem > (size_t)ctx->smem_optin)
    return fail(ctx, KANSO_ERR_UNSUPPORTED, "gemm_tma: %zu bytes of shared memory needed", smem);
  const dim3 grid(tiles_n, ksplit);
  return dtype == KANSO_DTYPE_Q8_0 ? tm_launch_q8_0(ctx, grid, smem, tmap, a)
                                   : tm_launch_q4_k(ctx, grid, smem, tmap, a);
}

}  // namespace kanso
