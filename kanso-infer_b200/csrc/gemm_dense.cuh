// What the tile products of unquantised weights share (gemm_dense.cu, gemm_pair.cu): launch arguments,
// where results go, tensor maps.
#pragma once
#include "dense.cuh"
#include "tensor_map.h"

namespace kanso {

constexpr int GD_K = 64;  // columns per stage (128 bytes)

struct GemmDenseArgs {
  void* out;            // f32 results, or the element type for the experts' activations
  int64_t out_ld, part_stride;
  const uint32_t* offsets;
  int64_t T;
  int groups, rows, k_steps, steps_per_split;
  int* status;
  const float* bias;
  int64_t group_step;
  const uint32_t* row_list;
  int relu2, elem, n_end;  // n_end: columns that are written

  // The bias of column n, added once where the columns' sum is split.
  __device__ __forceinline__ float bias_of(int n) const {
    return bias && n < rows && blockIdx.z == 0 ? bias[n] : 0.f;
  }
};
// Where the rows of a tile's group go: row r at r * out_ld + shift, by the list if there is one.
struct RowPlace {
  int64_t shift = 0, first = 0;
  const uint32_t* list = nullptr;
  __device__ __forceinline__ RowPlace(const GemmDenseArgs& a, int group) {
    if (!a.group_step) return;
    const int64_t per = (uint32_t)a.T / (uint32_t)a.groups;
    shift = group * (a.row_list ? a.group_step : a.group_step - per * a.out_ld);
    first = group * per;
    list = a.row_list;
  }
  __device__ __forceinline__ int64_t at(int64_t row, int64_t out_ld) const {
    return (list ? (int64_t)list[row - first] : row) * out_ld + shift;
  }
};

// [groups][rows][ld] in boxes of `box_rows` rows x 64 columns
inline int32_t weight_map(kanso_cuda_ctx* ctx, const DenseMat& w, CUtensorMap* map,
                          int box_rows = 128) {
  TmEncodeFn encode = tm_encoder();
  if (!encode) return fail(ctx, KANSO_ERR_DEVICE, "the driver has no tensor-map encoder");
  const cuuint64_t dim[3] = {(cuuint64_t)w.cols, (cuuint64_t)w.rows, (cuuint64_t)w.groups};
  const cuuint64_t stride[2] = {(cuuint64_t)w.ld * 2, (cuuint64_t)(w.rows * w.ld) * 2};
  const cuuint32_t box[3] = {GD_K, (cuuint32_t)box_rows, 1}, es[3] = {1, 1, 1};
  if (encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, w.w, dim, stride, box, es,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
             CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
    return fail(ctx, KANSO_ERR_DEVICE, "tensor map of a [%lld x %lld] weight", (long long)w.rows,
                (long long)w.cols);
  return KANSO_OK;
}
// [T][ld] in boxes of nt rows x 64 columns
inline int32_t rows_map(kanso_cuda_ctx* ctx, const void* x, int64_t T, int64_t cols, int64_t ld,
                        int nt, CUtensorMap* map) {
  TmEncodeFn encode = tm_encoder();
  if (!encode) return fail(ctx, KANSO_ERR_DEVICE, "the driver has no tensor-map encoder");
  const cuuint64_t dim[2] = {(cuuint64_t)cols, (cuuint64_t)T};
  const cuuint64_t stride[1] = {(cuuint64_t)ld * 2};
  const cuuint32_t box[2] = {GD_K, (cuuint32_t)nt}, es[2] = {1, 1};
  if (encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(x), dim, stride, box, es,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
             CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
    return fail(ctx, KANSO_ERR_DEVICE, "tensor map of [%lld x %lld] activations", (long long)T,
                (long long)cols);
  return KANSO_OK;
}

// Products large enough for pairs of CTAs (gemm_pair.cu); *handled = false: not this one. up: silu(w x) *
// (up x) in bfloat16.
int32_t launch_gemm_pair(kanso_cuda_ctx* ctx, const DenseMat& w, const DenseMat* up, const void* x,
                         const GemmRows& r, GemmDenseArgs a, bool ext, bool* handled);

}  // namespace kanso
