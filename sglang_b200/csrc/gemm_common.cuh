// What the block-scaled GEMM kernels share: rasterization, TMA descriptors, the pipeline-wait setting.
#pragma once
#include <cuda.h>

#include "cluster_rule.h"
#include "common.cuh"

namespace sglb200 {

// tile index -> (m_tile, n_tile): groups of `group_m` m-tiles sweep over n together, m fastest inside a group.
// The activation rows of a group stay in L2 while the weight matrix streams past them once per group.
__device__ __forceinline__ void tile_coord(int t, int tiles_m, int tiles_n, int group_m, int& m_tile, int& n_tile) {
  const int per_group = group_m * tiles_n;
  const int g = t / per_group;
  const int first_m = g * group_m;
  const int gsz = min(tiles_m - first_m, group_m);
  const int r = t - g * per_group;
  m_tile = first_m + r % gsz;
  n_tile = r / gsz;
}

// uint8 tensor [d2][d1][d0] (d0 contiguous) described with `rank` (2 or 3) dimensions, box = 128 x box_rows (x 1),
// 128-byte swizzle, out-of-range elements read as zero.  Cached per argument tuple and thread.
int get_tensor_map(const void* ptr, uint64_t d0, uint64_t d1, uint64_t d2, uint32_t box_rows, uint32_t rank, CUtensorMap* out);

// Output tensor [rows][N] of 2-byte elements, box = 64 columns x box_rows, 128-byte swizzle (matches the staging layout
// written by the epilogues).  Cached likewise.
int get_out_map(const void* ptr, uint64_t N, uint64_t rows, int out_fp16, uint32_t box_rows, CUtensorMap* out);

// m-tiles per rasterization group for rows of K bytes (see gemm.cu).
int choose_group_m(int64_t rows, int64_t K, int tile_rows);

extern uint32_t g_gemm_wait_probes;  // probes after which a pipeline wait gives up (sglb200_gemm_set_wait_probes)

// quant.cu: the quantizers (arguments as the C ABI's).  `trigger`: the launch that follows may be scheduled early, as the
// outputs are this call's own intermediates (see quant.cu).
int quant_fp8(const void* input, int in_dtype, void* output_q, float* output_s, int64_t num_tokens, int64_t hidden,
              int group_size, float eps, float fp8_min, float fp8_max, int64_t s_stride_token, int64_t s_stride_group,
              bool trigger, cudaStream_t st);
int silu_mul_quant_fp8(const void* input, int dtype, void* output_q, float* output_s, int64_t rows, int64_t d, int group_size,
                       float eps, const int32_t* num_rows_dev, bool trigger, cudaStream_t st);

// moe_misc.cu: out[t] = factor * sum over k of the row of `src` at inverse[t * topk + k], where that is not negative.
int sum_sorted(const void* src, const int32_t* inverse, void* out, int dtype, int64_t tokens, int64_t topk, int64_t hidden,
               float factor, cudaStream_t st);

// quant.cu: the quantizer (groups of 128) of a layer's activations with every row's codes and scales written to its `topk`
// places in the sorted order (`inverse` of the sort, -1 = nowhere), and zeros to the padding rows of 32-row quadrants that
// hold rows; other padding is not written.  `starts`: the first row of each of the sort's `buckets`, which take whole blocks of
// 128 rows, and the end.
int quant_sorted(const void* x, int dtype, void* out_q, float* out_s, const int32_t* inverse, const int32_t* sorted_ids,
                 const int32_t* starts, int buckets, int64_t tokens, int topk, int64_t hidden, float eps, cudaStream_t st);

// moe_align.cu: the sort (arguments as sglb200_moe_align_block_size).  `inverse` (or nullptr): the place of every flat index in
// the order, -1 for an id that is no bucket's.  `zeros` (or nullptr): zeros[0] and zeros[1] are set to 0.
int align_block_size(const int32_t* topk_ids, int64_t numel, int num_experts, int block_size, int32_t* sorted_token_ids,
                     int32_t* expert_ids, int32_t* num_tokens_post_pad, int32_t* cumsum_buffer, int pad_sorted_token_ids,
                     void* workspace, int64_t workspace_bytes, int32_t* inverse, int32_t* zeros, cudaStream_t st);

// moe_align.cu: the sort of few ids (as sglb200_moe_align_block_size, padding written) and the quantizer of the same layer's
// activations (groups of 128) in one launch, where `align_quant_fits`.  `inverse` and `zeros` as above.
bool align_quant_fits(const void* x, int64_t numel, int buckets);
int align_quant(const int32_t* ids, int64_t numel, int buckets, int block_size, int32_t* sorted, int32_t* expert_ids,
                int32_t* post_pad, int32_t* cumsum, const void* x, int dtype, void* out_q, float* out_s, int64_t tokens,
                int64_t hidden, float eps, float fp8_max, int32_t* inverse, int32_t* zeros, cudaStream_t st);

// What the current GPU holds of clusters (the driver is asked once per device).
const ClusterFits& cluster_fits();

// gemm.cu: the dense product (arguments as sglb200_fp8_blockwise_scaled_mm).  `after_quantizer`: the kernel before it in
// the stream is this library's quantizer, launched by the same call, so that the weights may be fetched while that runs.
int scaled_mm(const void* A, const void* B, const float* a_s, const float* b_s, void* C, const void* bias, int64_t M, int64_t N,
              int64_t K, int64_t as_stride_m, int64_t as_stride_k, int out_dtype, void* workspace, int64_t workspace_bytes,
              bool after_quantizer, cudaStream_t st);

// gemm.cu: the product of sorted rows with their experts (arguments as sglb200_fp8_blockwise_grouped_mm).  Padding other than
// kKept: the rows are as the sort leaves them, every expert's padding after its rows, and nobody reads what belongs to a padding
// row; without `scatter`, `row_weights` then apply to the sorted rows.  kSkipped: 32-row quadrants of padding may hold anything
// and are not stored.
enum class Padding { kKept, kUnread, kSkipped };
int grouped_mm_any(const void* A, const float* a_s, const void* B, const float* b_s, void* C, const int32_t* sorted_token_ids,
                   const int32_t* expert_ids, const int32_t* num_rows_dev, const float* row_weights, int64_t max_rows,
                   int64_t numel, int num_experts, int64_t N, int64_t K, int scatter, int out_dtype, Padding padding,
                   cudaStream_t st);
// The experts' first product with activation and re-quantisation in its epilogue (see there).
int grouped_act_mm(const void* A, const float* a_s, const void* w13, const float* b_s, void* out_q, float* out_s,
                   const int32_t* sorted_ids, const int32_t* expert_ids, const int32_t* num_rows_dev, int64_t max_rows,
                   int64_t numel, int num_experts, int64_t I, int64_t K, int dtype, cudaStream_t st);

// gemm_rows.cu: the dense product for few activation rows, and the expert-grouped one on rows sorted with a padding of
// 16 (`cumsum` = padded starts of the buckets, as the sort writes them; bucket 0 = filtered ids is skipped).
// `gather_topk` > 0: A and a_s have a row per token, fetched by sorted slot / gather_topk; 0: a row per sorted row.
// `nt` = activation rows per tile: 32 or 64.  `next_tile`: a zero (or nullptr), see RowsParams.
// `rows_grouped_single`: such a product has no more tiles than CTAs.
int rows_dense_mm(const void* A, const void* B, const float* a_s, const float* b_s, void* C, const void* bias, int64_t M,
                  int64_t N, int64_t K, int64_t as_stride_m, int64_t as_stride_k, int out_dtype, bool after_quantizer,
                  cudaStream_t st);
int rows_grouped_mm(const void* A, int64_t a_rows, int64_t as_stride, const float* a_s, const void* B, const float* b_s, void* C,
                    const int32_t* cumsum, const int32_t* sorted_ids, const float* row_weights, int64_t max_rows,
                    int64_t numel, int num_experts, int64_t N, int64_t K, int gather_topk, int scatter, int out_dtype, int nt,
                    int32_t* next_tile, bool pdl, cudaStream_t st);
bool rows_grouped_single(int64_t max_rows, int num_experts, int64_t N, int nt);

// gemm_small.cu: quantise + multiply in one launch; whether a problem is one for it.
bool small_linear_fits(int64_t M, int64_t N, int64_t K);
int small_linear(const void* x, int dtype, const void* B, const float* b_s, void* C, const void* bias, int64_t M, int64_t N,
                 int64_t K, cudaStream_t st);
int small_linear_status();
int small_linear_status_clear();

// gemm_rows.cu: status word of its kernels (0 ok, 1 a wait expired, -1 not readable), and its reset.
int rows_gemm_status();
int rows_gemm_status_clear();

}  // namespace sglb200
