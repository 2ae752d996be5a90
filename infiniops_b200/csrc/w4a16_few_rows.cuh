// The W4A16 / W8A16 GEMM for at most 16 activation rows per weight matrix (decode): what the dispatch
// in w4a16_gemm.cu hands to the kernel in w4a16_few_rows.cu.
#ifndef INFINIOPS_B200_W4A16_FEW_ROWS_CUH_
#define INFINIOPS_B200_W4A16_FEW_ROWS_CUH_

#include "common.cuh"

namespace iob {

constexpr int kFewRows = 16;           // most activation rows of one weight matrix (or routing block)

struct FewRowsParams {
  const void* a;           // [rows][K], 16-byte aligned
  const uint32_t* wq;      // [E][K/16][2N] (4-bit) or [E][K/16][4N] (8-bit) words
  const void* scales;      // [E][G][N]
  const uint32_t* zeros;   // [E][G][N/8] (4-bit), [E][G][N/4] (8-bit) or null
  const void* bias;        // [E][N] or null
  void* out;               // [rows][out_ld], this problem's columns from out_col0 on
  int m, n, k, groups, group_size;
  int layout;              // scale / zero-point layout: 0 plain, 1 provider
  int out_ld, out_col0;
  // routed form
  const int32_t* sorted_ids;
  const int32_t* expert_ids;
  const int32_t* num_post_pad;
  const float* topk_weights;
  int top_k, block_size, mul_weights, out_rows, a_sorted, out_sorted, blocks, experts;
  int fuse_silu;           // columns are gate and up interleaved in runs of 16; stores silu(gate) * up, [rows][N/2]
};

enum class FewRowsWeights { kInt4, kInt8, kFloat8 };

// Launches the kernel (dense, or routed when `expert_ids` is set).
int FewRowsGemm(int a_dtype, FewRowsWeights weights, const FewRowsParams& p, cudaStream_t stream);

}  // namespace iob
#endif  // INFINIOPS_B200_W4A16_FEW_ROWS_CUH_
