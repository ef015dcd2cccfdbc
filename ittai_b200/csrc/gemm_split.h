// The split-K GEMM of gemm_split_sm100.cu: the rule that picks it and its launch.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>

#include "../../include/ittai_b200.h"

namespace ittai {
struct GemmArgs;
// ittai_gemm_bf16_launch with the RMSNorm in front of the GEMM done inside it: `gain` [K] bf16, row_stats the partial sums of
// A's rows.  Only where gemm_split_wins (ITTAI_E_ARG otherwise).
int gemm_normed_launch(const IttaiGemm* a, const void* gain, cudaStream_t st);
// Whether the split-K kernel is the faster one for this shape.
bool gemm_split_wins(int m, int n, int n_sms);
// Rows of a tile of A (32, 64 or 128), and of a box of its tensor map.
int gemm_split_rows(int m, int n, int k, int n_sms);
// `tm_w`: boxes of 128 rows; W is constant (fetched ahead of the kernels that may still be running).
int gemm_split_launch(const CUtensorMap& tm_a, const CUtensorMap& tm_w, const GemmArgs& g, int tile_rows, int n_sms, cudaStream_t st);
}  // namespace ittai
