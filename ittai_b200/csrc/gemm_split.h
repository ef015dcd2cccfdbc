// The split-K GEMM of gemm_split_sm100.cu: the rule that picks it and its launch.
#pragma once
#include <cuda.h>

namespace ittai {
struct GemmArgs;
// Whether the split-K kernel is the faster one for this shape.
bool gemm_split_wins(int m, int n, int n_sms);
// `tm_b`: boxes of 128 rows; W is constant (fetched ahead of the kernels that may still be running).
int gemm_split_launch(const CUtensorMap& tm_a, const CUtensorMap& tm_b, const GemmArgs& g, int n_sms, cudaStream_t st);
}  // namespace ittai
