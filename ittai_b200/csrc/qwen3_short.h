// Projections of forwards of at most kShortTokens tokens (qwen3_short.cu; up to kNarrowTokens on warp-level MMAs), queued by qwen3_prefill.cu.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>

#include "../../include/ittai_b200.h"

namespace ittai {
constexpr int kShortTokens = 48, kNarrowTokens = 32, kShortParts = ITTAI_Q3_D / 32;      // `stats`: [tokens][kShortParts] sums of squares of h's rows
struct ShortMaps { CUtensorMap qkv, o, gu, down; };                   // the stacked weights of all layers
int short_maps(ShortMaps* m, const IttaiQwen3Prefill* p);
int short_qkv(const ShortMaps& m, const IttaiQwen3Prefill* p, int layer, const IttaiQkRope& r, const void* gain, const float* stats, cudaStream_t st);
int short_o(const ShortMaps& m, const IttaiQwen3Prefill* p, int layer, float* stats, cudaStream_t st);
int short_gate_up(const ShortMaps& m, const IttaiQwen3Prefill* p, int layer, const void* gain, const float* stats, cudaStream_t st);
int short_down(const ShortMaps& m, const IttaiQwen3Prefill* p, int layer, float* stats, cudaStream_t st);
}  // namespace ittai
