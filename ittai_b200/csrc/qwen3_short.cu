// The four projections of a Qwen3 layer for forwards of at most 32 tokens (a search query, a short prompt), and below for 33 to 48.
//
// At this size a projection is its weights on their way and one chain of latencies.  As split-K GEMMs on tcgen05 (gemm_split_sm100.cu) the chain
// was 9000 cycles for 23 tokens: activations through TMA, row statistics, a pass that normalises the landed tile in shared memory and
// fences it for the async proxy, 16 MMAs that read the weights out of shared memory (40 cycles each), a commit, tensor memory back into
// registers, partials in 4-byte stores.  Here everything between the activations and the output stays with the threads:
//
// * A cluster of four CTAs shares K out; a CTA has 128 (QKV: one head), 192 (gate/up) or 32 (O, down) weight rows of its quarter, 32 to 96 KB,
//   on their way to shared memory ahead of griddepcontrol.wait, and holds them (gate/up: half of them) in registers as MMA operands by then.
// * The activations of the quarter come by plain loads, whole rows of a warp, are normalised in registers on the way to shared memory with the
//   rounding steps of rmsnorm_rows_kernel (1 / rms from 32 partial sums of squares, one a lane, that the kernel before left), and meet the
//   weights in mma.sync m16n8k16: 32 rows x one K chunk x 8 NT tokens a warp.
// * Chunks meet in shared memory, quarters through st.async, 16 bytes at a time, in the CTA that finishes the token (token n: rank n mod 4,
//   where a warp or eight lanes hold a whole row piece for the head norm, the rotation or the statistics); sums in the order of chunks, then
//   of ranks from the last one on.  No order is the better one: against the eager module's 64 tokens behind a prompt of 32, which near-ties decide,
//   0 1 2 3 / 3 2 1 0 / chunks in pairs agree in 60 / 62 / 62, at an rms distance of 9.5e-3 / 9.5e-3 / 9.4e-3, the split-K GEMMs in 62 at 10.0e-3; the
//   test of that fixture asks for 61, which the ascending order misses and this one does not (pairs cost 4 % at 17 to 24 tokens).  Over many
//   prompts, against 64 bits, the error is that of the kernels before (700 prompts of 47 and 31 more tokens: logits +0.01 +- 0.15 %).
//
// Measured on a B200, a forward of 3 / 8 / 16 / 23 / 32 tokens with attn_few_kernel, us, split-K GEMMs -> this: 555 / 568 / 587 / 602 / 671 ->
// 328 / 345 / 420 / 504 / 584.  What grows with the tokens are the MMAs (legacy ones: 8 cycles each, 1150
// of gate/up's 5800 cycles at 23 tokens), the sums' way through shared memory and the activations, which 32 CTAs read from the same lines of
// L2.  Other forms while they were built, us at 3 / 23 / 32 tokens, when this took 365 / 534 / 620: weights from shared memory as the 128-row operand of
// tcgen05.mma, everything else alike 455 / 582 / 618; tokens as the 128-row operand in tensor memory 603 / 692 / 744 (padded rows cost what real
// ones do: 54 cycles an MMA of 128 columns); one kernel for all four projections, its sizes arguments 528 / 654 / 697; QKV in 16 warps of 64
// registers instead of 8 of 128 (their sums meet in four chunks instead of two) 369 / 554 / 666.
#include <cuda.h>

#include "gemm2_common.cuh"
#include "qwen3_short.h"

namespace ittai {
namespace brief {

constexpr int D = ITTAI_Q3_D, HD = ITTAI_Q3_HD, NKV = ITTAI_Q3_NKV, DQ = ITTAI_Q3_DQ, DQKV = ITTAI_Q3_DQKV, DGU = ITTAI_Q3_DGU, FF = ITTAI_Q3_FF;
constexpr int kRanks = 4;                    // CTAs that share K out
constexpr int kParts = D / 32;               // partial sums of squares of a row: one per 32-column tile of O and down
constexpr uint32_t kSpin = 1u << 18;         // polls that park the warp for up to 2 us
enum { kQkv = 0, kGateUp = 1, kResidual = 2 };

template <int EPI, int K>
struct Shape {
    static constexpr int kSlice = K / kRanks;                                       // columns of a CTA
    static constexpr int kRows = EPI == kQkv ? 128 : EPI == kGateUp ? 192 : 32;      // weight rows of a CTA
    static constexpr int kChunk = EPI == kResidual ? 64 : 128;                         // columns of a warp
    static constexpr int kChunks = kSlice / kChunk, kGroups = kRows / 32;            // warps: a chunk x 32 rows each
    static constexpr int kWarps = kChunks * kGroups, kThreads = 32 * kWarps;
    static constexpr int kSteps = kChunk / 16;                                       // MMAs along K
    static constexpr int kHeld = EPI == kQkv ? 8 : 4;                                // of which as many have their weights in registers ahead of the wait
    static constexpr int kXLd = kSlice * 2 + 16;                                     // bytes per token in shared memory: eight rows on different banks
    static constexpr int kPartLd = kRows + 4;                                        // floats per token of a chunk's sums, likewise
    static constexpr int kPieces = kSlice / 256;                                     // 16-byte pieces of a token row per lane
    static_assert(kSlice % 256 == 0 && kSteps >= kHeld, "whole warps per token");
    static_assert(EPI != kQkv || kWarps >= 8, "a warp for every token that a CTA finishes");
};
template <int NT, int EPI, int K>
struct Plan {
    using S = Shape<EPI, K>;
    static constexpr uint32_t kW = S::kRows * S::kSlice * 2, kPart = S::kChunks * 8 * NT * S::kPartLd * 4;
    static constexpr uint32_t kX = kW > kPart ? kW : kPart;                          // offset: the sums of the chunks take the place of the weights
    static constexpr uint32_t kRecv = (kX + 8 * NT * S::kXLd + 127) / 128 * 128;     // offset: [ranks][2 NT tokens][rows] sums of the quarters
    static constexpr uint32_t kNeed = kRecv + kRanks * 2 * NT * S::kRows * 4 + 1024;
    // Asked for, whether needed or not, from 9 tokens on: O-proj so much that an SM takes two of its CTAs and nothing beside them, QKV (25 to 32 tokens)
    // so much that it takes one.  A kernel starts while the one in front holds 128 of the 148 SMs: what fits three times on an SM goes to the empty
    // ones by threes, and the slowest CTA is what the next kernel waits for.  Texts of 12 / 16 / 23 / 32 tokens through the embedder, us, O-proj as
    // little as needed 484 / 496 / 605 / 657, two and 74 KB (76 KB each) beside them 485 / 498 / 576 / 659, this and 106 KB 474 / 487 / 566 / 655, one a SM
    // 533 / 545 / 616 / 672: gate/up then finds no room beside it.  QKV as little as needed, 32 tokens in one and three texts 666 and 661, this 657 and
    // 639; at 9 and 16 tokens 3 and 1 % slower.  Up to 8 tokens every form lost 2 to 10 %.
    static constexpr uint32_t kAtLeast = EPI == kQkv && NT == 4 ? 114 << 10 : EPI == kResidual && K == DQ && NT > 1 ? 98 << 10 : 0;
    static constexpr uint32_t kSmem = kNeed > kAtLeast ? kNeed : kAtLeast;
};

struct Args {
    const bf16* x;           // [T][K]
    const bf16* gain;        // [D] norm in front of the projection (QKV, gate/up)
    const float* stats_in;   // [T][kParts] sums of squares of x's rows (QKV, gate/up)
    bf16* out;               // QKV: [T][DQKV], q heads; gate/up: [T][FF]; O, down: [T][D]
    const bf16* res;         // O, down: [T][D]
    float* stats_out;        // O, down: [T][kParts]
    int tokens, w_row;       // first weight row of this layer in the map
    float eps;
    uint32_t* status;
    IttaiQkRope rope;
};

__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldsm2(uint32_t& r0, uint32_t& r1, uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x2.shared.b16 {%0,%1}, [%2];" : "=r"(r0), "=r"(r1) : "r"(addr) : "memory");
}
__device__ __forceinline__ void mma16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ float4 lds_f4(uint32_t addr) {
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ void st_async_f32x4(uint32_t dst, float4 v, uint32_t bar) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%1, %2, %3, %4}, [%5];"
                 ::"r"(dst), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w), "r"(bar) : "memory");
}
__device__ __forceinline__ uint32_t map_addr(uint32_t addr, int rank) {
    uint32_t a;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(addr), "r"(rank));
    return a;
}
__device__ __forceinline__ float4 add4(float4 a, float4 b) { return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w); }

template <int NT, int EPI, int K>
__global__ void __launch_bounds__(Shape<EPI, K>::kThreads, 2) proj_kernel(const __grid_constant__ CUtensorMap tm_w, const Args a) {
    using S = Shape<EPI, K>;
    using P = Plan<NT, EPI, K>;
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char* sm = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    __shared__ unsigned long long landed, arrived;
    const int warp = warp_index(), lane = threadIdx.x & 31;
    const int rank = blockIdx.x % kRanks, tile = blockIdx.x / kRanks;
    const int own = (a.tokens - rank + kRanks - 1) / kRanks;         // tokens that this CTA finishes (0 where there are fewer than ranks)
    if (threadIdx.x == 0) {
        mbar_init(&landed, 1);
        mbar_init(&arrived, 1);
        fence_mbar_init();
        mbar_expect_tx(&landed, P::kW);
        mbar_expect_tx(&arrived, (uint32_t)(own > 0 ? own : 0) * S::kRows * 4 * kRanks);
#pragma unroll 1
        for (int j = 0; j < S::kSlice / 64; ++j)
            tma_load_2d(sm + j * S::kRows * 128, &tm_w, rank * S::kSlice + 64 * j, a.w_row + tile * S::kRows, &landed);
    }
    __syncthreads();
    // another CTA's shared memory may be written only once that CTA runs; waited for ahead of the first write
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    pdl_trigger();

    const int chunk = warp / S::kGroups, group = warp % S::kGroups;
    const uint32_t w0 = smem_u32(sm), x0 = w0 + P::kX;
    // row of this lane in the ldmatrix of a 16 x 16 tile of weights: rows 0-7, 8-15, then the same with the upper eight columns
    const int wrow = 32 * group + (lane & 15), whalf = lane >> 4;
    auto load_w = [&](uint32_t (&f)[4], int mt, int ks) {
        const int c = chunk * S::kChunk + 16 * ks;                    // column of the slice
        const int row = wrow + 16 * mt;
        ldsm4(f, w0 + (uint32_t)(c >> 6) * (S::kRows * 128) + (uint32_t)row * 128 + (uint32_t)((((c & 63) >> 3) + whalf) ^ (row & 7)) * 16);
    };
    uint4 gain = make_uint4(0u, 0u, 0u, 0u);
    if constexpr (EPI != kResidual) gain = *reinterpret_cast<const uint4*>(a.gain + rank * S::kSlice + 8 * lane);
    // The rotary arguments lie in a line of the kernel's parameters that nothing ahead of the wait has read: fetched behind it, they cost 500
    // cycles: forwards of 3 / 8 / 23 / 32 tokens 365 / 390 / 534 / 621 -> 351 / 372 / 537 / 617 us.  The head norm's gain comes from HBM like the other one.
    IttaiQkRope rope;
    uint2 hgain = make_uint2(0u, 0u);
    if constexpr (EPI == kQkv) {
        rope = a.rope;
        asm volatile("" : "+l"(rope.pos), "+l"(rope.seq), "+l"(rope.slot), "+l"(rope.rope));
        if (tile < 24) hgain = *reinterpret_cast<const uint2*>(reinterpret_cast<const bf16*>(tile < 16 ? rope.qn : rope.kn) + 4 * lane);
    }
    bool ok = mbar_wait_bounded(&landed, 0, kSpin);
    __syncwarp();                                                     // the lanes left the wait one by one
    uint32_t wf[S::kHeld][2][4];
#pragma unroll
    for (int ks = 0; ks < S::kHeld; ++ks) { load_w(wf[ks][0], 0, ks); load_w(wf[ks][1], 1, ks); }
    if constexpr (EPI == kQkv) asm volatile("" : "+r"(hgain.x), "+r"(hgain.y));
    if constexpr (EPI != kResidual) asm volatile("" : "+r"(gain.x), "+r"(gain.y), "+r"(gain.z), "+r"(gain.w));    // arrived: a load left open may be scheduled behind the wait
    // addresses ahead of the wait: behind it only requests with constant offsets
    const bf16* xp = a.x + (size_t)warp * K + rank * S::kSlice + 8 * lane;
    const float* sp = EPI != kResidual ? a.stats_in + warp * kParts + lane : nullptr;
    asm volatile("" : "+l"(xp), "+l"(sp));
    pdl_wait();

    // ---- activations: a warp takes whole token rows of the slice
    constexpr int kRounds = (8 * NT + S::kWarps - 1) / S::kWarps;
    uint4 xv[kRounds][S::kPieces];
    float ss[kRounds];
#pragma unroll
    for (int i = 0; i < kRounds; ++i) {
        const int n = warp + i * S::kWarps;
        ss[i] = 0.f;
#pragma unroll
        for (int p = 0; p < S::kPieces; ++p) xv[i][p] = make_uint4(0u, 0u, 0u, 0u);
        if (n < a.tokens) {
#pragma unroll
            for (int p = 0; p < S::kPieces; ++p) xv[i][p] = ldcg128(xp + (size_t)i * S::kWarps * K + 256 * p);
            if constexpr (EPI != kResidual) ss[i] = ldcgf(sp + i * S::kWarps * kParts);
        }
    }
    // what the epilogue reads, ahead of the main loop.  O, down: eight lanes a token, four columns each; QKV: a warp a token
    const int quad = threadIdx.x & 7, slot8 = threadIdx.x >> 3;
    uint2 res = make_uint2(0u, 0u), cosr = res, sinr = res;
    bf16* dst = nullptr;
    if constexpr (EPI == kResidual) {
        if (slot8 < own) res = *reinterpret_cast<const uint2*>(a.res + (size_t)(kRanks * slot8 + rank) * D + tile * 32 + 4 * quad);
    }
    int pos = 0, seq = 0, row = 0;
    const int n_own = kRanks * warp + rank;                           // QKV: the token of this warp
    if constexpr (EPI == kQkv) {
        if (warp < own) {
            pos = rope.pos[n_own];
            if (tile >= 16) { seq = rope.seq[n_own]; row = rope.slot[n_own]; }
        }
    }
#pragma unroll
    for (int i = 0; i < kRounds; ++i) {
        const int n = warp + i * S::kWarps;
        if (n < 8 * NT) {
            if constexpr (EPI != kResidual) {
                const float rstd = rsqrt_full(warp_sum(ss[i]) * (1.0f / D) + a.eps);
                uint32_t* u = reinterpret_cast<uint32_t*>(&xv[i][0]);
                const uint32_t gw[4] = {gain.x, gain.y, gain.z, gain.w};
#pragma unroll
                for (int j = 0; j < 4; ++j) u[j] = mul_bf16x2(pack_bf16x2(bf_lo(u[j]) * rstd, bf_hi(u[j]) * rstd), gw[j]);
            }
#pragma unroll
            for (int p = 0; p < S::kPieces; ++p) *reinterpret_cast<uint4*>(sm + P::kX + n * S::kXLd + 512 * p + 16 * lane) = xv[i][p];
        }
    }
    if constexpr (EPI == kQkv) {
        if (warp < own) {
            if (tile < 24) {
                const bf16* rp = reinterpret_cast<const bf16*>(rope.rope) + (size_t)pos * HD + 4 * (lane & 15);
                cosr = *reinterpret_cast<const uint2*>(rp); sinr = *reinterpret_cast<const uint2*>(rp + HD / 2);
            }
            dst = tile < 16 ? a.out + (size_t)n_own * DQKV + tile * HD + 4 * lane
                            : reinterpret_cast<bf16*>(tile < 24 ? rope.kcache_layer : rope.vcache_layer) + (((size_t)seq * NKV + (tile & 7)) * rope.kv_cap + row) * HD + 4 * lane;
        }
    }
    __syncthreads();

    // ---- 32 rows x chunk x 8 NT tokens
    float acc[2][NT][4];
#pragma unroll
    for (int m = 0; m < 2; ++m)
#pragma unroll
        for (int n = 0; n < NT; ++n) acc[m][n][0] = acc[m][n][1] = acc[m][n][2] = acc[m][n][3] = 0.f;
    const uint32_t xl = x0 + (uint32_t)((lane & 7) + 8 * (lane >> 4)) * S::kXLd + chunk * S::kChunk * 2 + 16 * ((lane >> 3) & 1);
#pragma unroll
    for (int ks = 0; ks < S::kSteps; ++ks) {
        uint32_t b[NT][2];
#pragma unroll
        for (int n = 0; n + 1 < NT; n += 2) {
            uint32_t f[4];
            ldsm4(f, xl + 8 * n * S::kXLd + 32 * ks);
            b[n][0] = f[0]; b[n][1] = f[1]; b[n + 1][0] = f[2]; b[n + 1][1] = f[3];
        }
        if constexpr (NT & 1) ldsm2(b[NT - 1][0], b[NT - 1][1], x0 + (uint32_t)((lane & 7) + 8 * (NT - 1)) * S::kXLd + chunk * S::kChunk * 2 + 16 * ((lane >> 3) & 1) + 32 * ks);
        if (ks >= S::kHeld) { load_w(wf[ks % S::kHeld][0], 0, ks); load_w(wf[ks % S::kHeld][1], 1, ks); }
#pragma unroll
        for (int n = 0; n < NT; ++n) {
            mma16816(acc[0][n], wf[ks % S::kHeld][0], b[n][0], b[n][1]);
            mma16816(acc[1][n], wf[ks % S::kHeld][1], b[n][0], b[n][1]);
        }
    }
    if constexpr (S::kSteps > S::kHeld) __syncthreads();              // the weights in shared memory have been read by all
    float* part = reinterpret_cast<float*>(sm) + (size_t)chunk * 8 * NT * S::kPartLd;
    const int g = lane >> 2, t = lane & 3;
#pragma unroll
    for (int m = 0; m < 2; ++m)
#pragma unroll
        for (int n = 0; n < NT; ++n)
#pragma unroll
            for (int i = 0; i < 4; ++i) part[(8 * n + 2 * t + (i & 1)) * S::kPartLd + 32 * group + 16 * m + g + 8 * (i >> 1)] = acc[m][n][i];
    __syncthreads();

    // ---- sums of the chunks, four rows of a token at a time, to the rank that finishes the token
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    constexpr int kQuads = S::kRows / 4;
    const uint32_t recv = w0 + P::kRecv;
#pragma unroll 1
    for (int i = threadIdx.x; i < a.tokens * kQuads; i += S::kThreads) {
        const int n = i / kQuads, q = i % kQuads;
        float4 v = lds_f4(w0 + (uint32_t)(n * S::kPartLd + 4 * q) * 4);
#pragma unroll
        for (int c = 1; c < S::kChunks; ++c) v = add4(v, lds_f4(w0 + (uint32_t)((c * 8 * NT + n) * S::kPartLd + 4 * q) * 4));
        const int to = n % kRanks;
        st_async_f32x4(map_addr(recv + (uint32_t)((rank * 2 * NT + n / kRanks) * S::kRows + 4 * q) * 4, to), v, map_addr(smem_u32(&arrived), to));
    }
    bool came = true;
    {
        uint32_t spins = 0;
        while (!mbar_try_wait_cluster(&arrived, 0)) { if (++spins >= (kSpin << 4)) { came = false; break; } }
    }
    __syncwarp();
    auto total = [&](int slot, int q) {                              // sums of the ranks, the last one's first
        float4 v = lds_f4(recv + (uint32_t)(((kRanks - 1) * 2 * NT + slot) * S::kRows + 4 * q) * 4);
#pragma unroll
        for (int r = kRanks - 2; r >= 0; --r) v = add4(v, lds_f4(recv + (uint32_t)((r * 2 * NT + slot) * S::kRows + 4 * q) * 4));
        return v;
    };
    if constexpr (EPI == kQkv) {
        if (warp < own) {
            const float4 v = total(warp, lane);
            uint32_t y0 = pack_bf16x2(v.x, v.y), y1 = pack_bf16x2(v.z, v.w);
            if (tile < 24) {
                // the rounding steps of qk_rope_scatter_kernel on packed pairs; the partner element 64 columns away is 16 lanes away
                const float f0 = bf_lo(y0), f1 = bf_hi(y0), f2 = bf_lo(y1), f3 = bf_hi(y1);
                const float rstd = rsqrt_full(warp_sum(fmaf(f0, f0, fmaf(f1, f1, fmaf(f2, f2, f3 * f3)))) * (1.0f / HD) + rope.eps);
                const uint32_t n0 = mul_bf16x2(pack_bf16x2(f0 * rstd, f1 * rstd), hgain.x), n1 = mul_bf16x2(pack_bf16x2(f2 * rstd, f3 * rstd), hgain.y);
                const uint32_t neg = lane < 16 ? 0x80008000u : 0u;
                const uint32_t o0 = __shfl_xor_sync(0xffffffffu, n0, 16) ^ neg, o1 = __shfl_xor_sync(0xffffffffu, n1, 16) ^ neg;
                y0 = add_bf16x2(mul_bf16x2(n0, cosr.x), mul_bf16x2(o0, sinr.x));
                y1 = add_bf16x2(mul_bf16x2(n1, cosr.y), mul_bf16x2(o1, sinr.y));
            }
            *reinterpret_cast<uint2*>(dst) = make_uint2(y0, y1);
        }
    } else if constexpr (EPI == kGateUp) {
#pragma unroll 1
        for (int i = threadIdx.x; i < own * kQuads; i += S::kThreads) {
            const int slot = i / kQuads, q = i % kQuads;
            const float4 v = total(slot, q);
            // adjacent rows are (gate, up): act = bf16(bf16(silu(bf16 gate)) * bf16 up)
            const float g0 = bf16r(v.x), u0 = bf16r(v.y), g1 = bf16r(v.z), u1 = bf16r(v.w);
            *reinterpret_cast<uint32_t*>(a.out + (size_t)(kRanks * slot + rank) * FF + tile * (S::kRows / 2) + 2 * q) =
                pack_bf16x2(bf16r(g0 / (1.0f + expf(-g0))) * u0, bf16r(g1 / (1.0f + expf(-g1))) * u1);
        }
    } else {
        if (warp < (own + 3) / 4) {                                   // whole warps: four tokens each
            const float4 v = total(slot8 < own ? slot8 : 0, quad);
            const uint2 o = make_uint2(pack_bf16x2(bf_lo(res.x) + bf16r(v.x), bf_hi(res.x) + bf16r(v.y)), pack_bf16x2(bf_lo(res.y) + bf16r(v.z), bf_hi(res.y) + bf16r(v.w)));
            const float a0 = bf_lo(o.x), a1 = bf_hi(o.x), a2 = bf_lo(o.y), a3 = bf_hi(o.y);
            float s = fmaf(a0, a0, fmaf(a1, a1, fmaf(a2, a2, a3 * a3)));
#pragma unroll
            for (int m = 1; m < 8; m <<= 1) s += __shfl_xor_sync(0xffffffffu, s, m);
            if (slot8 < own) {
                const int n = kRanks * slot8 + rank;
                *reinterpret_cast<uint2*>(a.out + (size_t)n * D + tile * 32 + 4 * quad) = o;
                if (quad == 0) a.stats_out[n * kParts + tile] = s;
            }
        }
    }
    if (!__syncthreads_and(ok && came)) {
        // A CTA that gave up must not leave before what is owed to it has come: all send, also where their waits ran out.  Should a send take
        // longer than this wait, the barrier holds the CTA until the others have left (threads that have exited count as arrived).
        bool all = false;
        for (uint32_t spins = 0; !all && spins < (kSpin << 4); ++spins) all = mbar_try_wait_cluster(&arrived, 0);
        if (!__syncthreads_and(all)) {
            asm volatile("barrier.cluster.arrive.release;" ::: "memory");
            asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
        }
        if (threadIdx.x == 0) {
            if (atomicCAS(&a.status[0], 0u, (uint32_t)ITTAI_ST_GEMM_TIMEOUT) == 0u) { a.status[1] = blockIdx.x; a.status[2] = (uint32_t)K; }
            const long long t0 = clock64();                           // copies still in flight land before the shared memory is handed back
            while (clock64() - t0 < 2000000) {}
        }
        __syncthreads();
    }
}

// ---- 33 to 48 tokens ------------------------------------------------------------------------------------------------------
// The same flow on tcgen05, whose MMA costs the same 40 cycles for 16 and for 64 tokens (it is the weights' 4 KB a step, read out of shared memory,
// that take them): weights as the 128-row operand, activations normalised in registers on the way to where the MMA reads them, the
// accumulator through shared memory, so that a token's sums lie side by side.  A cluster of eight shares the K of O and down (64 rows a CTA).
// Forwards of 33 / 40 / 48 tokens with attn_few_kernel, us: split-K GEMMs 725 / 742 / 769, this 649 / 679 / 710 (up to 32 tokens see the top of the
// file).  The line at 48: an instantiation for 64 tokens, whose gate/up leaves no room in shared memory for its neighbours, took 986 against 957
// when it was tried.  Sums of the ranks in ascending order.
constexpr int kWideThreads = 256;
template <int TN, int EPI, int K>
struct WideShape {
    static constexpr int kRanks = EPI == kResidual ? 8 : 4;                          // CTAs that share K out
    static constexpr int kSlice = K / kRanks, kBlocks = kSlice / 64;                 // columns of a CTA
    static constexpr int kRows = EPI == kQkv ? 128 : EPI == kGateUp ? 192 : 64;      // weight rows of a CTA
    static constexpr int kAccs = kRows > 128 ? 2 : 1;                                // MMAs of 128 rows: the second one starts at row 64
    static constexpr int kSlots = TN / kRanks;                                       // tokens that a CTA finishes at most
    static constexpr int kPieces = kSlice / 8;                                       // 16-byte pieces of a token row
    static constexpr int kRounds = TN * kPieces / kWideThreads;
    static constexpr int kMine = (kSlots + kWideThreads / 32 - 1) / (kWideThreads / 32);       // QKV: tokens that a warp finishes
    static constexpr int kPartLd = kRows + 4;                                        // floats per token on the way from the accumulator
    static constexpr int kQuads = kRows / 4;
    static constexpr uint32_t kW = kRows * kSlice * 2, kX = TN * kSlice * 2, kPart = TN * kPartLd * 4, kRecv = kRanks * kSlots * kRows * 4;
    static constexpr uint32_t kSmem = kW + kX + kRecv + 1024;
    static constexpr uint32_t kCols = TN * kAccs <= 64 ? 64 : 128;                      // of tensor memory: a power of two
    static_assert(kPart <= kW, "the accumulator's way out takes the place of the weights");
    static_assert(kRows >= 128 || kX >= 64 * 128, "an MMA reads 128 rows: those past the tile lie in the next block or in x");
    static_assert(TN * kPieces % kWideThreads == 0 && TN % 16 == 0, "");
};

template <int TN, int EPI, int K>
__global__ void __launch_bounds__(kWideThreads, 2) wide_kernel(const __grid_constant__ CUtensorMap tm_w, const Args a) {
    using S = WideShape<TN, EPI, K>;
    constexpr int kRanks = S::kRanks, kThreads = kWideThreads, kWarps = kThreads / 32;
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char* sm = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    unsigned char* sx = sm + S::kW;
    __shared__ unsigned long long landed, acc_full, arrived;
    __shared__ uint32_t tmem_slot;
    __shared__ volatile uint32_t failed;
    const int warp = warp_index(), lane = threadIdx.x & 31;
    const int rank = blockIdx.x % kRanks, tile = blockIdx.x / kRanks;
    const int own = (a.tokens - rank + kRanks - 1) / kRanks;         // tokens that this CTA finishes (0 where there are fewer than ranks)
    if (threadIdx.x == 0) {
        mbar_init(&landed, 1);
        mbar_init(&acc_full, 1);
        mbar_init(&arrived, 1);
        failed = 0;
        fence_mbar_init();
        mbar_expect_tx(&landed, S::kW);
        mbar_expect_tx(&arrived, (uint32_t)own * S::kRows * 4 * kRanks);
#pragma unroll
        for (int j = 0; j < S::kBlocks; ++j)
            tma_load_2d(sm + j * S::kRows * 128, &tm_w, rank * S::kSlice + 64 * j, a.w_row + tile * S::kRows, &landed);
    }
    if (warp == 1) tmem_alloc(&tmem_slot, S::kCols);                  // ahead of the trigger: a later kernel on this SM cannot take them first
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    // another CTA's shared memory may be written only once that CTA runs; waited for ahead of the first write
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    pdl_trigger();
    const uint32_t tmem = tmem_slot;
    uint4 gain = make_uint4(0u, 0u, 0u, 0u);
    IttaiQkRope rope;
    uint2 hgain = make_uint2(0u, 0u);
    if constexpr (EPI == kQkv) {                                      // see proj_kernel
        rope = a.rope;
        asm volatile("" : "+l"(rope.pos), "+l"(rope.seq), "+l"(rope.slot), "+l"(rope.rope));
        if (tile < 24) hgain = *reinterpret_cast<const uint2*>(reinterpret_cast<const bf16*>(tile < 16 ? rope.qn : rope.kn) + 4 * lane);
        asm volatile("" : "+r"(hgain.x), "+r"(hgain.y));
    }
    if constexpr (EPI != kResidual) {
        gain = *reinterpret_cast<const uint4*>(a.gain + rank * S::kSlice + 8 * lane);
        asm volatile("" : "+r"(gain.x), "+r"(gain.y), "+r"(gain.z), "+r"(gain.w));     // arrived: a load left open may be scheduled behind the wait
    }
    pdl_wait();

    // ---- activations: piece i of the slice is 16 bytes of token i / kPieces (with a norm a warp has a whole row)
    uint4 xv[S::kRounds];
    float ss[S::kRounds];
#pragma unroll
    for (int i = 0; i < S::kRounds; ++i) {
        const int p = threadIdx.x + i * kThreads, n = p / S::kPieces;
        xv[i] = make_uint4(0u, 0u, 0u, 0u);
        ss[i] = 0.f;
        if (n < a.tokens) {
            xv[i] = ldcg128(a.x + (size_t)n * K + rank * S::kSlice + 8 * (p % S::kPieces));
            if constexpr (EPI != kResidual) ss[i] = ldcgf(a.stats_in + n * kParts + lane);
        }
    }
    // What the epilogue reads, ahead of the main loop.  O, down: 16 lanes a token, four columns each; QKV: a warp a token
    const int quad = threadIdx.x & 15, slot16 = threadIdx.x >> 4;
    uint2 res = make_uint2(0u, 0u), cosr[S::kMine], sinr[S::kMine];
    bf16* dst[S::kMine];
    if constexpr (EPI == kResidual) {
        if (slot16 < own) res = *reinterpret_cast<const uint2*>(a.res + (size_t)(kRanks * slot16 + rank) * D + tile * 64 + 4 * quad);
    }
    int pos[S::kMine], seq[S::kMine], row[S::kMine];
    if constexpr (EPI == kQkv) {
#pragma unroll
        for (int u = 0; u < S::kMine; ++u) {
            const int n = kRanks * (warp + kWarps * u) + rank;        // the u-th token of this warp
            pos[u] = seq[u] = row[u] = 0;
            if (n < a.tokens) {
                pos[u] = rope.pos[n];
                if (tile >= 16) { seq[u] = rope.seq[n]; row[u] = rope.slot[n]; }
            }
        }
    }
#pragma unroll
    for (int i = 0; i < S::kRounds; ++i) {
        const int p = threadIdx.x + i * kThreads, n = p / S::kPieces, c = p % S::kPieces;
        if (n < a.tokens) {                                           // rows past the last token: whatever lies there, their sums are not read
            if constexpr (EPI != kResidual) {
                const float rstd = rsqrt_full(warp_sum(ss[i]) * (1.0f / D) + a.eps);
                uint32_t* u = reinterpret_cast<uint32_t*>(&xv[i]);
                const uint32_t gw[4] = {gain.x, gain.y, gain.z, gain.w};
#pragma unroll
                for (int j = 0; j < 4; ++j) u[j] = mul_bf16x2(pack_bf16x2(bf_lo(u[j]) * rstd, bf_hi(u[j]) * rstd), gw[j]);
            }
            *reinterpret_cast<uint4*>(sx + (c >> 3) * (TN * 128) + n * 128 + (((c & 7) ^ (n & 7)) << 4)) = xv[i];
        }
    }
    fence_proxy_async_smem();                                         // the MMAs read through the async proxy
    if constexpr (EPI == kQkv) {
#pragma unroll
        for (int u = 0; u < S::kMine; ++u) {
            const int n = kRanks * (warp + kWarps * u) + rank;
            cosr[u] = sinr[u] = make_uint2(0u, 0u);
            if (n < a.tokens && tile < 24) {
                const bf16* rp = reinterpret_cast<const bf16*>(rope.rope) + (size_t)pos[u] * HD + 4 * (lane & 15);
                cosr[u] = *reinterpret_cast<const uint2*>(rp); sinr[u] = *reinterpret_cast<const uint2*>(rp + HD / 2);
            }
            dst[u] = tile < 16 ? a.out + (size_t)n * DQKV + tile * HD + 4 * lane
                               : reinterpret_cast<bf16*>(tile < 24 ? rope.kcache_layer : rope.vcache_layer) + (((size_t)seq[u] * NKV + (tile & 7)) * rope.kv_cap + row[u]) * HD + 4 * lane;
        }
    }
    __syncthreads();
    if (warp == 0) {
        if (elect_one()) {
            if (mbar_wait_bounded(&landed, 0, kSpin)) {
                tc_fence_after();
                constexpr uint32_t idesc = umma_idesc_bf16(128, TN);
#pragma unroll
                for (int kb = 0; kb < S::kBlocks; ++kb) {
                    const uint64_t dw = umma_desc_sw128(sm + kb * S::kRows * 128), dx = umma_desc_sw128(sx + kb * TN * 128);
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        umma_bf16(tmem, dw + 2 * k, dx + 2 * k, idesc, kb > 0 || k > 0 ? 1u : 0u);
                        if constexpr (S::kAccs == 2) umma_bf16(tmem + TN, dw + 2 * k + (64 * 128 >> 4), dx + 2 * k, idesc, kb > 0 || k > 0 ? 1u : 0u);
                    }
                }
                umma_commit(&acc_full);
            } else {
                failed = 1;
            }
        }
        __syncwarp();
    }
    {
        bool ok = true;
        uint32_t spins = 0;
        while (!mbar_try_wait_parked(&acc_full, 0)) { if (failed || ++spins >= kSpin) { ok = false; break; } }
        if (!__all_sync(0xffffffffu, ok)) failed = 1;
        __syncwarp();
    }
    tc_fence_after();
    // ---- accumulator: warp w may touch lanes 32 (w % 4) .. + 31, a weight row each; the two warps of a lane quarter share the tokens out
    {
        float* part = reinterpret_cast<float*>(sm);                   // in place of the weights: the MMAs have read them
        const int q = warp & 3, half = (warp >> 2) * (TN / 2);
#pragma unroll
        for (int m = 0; m < S::kAccs; ++m) {
            if ((S::kRows == 64 && q >= 2) || (m == 1 && q < 2)) continue;          // no rows of this tile, or the first MMA's
#pragma unroll
            for (int c = 0; c < TN / 2; c += 8) {
                if (half + c < a.tokens) {
                    uint32_t r[8];
                    tmem_ld_32x8(tmem + ((uint32_t)(32 * q) << 16) + m * TN + half + c, r);
                    tmem_ld_wait();
#pragma unroll
                    for (int i = 0; i < 8; ++i) part[(half + c + i) * S::kPartLd + 64 * m + 32 * q + lane] = __uint_as_float(r[i]);
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) tmem_dealloc(tmem, S::kCols);
    // ---- to the ranks that finish the tokens
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    const uint32_t w0 = smem_u32(sm), recv = smem_u32(sx) + S::kX;
    for (int i = threadIdx.x; i < a.tokens * S::kQuads; i += kThreads) {
        const int n = i / S::kQuads, q = i % S::kQuads, to = n % kRanks;
        st_async_f32x4(map_addr(recv + (uint32_t)((rank * S::kSlots + n / kRanks) * S::kRows + 4 * q) * 4, to), lds_f4(w0 + (uint32_t)(n * S::kPartLd + 4 * q) * 4),
                       map_addr(smem_u32(&arrived), to));
    }
    {
        uint32_t spins = 0;
        while (!mbar_try_wait_cluster(&arrived, 0)) { if (++spins >= (kSpin << 4)) { failed = 1; break; } }
        __syncwarp();
    }
    auto total = [&](int slot, int q) {                              // sums of the ranks, in their order
        float4 v = lds_f4(recv + (uint32_t)(slot * S::kRows + 4 * q) * 4);
#pragma unroll
        for (int r = 1; r < kRanks; ++r) v = add4(v, lds_f4(recv + (uint32_t)((r * S::kSlots + slot) * S::kRows + 4 * q) * 4));
        return v;
    };
    if constexpr (EPI == kQkv) {
#pragma unroll
        for (int u = 0; u < S::kMine; ++u) {
            if (warp + kWarps * u >= own) break;
            const float4 v = total(warp + kWarps * u, lane);
            uint32_t y0 = pack_bf16x2(v.x, v.y), y1 = pack_bf16x2(v.z, v.w);
            if (tile < 24) {
                // the rounding steps of qk_rope_scatter_kernel on packed pairs; the partner element 64 columns away is 16 lanes away
                const float f0 = bf_lo(y0), f1 = bf_hi(y0), f2 = bf_lo(y1), f3 = bf_hi(y1);
                const float rstd = rsqrt_full(warp_sum(fmaf(f0, f0, fmaf(f1, f1, fmaf(f2, f2, f3 * f3)))) * (1.0f / HD) + rope.eps);
                const uint32_t n0 = mul_bf16x2(pack_bf16x2(f0 * rstd, f1 * rstd), hgain.x), n1 = mul_bf16x2(pack_bf16x2(f2 * rstd, f3 * rstd), hgain.y);
                const uint32_t neg = lane < 16 ? 0x80008000u : 0u;
                const uint32_t o0 = __shfl_xor_sync(0xffffffffu, n0, 16) ^ neg, o1 = __shfl_xor_sync(0xffffffffu, n1, 16) ^ neg;
                y0 = add_bf16x2(mul_bf16x2(n0, cosr[u].x), mul_bf16x2(o0, sinr[u].x));
                y1 = add_bf16x2(mul_bf16x2(n1, cosr[u].y), mul_bf16x2(o1, sinr[u].y));
            }
            *reinterpret_cast<uint2*>(dst[u]) = make_uint2(y0, y1);
        }
    } else if constexpr (EPI == kGateUp) {
        for (int i = threadIdx.x; i < own * S::kQuads; i += kThreads) {
            const int slot = i / S::kQuads, q = i % S::kQuads;
            const float4 v = total(slot, q);
            // adjacent rows are (gate, up): act = bf16(bf16(silu(bf16 gate)) * bf16 up)
            const float g0 = bf16r(v.x), u0 = bf16r(v.y), g1 = bf16r(v.z), u1 = bf16r(v.w);
            *reinterpret_cast<uint32_t*>(a.out + (size_t)(kRanks * slot + rank) * FF + tile * (S::kRows / 2) + 2 * q) =
                pack_bf16x2(bf16r(g0 / (1.0f + expf(-g0))) * u0, bf16r(g1 / (1.0f + expf(-g1))) * u1);
        }
    } else {
        if (2 * warp < own) {                                         // whole warps: two tokens each
            const float4 v = total(slot16 < own ? slot16 : 0, quad);
            const uint2 o = make_uint2(pack_bf16x2(bf_lo(res.x) + bf16r(v.x), bf_hi(res.x) + bf16r(v.y)), pack_bf16x2(bf_lo(res.y) + bf16r(v.z), bf_hi(res.y) + bf16r(v.w)));
            const float a0 = bf_lo(o.x), a1 = bf_hi(o.x), a2 = bf_lo(o.y), a3 = bf_hi(o.y);
            float s = fmaf(a0, a0, fmaf(a1, a1, fmaf(a2, a2, a3 * a3)));
#pragma unroll
            for (int m = 1; m < 8; m <<= 1) s += __shfl_xor_sync(0xffffffffu, s, m);
            if (slot16 < own) {
                const int n = kRanks * slot16 + rank;
                *reinterpret_cast<uint2*>(a.out + (size_t)n * D + tile * 64 + 4 * quad) = o;
                if ((quad & 7) == 0) a.stats_out[n * kParts + 2 * tile + (quad >> 3)] = s;
            }
        }
    }
    __syncthreads();
    if (failed) {
        // A CTA that gave up must not leave before what is owed to it has come: all send, also where their waits ran out.  Should a send take
        // longer than this wait, the barrier holds the CTA until the others have left (threads that have exited count as arrived).
        bool all = false;
        for (uint32_t spins = 0; !all && spins < (kSpin << 4); ++spins) all = mbar_try_wait_cluster(&arrived, 0);
        if (!__syncthreads_and(all)) {
            asm volatile("barrier.cluster.arrive.release;" ::: "memory");
            asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
        }
        if (threadIdx.x == 0) {
            if (atomicCAS(&a.status[0], 0u, (uint32_t)ITTAI_ST_GEMM_TIMEOUT) == 0u) { a.status[1] = blockIdx.x; a.status[2] = (uint32_t)K; }
            const long long t0 = clock64();                           // copies still in flight land before the shared memory is handed back
            while (clock64() - t0 < 2000000) {}
        }
        __syncthreads();
    }
}

template <typename F>
static cudaError_t start(F* kernel, int threads, uint32_t smem, int ranks, int rows, const CUtensorMap& tm, const Args& a, int n_rows, int* attr_dev, cudaStream_t st) {
    int dev = 0;
    cudaGetDevice(&dev);
    if (*attr_dev != dev) {
        const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
        *attr_dev = dev;
    }
    return launch_pdl(kernel, dim3(ranks * (n_rows / rows)), dim3(threads), smem, st, ranks, tm, a);
}
template <int NT, int EPI, int K>
static cudaError_t launch_narrow(const CUtensorMap& tm, const Args& a, int n_rows, cudaStream_t st) {
    using S = Shape<EPI, K>;
    static thread_local int attr_dev = -1;
    return start(proj_kernel<NT, EPI, K>, S::kThreads, Plan<NT, EPI, K>::kSmem, kRanks, S::kRows, tm, a, n_rows, &attr_dev, st);
}
template <int TN, int EPI, int K>
static cudaError_t launch_wide(const CUtensorMap& tm, const Args& a, int n_rows, cudaStream_t st) {
    using S = WideShape<TN, EPI, K>;
    static thread_local int attr_dev = -1;
    return start(wide_kernel<TN, EPI, K>, kWideThreads, S::kSmem, S::kRanks, S::kRows, tm, a, n_rows, &attr_dev, st);
}
template <int EPI, int K>
static cudaError_t launch_any(const CUtensorMap& tm, const Args& a, int n_rows, cudaStream_t st) {
    if (a.tokens > kNarrowTokens) return launch_wide<48, EPI, K>(tm, a, n_rows, st);
    switch ((a.tokens + 7) / 8) {
        case 1: return launch_narrow<1, EPI, K>(tm, a, n_rows, st);
        case 2: return launch_narrow<2, EPI, K>(tm, a, n_rows, st);
        case 3: return launch_narrow<3, EPI, K>(tm, a, n_rows, st);
        default: return launch_narrow<4, EPI, K>(tm, a, n_rows, st);
    }
}

}  // namespace brief

int cuda_fail(cudaError_t e, const char* what);

void set_error(const char* fmt, ...);

int short_maps(ShortMaps* m, const IttaiQwen3Prefill* p) {
    using namespace brief;
    // what the GEMMs of longer forwards ask of their operands: rows are read 16 bytes at a time
    const void* rows[] = {p->wqkv, p->wo, p->wgu, p->wd, p->ln1, p->ln2, p->h, p->xn, p->qkv, p->attn, p->act};
    for (const void* r : rows) if ((uintptr_t)r & 15) { set_error("prefill: weights, gains and activations must be 16-byte aligned"); return ITTAI_E_ARG; }
    const long long L = p->n_layers;
    const bool wide = p->tokens > kNarrowTokens;
    int rc = make_tmap_bf16(&m->qkv, p->wqkv, L * DQKV, D, D, Shape<kQkv, D>::kRows);
    if (rc == ITTAI_OK) rc = make_tmap_bf16(&m->o, p->wo, L * D, DQ, DQ, wide ? WideShape<48, kResidual, DQ>::kRows : Shape<kResidual, DQ>::kRows);
    if (rc == ITTAI_OK) rc = make_tmap_bf16(&m->gu, p->wgu, L * DGU, D, D, Shape<kGateUp, D>::kRows);
    if (rc == ITTAI_OK) rc = make_tmap_bf16(&m->down, p->wd, L * D, FF, FF, wide ? WideShape<48, kResidual, FF>::kRows : Shape<kResidual, FF>::kRows);
    return rc;
}

static int done(cudaError_t e) { return e == cudaSuccess ? ITTAI_OK : cuda_fail(e, "launch of a short projection"); }

int short_qkv(const ShortMaps& m, const IttaiQwen3Prefill* p, int layer, const IttaiQkRope& r, const void* gain, const float* stats, cudaStream_t st) {
    brief::Args a{(const bf16*)p->h, (const bf16*)gain, stats, (bf16*)p->qkv, nullptr, nullptr, p->tokens, layer * brief::DQKV, p->eps, p->status, r};
    return done(brief::launch_any<brief::kQkv, brief::D>(m.qkv, a, brief::DQKV, st));
}
int short_gate_up(const ShortMaps& m, const IttaiQwen3Prefill* p, int layer, const void* gain, const float* stats, cudaStream_t st) {
    brief::Args a{(const bf16*)p->h, (const bf16*)gain, stats, (bf16*)p->act, nullptr, nullptr, p->tokens, layer * brief::DGU, p->eps, p->status, {}};
    return done(brief::launch_any<brief::kGateUp, brief::D>(m.gu, a, brief::DGU, st));
}
int short_o(const ShortMaps& m, const IttaiQwen3Prefill* p, int layer, float* stats, cudaStream_t st) {
    brief::Args a{(const bf16*)p->attn, nullptr, nullptr, (bf16*)p->h, (const bf16*)p->h, stats, p->tokens, layer * brief::D, p->eps, p->status, {}};
    return done(brief::launch_any<brief::kResidual, brief::DQ>(m.o, a, brief::D, st));
}
int short_down(const ShortMaps& m, const IttaiQwen3Prefill* p, int layer, float* stats, cudaStream_t st) {
    brief::Args a{(const bf16*)p->act, nullptr, nullptr, (bf16*)p->h, (const bf16*)p->h, stats, p->tokens, layer * brief::D, p->eps, p->status, {}};
    return done(brief::launch_any<brief::kResidual, brief::FF>(m.down, a, brief::D, st));
}

}  // namespace ittai
