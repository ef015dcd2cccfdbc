// Split-K bf16 GEMM for problems with few output tiles: C[M,N] = A[M,K] * W[N,K]^T (+ fused epilogue).
//
// A prompt of 23 tokens or a single image gives the persistent kernels a handful of tiles: 128 x 64 tiles of one row block
// are 16 CTAs for N = 1024, 256 x 256 pair tiles of 196 rows are 3 pairs for N = 768, and each walks the whole K alone.
// Such a GEMM is bound by how many SMs fetch weights and by the length of the serial chain, not by the tensor cores.  Here an
// output tile is 128 columns x 32, 64 or 128 token rows and belongs to a cluster of up to 8 CTAs that share its K out:
//
// * the weights are the M operand of the MMA and the token rows its N, so that a few rows cost a narrow MMA and little shared
//   memory instead of a padded 128-row operand;
// * warp 0 (one lane) streams k-blocks of 64 columns of W and A through a ring of three or four stages.  The W tiles of the first
//   stages are requested BEFORE griddepcontrol.wait: the caller has declared W constant (ITTAI_GEMM_STATIC_W), and two CTAs fit
//   an SM, so the next GEMM's weights arrive while this one's epilogue runs;
// * warp 1 (one lane) issues tcgen05.mma M128 N<rows> K16 into <rows> columns of tensor memory;
// * with GemmArgs::a_gain the other warps RMS-normalise each landed A tile in place (valid rows only, the rounding steps of
//   rmsnorm_rows_kernel) before the MMAs read it: the norm's own launch, a kernel boundary and a round trip of the activations
//   through L2 twice per layer, goes.  All six take every k-block where there are no more of them than stages, otherwise one or two keep
//   to a stage;
// * a thread holds one column of the accumulator, a warp 32 neighbouring ones of every row: they are stored straight from the
//   registers into the shared memory of the CTA that finishes the row (row r: rank r mod splits), counted there on a barrier (32 rows) or
//   ahead of a cluster barrier, and the epilogue reads only its own shared memory.  (With the partials kept where they arise, the meeting was a store, a
//   barrier, loads through distributed shared memory at each one's latency, and a second barrier before anyone might leave);
// * a warp takes a row, lane l its columns 4l .. 4l+3, one to four rows side by side.  A row in one warp makes the head norm and
//   the rotary partner of the QKV projection, the output statistics of a folded norm and coalesced 256-byte stores plain
//   shuffles.  What the epilogue reads from memory (residual, row statistics, rotary rows, bias) is requested while the
//   accumulator fills.
//
// Measured on a B200 inside a CUDA graph, weights from HBM, us, the layout described in brackets (A as a 128-row M operand, one
// row of a warp at a time, its loads behind the accumulator) -> this one, M 23 / 128 / 196 / 512: N 4096 K 1024 6.1 -> 4.7,
// 8.5 -> 6.6, 9.0 -> 8.1; N 6144 K 1024 7.2 -> 5.4, 9.1 -> 7.9; N 1024 K 3072 6.0 -> 5.4, 8.6 -> 7.2, 9.1 -> 8.1, 12.0 -> 9.9;
// N 768 K 768 4.4 -> 4.1, 6.4 -> 4.4, 6.7 -> 4.7, 7.6 -> 5.6; N 768 K 3072 6.0 -> 5.3, 8.9 -> 6.2, 9.9 -> 6.9, 10.9 -> 9.2.  It is
// bound by its own chain: a kernel boundary (0.8 us), the activations through TMA, 12 to 48 dependent MMAs, one exchange.  Of the 10300
// cycles of a QKV projection of 23 tokens 2000 were gains on their way from HBM behind the wait, 1000 a serial sum of the row statistics and
// 1300 the cluster barrier behind the partials; without them a query of 23 tokens takes 677 us instead of 707, a prompt of 47 tokens 1473
// instead of 1571 (with the smaller code), one image 402 instead of 406.  Four rows of a column as one 16-byte store, with the sums put back
// into rows by all threads: 693 and 427 us.
//
// The tensor memory is allocated BEFORE launch_dependents: a later kernel that shares the SM can then never hold columns
// this one still waits for (an SM holds two such CTAs, or one and an attention CTA of 256 columns, of its 512).
// Waits are bounded as in the other GEMM kernels.
#include <cuda.h>

#include "gemm_epilogue.cuh"
#include "gemm_split.h"
#include "launch.h"

namespace ittai {

constexpr int SN = 128, SK = 64;                                 // weight rows of a tile (the M of the MMA), k-block
constexpr int kSplitThreads = 256, kMaxSplit = 8;
constexpr uint32_t kSplitW = SN * SK * 2;
constexpr int kNormWarps = kSplitThreads / 32 - 2;
constexpr uint32_t kSplitSpin = 1u << 22;
// TN token rows (the N of the MMA).  The partials of a cluster go to the CTA that finishes the row: up to 64 rows into a buffer of
// their own, 128 rows into the ring, once every CTA of the cluster has stopped using it (kAlias).
template <int TN>
struct SplitCfg {
    static constexpr bool kAlias = TN > 64;
    // Tiles of 32 rows send by st.async to a barrier of the receiver (one way; a rank's 16 stores a warp take 1000 cycles to leave and 640
    // more to arrive), the others by plain stores ahead of a cluster barrier: twice as many st.async leave at half the rate of stores
    // (64 rows: 2200 cycles against 1300, which is what the barrier's 1700 against 800 gives back; one image 408 us against 406).
    static constexpr bool kAsync = TN == 32;
    static constexpr int kStages = TN == 32 ? 4 : 3;
    static constexpr int kRows = TN / 32;                        // output rows a warp works on side by side
    // Warps that normalise a k-block, in as many groups as stages: a group keeps to one stage and so waits for every use of its
    // barrier, one after the other.  (A group that skips uses, or that first looks at a later one, is let through by the parity of
    // the phase before and normalises what has not landed.)
    static constexpr int kNormGroup = kNormWarps / kStages;
    static_assert(kNormGroup >= 1, "a group for every stage");
    static constexpr uint32_t kA = TN * SK * 2;
    static constexpr uint32_t kRing = kStages * (kA + kSplitW);
    static constexpr uint32_t kRecv = kAlias ? 0 : TN * SN * 4;
    static constexpr uint32_t kSmem = kRing + kRecv + 1024 /*alignment*/ + 192 /*barriers*/ + TN * 8 /*row statistics*/ + kStages * SK * 2 /*gains*/;
    static_assert(!kAlias || TN * SN * 4 <= kRing, "the partial tiles reuse the ring");
    static_assert(2 * (kSmem + 1024) <= 228 * 1024, "two CTAs per SM");
};

__device__ __forceinline__ void split_cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void split_cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ float4 lds_f4(uint32_t addr) {
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ uint32_t split_mapa(uint32_t addr, int rank) {
    uint32_t a;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(addr), "r"(rank));
    return a;
}

// What the epilogue of one output row needs besides the sums.  Requested by every warp as soon as the kernels before have ended,
// ahead of its share of the main loop: behind the accumulator each of these loads is a round trip to L2 on the critical path.
struct SplitRow {
    uint2 res;               // four residual values
    uint2 cos, sin;          // rotary row (q and k heads)
    bf16* cache;             // cache row of a k or v head
};
struct SplitIndex { int pos, seq, slot; };
struct SplitCols {           // the same for every row: a lane keeps to its four columns
    float4 bias, csum;
    uint2 gain;
};

template <int EPI>
__device__ __forceinline__ SplitCols split_cols(const GemmArgs& g, int col0, int lane) {
    SplitCols k;
    const int c = col0 + 4 * lane;
    k.bias = g.bias != nullptr ? *reinterpret_cast<const float4*>(g.bias + c) : make_float4(0.f, 0.f, 0.f, 0.f);
    k.csum = g.row_stats != nullptr && g.a_gain == nullptr ? *reinterpret_cast<const float4*>(g.col_sums + c) : make_float4(0.f, 0.f, 0.f, 0.f);
    k.gain = make_uint2(0u, 0u);
    if (EPI == ITTAI_EPI_QKROPE && col0 / ITTAI_Q3_HD < 24)
        k.gain = *reinterpret_cast<const uint2*>(reinterpret_cast<const bf16*>(col0 / ITTAI_Q3_HD < 16 ? g.rope.qn : g.rope.kn) + 4 * lane);
    return k;
}

// Rows row0 + u * step (u < U) below `end`; whole warp, converged.  In two parts because the rotary rows and the cache rows hang
// on loads of their own: what a warp does between the two is not held up by the first.
template <int EPI, int U>
__device__ __forceinline__ void split_load_index(const GemmArgs& g, SplitIndex (&ix)[U], int row0, int step, int end, int col0) {
    if constexpr (EPI == ITTAI_EPI_QKROPE) {
        const int head = col0 / ITTAI_Q3_HD;
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int row = row0 + u * step;
            ix[u].pos = ix[u].seq = ix[u].slot = 0;
            if (row < end) {
                if (head < 24) ix[u].pos = g.rope.pos[row];
                if (head >= 16) { ix[u].seq = g.rope.seq[row]; ix[u].slot = g.rope.slot[row]; }
            }
        }
    }
}
template <int EPI, int U>
__device__ __forceinline__ void split_load_rows(const GemmArgs& g, const SplitIndex (&ix)[U], SplitRow (&in)[U], int row0, int step, int end, int col0, int lane) {
    if constexpr (EPI == ITTAI_EPI_QKROPE) {
        constexpr int HD = ITTAI_Q3_HD, NKV = ITTAI_Q3_NKV;
        const int head = col0 / HD;
        if (head < 24) {
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const bf16* rp = reinterpret_cast<const bf16*>(g.rope.rope) + (size_t)ix[u].pos * HD + 4 * (lane & 15);
                in[u].cos = make_uint2(0u, 0u); in[u].sin = in[u].cos;
                if (row0 + u * step < end) { in[u].cos = *reinterpret_cast<const uint2*>(rp); in[u].sin = *reinterpret_cast<const uint2*>(rp + HD / 2); }
            }
        }
        if (head >= 16) {
            bf16* cache = reinterpret_cast<bf16*>(head < 24 ? g.rope.kcache_layer : g.rope.vcache_layer);
#pragma unroll
            for (int u = 0; u < U; ++u) in[u].cache = cache + (((size_t)ix[u].seq * NKV + (head < 24 ? head - 16 : head - 24)) * g.rope.kv_cap + ix[u].slot) * HD + 4 * lane;
        }
    }
    if (g.residual != nullptr) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int row = row0 + u * step;
            in[u].res = row < end ? *reinterpret_cast<const uint2*>(g.residual + (size_t)row * g.ld_res + col0 + 4 * lane) : make_uint2(0u, 0u);
        }
    }
}

// Epilogue of one row piece: lane l holds columns col0 + 4l .. + 3 of row `row` (whole warp, converged).  `norm`: mean and 1 / standard
// deviation of a folded norm.  `store`: the row exists
// (uniform; rows past the end take part in the arithmetic so that the rows of a batch are one straight run of instructions).
template <int EPI>
__device__ __forceinline__ void split_epilogue_row(const GemmArgs& g, const SplitCols& k, const SplitRow& in, float2 norm, float (&v)[4], int row, bool store, int col0, int lane) {
    const int c = col0 + 4 * lane;
    if (g.row_stats != nullptr && g.a_gain == nullptr) {
        v[0] = norm.y * fmaf(-norm.x, k.csum.x, v[0]); v[1] = norm.y * fmaf(-norm.x, k.csum.y, v[1]);
        v[2] = norm.y * fmaf(-norm.x, k.csum.z, v[2]); v[3] = norm.y * fmaf(-norm.x, k.csum.w, v[3]);
    }
    if (g.bias != nullptr) { v[0] += k.bias.x; v[1] += k.bias.y; v[2] += k.bias.z; v[3] += k.bias.w; }
    if constexpr (EPI == ITTAI_EPI_SWIGLU) {
        const float g0 = bf16r(v[0]), u0 = bf16r(v[1]), g1 = bf16r(v[2]), u1 = bf16r(v[3]);
        const uint32_t o = pack_bf16x2(bf16r(g0 / (1.0f + expf(-g0))) * u0, bf16r(g1 / (1.0f + expf(-g1))) * u1);
        if (store) *reinterpret_cast<uint32_t*>(g.out + (size_t)row * g.ld_out + c / 2) = o;
        return;
    }
    if constexpr (EPI == ITTAI_EPI_QKROPE) {
        // on packed pairs: the Linear output rounded, then (q and k heads) the head norm and the half-split rotary embedding with the rounding
        // steps of qk_rope_scatter_kernel; the partner element 64 columns away is 16 lanes away
        constexpr int HD = ITTAI_Q3_HD;
        const int head = col0 / HD;
        uint32_t x0 = pack_bf16x2(v[0], v[1]), x1 = pack_bf16x2(v[2], v[3]);
        if (head < 24) {
            const float f0 = bf_lo(x0), f1 = bf_hi(x0), f2 = bf_lo(x1), f3 = bf_hi(x1);
            const float rstd = rsqrt_full(warp_sum(fmaf(f0, f0, fmaf(f1, f1, fmaf(f2, f2, f3 * f3)))) * (1.0f / HD) + g.rope.eps);
            const uint32_t n0 = mul_bf16x2(pack_bf16x2(f0 * rstd, f1 * rstd), k.gain.x), n1 = mul_bf16x2(pack_bf16x2(f2 * rstd, f3 * rstd), k.gain.y);
            const uint32_t neg = lane < 16 ? 0x80008000u : 0u;
            const uint32_t o0 = __shfl_xor_sync(0xffffffffu, n0, 16) ^ neg, o1 = __shfl_xor_sync(0xffffffffu, n1, 16) ^ neg;
            x0 = add_bf16x2(mul_bf16x2(n0, in.cos.x), mul_bf16x2(o0, in.sin.x));
            x1 = add_bf16x2(mul_bf16x2(n1, in.cos.y), mul_bf16x2(o1, in.sin.y));
        }
        bf16* dst = head < 16 ? g.out + (size_t)row * g.ld_out + c : in.cache;
        if (store) *reinterpret_cast<uint2*>(dst) = make_uint2(x0, x1);
        return;
    }
    if constexpr (EPI == ITTAI_EPI_GELU) {
#pragma unroll
        for (int i = 0; i < 4; ++i) v[i] = gelu_tanh(bf16r(v[i]));
    }
    if (g.residual != nullptr) {
        v[0] = bf_lo(in.res.x) + bf16r(v[0]); v[1] = bf_hi(in.res.x) + bf16r(v[1]);
        v[2] = bf_lo(in.res.y) + bf16r(v[2]); v[3] = bf_hi(in.res.y) + bf16r(v[3]);
    }
    const uint2 o = make_uint2(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]));
    if (store) *reinterpret_cast<uint2*>(g.out + (size_t)row * g.ld_out + c) = o;
    if (g.stats_out != nullptr) {
        const float a0 = bf_lo(o.x), a1 = bf_hi(o.x), a2 = bf_lo(o.y), a3 = bf_hi(o.y);
        const float s1 = warp_sum((a0 + a1) + (a2 + a3)), s2 = warp_sum(fmaf(a0, a0, fmaf(a1, a1, fmaf(a2, a2, a3 * a3))));
        if (store && lane == 0) *reinterpret_cast<float2*>(g.stats_out + 2 * ((size_t)row * (g.N / SN) + col0 / SN)) = make_float2(s1, s2);
    }
}

// Grid (splits, N / 128, row tiles of tile_rows <= TN), clusters of `splits` CTAs along x.
template <int TN, int EPI>
__global__ void __launch_bounds__(kSplitThreads, 2)
gemm_split_kernel(const __grid_constant__ CUtensorMap tm_a, const __grid_constant__ CUtensorMap tm_w, const GemmArgs g, const int tile_rows, const int lg) {
    using Cfg = SplitCfg<TN>;
    constexpr int kStages = Cfg::kStages;
    extern __shared__ __align__(1024) unsigned char gsm_raw[];
    unsigned char* gsm = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(gsm_raw) + 1023) & ~(uintptr_t)1023);
    unsigned char* sw = gsm;                                         // [stages][128 weight rows][128 B]
    unsigned char* sa = gsm + kStages * kSplitW;                     // [stages][TN token rows][128 B]
    float* part = reinterpret_cast<float*>(Cfg::kAlias ? gsm : gsm + Cfg::kRing);   // [splits][TN / splits][128]: the partials of this CTA's rows
    unsigned long long* bars = reinterpret_cast<unsigned long long*>(gsm + Cfg::kRing + Cfg::kRecv);
    unsigned long long* full = bars;
    unsigned long long* empty = bars + kStages;
    unsigned long long* acc_full = bars + 2 * kStages;
    unsigned long long* ready = bars + 2 * kStages + 1;              // [stages] A normalised
    unsigned long long* arrived = bars + 3 * kStages + 1;            // partials of this CTA's rows have arrived
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 3 * kStages + 2);
    float* scale = reinterpret_cast<float*>(bars + 16);              // a_gain: [TN] 1 / rms of A's rows
    float2* norm = reinterpret_cast<float2*>(bars + 16);             // folded norm: [TN / splits] mean, 1 / standard deviation of this CTA's rows
    volatile uint32_t* abort_flag = tmem_slot + 1;
    unsigned char* gain_s = reinterpret_cast<unsigned char*>(bars) + 192 + TN * 8;      // a_gain, all_norm: [stages][64] the CTA's gains
    static_assert(3 * kStages + 3 <= 16, "barriers and flags end before the row scales");

    const int warp = warp_index(), lane = threadIdx.x & 31;
    const int rank = blockIdx.x, splits = 1 << lg, tile_n = blockIdx.y, row_base = blockIdx.z * tile_rows;
    const int n_kb_all = g.K / SK, kb0 = n_kb_all * rank >> lg, n_kb = (n_kb_all * (rank + 1) >> lg) - kb0;   // >= 1: splits <= K / 64
    const int rows = min(tile_rows, g.M - row_base);
    const bool all_norm = n_kb <= kStages;                           // no stage is used twice: see the normalising warps

    if (threadIdx.x == 0) {
        for (int s = 0; s < kStages; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); mbar_init(&ready[s], all_norm ? kNormWarps : Cfg::kNormGroup); }
        mbar_init(acc_full, 1);
        mbar_init(arrived, 1);
        *abort_flag = 0;
        fence_mbar_init();
        // the partials of this CTA's rows, those of its own included
        if (Cfg::kAsync && splits > 1) mbar_expect_tx(arrived, rank < rows ? (uint32_t)(((rows - 1 - rank) >> lg) + 1) * (SN * 4) << lg : 0u);
        tma_prefetch_desc(&tm_a);
        tma_prefetch_desc(&tm_w);
    }
    if (warp == 1) tmem_alloc(tmem_slot, TN);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    // another CTA's shared memory may be written only once that CTA runs; waited for ahead of the first write
    if (!Cfg::kAlias && splits > 1) split_cluster_arrive();
    pdl_trigger();
    const uint32_t tmem_base = *tmem_slot;

    // Row r of the tile belongs to rank r % splits and there to warp (r / splits) % 8, U of them at a time.
    constexpr int U = Cfg::kRows;
    const int col0 = tile_n * SN, first = rank + splits * warp, step = splits * (kSplitThreads / 32);
    const int ahead = min(kStages, n_kb);
    if (warp == 0 && elect_one()) {
        for (int kb = 0; kb < ahead; ++kb) {
            mbar_expect_tx(&full[kb], Cfg::kA + kSplitW);
            tma_load_2d(sw + kb * kSplitW, &tm_w, (kb0 + kb) * SK, tile_n * SN, &full[kb]);
        }
    }
    __syncwarp();
    const bool normalises = warp >= 2 && g.a_gain != nullptr;
    // its k-blocks: group, group + kStages, ... (none for the warps left over); a thread keeps to one 16-byte column piece (eight
    // pieces a row), so its gains are one vector per k-block, the first of them fetched ahead of the wait like the weights
    constexpr int kNormThreads = 32 * Cfg::kNormGroup;
    const int group = all_norm ? 0 : warp - 2 < kStages * Cfg::kNormGroup ? (warp - 2) / Cfg::kNormGroup : n_kb;
    const int nt = all_norm ? threadIdx.x - 64 : (threadIdx.x - 64) % kNormThreads, piece = nt & 7;
    const uint4* gains = reinterpret_cast<const uint4*>(g.a_gain + (size_t)kb0 * SK) + piece;
    uint4 gain = make_uint4(0u, 0u, 0u, 0u);
    // Ahead of the wait, and in shared memory where that can be, so that they have arrived: a load that nothing uses before the wait is
    // scheduled behind it, and gains come from HBM (1500 to 2000 cycles a k-block on the critical path).
    float inv_k = 0.f;
    if (normalises) {
        asm volatile("rcp.rn.f32 %0, %1;" : "=f"(inv_k) : "f"((float)g.K));
        if (!all_norm) { if (group < n_kb) gain = gains[8 * group]; }
        else if (nt < 8 * n_kb) *reinterpret_cast<uint4*>(gain_s + nt * 16) = reinterpret_cast<const uint4*>(g.a_gain + (size_t)kb0 * SK)[nt];
    }
    pdl_wait();                                                      // from here on what the kernels before wrote
    if (warp == 0 && elect_one()) {
        for (int kb = 0; kb < ahead; ++kb) tma_load_2d(sa + kb * Cfg::kA, &tm_a, (kb0 + kb) * SK, row_base, &full[kb]);
    }
    __syncwarp();
    SplitRow in[U];
    SplitIndex ix[U];
    split_load_index<EPI, U>(g, ix, row_base + first, step, row_base + rows, col0);
    const SplitCols cols = split_cols<EPI>(g, col0, lane);
    if (!normalises) split_load_rows<EPI, U>(g, ix, in, row_base + first, step, row_base + rows, col0, lane);

    if (warp == 0) {
        if (elect_one()) {
            for (int kb = ahead; kb < n_kb && !*abort_flag; ++kb) {
                const int s = kb % kStages, use = kb / kStages;
                if (!mbar_wait_bounded(&empty[s], (use - 1) & 1, kSplitSpin)) { *abort_flag = 1; break; }
                mbar_expect_tx(&full[s], Cfg::kA + kSplitW);
                tma_load_2d(sw + s * kSplitW, &tm_w, (kb0 + kb) * SK, tile_n * SN, &full[s]);
                tma_load_2d(sa + s * Cfg::kA, &tm_a, (kb0 + kb) * SK, row_base, &full[s]);
            }
        }
    } else if (warp == 1) {
        if (elect_one()) {
            constexpr uint32_t idesc = umma_idesc_bf16(SN, TN);
            unsigned long long* landed = g.a_gain != nullptr ? ready : full;
            bool ok = true, next = false;
            for (int kb = 0; kb < n_kb; ++kb) {
                const int s = kb % kStages, use = kb / kStages;
                if (!next) ok = mbar_wait_bounded(&landed[s], use & 1, kSplitSpin) && !*abort_flag;
                if (!ok) break;
                tc_fence_after();
                next = mbar_test(&landed[(kb + 1) % kStages], ((kb + 1) / kStages) & 1);
                const uint64_t dw = umma_desc_sw128(sw + s * kSplitW), da = umma_desc_sw128(sa + s * Cfg::kA);
#pragma unroll
                for (int k = 0; k < SK / 16; ++k) umma_bf16(tmem_base, dw + 2 * k, da + 2 * k, idesc, (kb > 0 || k > 0) ? 1u : 0u);
                umma_commit(&empty[s]);
            }
            if (ok) umma_commit(acc_full); else *abort_flag = 1;
        }
    } else if (g.a_gain != nullptr) {
        // eight lanes a row, each every eighth partial sum
        const int t = threadIdx.x - 64;
        for (int r0 = 0; r0 < rows; r0 += 4 * kNormWarps) {
            const int r = r0 + (t >> 3);
            float ss = 0.f;
            if (r < rows) {
                const float2* ps = reinterpret_cast<const float2*>(g.row_stats) + (size_t)(row_base + r) * g.stats_parts;
                for (int i = t & 7; i < g.stats_parts; i += 8) ss += ps[i].y;
            }
#pragma unroll
            for (int o = 1; o < 8; o <<= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
            if (r < rows && (t & 7) == 0) scale[r] = rsqrt_full(ss * inv_k + g.stats_eps);
        }
        asm volatile("bar.sync 1, %0;" ::"n"(32 * kNormWarps) : "memory");
        // Up to as many k-blocks as stages (a short K, or one that many CTAs share) all warps take each of them.  Beyond that the groups.
        const int kb_step = all_norm ? 1 : kStages, row_step = (all_norm ? 32 * kNormWarps : kNormThreads) / 8;
#pragma unroll 1
        for (int kb = group; kb < n_kb; kb += kb_step) {
            const int s = kb % kStages, use = kb / kStages;
            const uint4 gq = all_norm ? *reinterpret_cast<const uint4*>(gain_s + kb * 128 + piece * 16) : gain;
            if (!all_norm && kb + kb_step < n_kb) gain = gains[8 * (kb + kb_step)];
            bool ok = true;
            uint32_t spins = 0;
            while (!mbar_try_wait_parked(&full[s], use & 1)) {
                if (((++spins) & 255u) == 0u && (*abort_flag || spins >= kSplitSpin)) { ok = false; break; }
            }
            if (!__all_sync(0xffffffffu, ok)) { *abort_flag = 1; break; }      // one answer for all lanes: warp-wide steps follow
            const uint32_t gw[4] = {gq.x, gq.y, gq.z, gq.w};
#pragma unroll 2
            for (int r = nt >> 3; r < rows; r += row_step) {
                uint4* p = reinterpret_cast<uint4*>(sa + s * Cfg::kA + r * 128 + ((piece ^ (r & 7)) << 4));
                const uint4 x = *p;
                const uint32_t xw[4] = {x.x, x.y, x.z, x.w};
                const float rs = scale[r];
                uint32_t o[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) o[j] = mul_bf16x2(pack_bf16x2(bf_lo(xw[j]) * rs, bf_hi(xw[j]) * rs), gw[j]);
                *p = make_uint4(o[0], o[1], o[2], o[3]);
            }
            fence_proxy_async_smem();                                // the MMAs read through the async proxy
            __syncwarp();
            if (lane == 0) mbar_arrive(&ready[s]);
        }
        split_load_rows<EPI, U>(g, ix, in, row_base + first, step, row_base + rows, col0, lane);
    } else if (g.row_stats != nullptr) {
        // a thread per row; the barrier behind the main loop hands the results to the epilogue
        const int t = threadIdx.x - 64, row = rank + splits * t;
        if (row < rows) {
            float2 ms;
            if (g.stats_parts == 0) ms = *reinterpret_cast<const float2*>(g.row_stats + 2 * (size_t)(row_base + row));
            else {
                const float2 ss = row_sums(g, row_base + row);
                const float inv_k = 1.0f / (float)(g.stats_k > 0 ? g.stats_k : g.K);
                ms.x = g.stats_rms ? 0.f : ss.x * inv_k;
                ms.y = rsqrtf(fmaxf(ss.y * inv_k - ms.x * ms.x, 0.f) + g.stats_eps);
            }
            norm[t] = ms;
        }
    }
    __syncwarp();
    // Warp w reads TMEM lanes 32 (w % 4) .. + 31, one weight row = output column per thread; the two warps of a lane quarter
    // take half of the token rows each.  A warp's store is 32 consecutive floats of one row, into the owner's buffer.
    const int half = (warp >> 2) * (TN / 2);
    const uint32_t src = smem_u32(part) + (uint32_t)rank * (TN >> lg) * (SN * 4) + 4u * ((warp & 3) * 32 + lane);
    uint32_t to[kMaxSplit], to_bar[Cfg::kAsync ? kMaxSplit : 1];     // the owners of eight neighbouring rows
#pragma unroll
    for (int i = 0; i < kMaxSplit; ++i) {
        to[i] = split_mapa(src, i & (splits - 1));
        if (Cfg::kAsync) to_bar[Cfg::kAsync ? i : 0] = split_mapa(smem_u32(arrived), i & (splits - 1));
    }
    bool ok = true;
    {
        uint32_t spins = 0;
        while (!mbar_try_wait_parked(acc_full, 0)) {
            if (((++spins) & 255u) == 0u && (*abort_flag || spins >= kSplitSpin)) { ok = false; break; }
        }
    }
    ok = __all_sync(0xffffffffu, ok);
    if (!ok) *abort_flag = 1;
    __syncwarp();
    tc_fence_after();
    if (splits > 1) {                // every CTA of the cluster runs; kAlias: and its MMAs have read its ring
        if (Cfg::kAlias) split_cluster_arrive();
        split_cluster_wait();
    } else if (Cfg::kAlias) {
        __syncthreads();
    }
#pragma unroll
    for (int c = 0; c < TN / 2; c += 16) {
        if (half + c >= rows) break;                // where the wait ran out too: the owners count on the bytes, the status tells the caller
        uint32_t acc[16];
        tmem_ld_32x16(tmem_base + ((uint32_t)((warp & 3) * 32) << 16) + half + c, acc);
        tmem_ld_wait16(acc);
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            const int n = half + c + i;
            if (n < rows) {
                const uint32_t dst = to[i % kMaxSplit] + (uint32_t)(n >> lg) * (SN * 4);
                // a launch without clusters (splits == 1) may not use st.async: it is an illegal instruction there
                if (!Cfg::kAsync || splits == 1) asm volatile("st.shared::cluster.b32 [%0], %1;" ::"r"(dst), "r"(acc[i]) : "memory");
                else asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];" ::"r"(dst), "r"(acc[i]), "r"(to_bar[Cfg::kAsync ? i % kMaxSplit : 0]) : "memory");
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) tmem_dealloc(tmem_base, TN);
    if (!Cfg::kAsync) {
        if (splits > 1) { split_cluster_arrive(); split_cluster_wait(); }
    } else if (splits > 1) {
        uint32_t spins = 0;
        while (!mbar_try_wait_cluster(arrived, 0)) {
            if (((++spins) & 255u) == 0u && (*abort_flag || spins >= kSplitSpin)) { *abort_flag = 1; break; }
        }
        __syncwarp();
    }
    const uint32_t mine = smem_u32(part) + 16u * lane;
    const bool folded = g.row_stats != nullptr && g.a_gain == nullptr;
    for (int r0 = first; r0 < rows; r0 += U * step) {
        if (r0 != first) {
            split_load_index<EPI, U>(g, ix, row_base + r0, step, row_base + rows, col0);
            split_load_rows<EPI, U>(g, ix, in, row_base + r0, step, row_base + rows, col0, lane);
        }
        uint32_t off[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            off[u] = (uint32_t)(min(r0 + u * step, TN - 1) >> lg) * (SN * 4);      // rows past the end: whatever lies there
        }
        float v[U][4];
#pragma unroll
        for (int s = 0; s < kMaxSplit; ++s) {
            if (s < splits) {
                const uint32_t base = mine + (uint32_t)s * (TN >> lg) * (SN * 4);
                float4 p[U];
#pragma unroll
                for (int u = 0; u < U; ++u) p[u] = lds_f4(base + off[u]);
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    if (s == 0) { v[u][0] = p[u].x; v[u][1] = p[u].y; v[u][2] = p[u].z; v[u][3] = p[u].w; }
                    else { v[u][0] += p[u].x; v[u][1] += p[u].y; v[u][2] += p[u].z; v[u][3] += p[u].w; }
                }
            }
        }
#pragma unroll
        for (int u = 0; u < U; ++u) split_epilogue_row<EPI>(g, cols, in[u], folded ? norm[min(r0 + u * step, TN - 1) >> lg] : make_float2(0.f, 1.f), v[u], row_base + r0 + u * step, r0 + u * step < rows, col0, lane);
    }
    __syncthreads();
    if (*abort_flag) {
        // A CTA that gave up may be ahead of others that have yet to write here, and must not leave before they have.  All send, also where
        // their waits ran out, so the bytes come; should one take longer than this wait, the barrier holds this CTA until the others have left
        // (threads that have exited count as arrived).  Only here: an arrival by everyone behind the sends costs each launch 0.5 us.
        if (Cfg::kAsync && splits > 1) {
            bool all = false;
            for (uint32_t spins = 0; !all && spins < kSplitSpin; ++spins) all = mbar_try_wait_cluster(arrived, 0);
            if (!__syncthreads_and(all)) { split_cluster_arrive(); split_cluster_wait(); }
        }
        if (threadIdx.x == 0) {
            if (atomicCAS(&g.status[0], 0u, (uint32_t)ITTAI_ST_GEMM_TIMEOUT) == 0u) { g.status[1] = blockIdx.x; g.status[2] = (uint32_t)n_kb; }
            // let copies that may still be in flight land before the shared memory is handed back
            const long long t0 = clock64();
            while (clock64() - t0 < 2000000) {}
        }
        __syncthreads();
    }
}

int cuda_fail(cudaError_t e, const char* what);

// CTAs that share a tile's K: a power of two (clusters of 3, 5 or 7 cost 5-15 % more than the next smaller power, measured with
// tiles of 128 x 128), at least three k-blocks each (N 768 K 768, us in two / four / eight parts: M 128, 24 tiles, 4.3 / 3.5 / 3.8;
// M 196, 48 tiles, 5.1 / 4.2 / 4.6), and no more CTAs than 7/4 per SM: beyond two per SM some run after the others (N 1024 K 3072 in
// tiles of 64 rows: M 512, 128 tiles as 128 / 256 / 512 CTAs 11.1 / 8.9 / 15.0; M 1280, 160 / 320 CTAs 19.0 / 21.1).  The shapes between
// 7/4 and two per SM, which 128 x 128 tiles lost on, would gain with today's (288 CTAs against what the line gives: N 1024 K 3072 at
// M 1152 12.6 / 14.2, N 768 K 768 at M 1536 6.7 / 7.6, N 2304 K 768 at M 512 6.8 / 7.7).
static int split_log2(int tiles, int n_kb, int n_sms) {
    int lg = 0;
    while (2 << lg <= kMaxSplit && (2 << lg) * tiles * 4 <= 7 * n_sms && (2 << lg) * 3 <= n_kb) ++lg;
    return lg;
}

// Up to half as many tiles of 128 x 128 as SMs.  Measured on a B200 with weights from HBM inside a CUDA graph, us, the kernel that
// would run otherwise -> this one.  Pair kernel: N 1024 K 3072 at M 196 / 512 / 1024 / 1152 19.1 -> 7.3, 19.0 -> 8.9, 19.3 -> 11.9,
// 19.5 -> 14.2, beyond the line at 1536 19.1 -> 15.9; N 768 K 768 at M 196 / 1024 / 1536 8.7 -> 3.7, 8.7 -> 5.7, 8.8 -> 7.6, beyond it at
// 2048 8.8 -> 7.9; N 2304 K 768 at M 512 8.9 -> 7.7, beyond it at 784 9.0 -> 8.1.  128 x 64 tiles of one CTA each (M <= 128, which bring W into L2
// first): N 1024 K 3072 at M 32 / 128 9.7 -> 4.3, 10.3 -> 6.6; N 768 K 768 3.8 -> 2.9, 4.6 -> 3.3; N 4096 K 1024 at M 32 / 64 / 128 4.7 -> 3.9, 4.9 -> 5.5,
// 5.2 -> 6.3, N 6144 5.4 -> 4.5, 5.7 -> 5.8, 6.2 -> 6.7 (where this one is the slower it still spares a norm's pass, or the rotation's).
// The line dates from an earlier form of both kernels and lies on the safe side of today's crossing with the pair kernel.  The
// one-CTA tiles, which only unsplit GEMMs reach above 128 rows, are the fastest of the three where they fill most of one round of the
// SMs: 5.1 us for N 768 K 768 at M 1536, 10.3 for N 1024 K 3072 at M 1152, 5.4 for N 2304 K 768 at M 512.
bool gemm_split_wins(int m, int n, int n_sms) { return m > 0 && n > 0 && 2ll * ((m + 127) / 128) * (n / SN) <= n_sms; }

// Rows of a tile.  32 rows are the shortest chain while they cost nothing in splits and leave most SMs one CTA (N 768 K 768 at
// M 128 / 196: 4.4 and 4.7 us against 4.7 and 4.9; N 768 K 3072 at M 128: 6.2 against 7.2; but N 2304 K 768 at M 128, two splits
// instead of four, 5.6 against 5.2, and N 4096 K 1024 at M 64, 256 CTAs instead of 128, 5.9 against 5.6).  128 rows are
// for a long K that smaller tiles leave too few splits for: N 1024 K 3072 at M 640 / 1024 12.4 and 12.8 against 13.5 and 14.4 (24
// k-blocks to a CTA become 12); with 16 k-blocks left it is no matter (N 1024 K 2048: 11.0 and 11.1 against 10.5 and 11.5).
int gemm_split_rows(int m, int n, int k, int n_sms) {
    const int tiles_n = n / SN, n_kb = k / SK;
    const auto tiles = [&](int tn) { return (m + tn - 1) / tn * tiles_n; };
    const auto lg = [&](int tn) { return split_log2(tiles(tn), n_kb, n_sms); };
    if (m <= 32 || (lg(32) == lg(64) && 3 * (tiles(32) << lg(32)) <= 4 * n_sms)) return 32;
    const int share = n_kb >> lg(64);
    return share > 16 && n_kb >> lg(128) < share ? 128 : 64;
}

template <int TN, int EPI>
static cudaError_t split_launch(const CUtensorMap& tm_a, const CUtensorMap& tm_w, const GemmArgs& g, int n_sms, cudaStream_t st) {
    constexpr uint32_t kLone = SplitCfg<TN>::kSmem > 115u * 1024 ? SplitCfg<TN>::kSmem : 115u * 1024;      // one CTA per SM
    static thread_local int attr_dev = -1;
    int dev = 0;
    cudaGetDevice(&dev);
    if (attr_dev != dev) {
        const cudaError_t e = cudaFuncSetAttribute(gemm_split_kernel<TN, EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kLone);
        if (e != cudaSuccess) return e;
        attr_dev = dev;
    }
    const int tiles_m = (g.M + TN - 1) / TN, tiles_n = g.N / SN, lg = split_log2(tiles_m * tiles_n, g.K / SK, n_sms);
    // A tower's QKV projection whose CTAs all find an SM of their own gets it, by shared memory that it does not need; otherwise SMs that the kernel in
    // front leaves empty take two.  One image of ViT-B/16 403.5 -> 391.2 us, of the variable-resolution tower 445 -> 429.  Not the others: two such
    // kernels in a row share no SM, and the second one's weights then come only when the first has ended (language, O-proj or down this way
    // 880 -> 980 us at 64 tokens; its QKV projection 805 -> 813 at 49, 876 -> 866 at 64, 1159 -> 1164 at 128).
    const bool lone = EPI == ITTAI_EPI_NONE && g.row_stats != nullptr && g.a_gain == nullptr && (tiles_m * tiles_n) << lg <= n_sms;
    // even row tiles: 196 rows are 98 and 98, not 128 and 68
    return launch_pdl(gemm_split_kernel<TN, EPI>, dim3(1 << lg, tiles_n, tiles_m), dim3(kSplitThreads), lone ? kLone : SplitCfg<TN>::kSmem, st, 1 << lg, tm_a, tm_w, g,
                      (g.M + tiles_m - 1) / tiles_m, lg);
}
template <int TN>
static cudaError_t split_launch_epi(const CUtensorMap& tm_a, const CUtensorMap& tm_w, const GemmArgs& g, int n_sms, cudaStream_t st) {
    switch (g.epi) {
        case ITTAI_EPI_GELU: return split_launch<TN, ITTAI_EPI_GELU>(tm_a, tm_w, g, n_sms, st);
        case ITTAI_EPI_SWIGLU: return split_launch<TN, ITTAI_EPI_SWIGLU>(tm_a, tm_w, g, n_sms, st);
        case ITTAI_EPI_QKROPE: return split_launch<TN, ITTAI_EPI_QKROPE>(tm_a, tm_w, g, n_sms, st);
        default: return split_launch<TN, ITTAI_EPI_NONE>(tm_a, tm_w, g, n_sms, st);
    }
}

int gemm_split_launch(const CUtensorMap& tm_a, const CUtensorMap& tm_w, const GemmArgs& g, int tile_rows, int n_sms, cudaStream_t st) {
    const cudaError_t e = tile_rows == 32 ? split_launch_epi<32>(tm_a, tm_w, g, n_sms, st) : tile_rows == 64 ? split_launch_epi<64>(tm_a, tm_w, g, n_sms, st)
                                                                                   : split_launch_epi<128>(tm_a, tm_w, g, n_sms, st);
    return e == cudaSuccess ? ITTAI_OK : cuda_fail(e, "launch gemm_split_kernel");
}

}  // namespace ittai
