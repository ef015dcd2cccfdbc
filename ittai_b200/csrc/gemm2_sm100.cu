// Two-SM bf16 GEMM: C[M,N] = A[M,K] * W[N,K]^T (+ fused epilogue) with tcgen05.mma.cta_group::2.  A cluster of two CTAs
// owns a 256 x 256 output tile: each CTA loads 128 rows of A and 128 rows of W per 64-wide k-block (32 KB instead of the
// 48 KB a lone CTA needs for its 128 x 256 tile: 64 bytes per clock and SM instead of 96), the leader CTA issues M256 N256 K16 MMAs that read both CTAs' shared memory, and each CTA
// keeps the accumulator rows of its own 128 rows of A in its own tensor memory (two 256-column buffers, so the epilogue of
// one tile overlaps the main loop of the next).
//
// Roles per CTA: warp 0 (one lane) TMA producer for this CTA's half of every stage, completion counted on the LEADER's
// full barrier; warp 1 allocates tensor memory and, in the leader only, issues the MMAs, releasing stages and
// publishing accumulators with multicast commits that arrive in both CTAs; warps 2-9 are the epilogue, 32 columns at a
// time: accumulator -> bias / activation / rounding in the row-per-thread layout tcgen05.ld gives -> residual add from
// a TMA-prefetched tile -> a swizzled staging tile in shared memory -> TMA store (row-per-thread global stores write
// half sectors of 32 different lines per instruction and slow the main loop's loads down).  The peer's epilogue warps
// arrive on the leader's accumulator-free barrier through the cluster's shared window.  Every wait is bounded.
#include "gemm2_common.cuh"

namespace ittai {

__device__ __forceinline__ __nv_bfloat162 as_bf162(uint32_t u) { __nv_bfloat162 v; memcpy(&v, &u, 4); return v; }
__device__ __forceinline__ uint32_t as_u32(__nv_bfloat162 v) { uint32_t u; memcpy(&u, &v, 4); return u; }

// The cos | sin rows (256 bytes) of the 32 tokens of a lane quarter: the quarter's two warps (two heads of the same tokens) bring 16
// rows each, two whole rows per load instruction, 16-byte pieces XOR-swizzled by the row.  (Row-per-thread loads of both heads
// are 64 pieces of 32 different lines each per warp, out of the L2 that feeds the main loop.)
__device__ __forceinline__ void stage_rope_rows(const GemmArgs& g, unsigned char* rows, int row0, int cq, int lane) {
    const int t = row0 + 16 * cq + (lane & 15);
    const int p = t < g.M ? g.rope.pos[t] : 0;
    const uint4* table = reinterpret_cast<const uint4*>(g.rope.rope);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int rr = 2 * i + (lane >> 4);
        const uint4 v = table[(size_t)__shfl_sync(0xffffffffu, p, rr) * (ITTAI_Q3_HD / 8) + (lane & 15)];
        *reinterpret_cast<uint4*>(rows + (16 * cq + rr) * 256 + (((lane & 15) ^ rr) << 4)) = v;
    }
}

// ITTAI_EPI_QKROPE: one warp = 32 tokens x one head (its 128 accumulator columns).  The thread that owns a token's row
// rounds the 128 values to bf16 (the Linear output), and for q / k heads applies the head RMSNorm and the half-split
// rotary embedding with the rounding steps of the eager modules (the arithmetic of qk_rope_scatter_kernel); q goes
// to the output matrix through the staging tiles and TMA stores, k and v from there to their cache rows; `cache_row`: row of the
// layer's store, without the head, of this lane's token.  `release` hands the accumulator back once it is in registers.
template <typename F>
__device__ __forceinline__ void epilogue_qkrope(const GemmArgs& g, const CUtensorMap* tm_out, uint32_t t_addr, unsigned char* so,
                                                const unsigned char* rope_rows, const uint32_t* sgain, uint32_t cache_row,
                                                int row0, int col0, int lane, float row_scale, F release) {
    constexpr int HD = ITTAI_Q3_HD;
    const int head = col0 / HD;
    uint32_t pk[64];
#pragma unroll
    for (int ch = 0; ch < 4; ++ch) {
        uint32_t r[32];
        tmem_ld_32x32(t_addr + 32 * ch, r);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 16; ++i) pk[16 * ch + i] = pack_bf16x2(__uint_as_float(r[2 * i]) * row_scale, __uint_as_float(r[2 * i + 1]) * row_scale);   // a folded RMSNorm's rstd of the row, else 1
    }
    release();
    if (head < 24) {
        float2 st = make_float2(0.f, 0.f);
#pragma unroll
        for (int i = 0; i < 64; ++i) { const float2 v = make_float2(bf_lo(pk[i]), bf_hi(pk[i])); st = __ffma2_rn(v, v, st); }
        const float rstd = 1.0f / sqrtf((st.x + st.y) * (1.0f / HD) + g.rope.eps);
        const unsigned char* rp = rope_rows + lane * 256;
#pragma unroll
        for (int i = 0; i < 64; ++i) asm("" : "+r"(pk[i]));      // unpacked again below: kept from above, the fp32 values would spill
        // Only x * rstd is an fp32 product; every later step is a product or a sum of two bf16 values rounded to bf16, which is
        // one packed instruction for two elements (the _rn forms: never contracted into an FMA).  Through fp32 and back each step was a conversion per element, ten per
        // pair on a pipe of 16 lanes per SM: 10 k cycles of a tile's 14 k (main loop: 8 k).
#pragma unroll
        for (int jj = 0; jj < 8; ++jj) {                  // elements 8jj .. 8jj+7 and their partners 64 + the same
            const uint4 cw = *reinterpret_cast<const uint4*>(rp + ((jj ^ (lane & 15)) << 4)), sw = *reinterpret_cast<const uint4*>(rp + (((jj + 8) ^ (lane & 15)) << 4));
            const uint4 ga = *reinterpret_cast<const uint4*>(sgain + 4 * jj), gb = *reinterpret_cast<const uint4*>(sgain + 32 + 4 * jj);
            const uint32_t wc[4] = {cw.x, cw.y, cw.z, cw.w}, ws[4] = {sw.x, sw.y, sw.z, sw.w};
            const uint32_t wga[4] = {ga.x, ga.y, ga.z, ga.w}, wgb[4] = {gb.x, gb.y, gb.z, gb.w};
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const uint32_t ua = pk[4 * jj + j], ub = pk[32 + 4 * jj + j];
                const __nv_bfloat162 x0 = __hmul2_rn(as_bf162(pack_bf16x2(bf_lo(ua) * rstd, bf_hi(ua) * rstd)), as_bf162(wga[j]));
                const __nv_bfloat162 x1 = __hmul2_rn(as_bf162(pack_bf16x2(bf_lo(ub) * rstd, bf_hi(ub) * rstd)), as_bf162(wgb[j]));
                const __nv_bfloat162 cs = as_bf162(wc[j]), sn = as_bf162(ws[j]);
                pk[4 * jj + j] = as_u32(__hsub2_rn(__hmul2_rn(x0, cs), __hmul2_rn(x1, sn)));
                pk[32 + 4 * jj + j] = as_u32(__hadd2_rn(__hmul2_rn(x1, cs), __hmul2_rn(x0, sn)));
            }
        }
    }
    // four staging tiles of 32 columns, so that the tile is fenced and stored at once
    const int swz = (lane >> 1) & 3;
    // The tile before has left them.  For k and v heads too, although they store nothing through TMA: in a run of consecutive tiles
    // the first k tile of a row block follows the last q tile, whose stores may still be reading.  At once where none is pending.
    if (lane == 0) tma_store_wait_read<0>();
    __syncwarp();
#pragma unroll
    for (int ch = 0; ch < 4; ++ch)
#pragma unroll
        for (int j = 0; j < 4; ++j)
            *reinterpret_cast<uint4*>(so + ch * 2048 + lane * 64 + ((j ^ swz) << 4)) = make_uint4(pk[16 * ch + 4 * j], pk[16 * ch + 4 * j + 1], pk[16 * ch + 4 * j + 2], pk[16 * ch + 4 * j + 3]);
    if (head < 16) {
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) {
#pragma unroll
            for (int ch = 0; ch < 4; ++ch) tma_store_2d(tm_out, so + ch * 2048, col0 + 32 * ch, row0);
            tma_store_commit();
        }
    } else {
        // 16 lanes per token: a whole 256-byte cache row
        __syncwarp();
        bf16* cache = reinterpret_cast<bf16*>(head < 24 ? g.rope.kcache_layer : g.rope.vcache_layer) + (size_t)(head < 24 ? head - 16 : head - 24) * g.rope.kv_cap * HD;
        const int piece = lane & 15;
#pragma unroll 4
        for (int i = 0; i < 16; ++i) {
            const int rr = 2 * i + (lane >> 4);
            const uint32_t row = __shfl_sync(0xffffffffu, cache_row, rr);
            const uint4 val = *reinterpret_cast<const uint4*>(so + (piece >> 2) * 2048 + rr * 64 + (((piece & 3) ^ ((rr >> 1) & 3)) << 4));
            if (row0 + rr < g.M) *reinterpret_cast<uint4*>(cache + (size_t)row * HD + 8 * piece) = val;
        }
        __syncwarp();
    }
}

// ROPE: ITTAI_EPI_QKROPE, else every other epilogue.  The rotary kernel gives one of the five stages up for the rotary rows of the
// CTA's 128 tokens.
//
// Where an epilogue needs something per token (rotary rows, cache rows, row statistics) a pair takes CONSECUTIVE tiles, the column
// tiles of a row block one after the other, and fetches it once per row block; otherwise the tiles are dealt out round-robin.  Fetched
// per tile it stood on the epilogue's path, which then was longer than the main loop: QKV projection with a folded norm at 8192 /
// 16384 / 32768 tokens 62.2 -> 55.0, 119.5 -> 106.4, 268.6 -> 230.8 us, without one 59.2 -> 54.5, 113.7 -> 105.7, 220.8 -> 218.9 (and 50,
// 97, 186 with no epilogue but the store).  A tile's 128 columns are staged, fenced and stored at once for the same reason (a fence
// per 32 columns: 1.5 k of the 12 k cycles that a tile's epilogue took).
template <bool ROPE>
struct Gemm2Cfg {
    static constexpr int kStages = ROPE ? kStages2 - 1 : kStages2;
    static constexpr uint32_t kStageOut = ROPE ? 4 * 2048 : ittai::kStageOut;          // per epilogue warp
    static constexpr uint32_t kColumns = ROPE ? 512 : 2 * 4096;                        // what the epilogue keeps per column
    static constexpr uint32_t kSmem = kStages2 * (kHalfA + kHalfB) + kEpiWarps * kStageOut + kColumns + 1024 /*alignment*/ + 512 /*barriers*/;
    static_assert(kSmem <= 227 * 1024, "shared memory of a CTA");
};
template <bool ROPE>
__global__ void __launch_bounds__(kThreads2, 1)
gemm2_bf16_kernel(const __grid_constant__ CUtensorMap tm_a, const __grid_constant__ CUtensorMap tm_b,
                  const __grid_constant__ CUtensorMap tm_out, const __grid_constant__ CUtensorMap tm_res, const GemmArgs g) {
    using Cfg = Gemm2Cfg<ROPE>;
    constexpr int kStages = Cfg::kStages;
    static_assert(kHalfA + kHalfB == 4 * 32 * 256, "a stage holds the rotary rows of 128 tokens");
    extern __shared__ __align__(1024) unsigned char gsm_raw[];
    unsigned char* gsm = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(gsm_raw) + 1023) & ~(uintptr_t)1023);
    unsigned char* sa = gsm;                                         // [stages][128 rows][128 B]
    unsigned char* sb = gsm + kStages * kHalfA;                     // [stages][128 rows][128 B]
    unsigned char* srope = sb + kStages * kHalfB;                    // ROPE: [4 lane quarters][32 rows][256 B]
    unsigned char* sout = gsm + kStages2 * (kHalfA + kHalfB);        // [epilogue warps] staging tiles, then their bias slices
    unsigned long long* bars = reinterpret_cast<unsigned long long*>(sout + kEpiWarps * Cfg::kStageOut + Cfg::kColumns);
    unsigned long long* full = bars;                                 // [stages]  both producers -> leader's MMA
    unsigned long long* empty = bars + kStages;                     // [stages]  MMA -> this CTA's producer
    unsigned long long* acc_full = bars + 2 * kStages;              // [2]       MMA -> this CTA's epilogue
    unsigned long long* acc_empty = bars + 2 * kStages + 2;         // [2]       both epilogues -> leader's MMA
    unsigned long long* res_bars = bars + 2 * kStages + 4;          // [epilogue warps][2] residual chunk landed
    unsigned long long* rope_full = res_bars + 2 * kEpiWarps;        // [4] both warps of a lane quarter have brought their rotary rows
    unsigned long long* rope_free = rope_full + 4;                   // [4] both have done with them
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(rope_free + 4);
    volatile uint32_t* abort_flag = tmem_slot + 1;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = cluster_ctarank();                         // 0 = leader
    const int pair = blockIdx.x >> 1, n_pairs = gridDim.x >> 1;
    const int tiles_n = g.N / PN, tiles_m = (g.M + PM - 1) / PM, n_tiles = tiles_m * tiles_n;
    const int n_kb = g.K / PK;
    const bool runs = ROPE || g.row_stats != nullptr;                // consecutive tiles
    const int t_first = runs ? (int)((long long)n_tiles * pair / n_pairs) : pair, t_end = runs ? (int)((long long)n_tiles * (pair + 1) / n_pairs) : n_tiles;
    const int t_step = runs ? 1 : n_pairs;

    if (threadIdx.x == 0) {
        for (int s = 0; s < kStages; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
        for (int b = 0; b < 2; ++b) { mbar_init(&acc_full[b], 1); mbar_init(&acc_empty[b], 2 * kEpiWarps); }
        for (int b = 0; b < 2 * kEpiWarps; ++b) mbar_init(&res_bars[b], 1);
        for (int b = 0; b < 8; ++b) mbar_init(&rope_full[b], 2);
        *abort_flag = 0;
        fence_mbar_init();
        tma_prefetch_desc(&tm_a);
        tma_prefetch_desc(&tm_b);
    }
    pdl_trigger();
    if (warp == 1) tmem_alloc_pair(tmem_slot, kTmemCols2);
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();                                              // the peer's barriers exist before anything targets them
    tc_fence_after();
    pdl_wait();                                                      // operands come from the kernels before this one
    const uint32_t tmem_base = *tmem_slot;

    if (warp == 0) {
        if (elect_one()) {
            // ---- TMA producer for this CTA's halves; one running k-block counter across all of the pair's tiles
            int it = 0;
            for (int tile = t_first; tile < t_end && !*abort_flag; tile += t_step) {
                const int tile_m = TILE_M(tile), tile_n = TILE_N(tile);
                for (int kb = 0; kb < n_kb; ++kb, ++it) {
                    const int s = it % kStages, use = it / kStages;
                    if (use > 0 && !mbar_wait_bounded(&empty[s], (use - 1) & 1, kSpin2)) { *abort_flag = 1; break; }
                    if (*abort_flag) break;
                    if (rank == 0) mbar_expect_tx(&full[s], 2 * (kHalfA + kHalfB));
                    const uint32_t leader_full = map_to_cta(&full[s], 0);
                    tma_load_2d_pair(sa + s * kHalfA, &tm_a, kb * PK, tile_m * PM + (int)rank * 128, leader_full);
                    tma_load_2d_pair(sb + s * kHalfB, &tm_b, kb * PK, tile_n * PN + (int)rank * 128, leader_full);
                }
            }
        }
    } else if (warp == 1) {
        if (rank == 0 && elect_one()) {
            // ---- MMA issuer (leader only)
            constexpr uint32_t idesc = umma_idesc_bf16(PM, PN);
            int it = 0, local = 0;
            bool ok = true, next = false;
            for (int tile = t_first; tile < t_end && ok; tile += t_step, ++local) {
                const int buf = local & 1, round = local >> 1;
                ok = (round == 0 || mbar_wait_bounded(&acc_empty[buf], (round - 1) & 1, kSpin2)) && !*abort_flag;
                if (!ok) break;
                tc_fence_after();
                const uint32_t d_tmem = tmem_base + (uint32_t)(buf * PN);
                for (int kb = 0; kb < n_kb; ++kb, ++it) {
                    const int s = it % kStages, use = it / kStages;
                    if (!next) ok = mbar_wait_bounded(&full[s], use & 1, kSpin2) && !*abort_flag;
                    if (!ok) break;
                    tc_fence_after();
                    next = mbar_test(&full[(it + 1) % kStages], ((it + 1) / kStages) & 1);
                    const uint64_t da = umma_desc_sw128(sa + s * kHalfA), db = umma_desc_sw128(sb + s * kHalfB);
#pragma unroll
                    for (int k = 0; k < PK / 16; ++k)
                        umma_bf16_pair(d_tmem, da + 2 * k, db + 2 * k, idesc, (kb > 0 || k > 0) ? 1u : 0u);
                    umma_commit_pair(&empty[s]);               // both CTAs' producers may refill the stage
                }
                if (!ok) break;
                umma_commit_pair(&acc_full[buf]);              // both CTAs' epilogues may read their rows
            }
            if (!ok) *abort_flag = 1;
        }
    } else {
        // ---- epilogue: warp w may touch TMEM lanes 32*(w%4)..+31 = 32 rows of this CTA's half tile; the two warps that
        //      share a lane quarter split the 256 columns
        const int ew = warp - 2, q = warp & 3, cq = ew >> 2;         // TMEM lane quarter, column slice (kEpiCols columns)
        unsigned char* so = sout + ew * Cfg::kStageOut;              // three (ROPE: four) [32 rows][64 B] tiles, 64-byte swizzle
        const unsigned char* sgain = sout + kEpiWarps * Cfg::kStageOut;   // ROPE: head norm gains of q and k, 128 bf16 each
        float* sbias = reinterpret_cast<float*>(sout + kEpiWarps * kStageOut) + ew * kEpiCols;   // this warp's bias values
        float* scsum = sbias + kEpiWarps * kEpiCols;                 // and, with a folded LayerNorm, its column sums
        const bool fold = g.row_stats != nullptr;
        unsigned long long* res_bar = res_bars + 2 * ew;
        const bool swiglu = g.epi == ITTAI_EPI_SWIGLU, has_res = g.residual != nullptr;
        const int swz = (lane >> 1) & 3;                             // 64-byte swizzle of this thread's staging row
        constexpr uint32_t kChunks = kEpiCols / 32;                  // 32-column chunks per tile for this warp
        // With a residual, tile 0 stages the output and tiles 1-2 receive residual chunks by TMA, two chunks ahead of
        // their use and across tile boundaries: chunk n of this warp's running sequence is chunk n % kChunks of its
        // (n / kChunks)-th tile and lands in buffer n % 2.  Without one, the three tiles rotate as output staging.
        auto prefetch_res = [&](uint32_t n) {
            const int t = t_first + (int)(n / kChunks) * t_step;
            if (t < t_end) {
                mbar_expect_tx(&res_bar[n & 1], 2048);
                tma_load_2d(so + 2048 + (n & 1) * 2048, &tm_res, TILE_N(t) * PN + kEpiCols * cq + 32 * (int)(n % kChunks),
                            TILE_M(t) * PM + (int)rank * 128 + q * 32, &res_bar[n & 1]);
            }
        };
        if (has_res && lane == 0) { prefetch_res(0); prefetch_res(1); }
        if constexpr (ROPE) {                                         // every warp writes the same values
            reinterpret_cast<uint4*>(sout + kEpiWarps * Cfg::kStageOut)[lane] = lane < 16 ? reinterpret_cast<const uint4*>(g.rope.qn)[lane] : reinterpret_cast<const uint4*>(g.rope.kn)[lane - 16];
            __syncwarp();
        }
        uint32_t cc = 0;
        int local = 0, seen_m = -1, rope_m = -1;                     // row blocks that the statistics and cache rows, and the rotary rows, are of
        uint32_t rope_n = 0;
        float mean = 0.f, rstd = 1.f;
        uint32_t cache_row = 0;
        bool ok = true;
        auto wait = [&](void* bar, uint32_t parity) {                // whole warp; bounded, given up when another role aborted; one answer for all lanes
            bool done = true;
            uint32_t spins = 0;
            while (!mbar_try_wait_parked(bar, parity)) {
                if (((++spins) & 255u) == 0u && (*abort_flag || spins >= kSpin2)) { done = false; break; }
            }
            return __all_sync(0xffffffffu, done) != 0;
        };
        for (int tile = t_first; tile < t_end; tile += t_step, ++local) {
            const int buf = local & 1, round = local >> 1;
            const int tile_m = TILE_M(tile), tile_n = TILE_N(tile);
            const int row0 = tile_m * PM + (int)rank * 128 + q * 32;  // first row of this warp
            const int col0 = tile_n * PN + kEpiCols * cq;             // first accumulator column of this warp
            // the bias slice does not depend on the accumulator: fetched before waiting for it
            if (!ROPE && g.bias != nullptr && lane < kEpiCols / 4) *reinterpret_cast<float4*>(sbias + 4 * lane) = *reinterpret_cast<const float4*>(g.bias + col0 + 4 * lane);
            if (!ROPE && fold && lane < kEpiCols / 4) *reinterpret_cast<float4*>(scsum + 4 * lane) = *reinterpret_cast<const float4*>(g.col_sums + col0 + 4 * lane);
            if (runs && tile_m != seen_m) {
                seen_m = tile_m;
                if (fold && row0 + lane < g.M) {
                    if (g.stats_parts == 0) {
                        const float2 ms = *reinterpret_cast<const float2*>(g.row_stats + 2 * (size_t)(row0 + lane));
                        mean = ms.x; rstd = ms.y;
                    } else {
                        // partial (sum, sum of squares) of the K columns in slices, added in slice order
                        const float2 ss = row_sums(g, row0 + lane);
                        const float inv_k = 1.0f / (float)(g.stats_k > 0 ? g.stats_k : g.K);
                        mean = g.stats_rms ? 0.f : ss.x * inv_k;
                        rstd = rsqrtf(fmaxf(ss.y * inv_k - mean * mean, 0.f) + g.stats_eps);
                    }
                }
                if constexpr (ROPE) {
                    const int tt = row0 + lane;
                    if (tt < g.M) cache_row = (uint32_t)(g.rope.seq[tt] * ITTAI_Q3_NKV) * (uint32_t)g.rope.kv_cap + (uint32_t)g.rope.slot[tt];
                }
            }
            float st1 = 0.f, st2 = 0.f;                               // statistics of this row's output slice
            if constexpr (ROPE) {
                if (col0 < ITTAI_Q3_DQ + ITTAI_Q3_DKV) {
                    if (tile_m != rope_m) {
                        if (rope_m >= 0) {
                            if (lane == 0) mbar_arrive(&rope_free[q]);
                            ok = wait(&rope_free[q], (rope_n - 1) & 1);
                        }
                        if (ok) {
                            stage_rope_rows(g, srope + q * 8192, row0, cq, lane);
                            __syncwarp();
                            if (lane == 0) mbar_arrive(&rope_full[q]);
                            ok = wait(&rope_full[q], rope_n & 1);
                        }
                        if (!ok) { *abort_flag = 1; break; }
                        rope_m = tile_m;
                        ++rope_n;
                    }
                }
            }
            __syncwarp();
            ok = wait(&acc_full[buf], round & 1);
            __syncwarp();
            if (!ok) { *abort_flag = 1; break; }
            tc_fence_after();
            auto release = [&]() {                                    // this warp has read the accumulator
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive_cluster(map_to_cta(&acc_empty[buf], 0));
            };
            if constexpr (ROPE) {
                epilogue_qkrope(g, &tm_out, tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(buf * PN + kEpiCols * cq), so,
                                srope + q * 8192, reinterpret_cast<const uint32_t*>(sgain) + (col0 < ITTAI_Q3_DQ ? 0 : 64), cache_row, row0, col0, lane, rstd, release);
                continue;
            }
#pragma unroll 1
            for (uint32_t ch = 0; ch < kChunks && ok; ++ch, ++cc) {
                // 32 accumulator columns of this thread's row -> bias, activation, rounding -> 16 packed words
                uint32_t r[32], o[16];
                tmem_ld_32x32(tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(buf * PN + kEpiCols * cq + 32 * ch), r);
                tmem_ld_wait();
                epilogue_pack(g, r, g.bias != nullptr ? sbias + 32 * ch : nullptr, o, fold ? scsum + 32 * ch : nullptr, mean, rstd);
                if (swiglu) {
                    // 16 output columns per chunk: two consecutive chunks fill one 32-column staging tile, then one TMA store
                    const uint32_t half = ch & 1;
                    unsigned char* sto = so + ((cc >> 1) % 3u) * 2048;
                    if (half == 0) {
                        if (lane == 0) tma_store_wait_read<2>();
                        __syncwarp();
                    }
#pragma unroll
                    for (int j = 0; j < 2; ++j)
                        *reinterpret_cast<uint4*>(sto + lane * 64 + (((2 * half + j) ^ swz) << 4)) = make_uint4(o[4 * j], o[4 * j + 1], o[4 * j + 2], o[4 * j + 3]);
                    if (half == 1) {
                        fence_proxy_async_smem();
                        __syncwarp();
                        if (lane == 0) { tma_store_2d(&tm_out, sto, (col0 + 32 * ((int)ch - 1)) / 2, row0); tma_store_commit(); }
                    }
                    continue;
                }
                if (has_res) {
                    // out = bf16(residual + bf16(module output)); this thread's row piece of the TMA-filled buffer
                    const uint32_t b = cc & 1;
                    ok = wait(&res_bar[b], (cc >> 1) & 1);
                    if (!ok) { *abort_flag = 1; break; }
                    const unsigned char* rrow = so + 2048 + b * 2048 + lane * 64;
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const uint4 rs = *reinterpret_cast<const uint4*>(rrow + ((j ^ swz) << 4));
                        o[4 * j] = pack_bf16x2(bf_lo(rs.x) + bf_lo(o[4 * j]), bf_hi(rs.x) + bf_hi(o[4 * j]));
                        o[4 * j + 1] = pack_bf16x2(bf_lo(rs.y) + bf_lo(o[4 * j + 1]), bf_hi(rs.y) + bf_hi(o[4 * j + 1]));
                        o[4 * j + 2] = pack_bf16x2(bf_lo(rs.z) + bf_lo(o[4 * j + 2]), bf_hi(rs.z) + bf_hi(o[4 * j + 2]));
                        o[4 * j + 3] = pack_bf16x2(bf_lo(rs.w) + bf_lo(o[4 * j + 3]), bf_hi(rs.w) + bf_hi(o[4 * j + 3]));
                    }
                    __syncwarp();                                     // every lane has consumed the buffer: refill it
                    if (lane == 0) prefetch_res(cc + 2);
                }
                if (g.stats_out != nullptr) {
#pragma unroll
                    for (int i = 0; i < 16; ++i) {
                        const float lo = bf_lo(o[i]), hi = bf_hi(o[i]);
                        st1 += lo + hi;
                        st2 = fmaf(lo, lo, fmaf(hi, hi, st2));
                    }
                }
                // the store that last used this staging tile must have finished reading it
                unsigned char* sto = has_res ? so : so + (cc % 3u) * 2048;
                if (lane == 0) { if (has_res) tma_store_wait_read<0>(); else tma_store_wait_read<2>(); }
                __syncwarp();
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    *reinterpret_cast<uint4*>(sto + lane * 64 + ((j ^ swz) << 4)) = make_uint4(o[4 * j], o[4 * j + 1], o[4 * j + 2], o[4 * j + 3]);
                fence_proxy_async_smem();
                __syncwarp();
                if (lane == 0) { tma_store_2d(&tm_out, sto, col0 + 32 * (int)ch, row0); tma_store_commit(); }
            }
            if (!ok) break;
            if (g.stats_out != nullptr && row0 + lane < g.M)
                *reinterpret_cast<float2*>(g.stats_out + 2 * ((size_t)(row0 + lane) * (g.N / 128) + col0 / 128)) = make_float2(st1, st2);
            release();
        }
        if (lane == 0) tma_store_wait_all();                          // shared memory stays valid until the stores are done
    }
    tc_fence_before();
    __syncthreads();
    if (*abort_flag) {
        if (threadIdx.x == 0) {
            if (atomicCAS(&g.status[0], 0u, (uint32_t)ITTAI_ST_GEMM_TIMEOUT) == 0u) { g.status[1] = blockIdx.x; g.status[2] = (uint32_t)n_kb; }
            // let copies that may still be in flight land before the shared memory is handed back
            const long long t0 = clock64();
            while (clock64() - t0 < 2000000) {}
        }
        __syncthreads();
    }
    // neither CTA leaves while the other may still read its shared memory or signal its barriers
    cluster_sync_all();
    if (warp == 1) { __syncwarp(); tmem_dealloc_pair(tmem_base, kTmemCols2); }
}

int cuda_fail(cudaError_t e, const char* what);

template <bool ROPE>
static cudaError_t gemm2_launch(const CUtensorMap& tm_a, const CUtensorMap& tm_b, const CUtensorMap& tm_out, const CUtensorMap& tm_res, const GemmArgs& g, cudaStream_t st) {
    static thread_local int attr_dev = -1, max_pairs = 0;
    int dev = 0;
    cudaGetDevice(&dev);
    if (attr_dev != dev) {
        cudaError_t e = cudaFuncSetAttribute(gemm2_bf16_kernel<ROPE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Gemm2Cfg<ROPE>::kSmem);
        if (e != cudaSuccess) return e;
        int n_sms = 0;
        e = cudaDeviceGetAttribute(&n_sms, cudaDevAttrMultiProcessorCount, dev);
        if (e != cudaSuccess) return e;
        cudaLaunchConfig_t cfg = {};
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = 2; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
        cfg.blockDim = dim3(kThreads2);
        cfg.dynamicSmemBytes = Gemm2Cfg<ROPE>::kSmem;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        cfg.gridDim = dim3(n_sms & ~1);
        int n_clusters = 0;
        e = cudaOccupancyMaxActiveClusters(&n_clusters, gemm2_bf16_kernel<ROPE>, &cfg);
        if (e != cudaSuccess) return e;
        max_pairs = n_clusters < 1 ? 1 : (n_clusters > n_sms / 2 ? n_sms / 2 : n_clusters);
        attr_dev = dev;
    }
    const int tiles = ((g.M + PM - 1) / PM) * (g.N / PN);
    return launch_pdl(gemm2_bf16_kernel<ROPE>, dim3(2 * (tiles < max_pairs ? tiles : max_pairs)), dim3(kThreads2), Gemm2Cfg<ROPE>::kSmem, st, 2, tm_a, tm_b, tm_out, tm_res, g);
}

int gemm2_bf16_launch(const CUtensorMap& tm_a, const CUtensorMap& tm_b, const GemmArgs& g, cudaStream_t st) {
    // the epilogue stores 32-row x 32-column boxes through TMA (rows past M are dropped) and fetches the residual the same way
    CUtensorMap tm_out, tm_res;
    const bool swiglu = g.epi == ITTAI_EPI_SWIGLU;
    int rc = make_tmap_bf16(&tm_out, g.out, g.M, swiglu ? g.N / 2 : g.N, g.ld_out, 32, 32);
    if (rc != ITTAI_OK) return rc;
    if (g.residual != nullptr) rc = make_tmap_bf16(&tm_res, g.residual, g.M, g.N, g.ld_res, 32, 32);
    else tm_res = tm_out;
    if (rc != ITTAI_OK) return rc;
    const cudaError_t e = g.epi == ITTAI_EPI_QKROPE ? gemm2_launch<true>(tm_a, tm_b, tm_out, tm_res, g, st) : gemm2_launch<false>(tm_a, tm_b, tm_out, tm_res, g, st);
    return e == cudaSuccess ? ITTAI_OK : cuda_fail(e, "launch gemm2_bf16_kernel");
}

}  // namespace ittai
