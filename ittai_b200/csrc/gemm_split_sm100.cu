// Split-K bf16 GEMM for problems with few output tiles: C[M,N] = A[M,K] * W[N,K]^T (+ fused epilogue).
//
// A prompt of 23 tokens or a single image gives the persistent kernels a handful of tiles: 128 x 64 tiles of one row block
// are 16 CTAs for N = 1024, 256 x 256 pair tiles of 196 rows are 3 pairs for N = 768, and each walks the whole K alone.
// Such a GEMM is bound by how many SMs fetch weights and by the length of the serial chain, not by the tensor cores.  Here
// an output tile is 128 x 128 and belongs to a cluster of up to 8 CTAs that share its K out between them:
//
// * warp 0 (one lane) streams 128 x 64 tiles of A and W through a ring of three stages.  The W tiles of the
//   first stages are requested BEFORE griddepcontrol.wait: the caller has declared W constant (ITTAI_GEMM_STATIC_W), and two
//   CTAs fit an SM (97 KB each), so the next GEMM's weights arrive while this one's epilogue runs;
// * warp 1 (one lane) issues tcgen05.mma M128 N128 K16 into 128 columns of tensor memory;
// * with GemmArgs::a_gain the other six warps RMS-normalise each landed A tile in place (valid rows only, the rounding steps of
//   rmsnorm_rows_kernel) before the MMAs read it: the norm's own launch, a kernel boundary and a round trip of the activations
//   through L2 twice per layer, goes;
// * all eight warps then copy the valid rows of the partial tile to shared memory as fp32 (the ring is free by then), the
//   cluster meets, and the rows are dealt out over its CTAs: a warp takes a row, lane l its columns 4l .. 4l+3, adds the
//   splits in rank order through distributed shared memory and runs the epilogue.  A row in one warp makes the head norm
//   and the rotary partner of the QKV projection, the output statistics of a folded norm and coalesced 256-byte stores
//   plain shuffles.
//
// The tensor memory is allocated BEFORE launch_dependents: a later kernel that shares the SM can then never hold columns
// this one still waits for (an SM holds two such CTAs, or one and an attention CTA of 256 columns, of its 512).
// Waits are bounded as in the other GEMM kernels.
#include <cuda.h>

#include "gemm_epilogue.cuh"
#include "gemm_split.h"
#include "launch.h"

namespace ittai {

constexpr int SM_ = 128, SN = 128, SK = 64;
constexpr int kSplitStages = 3, kSplitThreads = 256, kMaxSplit = 8;
constexpr uint32_t kSplitA = SM_ * SK * 2, kSplitB = SN * SK * 2;
constexpr int kPartLd = SN + 4;                                  // fp32 per row of the partial tile: 16 bytes of padding keep
                                                                 // the row-per-thread 128-bit stores free of bank conflicts
constexpr uint32_t kSplitSmem = kSplitStages * (kSplitA + kSplitB) + 1024 /*alignment*/ + 128 /*barriers*/ + SM_ * 4 /*row scales*/;
static_assert(SM_ * kPartLd * 4 <= kSplitStages * (kSplitA + kSplitB), "the partial tile reuses the ring");
constexpr int kNormWarps = kSplitThreads / 32 - 2;
constexpr uint32_t kSplitSpin = 1u << 22;
constexpr uint32_t kSplitCols = 128;

__device__ __forceinline__ void split_cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ float4 ld_cluster_f4(uint32_t addr) {
    float4 v;
    asm volatile("ld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
    return v;
}

// Epilogue of one row piece: lane l holds columns col0 + 4l .. + 3 of row `row` (whole warp, converged).
__device__ __forceinline__ void split_epilogue_row(const GemmArgs& g, float (&v)[4], int row, int col0, int lane) {
    const int c = col0 + 4 * lane;
    if (g.row_stats != nullptr && g.a_gain == nullptr) {
        float mean, rstd;
        if (g.stats_parts == 0) {
            const float2 ms = *reinterpret_cast<const float2*>(g.row_stats + 2 * (size_t)row);
            mean = ms.x; rstd = ms.y;
        } else {
            const float2* ps = reinterpret_cast<const float2*>(g.row_stats) + (size_t)row * g.stats_parts;
            float s1 = 0.f, s2 = 0.f;
            for (int i = lane; i < g.stats_parts; i += 32) { const float2 t = ps[i]; s1 += t.x; s2 += t.y; }
            s1 = warp_sum(s1);
            s2 = warp_sum(s2);
            const float inv_k = 1.0f / (float)(g.stats_k > 0 ? g.stats_k : g.K);
            mean = g.stats_rms ? 0.f : s1 * inv_k;
            rstd = rsqrtf(fmaxf(s2 * inv_k - mean * mean, 0.f) + g.stats_eps);
        }
        const float4 cs = *reinterpret_cast<const float4*>(g.col_sums + c);
        v[0] = rstd * fmaf(-mean, cs.x, v[0]); v[1] = rstd * fmaf(-mean, cs.y, v[1]);
        v[2] = rstd * fmaf(-mean, cs.z, v[2]); v[3] = rstd * fmaf(-mean, cs.w, v[3]);
    }
    if (g.bias != nullptr) {
        const float4 b4 = *reinterpret_cast<const float4*>(g.bias + c);
        v[0] += b4.x; v[1] += b4.y; v[2] += b4.z; v[3] += b4.w;
    }
    if (g.epi == ITTAI_EPI_SWIGLU) {
        const float g0 = bf16r(v[0]), u0 = bf16r(v[1]), g1 = bf16r(v[2]), u1 = bf16r(v[3]);
        *reinterpret_cast<uint32_t*>(g.out + (size_t)row * g.ld_out + c / 2) =
            pack_bf16x2(bf16r(g0 / (1.0f + expf(-g0))) * u0, bf16r(g1 / (1.0f + expf(-g1))) * u1);
        return;
    }
    if (g.epi == ITTAI_EPI_QKROPE) {
        // the Linear output rounded, then (q and k heads) the head norm and the half-split rotary embedding with the rounding
        // steps of qk_rope_scatter_kernel; the partner element 64 columns away is 16 lanes away
        constexpr int HD = ITTAI_Q3_HD, NKV = ITTAI_Q3_NKV;
        const int head = col0 / HD;
        float x[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) x[i] = bf16r(v[i]);
        if (head < 24) {
            const float ss = warp_sum(fmaf(x[0], x[0], fmaf(x[1], x[1], fmaf(x[2], x[2], x[3] * x[3]))));
            const float rstd = 1.0f / sqrtf(ss * (1.0f / HD) + g.rope.eps);
            const bf16* gain = reinterpret_cast<const bf16*>(head < 16 ? g.rope.qn : g.rope.kn) + 4 * lane;
            const bf16* rp = reinterpret_cast<const bf16*>(g.rope.rope) + (size_t)g.rope.pos[row] * HD + 4 * (lane & 15);
            const uint2 gw = *reinterpret_cast<const uint2*>(gain), cw = *reinterpret_cast<const uint2*>(rp), sw = *reinterpret_cast<const uint2*>(rp + HD / 2);
            const float ga[4] = {bf_lo(gw.x), bf_hi(gw.x), bf_lo(gw.y), bf_hi(gw.y)}, cs[4] = {bf_lo(cw.x), bf_hi(cw.x), bf_lo(cw.y), bf_hi(cw.y)};
            const float sn[4] = {bf_lo(sw.x), bf_hi(sw.x), bf_lo(sw.y), bf_hi(sw.y)};
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float mine = bf16r(bf16r(x[i] * rstd) * ga[i]), other = __shfl_xor_sync(0xffffffffu, mine, 16);
                x[i] = bf16r(bf16r(mine * cs[i]) + bf16r((lane < 16 ? -other : other) * sn[i]));
            }
        }
        bf16* dst;
        if (head < 16) dst = g.out + (size_t)row * g.ld_out + c;
        else {
            bf16* cache = reinterpret_cast<bf16*>(head < 24 ? g.rope.kcache_layer : g.rope.vcache_layer);
            dst = cache + (((size_t)g.rope.seq[row] * NKV + (head < 24 ? head - 16 : head - 24)) * g.rope.kv_cap + g.rope.slot[row]) * HD + 4 * lane;
        }
        *reinterpret_cast<uint2*>(dst) = make_uint2(pack_bf16x2(x[0], x[1]), pack_bf16x2(x[2], x[3]));
        return;
    }
    if (g.epi == ITTAI_EPI_GELU) {
#pragma unroll
        for (int i = 0; i < 4; ++i) v[i] = gelu_tanh(bf16r(v[i]));
    }
    if (g.residual != nullptr) {
        const uint2 rs = *reinterpret_cast<const uint2*>(g.residual + (size_t)row * g.ld_res + c);
        v[0] = bf_lo(rs.x) + bf16r(v[0]); v[1] = bf_hi(rs.x) + bf16r(v[1]);
        v[2] = bf_lo(rs.y) + bf16r(v[2]); v[3] = bf_hi(rs.y) + bf16r(v[3]);
    }
    const uint2 o = make_uint2(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]));
    *reinterpret_cast<uint2*>(g.out + (size_t)row * g.ld_out + c) = o;
    if (g.stats_out != nullptr) {
        const float a0 = bf_lo(o.x), a1 = bf_hi(o.x), a2 = bf_lo(o.y), a3 = bf_hi(o.y);
        const float s1 = warp_sum((a0 + a1) + (a2 + a3)), s2 = warp_sum(fmaf(a0, a0, fmaf(a1, a1, fmaf(a2, a2, a3 * a3))));
        if (lane == 0) *reinterpret_cast<float2*>(g.stats_out + 2 * ((size_t)row * (g.N / SN) + col0 / SN)) = make_float2(s1, s2);
    }
}

// Grid (splits, N / 128, row blocks), clusters of `splits` CTAs along x.
__global__ void __launch_bounds__(kSplitThreads, 2)
gemm_split_kernel(const __grid_constant__ CUtensorMap tm_a, const __grid_constant__ CUtensorMap tm_b, const GemmArgs g) {
    extern __shared__ __align__(1024) unsigned char gsm_raw[];
    unsigned char* gsm = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(gsm_raw) + 1023) & ~(uintptr_t)1023);
    unsigned char* sa = gsm;                                         // [stages][128 rows][128 B]
    unsigned char* sb = gsm + kSplitStages * kSplitA;
    float* part = reinterpret_cast<float*>(gsm);                     // [128][kPartLd], once the ring is idle
    unsigned long long* bars = reinterpret_cast<unsigned long long*>(gsm + kSplitStages * (kSplitA + kSplitB));
    unsigned long long* full = bars;
    unsigned long long* empty = bars + kSplitStages;
    unsigned long long* acc_full = bars + 2 * kSplitStages;
    unsigned long long* ready = bars + 2 * kSplitStages + 1;          // [stages] A normalised
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 3 * kSplitStages + 1);
    float* scale = reinterpret_cast<float*>(bars + 16);              // [128] 1 / rms of A's rows
    volatile uint32_t* abort_flag = tmem_slot + 1;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rank = blockIdx.x, splits = gridDim.x, tile_n = blockIdx.y, tile_m = blockIdx.z;
    const int n_kb_all = g.K / SK, kb0 = n_kb_all * rank / splits, n_kb = n_kb_all * (rank + 1) / splits - kb0;   // >= 1: splits <= K / 64
    const int rows = min(SM_, g.M - tile_m * SM_);

    if (threadIdx.x == 0) {
        for (int s = 0; s < kSplitStages; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); mbar_init(&ready[s], kNormWarps); }
        mbar_init(acc_full, 1);
        *abort_flag = 0;
        fence_mbar_init();
        tma_prefetch_desc(&tm_a);
        tma_prefetch_desc(&tm_b);
    }
    if (warp == 1) tmem_alloc(tmem_slot, kSplitCols);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    pdl_trigger();
    const uint32_t tmem_base = *tmem_slot;

    if (warp == 0) {
        if (lane == 0) {
            const int ahead = min(kSplitStages, n_kb);
            for (int kb = 0; kb < ahead; ++kb) {
                mbar_expect_tx(&full[kb], kSplitA + kSplitB);
                tma_load_2d(sb + kb * kSplitB, &tm_b, (kb0 + kb) * SK, tile_n * SN, &full[kb]);
            }
            pdl_wait();
            for (int kb = 0; kb < n_kb && !*abort_flag; ++kb) {
                const int s = kb % kSplitStages, use = kb / kSplitStages;
                if (use > 0 && !mbar_wait_bounded(&empty[s], (use - 1) & 1, kSplitSpin)) { *abort_flag = 1; break; }
                if (kb >= ahead) {
                    mbar_expect_tx(&full[s], kSplitA + kSplitB);
                    tma_load_2d(sb + s * kSplitB, &tm_b, (kb0 + kb) * SK, tile_n * SN, &full[s]);
                }
                tma_load_2d(sa + s * kSplitA, &tm_a, (kb0 + kb) * SK, tile_m * SM_, &full[s]);
            }
        }
    } else if (warp == 1 && lane == 0) {
        constexpr uint32_t idesc = umma_idesc_bf16(SM_, SN);
        bool ok = true;
        for (int kb = 0; kb < n_kb; ++kb) {
            const int s = kb % kSplitStages, use = kb / kSplitStages;
            ok = mbar_wait_bounded(g.a_gain != nullptr ? &ready[s] : &full[s], use & 1, kSplitSpin) && !*abort_flag;
            if (!ok) break;
            tc_fence_after();
            const uint64_t da = umma_desc_sw128(sa + s * kSplitA), db = umma_desc_sw128(sb + s * kSplitB);
#pragma unroll
            for (int k = 0; k < SK / 16; ++k) umma_bf16(tmem_base, da + 2 * k, db + 2 * k, idesc, (kb > 0 || k > 0) ? 1u : 0u);
            umma_commit(&empty[s]);
        }
        if (ok) umma_commit(acc_full); else *abort_flag = 1;
    } else if (warp >= 2 && g.a_gain != nullptr) {
        // a thread keeps to one 16-byte column piece of the tiles (192 threads, eight pieces a row), so its gains are one
        // vector per k-block; the first is fetched ahead of the wait like the weights
        const int t = threadIdx.x - 64, piece = t & 7;
        const uint4* gains = reinterpret_cast<const uint4*>(g.a_gain + (size_t)kb0 * SK) + piece;
        uint4 next = gains[0];
        pdl_wait();
        if (t < rows) {
            const float2* ps = reinterpret_cast<const float2*>(g.row_stats) + (size_t)(tile_m * SM_ + t) * g.stats_parts;
            float ss = 0.f;
            for (int i = 0; i < g.stats_parts; ++i) ss += ps[i].y;
            scale[t] = 1.0f / sqrtf(ss * (1.0f / (float)g.K) + g.stats_eps);
        }
        asm volatile("bar.sync 1, %0;" ::"n"(32 * kNormWarps) : "memory");
        for (int kb = 0; kb < n_kb; ++kb) {
            const int s = kb % kSplitStages, use = kb / kSplitStages;
            const uint4 gq = next;
            if (kb + 1 < n_kb) next = gains[8 * (kb + 1)];
            bool ok = true;
            uint32_t spins = 0;
            while (!mbar_try_wait_parked(&full[s], use & 1)) {
                if (((++spins) & 255u) == 0u && (*abort_flag || spins >= kSplitSpin)) { ok = false; break; }
            }
            if (!ok) { *abort_flag = 1; break; }
            const uint32_t gw[4] = {gq.x, gq.y, gq.z, gq.w};
            for (int r = t >> 3; r < rows; r += 4 * kNormWarps) {
                uint4* p = reinterpret_cast<uint4*>(sa + s * kSplitA + r * 128 + ((piece ^ (r & 7)) << 4));
                const uint4 x = *p;
                const uint32_t xw[4] = {x.x, x.y, x.z, x.w};
                const float rs = scale[r];
                uint32_t o[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) o[j] = pack_bf16x2(bf16r(bf_lo(xw[j]) * rs) * bf_lo(gw[j]), bf16r(bf_hi(xw[j]) * rs) * bf_hi(gw[j]));
                *p = make_uint4(o[0], o[1], o[2], o[3]);
            }
            fence_proxy_async_smem();                                // the MMAs read through the async proxy
            __syncwarp();
            if (lane == 0) mbar_arrive(&ready[s]);
        }
    }
    __syncwarp();
    pdl_wait();                                                      // the epilogue reads what the kernels before wrote
    bool ok = true;
    {
        uint32_t spins = 0;
        while (!mbar_try_wait_parked(acc_full, 0)) {
            if (((++spins) & 255u) == 0u && (*abort_flag || spins >= kSplitSpin)) { ok = false; break; }
        }
    }
    if (!ok) *abort_flag = 1;
    __syncwarp();
    tc_fence_after();
    // every MMA has finished, so every stage has been read: the ring becomes the partial tile.  Warp w reads TMEM lanes
    // 32 (w % 4) .. + 31 (32 rows of the tile), the two warps of a lane quarter half of the columns each.
    const int q = warp & 3;
    if (ok && q * 32 < rows) {
        float* dst = part + (size_t)(q * 32 + lane) * kPartLd + (warp >> 2) * (SN / 2);
#pragma unroll
        for (int c0 = 0; c0 < SN / 2; c0 += 32) {
            uint32_t r[32];
            tmem_ld_32x32(tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)((warp >> 2) * (SN / 2) + c0), r);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 8; ++i) *reinterpret_cast<uint4*>(dst + c0 + 4 * i) = make_uint4(r[4 * i], r[4 * i + 1], r[4 * i + 2], r[4 * i + 3]);
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) tmem_dealloc(tmem_base, kSplitCols);
    if (splits > 1) split_cluster_sync();
    uint32_t base[kMaxSplit];
#pragma unroll
    for (int s = 0; s < kMaxSplit; ++s)
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(base[s]) : "r"(smem_u32(part) + 16u * lane), "r"(s < splits ? s : 0));
    const int col0 = tile_n * SN;
    for (int r = rank + splits * warp; r < rows; r += splits * (kSplitThreads / 32)) {
        float4 p[kMaxSplit];
#pragma unroll
        for (int s = 0; s < kMaxSplit; ++s)
            if (s < splits) p[s] = ld_cluster_f4(base[s] + (uint32_t)r * (kPartLd * 4));
        float v[4] = {p[0].x, p[0].y, p[0].z, p[0].w};
#pragma unroll
        for (int s = 1; s < kMaxSplit; ++s)
            if (s < splits) { v[0] += p[s].x; v[1] += p[s].y; v[2] += p[s].z; v[3] += p[s].w; }
        split_epilogue_row(g, v, tile_m * SM_ + r, col0, lane);
    }
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
    if (splits > 1) split_cluster_sync();                            // no CTA leaves while another may still read its part
}

int cuda_fail(cudaError_t e, const char* what);

// CTAs that share a tile's K: a power of two (clusters of 3, 5 or 7 cost 5-15 % more than the next smaller power), at least three
// k-blocks each (12 k-blocks, 36 tiles: 7.2 us in four parts, 12.6 in eight), and two CTAs per SM at most save for a few
// (48 tiles: 6.8 us as 192 CTAs, 7.1 as 96; 72 tiles: 10.0 us as 288 CTAs, 8.7 as 144).
static int split_count(int tiles, int n_kb, int n_sms) {
    int s = 1;
    while (s < kMaxSplit && 2 * s * tiles * 4 <= 7 * n_sms && 2 * s * 3 <= n_kb) s *= 2;
    return s;
}

// The persistent pair kernel is the faster one as soon as a tile's K cannot be shared.  Measured on a B200 with weights from
// HBM, us, pair kernel -> this one: N 1024 K 3072 at M 196 / 512 / 1024 / 1536: 22.0 -> 9.1, 22.0 -> 11.6, 22.3 -> 15.9,
// 22.2 -> 25.0; N 768 K 768 at M 196 / 1536 / 2048: 9.3 -> 5.9, 9.6 -> 8.7, 9.7 -> 11.0; N 2304 K 768 at M 512 / 784:
// 10.1 -> 8.8, 10.2 -> 11.6.  Against 128 x 64 tiles walked by one CTA each (M <= 128): N 1024 K 3072 at M 32 / 128 18.6 -> 6.1,
// 19.0 -> 8.3; N 768 K 768 6.2 -> 4.2, 6.9 -> 5.9.
bool gemm_split_wins(int m, int n, int n_sms) { return m > 0 && n > 0 && 2ll * ((m + SM_ - 1) / SM_) * (n / SN) <= n_sms; }

int gemm_split_launch(const CUtensorMap& tm_a, const CUtensorMap& tm_b, const GemmArgs& g, int n_sms, cudaStream_t st) {
    static thread_local int attr_dev = -1;
    int dev = 0;
    cudaGetDevice(&dev);
    if (attr_dev != dev) {
        const cudaError_t e = cudaFuncSetAttribute(gemm_split_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSplitSmem);
        if (e != cudaSuccess) return cuda_fail(e, "cudaFuncSetAttribute(gemm_split)");
        attr_dev = dev;
    }
    const int tiles_m = (g.M + SM_ - 1) / SM_, tiles_n = g.N / SN, splits = split_count(tiles_m * tiles_n, g.K / SK, n_sms);
    const cudaError_t e = launch_pdl(gemm_split_kernel, dim3(splits, tiles_n, tiles_m), dim3(kSplitThreads), kSplitSmem, st, splits, tm_a, tm_b, g);
    return e == cudaSuccess ? ITTAI_OK : cuda_fail(e, "launch gemm_split_kernel");
}

}  // namespace ittai
