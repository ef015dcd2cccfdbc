// Softmax attention for the prefill and SigLIP paths: flash-style, 64 query rows x 64 keys per step, causal (Qwen3,
// grouped-query, head_dim 128) or dense with a key-length mask (SigLIP, head_dim 64).  Same schedule as the
// reference's attention tasks (src/ittai/qwen3/sm80.py:274-403, src/ittai/siglip/kernel.py:366-500): Q tile resident,
// K/V blocks streamed, scores and softmax in fp32 in the log2 domain, P rounded to bf16 for the PV product.
// Tensor-core path: warp-level mma.sync m16n8k16 (bf16 in, fp32 accumulate) on ldmatrix fragments from swizzled
// shared memory.  Attention is a few percent of SigLIP's FLOPs and a third of a 4k prefill's.
#include <type_traits>

#include "common.cuh"
#include "launch.h"

namespace ittai {

struct AttnArgs {
    const bf16* q; const bf16* k; const bf16* v; bf16* o;
    long long q_row, q_head, k_row, k_head, k_seq, v_row, v_head, v_seq, o_row, o_head;   // strides in elements
    const int4* seqs;     // per sequence: {first q/o row, q rows, first k/v row, k/v rows}
    int group;            // query heads per kv head
    float scale_log2;     // head_dim^-0.5 * log2(e)
};

__device__ __forceinline__ void cp_async16(void* dst, const void* src, bool pred) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    const int n = pred ? 16 : 0;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ void ldsm_x4(uint32_t (&r)[4], const void* p) {
    const uint32_t a = (uint32_t)__cvta_generic_to_shared(p);
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a));
}
__device__ __forceinline__ void ldsm_x4_t(uint32_t (&r)[4], const void* p) {
    const uint32_t a = (uint32_t)__cvta_generic_to_shared(p);
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a));
}
__device__ __forceinline__ void mma16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

constexpr int kAttnBN = 64;     // keys per step; query rows per CTA = 16 per warp, 4 warps (head_dim 128) or 8 (head_dim 64)

// element offset of 16-byte chunk `ch` of row `r` in a [rows][HD] tile whose chunks are XOR-swizzled by the row
template <int HD>
__device__ __forceinline__ int sw(int r, int ch) { return r * HD + ((ch ^ (r & 7)) << 3); }

template <int HD, int ROWS, int THREADS>
__device__ __forceinline__ void load_tile(bf16* dst, const bf16* src, long long row_stride, int rows_valid, int tid) {
    constexpr int CH = HD / 8;
    for (int i = tid; i < ROWS * CH; i += THREADS) {
        const int r = i / CH, ch = i % CH;
        cp_async16(dst + sw<HD>(r, ch), src + (long long)r * row_stride + ch * 8, r < rows_valid);
    }
}

template <int HD, bool CAUSAL, int WARPS>
__global__ void __launch_bounds__(WARPS * 32) attn_fwd_kernel(const AttnArgs a) {
    pdl_trigger();
    pdl_wait();
    const int4 sinfo = a.seqs[blockIdx.z];
    constexpr int kAttnBM = 16 * WARPS, kAttnThreads = 32 * WARPS;
    // shared memory: Q tile, then two (K, V) tile pairs so that block kb+1 streams in while block kb is multiplied
    extern __shared__ __align__(128) unsigned char attn_smem[];
    bf16* sq = reinterpret_cast<bf16*>(attn_smem);
    bf16* skv = sq + kAttnBM * HD;                                    // [2][K | V][64 * HD]
    const int q_len = sinfo.y, kv_len = sinfo.w;
    const int qb = blockIdx.x * kAttnBM;
    if (qb >= q_len) return;
    const int head = blockIdx.y, kvh = head / a.group;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
    const bf16* qp = a.q + (long long)(sinfo.x + qb) * a.q_row + (long long)head * a.q_head;
    const bf16* kp = a.k + (long long)blockIdx.z * a.k_seq + (long long)kvh * a.k_head + (long long)sinfo.z * a.k_row;
    const bf16* vp = a.v + (long long)blockIdx.z * a.v_seq + (long long)kvh * a.v_head + (long long)sinfo.z * a.v_row;
    const int q_rows = q_len - qb < kAttnBM ? q_len - qb : kAttnBM;
    const int shift = kv_len - q_len;                       // query i sees keys j <= i + shift
    int kv_end = kv_len;
    if (CAUSAL) { const int lim = qb + q_rows + shift; kv_end = lim < kv_len ? lim : kv_len; }
    const bool warp_live = warp * 16 < q_rows;              // a warp whose 16 rows are all padding only helps loading

    auto load_kv = [&](int kb, int buf) {
        const int rows_valid = kv_len - kb < kAttnBN ? kv_len - kb : kAttnBN;
        load_tile<HD, kAttnBN, kAttnThreads>(skv + (size_t)buf * 2 * kAttnBN * HD, kp + (long long)kb * a.k_row, a.k_row, rows_valid, tid);
        load_tile<HD, kAttnBN, kAttnThreads>(skv + (size_t)buf * 2 * kAttnBN * HD + kAttnBN * HD, vp + (long long)kb * a.v_row, a.v_row, rows_valid, tid);
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    load_tile<HD, kAttnBM, kAttnThreads>(sq, qp, a.q_row, q_rows, tid);
    if (kv_end > 0) load_kv(0, 0); else asm volatile("cp.async.commit_group;" ::: "memory");
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    uint32_t qf[HD / 16][4];
#pragma unroll
    for (int ks = 0; ks < HD / 16; ++ks)
        ldsm_x4(qf[ks], sq + sw<HD>(warp * 16 + (lane & 7) + ((lane >> 3) & 1) * 8, ks * 2 + (lane >> 4)));

    float o[HD / 8][4];
#pragma unroll
    for (int i = 0; i < HD / 8; ++i) { o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.f; }
    float m0 = -INFINITY, m1 = -INFINITY, l0 = 0.f, l1 = 0.f;     // rows g and g + 8 of this warp's 16
    const int row0 = qb + warp * 16 + g, row1 = row0 + 8;

    int buf = 0;
    for (int kb = 0; kb < kv_end; kb += kAttnBN, buf ^= 1) {
        // block kb is in `buf` (waited for below or before the loop); start fetching the next one into the other half
        if (kb + kAttnBN < kv_end) load_kv(kb + kAttnBN, buf ^ 1);
        const bf16* sk = skv + (size_t)buf * 2 * kAttnBN * HD;
        const bf16* sv = sk + kAttnBN * HD;
        const int rows_valid = kv_len - kb < kAttnBN ? kv_len - kb : kAttnBN;
        const int n16 = (rows_valid + 15) / 16;              // 16-key groups that hold at least one real key
        if (warp_live) {
            // ---- S = Q K^T
            float s[kAttnBN / 8][4];
#pragma unroll
            for (int i = 0; i < kAttnBN / 8; ++i) { s[i][0] = s[i][1] = s[i][2] = s[i][3] = 0.f; }
#pragma unroll
            for (int ks = 0; ks < HD / 16; ++ks) {
#pragma unroll
                for (int np = 0; np < kAttnBN / 16; ++np) {
                    if (np < n16) {
                        uint32_t kf[4];
                        ldsm_x4(kf, sk + sw<HD>(np * 16 + (lane & 7) + (lane >> 4) * 8, ks * 2 + ((lane >> 3) & 1)));
                        mma16816(s[2 * np], qf[ks], kf[0], kf[1]);
                        mma16816(s[2 * np + 1], qf[ks], kf[2], kf[3]);
                    }
                }
            }
            // ---- mask, scale, online softmax
            float mx0 = -INFINITY, mx1 = -INFINITY;
#pragma unroll
            for (int i = 0; i < kAttnBN / 8; ++i) {
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int j = kb + i * 8 + 2 * t + (e & 1), r = (e < 2) ? row0 : row1;
                    const bool vis = j < kv_len && (!CAUSAL || j <= r + shift);
                    s[i][e] = vis ? s[i][e] * a.scale_log2 : -INFINITY;
                }
                mx0 = fmaxf(mx0, fmaxf(s[i][0], s[i][1]));
                mx1 = fmaxf(mx1, fmaxf(s[i][2], s[i][3]));
            }
            mx0 = fmaxf(mx0, __shfl_xor_sync(0xffffffffu, mx0, 1)); mx0 = fmaxf(mx0, __shfl_xor_sync(0xffffffffu, mx0, 2));
            mx1 = fmaxf(mx1, __shfl_xor_sync(0xffffffffu, mx1, 1)); mx1 = fmaxf(mx1, __shfl_xor_sync(0xffffffffu, mx1, 2));
            const float mn0 = fmaxf(m0, mx0), mn1 = fmaxf(m1, mx1);
            const float ms0 = mn0 == -INFINITY ? 0.f : mn0, ms1 = mn1 == -INFINITY ? 0.f : mn1;
            const float c0 = exp2f(m0 - ms0), c1 = exp2f(m1 - ms1);
            m0 = mn0; m1 = mn1;
            float ps0 = 0.f, ps1 = 0.f;
            uint32_t pf[kAttnBN / 16][4];
#pragma unroll
            for (int i = 0; i < kAttnBN / 8; ++i) {
                const float p0 = exp2f(s[i][0] - ms0), p1 = exp2f(s[i][1] - ms0), p2 = exp2f(s[i][2] - ms1), p3 = exp2f(s[i][3] - ms1);
                ps0 += p0 + p1; ps1 += p2 + p3;
                pf[i / 2][(i & 1) * 2] = pack_bf16x2(p0, p1);
                pf[i / 2][(i & 1) * 2 + 1] = pack_bf16x2(p2, p3);
            }
            l0 = l0 * c0 + ps0; l1 = l1 * c1 + ps1;
#pragma unroll
            for (int i = 0; i < HD / 8; ++i) { o[i][0] *= c0; o[i][1] *= c0; o[i][2] *= c1; o[i][3] *= c1; }
            // ---- O += P V
#pragma unroll
            for (int ks = 0; ks < kAttnBN / 16; ++ks) {
                if (ks < n16) {
#pragma unroll
                    for (int dp = 0; dp < HD / 16; ++dp) {
                        uint32_t vf[4];
                        ldsm_x4_t(vf, sv + sw<HD>(ks * 16 + (lane & 7) + ((lane >> 3) & 1) * 8, dp * 2 + (lane >> 4)));
                        mma16816(o[2 * dp], pf[ks], vf[0], vf[1]);
                        mma16816(o[2 * dp + 1], pf[ks], vf[2], vf[3]);
                    }
                }
            }
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");   // the next block has landed
        __syncthreads();                                      // and everyone is done reading this one
    }
    if (!warp_live) return;
    // ---- normalise and store
    l0 += __shfl_xor_sync(0xffffffffu, l0, 1); l0 += __shfl_xor_sync(0xffffffffu, l0, 2);
    l1 += __shfl_xor_sync(0xffffffffu, l1, 1); l1 += __shfl_xor_sync(0xffffffffu, l1, 2);
    const float i0 = l0 > 0.f ? 1.0f / l0 : 0.f, i1 = l1 > 0.f ? 1.0f / l1 : 0.f;
    bf16* op = a.o + (long long)sinfo.x * a.o_row + (long long)head * a.o_head;
#pragma unroll
    for (int i = 0; i < HD / 8; ++i) {
        const int d = i * 8 + 2 * t;
        if (row0 < q_len) *reinterpret_cast<uint32_t*>(op + (long long)row0 * a.o_row + d) = pack_bf16x2(o[i][0] * i0, o[i][1] * i0);
        if (row1 < q_len) *reinterpret_cast<uint32_t*>(op + (long long)row1 * a.o_row + d) = pack_bf16x2(o[i][2] * i1, o[i][3] * i1);
    }
}

// Few queries (at most 64 a sequence), causal, head_dim 128: a short prompt.  One CTA per (sequence, head, ROWS queries), 32 keys a step, the next
// step's on their way meanwhile.  It runs once per layer, so what attn_fwd_kernel spends here, its 64-key steps unrolled for keys that do not
// exist, is code to be fetched (see the attention of qwen3_chain.cu) and masks.  ROWS = 32: two warps per 16 queries that both compute the scores
// and share the output's 128 columns out, the shorter chain; ROWS = 64: a warp per 16 queries, half the loads and two thirds of the MMAs, where
// there are more tiles than SMs.  A query's values are the same bits in both.  How the CTAs are spread over the SMs: attn_few_launch_rows.
// Forwards of 3 / 8 / 23 / 32 / 48 / 64 tokens with split-K projections, us, attn_fwd_kernel -> this: 627 / 637 / 669 / 737 / 834 / 927 -> 555 / 568 /
// 602 / 671 / 769 / 852; 40 texts of 60 tokens 3086 -> 2937, 130 of 40 5574 -> 5440.  (Above 64 the key-loop kernel on tcgen05 takes over.)
constexpr int kFewMax = 64, kFewKeys = 32, kFewThreads = 128;
__device__ __forceinline__ float ex2_ftz(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
template <int ROWS>
__global__ void __launch_bounds__(kFewThreads) attn_few_kernel(const AttnArgs a, int seqs_ready) {
    constexpr int HD = 128, kShare = ROWS / 16 * 32 == kFewThreads ? 1 : 2, kCols = HD / kShare;   // warps that share 16 queries' columns out
    static_assert(ROWS / 16 * kShare * 32 == kFewThreads, "");
    extern __shared__ __align__(128) unsigned char attn_smem[];
    bf16* sq = reinterpret_cast<bf16*>(attn_smem);
    bf16* skv = sq + ROWS * HD;                                   // [2][K | V][32 * HD]
    const int tid = threadIdx.x, warp = warp_index(), lane = tid & 31, g = lane >> 2, t = lane & 3;
    pdl_trigger();
    // With records that may be read ahead of the wait the addresses are there behind it: 400 of the kernel's 3200 cycles at 23 tokens.
    if (!seqs_ready) pdl_wait();
    const int4 sinfo = a.seqs[blockIdx.z];
    const int q_len = sinfo.y, kv_len = sinfo.w, qb = blockIdx.x * ROWS;
    // an empty tile; a first one waits even so: behind a grid without any wait the next one would start ahead of what runs in front of this
    if (qb >= q_len) {
        if (seqs_ready && blockIdx.x == 0) pdl_wait();
        return;
    }
    const int head = blockIdx.y, kvh = head / a.group;
    const bf16* qp = a.q + (long long)(sinfo.x + qb) * a.q_row + (long long)head * a.q_head;
    const bf16* kp = a.k + (long long)blockIdx.z * a.k_seq + (long long)kvh * a.k_head + (long long)sinfo.z * a.k_row;
    const bf16* vp = a.v + (long long)blockIdx.z * a.v_seq + (long long)kvh * a.v_head + (long long)sinfo.z * a.v_row;
    const int q_rows = q_len - qb < ROWS ? q_len - qb : ROWS;
    const int shift = kv_len - q_len + qb;                            // row i of the tile sees keys j <= i + shift
    const int kv_end = q_rows + shift < kv_len ? q_rows + shift : kv_len;
    // thread: 16-byte piece tid % 16 of rows tid / 16 + 8 i
    const int lr = tid >> 4, lc = tid & 15;
    const bf16 *qt = qp + lr * a.q_row + lc * 8, *kt = kp + lr * a.k_row + lc * 8, *vt = vp + lr * a.v_row + lc * 8;
    long long q8 = 8 * a.q_row, k8 = 8 * a.k_row, v8 = 8 * a.v_row;
    asm volatile("" : "+l"(qt), "+l"(kt), "+l"(vt), "+l"(q8), "+l"(k8), "+l"(v8));
    // rows past the end: the first one's address, nothing read
    auto load = [&](bf16* dst, const bf16* src, long long step, int rows, auto pieces) {
#pragma unroll
        for (int i = 0; i < decltype(pieces)::value; ++i) cp_async16(dst + sw<HD>(lr + 8 * i, lc), lr + 8 * i < rows ? src + i * step : a.q, lr + 8 * i < rows);
    };
    auto load_kv = [&](int kb, int buf) {
        bf16* dst = skv + (size_t)buf * 2 * kFewKeys * HD;
        load(dst, kt, k8, kv_end - kb, std::integral_constant<int, kFewKeys / 8>());
        load(dst + kFewKeys * HD, vt, v8, kv_end - kb, std::integral_constant<int, kFewKeys / 8>());
        kt += 4 * k8; vt += 4 * v8;
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    if (seqs_ready) pdl_wait();
    load(sq, qt, q8, q_rows, std::integral_constant<int, ROWS / 8>());
    if (kv_end > 0) load_kv(0, 0); else asm volatile("cp.async.commit_group;" ::: "memory");
    const int rt = 16 * (warp / kShare), part = warp % kShare;        // this warp's 16 queries, and its share of the output columns
    float o[kCols / 8][4];
#pragma unroll
    for (int i = 0; i < kCols / 8; ++i) o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.f;
    float m0 = -INFINITY, m1 = -INFINITY, l0 = 0.f, l1 = 0.f;         // rows g and g + 8
    const int r0 = rt + g, r1 = r0 + 8;
    int buf = 0;
#pragma unroll 1
    for (int kb = 0; kb < kv_end; kb += kFewKeys, buf ^= 1) {
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();                                              // this step's keys are there, and the other buffer has been read
        if (kb + kFewKeys < kv_end) load_kv(kb + kFewKeys, buf ^ 1);
        const bf16* sk = skv + (size_t)buf * 2 * kFewKeys * HD;
        const bf16* sv = sk + kFewKeys * HD;
        float s[4][4];
#pragma unroll
        for (int i = 0; i < 4; ++i) s[i][0] = s[i][1] = s[i][2] = s[i][3] = 0.f;
#pragma unroll
        for (int ks = 0; ks < HD / 16; ++ks) {
            uint32_t qf[4], kf[4];
            ldsm_x4(qf, sq + sw<HD>(rt + (lane & 15), ks * 2 + (lane >> 4)));
#pragma unroll
            for (int np = 0; np < 2; ++np) {
                ldsm_x4(kf, sk + sw<HD>(np * 16 + (lane & 7) + (lane >> 4) * 8, ks * 2 + ((lane >> 3) & 1)));
                mma16816(s[2 * np], qf, kf[0], kf[1]);
                mma16816(s[2 * np + 1], qf, kf[2], kf[3]);
            }
        }
        float x0 = -INFINITY, x1 = -INFINITY;
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int j = kb + 8 * i + 2 * t + e;
                s[i][e] = j < kv_len && j <= r0 + shift ? s[i][e] * a.scale_log2 : -INFINITY;
                s[i][e + 2] = j < kv_len && j <= r1 + shift ? s[i][e + 2] * a.scale_log2 : -INFINITY;
                x0 = fmaxf(x0, s[i][e]); x1 = fmaxf(x1, s[i][e + 2]);
            }
        x0 = fmaxf(x0, __shfl_xor_sync(0xffffffffu, x0, 1)); x1 = fmaxf(x1, __shfl_xor_sync(0xffffffffu, x1, 1));
        x0 = fmaxf(x0, __shfl_xor_sync(0xffffffffu, x0, 2)); x1 = fmaxf(x1, __shfl_xor_sync(0xffffffffu, x1, 2));
        const float n0 = fmaxf(m0, x0), n1 = fmaxf(m1, x1);
        const float f0 = n0 == -INFINITY ? 0.f : n0, f1 = n1 == -INFINITY ? 0.f : n1;      // a row without keys so far
        const float c0 = ex2_ftz(m0 - f0), c1 = ex2_ftz(m1 - f1);
        m0 = n0; m1 = n1;
        uint32_t pf[2][4];
        float p0 = 0.f, p1 = 0.f;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float e0 = ex2_ftz(s[i][0] - f0), e1 = ex2_ftz(s[i][1] - f0), e2 = ex2_ftz(s[i][2] - f1), e3 = ex2_ftz(s[i][3] - f1);
            p0 += e0 + e1; p1 += e2 + e3;
            pf[i / 2][(i & 1) * 2] = pack_bf16x2(e0, e1);
            pf[i / 2][(i & 1) * 2 + 1] = pack_bf16x2(e2, e3);
        }
        l0 = l0 * c0 + p0; l1 = l1 * c1 + p1;
#pragma unroll
        for (int i = 0; i < kCols / 8; ++i) { o[i][0] *= c0; o[i][1] *= c0; o[i][2] *= c1; o[i][3] *= c1; }
#pragma unroll
        for (int ks = 0; ks < 2; ++ks)
#pragma unroll
            for (int dp = 0; dp < kCols / 16; ++dp) {
                uint32_t vf[4];
                ldsm_x4_t(vf, sv + sw<HD>(ks * 16 + (lane & 7) + ((lane >> 3) & 1) * 8, kCols / 8 * part + dp * 2 + (lane >> 4)));
                mma16816(o[2 * dp], pf[ks], vf[0], vf[1]);
                mma16816(o[2 * dp + 1], pf[ks], vf[2], vf[3]);
            }
    }
    if (rt >= q_rows) return;
    l0 += __shfl_xor_sync(0xffffffffu, l0, 1); l0 += __shfl_xor_sync(0xffffffffu, l0, 2);
    l1 += __shfl_xor_sync(0xffffffffu, l1, 1); l1 += __shfl_xor_sync(0xffffffffu, l1, 2);
    const float i0 = l0 > 0.f ? 1.0f / l0 : 0.f, i1 = l1 > 0.f ? 1.0f / l1 : 0.f;
    bf16* op = a.o + (long long)(sinfo.x + qb) * a.o_row + (long long)head * a.o_head + kCols * part + 2 * t;
#pragma unroll
    for (int i = 0; i < kCols / 8; ++i) {
        if (r0 < q_rows) *reinterpret_cast<uint32_t*>(op + (long long)r0 * a.o_row + 8 * i) = pack_bf16x2(o[i][0] * i0, o[i][1] * i0);
        if (r1 < q_rows) *reinterpret_cast<uint32_t*>(op + (long long)r1 * a.o_row + 8 * i) = pack_bf16x2(o[i][2] * i1, o[i][3] * i1);
    }
}

// Short sequences (at most 256 keys, dense): one CTA per (sequence, head) keeps the whole K and V in shared memory,
// loaded once, and every warp runs its 16 query rows against all keys with no CTA-wide barrier after the load: 13 warps
// for SigLIP's 196 tokens, two CTAs per SM.  K and V are read from HBM once per head instead of once per query block.
constexpr int kShortKeys = 256;
template <int HD>
__global__ void __launch_bounds__(512) attn_short_kernel(const AttnArgs a, int warps) {
    pdl_trigger();
    pdl_wait();
    extern __shared__ __align__(128) unsigned char attn_smem[];
    const int4 sinfo = a.seqs[blockIdx.z];
    const int q_len = sinfo.y, kv_len = sinfo.w;
    const int head = blockIdx.y, kvh = head / a.group;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
    const int q_rows_pad = warps * 16, threads = warps * 32;
    bf16* sq = reinterpret_cast<bf16*>(attn_smem);
    bf16* sk = sq + q_rows_pad * HD;
    bf16* sv = sk + kShortKeys * HD;
    const bf16* qp = a.q + (long long)sinfo.x * a.q_row + (long long)head * a.q_head;
    const bf16* kp = a.k + (long long)blockIdx.z * a.k_seq + (long long)kvh * a.k_head + (long long)sinfo.z * a.k_row;
    const bf16* vp = a.v + (long long)blockIdx.z * a.v_seq + (long long)kvh * a.v_head + (long long)sinfo.z * a.v_row;
    constexpr int CH = HD / 8;
    const int kv_pad = (kv_len + 15) & ~15;
    for (int i = tid; i < q_rows_pad * CH; i += threads) {
        const int r = i / CH, ch = i % CH;
        cp_async16(sq + sw<HD>(r, ch), qp + (long long)r * a.q_row + ch * 8, r < q_len);
    }
    for (int i = tid; i < kv_pad * CH; i += threads) {
        const int r = i / CH, ch = i % CH;
        cp_async16(sk + sw<HD>(r, ch), kp + (long long)r * a.k_row + ch * 8, r < kv_len);
        cp_async16(sv + sw<HD>(r, ch), vp + (long long)r * a.v_row + ch * 8, r < kv_len);
    }
    asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    if (warp * 16 >= q_len) return;
    uint32_t qf[HD / 16][4];
#pragma unroll
    for (int ks = 0; ks < HD / 16; ++ks)
        ldsm_x4(qf[ks], sq + sw<HD>(warp * 16 + (lane & 7) + ((lane >> 3) & 1) * 8, ks * 2 + (lane >> 4)));
    float o[HD / 8][4];
#pragma unroll
    for (int i = 0; i < HD / 8; ++i) { o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.f; }
    float m0 = -INFINITY, m1 = -INFINITY, l0 = 0.f, l1 = 0.f;
    for (int kb = 0; kb < kv_len; kb += kAttnBN) {
        const int rows_valid = kv_len - kb < kAttnBN ? kv_len - kb : kAttnBN;
        const int n16 = (rows_valid + 15) / 16;
        float s[kAttnBN / 8][4];
#pragma unroll
        for (int i = 0; i < kAttnBN / 8; ++i) { s[i][0] = s[i][1] = s[i][2] = s[i][3] = 0.f; }
#pragma unroll
        for (int ks = 0; ks < HD / 16; ++ks) {
#pragma unroll
            for (int np = 0; np < kAttnBN / 16; ++np) {
                if (np < n16) {
                    uint32_t kf[4];
                    ldsm_x4(kf, sk + sw<HD>(kb + np * 16 + (lane & 7) + (lane >> 4) * 8, ks * 2 + ((lane >> 3) & 1)));
                    mma16816(s[2 * np], qf[ks], kf[0], kf[1]);
                    mma16816(s[2 * np + 1], qf[ks], kf[2], kf[3]);
                }
            }
        }
        float mx0 = -INFINITY, mx1 = -INFINITY;
#pragma unroll
        for (int i = 0; i < kAttnBN / 8; ++i) {
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int j = kb + i * 8 + 2 * t + (e & 1);
                s[i][e] = j < kv_len ? s[i][e] * a.scale_log2 : -INFINITY;
            }
            mx0 = fmaxf(mx0, fmaxf(s[i][0], s[i][1]));
            mx1 = fmaxf(mx1, fmaxf(s[i][2], s[i][3]));
        }
        mx0 = fmaxf(mx0, __shfl_xor_sync(0xffffffffu, mx0, 1)); mx0 = fmaxf(mx0, __shfl_xor_sync(0xffffffffu, mx0, 2));
        mx1 = fmaxf(mx1, __shfl_xor_sync(0xffffffffu, mx1, 1)); mx1 = fmaxf(mx1, __shfl_xor_sync(0xffffffffu, mx1, 2));
        const float mn0 = fmaxf(m0, mx0), mn1 = fmaxf(m1, mx1);
        const float c0 = exp2f(m0 - mn0), c1 = exp2f(m1 - mn1);       // every block holds a real key, so mn is finite
        m0 = mn0; m1 = mn1;
        float ps0 = 0.f, ps1 = 0.f;
        uint32_t pf[kAttnBN / 16][4];
#pragma unroll
        for (int i = 0; i < kAttnBN / 8; ++i) {
            const float p0 = exp2f(s[i][0] - mn0), p1 = exp2f(s[i][1] - mn0), p2 = exp2f(s[i][2] - mn1), p3 = exp2f(s[i][3] - mn1);
            ps0 += p0 + p1; ps1 += p2 + p3;
            pf[i / 2][(i & 1) * 2] = pack_bf16x2(p0, p1);
            pf[i / 2][(i & 1) * 2 + 1] = pack_bf16x2(p2, p3);
        }
        l0 = l0 * c0 + ps0; l1 = l1 * c1 + ps1;
#pragma unroll
        for (int i = 0; i < HD / 8; ++i) { o[i][0] *= c0; o[i][1] *= c0; o[i][2] *= c1; o[i][3] *= c1; }
#pragma unroll
        for (int ks = 0; ks < kAttnBN / 16; ++ks) {
            if (ks < n16) {
#pragma unroll
                for (int dp = 0; dp < HD / 16; ++dp) {
                    uint32_t vf[4];
                    ldsm_x4_t(vf, sv + sw<HD>(kb + ks * 16 + (lane & 7) + ((lane >> 3) & 1) * 8, dp * 2 + (lane >> 4)));
                    mma16816(o[2 * dp], pf[ks], vf[0], vf[1]);
                    mma16816(o[2 * dp + 1], pf[ks], vf[2], vf[3]);
                }
            }
        }
    }
    l0 += __shfl_xor_sync(0xffffffffu, l0, 1); l0 += __shfl_xor_sync(0xffffffffu, l0, 2);
    l1 += __shfl_xor_sync(0xffffffffu, l1, 1); l1 += __shfl_xor_sync(0xffffffffu, l1, 2);
    const float i0 = l0 > 0.f ? 1.0f / l0 : 0.f, i1 = l1 > 0.f ? 1.0f / l1 : 0.f;
    const int row0 = warp * 16 + g, row1 = row0 + 8;
    bf16* op = a.o + (long long)sinfo.x * a.o_row + (long long)head * a.o_head;
#pragma unroll
    for (int i = 0; i < HD / 8; ++i) {
        const int d = i * 8 + 2 * t;
        if (row0 < q_len) *reinterpret_cast<uint32_t*>(op + (long long)row0 * a.o_row + d) = pack_bf16x2(o[i][0] * i0, o[i][1] * i0);
        if (row1 < q_len) *reinterpret_cast<uint32_t*>(op + (long long)row1 * a.o_row + d) = pack_bf16x2(o[i][2] * i1, o[i][3] * i1);
    }
}

// One query per sequence (the SigLIP MAP head: a learned probe attends over the tokens), head_dim 64: a CTA of 16 warps
// per (sequence, head); 8 lanes share a key (8 dims each, one 16-byte load), so the CTA's 64 groups have 196 keys in hand with four
// requests each, all of them on their way before the first score.  Each group keeps a private online softmax; the four groups of a
// warp meet through shuffles, the warps through shared memory.  Latency: with 16 groups walking the keys one after the other one image
// took 11.2 us and 8 images 14.5; 8 images take 4.2 this way.
constexpr int kQ1Warps = 16, kQ1Groups = 4 * kQ1Warps, kQ1Keys = 4;
__global__ void __launch_bounds__(32 * kQ1Warps) attn_q1_kernel(const AttnArgs a) {
    pdl_trigger();
    pdl_wait();
    const int head = blockIdx.x, kvh = head / a.group;
    const int4 sinfo = a.seqs[blockIdx.y];
    const int kv_len = sinfo.w;
    const int warp = threadIdx.x >> 5, grp = threadIdx.x >> 3, sub = threadIdx.x & 7;
    __shared__ float s_m[kQ1Warps], s_l[kQ1Warps], s_o[kQ1Warps][64];
    const bf16* qp = a.q + (long long)sinfo.x * a.q_row + (long long)head * a.q_head + 8 * sub;
    const uint4 qw = *reinterpret_cast<const uint4*>(qp);
    const uint32_t qq[4] = {qw.x, qw.y, qw.z, qw.w};
    float q[8];
#pragma unroll
    for (int j = 0; j < 4; ++j) { q[2 * j] = bf_lo(qq[j]) * a.scale_log2; q[2 * j + 1] = bf_hi(qq[j]) * a.scale_log2; }
    const bf16* kb = a.k + (long long)blockIdx.y * a.k_seq + (long long)kvh * a.k_head + (long long)sinfo.z * a.k_row + 8 * sub;
    const bf16* vb = a.v + (long long)blockIdx.y * a.v_seq + (long long)kvh * a.v_head + (long long)sinfo.z * a.v_row + 8 * sub;
    float m = -INFINITY, l = 0.f, acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    for (int j0 = 0; j0 < kv_len; j0 += kQ1Groups * kQ1Keys) {
        uint4 kw[kQ1Keys], vw[kQ1Keys];
#pragma unroll
        for (int u = 0; u < kQ1Keys; ++u) {
            const int j = j0 + grp + u * kQ1Groups;
            kw[u] = make_uint4(0, 0, 0, 0); vw[u] = kw[u];
            if (j < kv_len) {
                kw[u] = *reinterpret_cast<const uint4*>(kb + (long long)j * a.k_row);
                vw[u] = *reinterpret_cast<const uint4*>(vb + (long long)j * a.v_row);
            }
        }
#pragma unroll
        for (int u = 0; u < kQ1Keys; ++u) {
            const uint32_t kk[4] = {kw[u].x, kw[u].y, kw[u].z, kw[u].w}, vv[4] = {vw[u].x, vw[u].y, vw[u].z, vw[u].w};
            float sc = 0.f;
#pragma unroll
            for (int e = 0; e < 4; ++e) sc += q[2 * e] * bf_lo(kk[e]) + q[2 * e + 1] * bf_hi(kk[e]);
#pragma unroll
            for (int o = 4; o > 0; o >>= 1) sc += __shfl_xor_sync(0xffffffffu, sc, o);
            if (j0 + grp + u * kQ1Groups < kv_len) {
                const float mn = fmaxf(m, sc), c = exp2f(m - mn), pr = exp2f(sc - mn);
                l = l * c + pr;
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    acc[2 * e] = acc[2 * e] * c + pr * bf_lo(vv[e]);
                    acc[2 * e + 1] = acc[2 * e + 1] * c + pr * bf_hi(vv[e]);
                }
                m = mn;
            }
        }
    }
    // a group without keys has m = -inf and weighs nothing
#pragma unroll
    for (int o = 8; o < 32; o <<= 1) {
        const float m2 = __shfl_xor_sync(0xffffffffu, m, o), l2 = __shfl_xor_sync(0xffffffffu, l, o), mn = fmaxf(m, m2);
        const float c = m == -INFINITY ? 0.f : exp2f(m - mn), c2 = m2 == -INFINITY ? 0.f : exp2f(m2 - mn);
        l = l * c + l2 * c2;
#pragma unroll
        for (int e = 0; e < 8; ++e) acc[e] = acc[e] * c + __shfl_xor_sync(0xffffffffu, acc[e], o) * c2;
        m = mn;
    }
    if ((threadIdx.x & 31) < 8) {
        if (sub == 0) { s_m[warp] = m; s_l[warp] = l; }
#pragma unroll
        for (int e = 0; e < 8; ++e) s_o[warp][8 * sub + e] = acc[e];
    }
    __syncthreads();
    if (threadIdx.x < 64) {
        float M = -INFINITY;
#pragma unroll
        for (int g = 0; g < kQ1Warps; ++g) M = fmaxf(M, s_m[g]);
        float o = 0.f, L = 0.f;
        if (M != -INFINITY) {
#pragma unroll
            for (int g = 0; g < kQ1Warps; ++g) {
                const float w = exp2f(s_m[g] - M);        // a warp without keys has m = -inf: weight 0
                o = fmaf(s_o[g][threadIdx.x], w, o);
                L = fmaf(s_l[g], w, L);
            }
        }
        a.o[(long long)sinfo.x * a.o_row + (long long)head * a.o_head + threadIdx.x] = __float2bfloat16_rn(L > 0.f ? o / L : 0.f);
    }
}

static int attn_short_launch(const AttnArgs& a, int max_q_len, int n_heads, int n_seqs, cudaStream_t st) {
    const int warps = (max_q_len + 15) / 16;
    const size_t smem = (size_t)(warps * 16 + 2 * kShortKeys) * 64 * 2;
    static thread_local int attr_dev = -1;
    int dev = 0;
    cudaGetDevice(&dev);
    if (attr_dev != dev) {
        const cudaError_t e = cudaFuncSetAttribute(attn_short_kernel<64>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)((16 * 16 + 2 * kShortKeys) * 64 * 2));
        if (e != cudaSuccess) return (int)e;
        attr_dev = dev;
    }
    launch_pdl(attn_short_kernel<64>, dim3(1, n_heads, n_seqs), dim3(warps * 32), smem, st, 1, a, warps);
    return 0;
}

template <int HD, bool CAUSAL, int WARPS>
static int attn_launch(const AttnArgs& a, int max_q_len, int n_heads, int n_seqs, cudaStream_t st) {
    constexpr size_t smem = (size_t)(16 * WARPS + 4 * kAttnBN) * HD * 2;
    const dim3 grid((max_q_len + 16 * WARPS - 1) / (16 * WARPS), n_heads, n_seqs);
    static thread_local int attr_dev = -1;
    int dev = 0;
    cudaGetDevice(&dev);
    if (attr_dev != dev) {
        const cudaError_t e = cudaFuncSetAttribute(attn_fwd_kernel<HD, CAUSAL, WARPS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return (int)e;
        attr_dev = dev;
    }
    launch_pdl(attn_fwd_kernel<HD, CAUSAL, WARPS>, grid, dim3(WARPS * 32), smem, st, 1, a);
    return 0;
}

// A CTA asks for so much shared memory that an SM takes no more of them than its even share: they start while the kernel in front holds most SMs, and
// without that the empty ones filled up (five on an SM), which a long cache then paid for.  16 heads, one layer, us, attn_fwd_kernel / packed / spread:
// 16 sequences of 16 queries behind 1000 cached keys 39 / 51 / 31, four of 64 45 / 36 / 24.  Forwards of 28 layers, us: 4 x 2 tokens behind 7900 cached
// ones 8640 / 11 340 / 5650, 8 x 5 behind 1000 2010 / 2270 / 1570; texts of 40 and 64 tokens 874 / 756 / 732 and 996 / 940 / 921.
template <int ROWS>
static cudaError_t attn_few_launch_rows(const AttnArgs& a, int max_q_len, int n_heads, int n_seqs, int seqs_ready, int n_sms, cudaStream_t st) {
    constexpr int kNeed = (ROWS + 4 * kFewKeys) * 128 * 2, kSm = 228 * 1024, kLone = kSm / 2 + 128;
    static thread_local int attr_dev = -1;
    int dev = 0;
    cudaGetDevice(&dev);
    if (attr_dev != dev) {
        const cudaError_t e = cudaFuncSetAttribute(attn_few_kernel<ROWS>, cudaFuncAttributeMaxDynamicSharedMemorySize, kLone);
        if (e != cudaSuccess) return e;
        attr_dev = dev;
    }
    const dim3 grid((max_q_len + ROWS - 1) / ROWS, n_heads, n_seqs);
    const long long per_sm = ((long long)grid.x * grid.y * grid.z + n_sms - 1) / n_sms;
    const int room = kSm / (int)(per_sm < 8 ? per_sm + 1 : 9) - 1024 + 128;        // per_sm + 1 of them, with 1 KB each for the system, do not fit
    return launch_pdl(attn_few_kernel<ROWS>, grid, dim3(kFewThreads), (size_t)(room > kNeed ? room : kNeed), st, 1, a, seqs_ready);
}
static cudaError_t attn_few_launch(const AttnArgs& a, int max_q_len, int n_heads, int n_seqs, int seqs_ready, cudaStream_t st) {
    static thread_local int sm_dev = -1, n_sms = 0;
    int dev = 0;
    cudaGetDevice(&dev);
    if (sm_dev != dev) {
        const cudaError_t e = cudaDeviceGetAttribute(&n_sms, cudaDevAttrMultiProcessorCount, dev);
        if (e != cudaSuccess) return e;
        sm_dev = dev;
    }
    // More tiles of 32 queries than SMs: tiles of 64, if there are so many queries.  One layer, us, attn_fwd_kernel / tiles of 32 / of 64: 64 sequences of
    // 33 queries behind 1000 keys 180 / 187 / 121, of 64 behind 100 42 / 41 / 29, five (160 tiles of 32) of 33 behind 1000 44 / 32 / 25; but four (128)
    // 44 / 23.6 / 24.5.
    const bool whole = max_q_len > 32 && 2ll * n_heads * n_seqs > n_sms;
    return whole ? attn_few_launch_rows<64>(a, max_q_len, n_heads, n_seqs, seqs_ready, n_sms, st)
                 : attn_few_launch_rows<32>(a, max_q_len, n_heads, n_seqs, seqs_ready, n_sms, st);
}

void set_error(const char* fmt, ...);
int cuda_fail(cudaError_t e, const char* what);
bool attn_tc_supported(const IttaiAttention* p);          // attention_sm100.cu
int attn_tc_launch(const IttaiAttention* p, cudaStream_t st);
bool attn_fa_supported(const IttaiAttention* p);          // attention_fa_sm100.cu
int attn_fa_launch(const IttaiAttention* p, bool disjoint, cudaStream_t st);
static int attention_launch(const IttaiAttention* p, bool disjoint, cudaStream_t st);

}  // namespace ittai

using namespace ittai;

extern "C" int ittai_attention_launch(const IttaiAttention* p, void* stream) { return attention_launch(p, false, (cudaStream_t)stream); }
extern "C" int ittai_attention_packed_launch(const IttaiAttention* p, void* stream) { return attention_launch(p, true, (cudaStream_t)stream); }

// `disjoint`: the caller vouches that no two sequences share a query row.
static int ittai::attention_launch(const IttaiAttention* p, bool disjoint, cudaStream_t stream) {
    if (!p || !p->q || !p->k || !p->v || !p->o || !p->seqs) { set_error("attention: null pointer"); return ITTAI_E_ARG; }
    if (p->head_dim != 64 && p->head_dim != 128 && !(p->head_dim == 80 && attn_fa_supported(p))) {
        set_error("attention: head_dim %d (64, 128, or 80 in the packed layout of the key-loop kernel)", p->head_dim);
        return ITTAI_E_ARG;
    }
    if (p->n_seqs < 1 || p->n_heads < 1 || p->group < 1 || p->max_q_len < 1) { set_error("attention: bad sizes"); return ITTAI_E_ARG; }
    const long long strides[] = {p->q_row, p->q_head, p->k_row, p->k_head, p->k_seq, p->v_row, p->v_head, p->v_seq, p->o_row};
    for (long long s : strides) if (s % 8) { set_error("attention: strides must be multiples of 8 elements"); return ITTAI_E_ARG; }
    if (attn_tc_supported(p)) return attn_tc_launch(p, stream);
    if (attn_fa_supported(p)) return attn_fa_launch(p, disjoint, stream);
    AttnArgs a;
    a.q = (const bf16*)p->q; a.k = (const bf16*)p->k; a.v = (const bf16*)p->v; a.o = (bf16*)p->o;
    a.q_row = p->q_row; a.q_head = p->q_head; a.k_row = p->k_row; a.k_head = p->k_head; a.k_seq = p->k_seq;
    a.v_row = p->v_row; a.v_head = p->v_head; a.v_seq = p->v_seq; a.o_row = p->o_row; a.o_head = p->o_head;
    a.seqs = (const int4*)p->seqs; a.group = p->group;
    a.scale_log2 = 1.4426950408889634f / sqrtf((float)p->head_dim);
    cudaStream_t st = stream;
    const int ql = p->max_q_len, nh = p->n_heads, ns = p->n_seqs;
    int rc;
    if (p->head_dim == 64 && !p->causal && ql == 1) {
        const cudaError_t e1 = launch_pdl(attn_q1_kernel, dim3(nh, ns), dim3(32 * kQ1Warps), 0, st, 1, a);
        return e1 == cudaSuccess ? ITTAI_OK : cuda_fail(e1, "launch attn_q1_kernel");
    }
    if (p->head_dim == 128 && p->causal && ql <= kFewMax) {
        const cudaError_t e1 = attn_few_launch(a, ql, nh, ns, p->seqs_ready, st);
        return e1 == cudaSuccess ? ITTAI_OK : cuda_fail(e1, "launch attn_few_kernel");
    }
    if (p->head_dim == 128) rc = p->causal ? attn_launch<128, true, 4>(a, ql, nh, ns, st) : attn_launch<128, false, 4>(a, ql, nh, ns, st);
    else if (!p->causal && ql > 64 && ql <= 256 && p->max_kv_len > 0 && p->max_kv_len <= kShortKeys) rc = attn_short_launch(a, ql, nh, ns, st);
    else if (ql <= 64) rc = p->causal ? attn_launch<64, true, 4>(a, ql, nh, ns, st) : attn_launch<64, false, 4>(a, ql, nh, ns, st);
    else rc = p->causal ? attn_launch<64, true, 8>(a, ql, nh, ns, st) : attn_launch<64, false, 8>(a, ql, nh, ns, st);
    if (rc != 0) return cuda_fail((cudaError_t)rc, "cudaFuncSetAttribute(attn_fwd_kernel)");
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? ITTAI_OK : cuda_fail(e, "launch attn_fwd_kernel");
}
