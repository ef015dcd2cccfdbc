// Qwen3-0.6B greedy decode as a chain of small dependent kernels, one CUDA graph per token or per four (batch 1, 2, 4 or 8).
//
// A decoded token is 28 x (QKV, attention, O-proj, gate/up, down) + head + finish: 142 launches whose only dependency is
// one short vector.  With programmatic dependent launch every kernel is resident, and has fetched its weights, while its
// predecessor still runs; what remains per hand-off is a kernel boundary, 0.7-0.9 us in a graph on a B200 (last store of a
// kernel to the release of the next), against 1.4-2.9 us for a polled flag word that 148 CTAs read (qwen3_decode.cu).
//
// * GEMV kernels (gemv_kernel): 512 threads; a CTA's whole slice of a projection (32 to 96 KB) is on its way to
//   shared memory BEFORE griddepcontrol.wait (weights do not depend on the token); after the wait it is multiplied with
//   the activations of all sequences as mma.sync m16n8k16 tiles (the sequences are the N dimension), a warp taking 16 (or
//   8) rows x one K chunk.  CTAs of two neighbouring kernels fit an SM (the largest pair, gate/up and down at batch 8: 142 + 54
//   of 228 KB; attention and gate/up do not), so the next kernel's weights stream while this one waits.  The K chunks meet in
//   shared memory, in fixed order.
// * Attention (attn_kernel): a cluster of CS CTAs per (sequence, kv head) splits the cache; K/V tiles of 32 positions
//   arrive by TMA (128-byte swizzle), the first six before the wait; scores and P V on mma.sync, the splits meet
//   through distributed shared memory.  Probabilities enter P V as three bf16 parts in separate N columns (the columns
//   are idle anyway): 3 x 8 bits are all of an fp32 probability.  With two parts 1.5-3.3e-3 of the outputs were not the 64-bit
//   result rounded once, with three 0.6-3.6e-4, which is what fp32 sums leave, at the same time per step (batch 1, 4096: 523 us,
//   519; batch 2, 8000: 727, 730).
// * finish_kernel: argmax over the head's candidates, token feedback, positions, next token's embedding row.
//
// Rounding points are the eager modules' (the same as in qwen3_decode.cu).
//
// Measured on a B200, us per step, the persistent kernel of qwen3_decode.cu -> this chain: batch 1 at 47 / 4096 / 8100 cached
// positions 549 -> 370, 575 -> 455, 657 -> 568; batch 4 at 47 / 1000 / 8100 782 -> 419, 830 -> 478, 1419 -> 982; batch 8 at 1000 /
// 8100 1026 -> 611, 2211 -> 1545.  A layer takes 11.5 us at a short cache, from the last store of a kernel to that of the next: attention 3.3,
// gate/up 2.7, QKV 2.0, down 2.0, O-proj 1.5, of each of which 0.6 to 0.8 are the boundary; the head 47 us at 6.6 TB/s.  What had
// to go on the way (batch 1, 47 positions): weights through registers (800 us: a kernel's activation loads stand behind the
// next kernel's weight loads in the load pipe), normalisation in every warp's fragments (509: issue-bound), constants
// loaded ahead of the wait but scheduled behind it, the head through registers (93 us instead of 47).
#include <mutex>
#include <new>

#include "gemm2_common.cuh"
#include "launch.h"
#include "tcgen05.cuh"
#include "tmap.h"

namespace ittai {
namespace chain {

constexpr int D = ITTAI_Q3_D, HD = ITTAI_Q3_HD, NKV = ITTAI_Q3_NKV, DQ = ITTAI_Q3_DQ, DQKV = ITTAI_Q3_DQKV, DGU = ITTAI_Q3_DGU, FF = ITTAI_Q3_FF;
constexpr int kGemvThreads = 512;
constexpr int kMaxHeadCtas = 1024;
constexpr uint32_t kSpin = 1u << 22;         // polls of a copy that does not land
constexpr uint32_t kSpinParked = 1u << 18;   // the same where a poll parks the warp for up to 2 us

// Device-side state of one decode call (in the caller's workspace).
struct State {
    int32_t step, n_steps, n_forced, abort;
    int32_t* out_ids;
    const int32_t* forced;
    uint64_t* step_ns;
    int32_t cur_pos[ITTAI_MAX_BATCH];    // cache row of the token being computed; -1 once the call has aborted
};
struct Buffers {
    State* st;
    bf16 *h, *hmid, *qkv, *attn, *act;   // [B, width]
    float* cand_val;                     // [head CTAs, B]
    int32_t* cand_idx;
};
inline size_t layout(int batch, char* base, Buffers* w) {
    size_t off = 0;
    auto take = [&](size_t n) { char* p = base + off; off += (n + 255) / 256 * 256; return p; };
    w->st = reinterpret_cast<State*>(take(sizeof(State)));
    w->h = reinterpret_cast<bf16*>(take((size_t)batch * D * 2));
    w->hmid = reinterpret_cast<bf16*>(take((size_t)batch * D * 2));
    w->qkv = reinterpret_cast<bf16*>(take((size_t)batch * DQKV * 2));
    w->attn = reinterpret_cast<bf16*>(take((size_t)batch * DQ * 2));
    w->act = reinterpret_cast<bf16*>(take((size_t)batch * FF * 2));
    w->cand_val = reinterpret_cast<float*>(take((size_t)kMaxHeadCtas * batch * 4));
    w->cand_idx = reinterpret_cast<int32_t*>(take((size_t)kMaxHeadCtas * batch * 4));
    return off;
}

__device__ __forceinline__ void mma16816(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// bf16 pair of x -> bf16(bf16(x * rstd) * gain)
__device__ __forceinline__ uint32_t norm_pair(uint32_t x, uint32_t g, float rstd) {
    return pack_bf16x2(bf16r(bf_lo(x) * rstd) * bf_lo(g), bf16r(bf_hi(x) * rstd) * bf_hi(g));
}
// RMSNorm of the NB rows of x (width D) into xs[b][..] (rows padded by 64 bytes, see the weight rows): the 512 threads share
// the rows out, 2 NB values each, so that every value is normalised once per CTA.  Contains the two barriers after which xs
// may be read.
constexpr int kXsLd = D + 32;             // bf16 per row of xs
__device__ __forceinline__ void gemv_sync() { asm volatile("bar.sync 1, %0;" ::"n"(kGemvThreads) : "memory"); }   // not the head's feeding warp
template <int NB, typename F>
__device__ __forceinline__ void norm_rows(const bf16* x, const bf16* gain_s, bf16* xs, float* ss_s, int tid, float eps, F&& meanwhile) {
    constexpr int W = 16 / NB, E = 2 * NB;             // warps per row, values per thread
    const int warp = tid >> 5, b = warp / W, e0 = (tid - b * W * 32) * E;
    uint32_t u[NB];
    const bf16* src = x + (size_t)b * D + e0;
    if constexpr (NB == 1) u[0] = ldcg32(src);
    else if constexpr (NB == 2) asm volatile("ld.global.cg.v2.u32 {%0,%1}, [%2];" : "=r"(u[0]), "=r"(u[1]) : "l"(src));
    else {
#pragma unroll
        for (int i = 0; i < NB / 4; ++i) {
            const uint4 q = ldcg128(src + 8 * i);
            u[4 * i] = q.x; u[4 * i + 1] = q.y; u[4 * i + 2] = q.z; u[4 * i + 3] = q.w;
        }
    }
    meanwhile();
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < NB; ++i) s = fmaf(bf_lo(u[i]), bf_lo(u[i]), fmaf(bf_hi(u[i]), bf_hi(u[i]), s));
    s = warp_sum(s);
    if ((tid & 31) == 0) ss_s[warp] = s;
    gemv_sync();
    float tot = 0.f;
#pragma unroll
    for (int i = 0; i < W; ++i) tot += ss_s[b * W + i];
    const float rstd = rsqrt_full(tot * (1.0f / D) + eps);
    const uint32_t* gw = reinterpret_cast<const uint32_t*>(gain_s + e0);
    uint32_t* dst = reinterpret_cast<uint32_t*>(xs + b * kXsLd + e0);
#pragma unroll
    for (int i = 0; i < NB; ++i) dst[i] = norm_pair(u[i], gw[i], rstd);
    gemv_sync();
}

__device__ __forceinline__ uint4 lds128(const void* p) {          // volatile: stays where it is written
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(smem_u32(p)) : "memory");
    return v;
}

enum { kPlain = 0, kSwiglu = 1, kResidual = 2 };

struct GemvArgs {
    const bf16* w;          // [rows][K]
    const bf16* x;          // [B][K]
    const bf16* gain;       // norm in front of the projection, or unused
    const bf16* res;        // kResidual: [B][D]
    bf16* out;              // [B][ld_out]
    int ld_out;
    float eps;
    uint32_t* status;
    const State* st;        // gate/up, or down at batch 1: the next layer's cache rows to bring into L2 (k_next [B * 8][kv_cap][128]); nullptr: none
    const bf16 *k_next, *v_next;
    int kv_cap;
    const unsigned char* ahead;      // O-proj: weights to bring into L2, eight pieces of ahead_bytes per CTA (nullptr: none)
    uint32_t ahead_bytes;
    int late_trigger;       // first kernel of a token: dependents start only once everything before this kernel is complete
    int drop;               // test hook: CTA 0 leaves its weight rows out, so that its wait runs out
    uint32_t limit;         // polls before the wait for the weights gives up
};

// out = epilogue(W x).  ROWS = 32 or 48: 16-row tiles; ROWS = 8: half a tile.  KC K chunks x (16 / KC) tile groups over the 16
// warps.  QKV: 128 CTAs of 32 rows (64 KB), gate/up: 128 of 48 (96 KB), O-proj: 128 of 8 (32 KB), down: 128 of 8 (48 KB).
// The weight rows come by bulk copies (they bypass the load pipe, in which the next kernel's weights would otherwise
// stand in front of this one's activations) into rows padded by 64 bytes, so that the eight rows a warp reads at once fall
// on different banks.  A lane reads 16-byte pieces of its rows: columns 32 j + 8 t .. + 7 of the chunk, which serve as the
// k-indices of two MMAs (which column a k-index stands for is free as long as A and B agree).
template <int K, int ROWS>
constexpr uint32_t gemv_smem() { return (uint32_t)ROWS * (K * 2 + 64); }

template <int NB, int K, int ROWS, int EPI, int EARLY = 0>
__global__ void __launch_bounds__(kGemvThreads, 2) gemv_kernel(const GemvArgs a) {
    constexpr int KC = ROWS == 32 ? 8 : 16, KW = K / KC, NJ = KW / 32, NR = ROWS == 8 ? 1 : 2, NT = ROWS == 48 ? 3 : 1;
    constexpr int LD = K * 2 + 64;                      // bytes per weight row in shared memory
    constexpr bool kNorm = EPI != kResidual;
    static_assert(KW % 32 == 0, "K chunk");
    extern __shared__ __align__(128) unsigned char w_s[];
    __shared__ float part[KC][NB][ROWS];
    __shared__ float ss_s[16];
    __shared__ __align__(16) bf16 gain_s[kNorm ? D : 8];
    __shared__ __align__(16) bf16 xs[kNorm ? NB * kXsLd : 8];
    __shared__ unsigned long long landed;
    const int tid = threadIdx.x, warp = warp_index(), lane = tid & 31, g = lane >> 2, t = lane & 3;
    const int kc = ROWS == 32 ? warp & 7 : warp, tile = ROWS == 32 ? warp >> 3 : 0;
    const int row0 = blockIdx.x * ROWS;
    const int col = kc * KW + 8 * t;
    if (tid == 0) { mbar_init(&landed, 1); fence_mbar_init(); mbar_expect_tx(&landed, ROWS * K * 2); }
    __syncwarp();
    if (warp == 0 && !(a.drop && blockIdx.x == 0)) {
        for (int r = lane; r < ROWS; r += 32) bulk_g2s(w_s + r * LD, a.w + (size_t)(row0 + r) * K, K * 2, &landed);
    }
    if (!a.late_trigger) pdl_trigger();
    // By gate/up, or at batch 1 by the down projection, which has more time before its wait (gate/up's last CTAs find room only when attention
    // ends): batch 1 at 60 / 800 / 4096 / 6500 positions 381 / 377, 394 / 390, 469 / 462, 527 / 521; batch 2 at 1000 / 4000 423 / 419, 540 / 545;
    // batch 4 at 1000 484 / 493.
    if ((EPI == kSwiglu || (EPI == kResidual && NB == 1)) && a.k_next != nullptr && warp == 1) {
        // an even share of every sequence's cached rows; positions are stable here (see attn_kernel)
        constexpr int kItems = NB * NKV, kParts = DGU / 48 / kItems;                  // both have 128 CTAs
        static_assert(DGU / 48 == D / 8, "an even share for every CTA");
        const int item = blockIdx.x % kItems, piece = blockIdx.x / kItems;
        int pos = (int)ld_relaxed(reinterpret_cast<const uint32_t*>(&a.st->cur_pos[item / NKV]));
        // More than L2 keeps until it is read.  us per step without / with it: batch 1 at 6500 / 8000 positions (27 / 33 MB a layer) 554 / 531
        // and 588 / 570, batch 2 at 3500 / 5000 (29 / 41 MB) 548 / 532 and 595 / 606, batch 4 at 1800 (29 MB) 549 / 550, batch 8 at 1000 (33 MB) 614 / 645.
        if ((long long)NB * NKV * pos * HD * 4 > ((NB <= 2 ? 36 : 24) << 20)) pos = 0;
        const int q0 = (int)((long long)pos * piece / kParts), q1 = (int)((long long)pos * (piece + 1) / kParts);
        for (int q = q0 + 32 * lane; q < q1; q += 32 * 32) {
            const uint32_t n = (uint32_t)(q1 - q < 32 ? q1 - q : 32) * HD * 2;
            l2_prefetch(a.k_next + ((size_t)item * a.kv_cap + q) * HD, n);
            l2_prefetch(a.v_next + ((size_t)item * a.kv_cap + q) * HD, n);
        }
    }
    if (EPI == kResidual && a.ahead != nullptr && warp == 1 && lane < 8)
        l2_prefetch(a.ahead + ((size_t)blockIdx.x * 8 + lane) * a.ahead_bytes, a.ahead_bytes);
    const unsigned char* wr = w_s + (tile * 16 + g) * LD + col * 2;
    if constexpr (kNorm) reinterpret_cast<uint32_t*>(gain_s)[tid] = reinterpret_cast<const uint32_t*>(a.gain)[tid];
    __syncthreads();                                   // the barrier exists for every warp, and the gain has arrived: a load
                                                       // left open here may be scheduled behind the wait
    // A warp's weights in registers ahead of the wait: 64 KB of a QKV slice take the shared memory 512 cycles, which stood between the
    // activations and the sums.  Gate/up would need 48 registers for it on top of its own and starts late (its last CTAs find room when
    // attention ends): held there too, us per step 512 instead of 485 (batch 1, 4096), 499 instead of 482 (batch 4, 1000); see hold_tiles for what it does.  Waiting for the
    // weights in front of the dependency costs nothing where they are late: asking once and loading the activations first
    // 413 instead of 400 (batch 1, 800).  None held -> this: batch 1 at 47 / 4096 391 -> 380, 498 -> 485, batch 4 and 8 at 1000 497 -> 482, 629 -> 614.
    constexpr bool kHeld = ROWS != 48;
    constexpr int kEarly = kHeld ? NT : EARLY, kRegs = kEarly > 0 ? kEarly : 1;
    uint4 wl[kRegs][NJ], wh[NR == 2 ? kRegs : 1][NR == 2 ? NJ : 1];
    auto hold = [&]() {
#pragma unroll
        for (int n = 0; n < kEarly; ++n)
#pragma unroll
            for (int j = 0; j < NJ; ++j) {
                wl[n][j] = lds128(wr + 16 * n * LD + 64 * j);
                if constexpr (NR == 2) wh[n][j] = lds128(wr + (16 * n + 8) * LD + 64 * j);
            }
    };
    bool ok = true;
    if constexpr (kHeld) {
        ok = mbar_wait_bounded(&landed, 0, a.limit);
        __syncwarp();                                  // the lanes left the wait one by one
        hold();
    }
    pdl_wait();
    if (a.late_trigger) pdl_trigger();
    uint4 x[NJ];
    // Gate/up, EARLY tiles: while the activations travel, if the weights are there
    bool there = kHeld || EARLY == 0;
    auto early = [&]() { if constexpr (!kHeld && EARLY > 0) { there = __all_sync(0xffffffffu, mbar_test(&landed, 0)); if (there) hold(); } };
    if constexpr (kNorm) norm_rows<NB>(a.x, gain_s, xs, ss_s, tid, a.eps, early);
#pragma unroll
    for (int j = 0; j < NJ; ++j) {
        if constexpr (kNorm) x[j] = g < NB ? *reinterpret_cast<const uint4*>(xs + g * kXsLd + col + 32 * j) : make_uint4(0u, 0u, 0u, 0u);
        else x[j] = g < NB ? ldcg128(a.x + (size_t)g * K + col + 32 * j) : make_uint4(0u, 0u, 0u, 0u);
    }
    float res = 0.f;
    if constexpr (EPI == kResidual) {
        if (tid < 8 * NB) res = ldcg_bf16(a.res + (size_t)(tid >> 3) * D + row0 + (tid & 7));
    }
    if constexpr (!kHeld) {
        ok = mbar_wait_bounded(&landed, 0, a.limit);
        __syncwarp();
        if (!there) hold();
    }
#pragma unroll
    for (int n = 0; n < NT; ++n) {
        float d0[4] = {0.f, 0.f, 0.f, 0.f}, d1[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int j = 0; j < NJ; ++j) {
            uint4 lo, hi = make_uint4(0u, 0u, 0u, 0u);
            if (n < kEarly) { lo = wl[n < kRegs ? n : 0][j]; if constexpr (NR == 2) hi = wh[n < kRegs ? n : 0][j]; }
            else { lo = lds128(wr + 16 * n * LD + 64 * j); if constexpr (NR == 2) hi = lds128(wr + (16 * n + 8) * LD + 64 * j); }
            mma16816(d0, lo.x, hi.x, lo.y, hi.y, x[j].x, x[j].y);
            mma16816(d1, lo.z, hi.z, lo.w, hi.w, x[j].z, x[j].w);
        }
        float* p = &part[kc][0][(tile + n) * 16 + g];
        if (2 * t < NB) { p[2 * t * ROWS] = d0[0] + d1[0]; if (NR == 2) p[2 * t * ROWS + 8] = d0[2] + d1[2]; }
        if (2 * t + 1 < NB) { p[(2 * t + 1) * ROWS] = d0[1] + d1[1]; if (NR == 2) p[(2 * t + 1) * ROWS + 8] = d0[3] + d1[3]; }
    }
    __syncthreads();
    if constexpr (ROWS >= 32) {
        // two threads of a warp side by side hold two rows of one sequence
#pragma unroll
        for (int i0 = 0; i0 < ROWS * NB; i0 += kGemvThreads) {
            const int i = i0 + tid;
            if (i0 + 32 * warp < ROWS * NB) {
                const int b = i / ROWS, r = i % ROWS;      // a warp may span two sequences, an aligned group of 16 never does
                float s = 0.f;
                if (i < ROWS * NB) {
#pragma unroll
                    for (int k = 0; k < KC; ++k) s += part[k][b][r];
                }
                if constexpr (EPI == kPlain) {
                    const float o = __shfl_down_sync(0xffffffffu, s, 1);
                    if ((lane & 1) == 0 && i < ROWS * NB) *reinterpret_cast<uint32_t*>(a.out + (size_t)b * a.ld_out + row0 + r) = pack_bf16x2(s, o);
                } else {
                    // rows 2i, 2i + 1 are (gate, up): act = bf16(bf16(silu(bf16 gate)) * bf16 up)
                    const float up = bf16r(__shfl_down_sync(0xffffffffu, s, 1)), gate = bf16r(s);
                    const float v = bf16r(gate / (1.0f + expf(-gate))) * up;
                    const float v2 = __shfl_down_sync(0xffffffffu, v, 2);
                    if ((lane & 3) == 0 && i < ROWS * NB) *reinterpret_cast<uint32_t*>(a.out + (size_t)b * a.ld_out + (row0 + r) / 2) = pack_bf16x2(v, v2);
                }
            }
        }
    } else {
        if (tid < 8 * NB) {                             // eight rows of a sequence side by side
            const int b = tid >> 3, r = tid & 7;
            float s = 0.f;
#pragma unroll
            for (int k = 0; k < KC; ++k) s += part[k][b][r];
            a.out[(size_t)b * a.ld_out + row0 + r] = __float2bfloat16_rn(res + bf16r(s));
        }
    }
    if (!ok) {
        if (lane == 0 && atomicCAS(&a.status[0], 0u, (uint32_t)ITTAI_ST_STREAM_TIMEOUT) == 0u) { a.status[1] = row0; a.status[2] = blockIdx.x; }
        const long long t0 = clock64();                    // copies still in flight land before the shared memory is handed back
        while (clock64() - t0 < 2000000) {}
    }
}

// ---- lm_head: logits = E bf16(norm(h)), with the arg-max candidates of this CTA's rows ----------------------------------
// One CTA per SM walks its contiguous share of the table, 16 rows (32 KB) per ring stage, five stages: at batch 1 and 2 they fit
// beside a CTA of the last down-projection (222 and 227 of 228 KB), so that the ring is full when the hidden state arrives; at
// batch 4 and 8 (236 and 254 KB) it starts to fill when that kernel ends.  A warp multiplies the 16 rows with one of
// 16 K chunks; 311 MB of weights at the memory rate are the whole of it (loads through registers, two 64 KB steps ahead,
// gave 93 us instead of 47).
struct HeadArgs {
    const bf16* w;          // [V][D]
    const bf16* x;          // [B][D]
    const bf16* gain;
    bf16* logits;           // [B][V] or nullptr
    float* cand_val;        // [CTAs][B]
    int32_t* cand_idx;
    uint32_t* status;
    int vocab;
    float eps;
    uint32_t limit;
};
constexpr int kHeadRing = 5, kHeadRows = 16, kHeadLd = D * 2 + 64;
constexpr uint32_t kHeadSmem = kHeadRing * kHeadRows * kHeadLd;
template <int NB>
__global__ void __launch_bounds__(kGemvThreads + 32, 1) head_kernel(const HeadArgs a) {
    constexpr int KW = D / 16, NJ = KW / 32;
    extern __shared__ __align__(128) unsigned char w_s[];
    __shared__ float part[2][16][NB][kHeadRows];
    __shared__ float ss_s[16];
    __shared__ __align__(16) bf16 gain_s[D];
    __shared__ __align__(16) bf16 xs[NB * kXsLd];
    __shared__ unsigned long long full[kHeadRing], empty[kHeadRing];
    __shared__ volatile uint32_t failed;
    const int tid = threadIdx.x, warp = warp_index(), lane = tid & 31, g = lane >> 2, t = lane & 3;
    const int r_lo = (int)((long long)a.vocab * blockIdx.x / gridDim.x), r_hi = (int)((long long)a.vocab * (blockIdx.x + 1) / gridDim.x);
    const int n_it = (r_hi - r_lo + kHeadRows - 1) / kHeadRows;
    if (tid == 0) {
        for (int s = 0; s < kHeadRing; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 16); }
        failed = 0;
        fence_mbar_init();
    }
    __syncthreads();
    pdl_trigger();
    if (warp == 16) {                    // the feeding warp: one row per lane
        for (int it = 0; it < n_it && !failed; ++it) {
            const int s = it % kHeadRing, r0 = r_lo + it * kHeadRows, n = r_hi - r0 < kHeadRows ? r_hi - r0 : kHeadRows;
            if (it >= kHeadRing && !__all_sync(0xffffffffu, mbar_wait_bounded(&empty[s], ((it / kHeadRing) - 1) & 1, a.limit))) { failed = 1; break; }
            if (lane == 0) mbar_expect_tx(&full[s], (uint32_t)n * D * 2);
            __syncwarp();
            if (lane < n) bulk_g2s(w_s + (s * kHeadRows + lane) * kHeadLd, a.w + (size_t)(r0 + lane) * D, D * 2, &full[s]);
        }
        pdl_wait();
        return;
    }
    reinterpret_cast<uint32_t*>(gain_s)[tid] = reinterpret_cast<const uint32_t*>(a.gain)[tid];
    gemv_sync();                         // the gain has arrived (see gemv_kernel)
    pdl_wait();
    norm_rows<NB>(a.x, gain_s, xs, ss_s, tid, a.eps, []() {});
    const int col = warp * KW + 8 * t;
    uint4 x[NJ];
#pragma unroll
    for (int j = 0; j < NJ; ++j) x[j] = g < NB ? *reinterpret_cast<const uint4*>(xs + g * kXsLd + col + 32 * j) : make_uint4(0u, 0u, 0u, 0u);
    float best = -INFINITY;
    int best_i = 0x7fffffff;
    const int rb = tid / kHeadRows, rr = tid % kHeadRows;          // reducing threads: sequence, row of the stage
    for (int it = 0; it < n_it; ++it) {
        const int s = it % kHeadRing, buf = it & 1;
        bool ok = true;
        uint32_t spins = 0;
        while (!mbar_try_wait_parked(&full[s], (it / kHeadRing) & 1)) { if (++spins >= a.limit || failed) { ok = false; break; } }
        if (!ok) failed = 1;
        __syncwarp();                    // the lanes left the wait one by one
        const unsigned char* wr = w_s + (s * kHeadRows + g) * kHeadLd + col * 2;
        float d0[4] = {0.f, 0.f, 0.f, 0.f}, d1[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int j = 0; j < NJ; ++j) {
            const uint4 lo = *reinterpret_cast<const uint4*>(wr + 64 * j), hi = *reinterpret_cast<const uint4*>(wr + 8 * kHeadLd + 64 * j);
            mma16816(d0, lo.x, hi.x, lo.y, hi.y, x[j].x, x[j].y);
            mma16816(d1, lo.z, hi.z, lo.w, hi.w, x[j].z, x[j].w);
        }
        __syncwarp();
        if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&empty[s])) : "memory");
        float* p = &part[buf][warp][0][g];
        if (2 * t < NB) { p[2 * t * kHeadRows] = d0[0] + d1[0]; p[2 * t * kHeadRows + 8] = d0[2] + d1[2]; }
        if (2 * t + 1 < NB) { p[(2 * t + 1) * kHeadRows] = d0[1] + d1[1]; p[(2 * t + 1) * kHeadRows + 8] = d0[3] + d1[3]; }
        gemv_sync();                     // readers of the other buffer have passed the barrier before this one
        if (tid < kHeadRows * NB) {
            float sum = 0.f;
#pragma unroll
            for (int k = 0; k < 16; ++k) sum += part[buf][k][rb][rr];
            const int row = r_lo + it * kHeadRows + rr;
            if (row < r_hi) {
                const float v = bf16r(sum);
                if (a.logits != nullptr) a.logits[(size_t)rb * a.vocab + row] = __float2bfloat16_rn(v);
                if (v > best) { best = v; best_i = row; }        // rows ascend: the first maximum is kept
            }
        }
    }
    if (tid < (kHeadRows * NB < 32 ? 32 : kHeadRows * NB)) {
#pragma unroll
        for (int o = kHeadRows / 2; o > 0; o >>= 1) {       // highest value, lowest row on ties
            const float ov = __shfl_xor_sync(0xffffffffu, best, o);
            const int oi = __shfl_xor_sync(0xffffffffu, best_i, o);
            if (ov > best || (ov == best && oi < best_i)) { best = ov; best_i = oi; }
        }
        if (rr == 0 && rb < NB) { a.cand_val[blockIdx.x * NB + rb] = best; a.cand_idx[blockIdx.x * NB + rb] = best_i; }
    }
    if (failed && tid == 0) {
        if (atomicCAS(&a.status[0], 0u, (uint32_t)ITTAI_ST_STREAM_TIMEOUT) == 0u) { a.status[1] = (uint32_t)r_lo; a.status[2] = blockIdx.x; }
        const long long t0 = clock64();                    // copies still in flight land before the shared memory is handed back
        while (clock64() - t0 < 2000000) {}
    }
}

// ---- token feedback -------------------------------------------------------------------------------------------------------
struct TokenArgs {
    State* st;
    const bf16* embed;
    bf16* h;
    const float* cand_val;
    const int32_t* cand_idx;
    int n_cand;
    int32_t* pos;
    int32_t* next_id;
    uint32_t* status;
    int vocab, kv_cap;
};
__device__ __forceinline__ void bad_token(const TokenArgs& a, int id, int step, int pos, int b) {
    if (atomicCAS(&a.status[0], 0u, (uint32_t)ITTAI_ST_BAD_TOKEN) == 0u) {
        a.status[1] = (uint32_t)id; a.status[2] = (uint32_t)step; a.status[3] = (uint32_t)pos; a.status[4] = (uint32_t)b;
    }
}
// Embedding row of sequence b's next token.  One warp.
__device__ __forceinline__ void embed_row(const TokenArgs& a, int b, int id, int lane) {
    const int row = id < 0 ? 0 : (id >= a.vocab ? a.vocab - 1 : id);
#pragma unroll
    for (int i = 0; i < 4; ++i)
        *reinterpret_cast<uint4*>(a.h + (size_t)b * D + (lane + 32 * i) * 8) = *reinterpret_cast<const uint4*>(a.embed + (size_t)row * D + (lane + 32 * i) * 8);
}

// First kernel of a call: one warp per sequence.  Takes the call's parameters into the device state, checks the first ids
// and positions, gathers the first embedding rows.
template <int NB>
__global__ void __launch_bounds__(32 * NB) begin_kernel(const TokenArgs a, int32_t* out_ids, const int32_t* forced, uint64_t* step_ns, int n_steps, int n_forced) {
    const int b = warp_index(), lane = threadIdx.x & 31;
    __shared__ int bad;
    if (threadIdx.x < ITTAI_STATUS_WORDS) a.status[threadIdx.x] = 0u;
    if (threadIdx.x == 0) {
        bad = 0;
        State s;
        s.step = 0; s.n_steps = n_steps; s.n_forced = n_forced; s.abort = 0;
        s.out_ids = out_ids; s.forced = forced; s.step_ns = step_ns;
        a.st->step = s.step; a.st->n_steps = s.n_steps; a.st->n_forced = s.n_forced;
        a.st->out_ids = s.out_ids; a.st->forced = s.forced; a.st->step_ns = s.step_ns;
    }
    __syncthreads();
    const int id = n_forced > 0 ? forced[b] : a.next_id[b], pos = a.pos[b];
    if (id < 0 || id >= a.vocab || pos < 0 || pos >= a.kv_cap) {
        if (lane == 0) { bad_token(a, id, 0, pos, b); bad = 1; }
    }
    __syncthreads();
    if (lane == 0) a.st->cur_pos[b] = bad ? -1 : pos;
    if (threadIdx.x == 0) a.st->abort = bad;
    embed_row(a, b, id, lane);
}

// Last kernel of a token, one warp per sequence.  With HEAD: arg-max over the head's candidates, stored as the step's id and
// fed back.  Without: a forced step whose logits nobody asked for.  Then the next token's row and position; after the last
// step of the call the cache lengths `pos` advance, unless a step found an id or a position out of range or a wait of one of its
// kernels ran out: from there on nothing that was computed is stored as an id, fed back or counted.
template <int NB, bool HEAD>
__global__ void __launch_bounds__(32 * NB) finish_kernel(const TokenArgs a) {
    pdl_trigger();
    pdl_wait();
    const int b = warp_index(), lane = threadIdx.x & 31;
    __shared__ int bad, stopped;
    State* st = a.st;
    const int step = st->step, n_steps = st->n_steps, pos = st->cur_pos[b];
    int32_t* out_ids = st->out_ids;
    if (threadIdx.x == 0) bad = stopped = st->abort != 0 || ld_relaxed(a.status) != 0u;
    __syncthreads();
    const bool abort = stopped != 0;                   // as it was before this kernel reported anything itself
    int id = -1;
    if constexpr (HEAD) {
        float v = -INFINITY;
        int ix = 0x7fffffff;
        for (int k = lane; k < a.n_cand; k += 32) {
            const float vk = a.cand_val[k * NB + b];
            const int ik = a.cand_idx[k * NB + b];
            if (vk > v || (vk == v && ik < ix)) { v = vk; ix = ik; }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float ov = __shfl_xor_sync(0xffffffffu, v, o);
            const int oi = __shfl_xor_sync(0xffffffffu, ix, o);
            if (ov > v || (ov == v && oi < ix)) { v = ov; ix = oi; }
        }
        id = ix;
        // no logit compared greater than -inf (a row of NaNs): reported instead of fed back
        if (ix == 0x7fffffff && lane == 0 && !abort) { bad_token(a, ix, step, pos, b); bad = 1; }
    }
    if (lane == 0 && !abort) {
        out_ids[(size_t)step * NB + b] = id;
        if (HEAD) a.next_id[b] = id;
    }
    const bool last = step + 1 >= n_steps;
    int next = id;
    if (!last) {
        if (step + 1 < st->n_forced) next = st->forced[(size_t)(step + 1) * NB + b];
        if (!HEAD && step + 1 >= st->n_forced) next = a.next_id[b];
        if (lane == 0 && !abort && (next < 0 || next >= a.vocab || pos + 1 >= a.kv_cap)) { bad_token(a, next, step + 1, pos + 1, b); bad = 1; }
    }
    __syncthreads();
    if (lane == 0) {
        st->cur_pos[b] = bad ? -1 : pos + 1;
        if (last && !bad) a.pos[b] = pos + 1;
    }
    if (threadIdx.x == 0) {
        st->step = step + 1;
        st->abort = bad;
        if (st->step_ns != nullptr) st->step_ns[step] = globaltimer_ns();
    }
    if (!last) embed_row(a, b, next, lane);
}

// ---- attention ------------------------------------------------------------------------------------------------------------
// One cluster of CS CTAs per (sequence, kv head); rank r takes the r-th piece of the cached positions (if the sequence is long
// enough for so many, see pieces), rank 0 also the new one (norm, rotation, append, and its own score).  Three groups of two
// compute warps take turns on 32-position tiles, a warp 16 positions of each with its own softmax; a seventh warp feeds a ring
// of six 16 KB tiles (two CTAs per SM).  A warp's 16 positions are 16 MMAs: scores with the keys as A (M = positions) and the two query heads as N columns, P V with
// V^T as A (ldmatrix.trans on the swizzled tile) and P as B, its middle, low and high parts in columns 0-1, 2-3 and 4-5.
// A tile is about 1000 dependent cycles for a warp the first time and 600 from then on, which is why the tiles are small and the warps
// many; the difference is instruction supply.  Every kernel of a layer runs once, so its code comes from the second-level instruction
// cache at about three cycles an instruction: code off the straight path costs the same as data that has to be fetched.  Hence the warp
// index as a uniform value, rolled loops where nothing is gained by unrolling, packed bf16 arithmetic in the rotation, the operand words
// of q in the order in which a lane reads them, and one pass over the merge: 34.9 -> 19.7 KB.  With the partials sent by st.async instead
// of stored ahead of a second cluster barrier (1500 cycles of 6300), us per step before -> after: batch 1 at 47 / 800 / 4096 / 8000
// positions 420 -> 390, 440 -> 409, 520 -> 498, 584 -> 573; batch 2 and 4 at 1000 475 -> 450 and 530 -> 497; batch 8 at 1000 / 8100
// 681 -> 629 and 1587 -> 1563.
constexpr int kGroups = 3, kAttnWarps = 2 * kGroups, kAttnThreads = 32 * kAttnWarps + 32, kTilePos = 32, kRing = 2 * kGroups;
// Tile `it` belongs to group it % 3, which has two ring slots of its own: a slot's phases are waited for by the same two
// warps in order (a slot shared by groups that skip each other's phases cannot be told apart by parity).
__device__ __forceinline__ int ring_slot(int it) { return (it % kGroups) * 2 + ((it / kGroups) & 1); }
__device__ __forceinline__ uint32_t ring_parity(int it) { return (uint32_t)(it / (2 * kGroups)) & 1u; }
constexpr uint32_t kHalfTile = kTilePos * 128;                 // 32 positions x 64 dims
constexpr uint32_t kTileBytes = 4 * kHalfTile;                 // K low / high dims, V low / high dims
constexpr uint32_t kAttnSmem = kRing * kTileBytes + 1024;
constexpr float kScoreScale = 0.08838834764831845f * 1.4426950408889634f;   // head_dim^-0.5 * log2(e)

struct AttnChainArgs {
    const State* st;
    const bf16* qkv;        // [B][DQKV]
    const bf16* qn;
    const bf16* kn;
    const bf16* rope;
    bf16* kcache;           // this layer [B][8][cap][128]
    bf16* vcache;
    bf16* attn;             // [B][DQ]
    uint32_t* status;
    int layer, batch, kv_cap;
    float eps;
    uint32_t limit, limit_parked;
};

__device__ __forceinline__ float ex2f(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldsm4_t(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ uint32_t movm_t(uint32_t a) {
    uint32_t d;
    asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(d) : "r"(a));
    return d;
}
__device__ __forceinline__ void compute_sync() { asm volatile("bar.sync 1, %0;" ::"n"(32 * kAttnWarps) : "memory"); }
__device__ __forceinline__ void tma_load_2d_hint(void* dst, const void* tmap, int x, int y, void* bar, uint64_t policy) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1, {%2, %3}], [%4], %5;"
                 ::"r"(smem_u32(dst)), "l"(tmap), "r"(x), "r"(y), "r"(smem_u32(bar)), "l"(policy) : "memory");
}
// Byte address of the 16-byte chunk `chunk` (0..7) of row `row` of a half tile under the 128-byte swizzle.
__device__ __forceinline__ uint32_t swz(uint32_t base, int row, int chunk) { return base + (uint32_t)row * 128u + (uint32_t)((chunk ^ (row & 7)) << 4); }
// Two floats into rank `rank`'s copy of `p`, counted on its copy of `bar`.
__device__ __forceinline__ void st_async_f32x2(void* p, int rank, float x, float y, void* bar) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v2.f32 [%0], {%1, %2}, [%3];"
                 ::"r"(map_to_cta(p, (uint32_t)rank)), "f"(x), "f"(y), "r"(map_to_cta(bar, (uint32_t)rank)) : "memory");
}

// The pieces that the cache of a sequence with `len` positions is cut into, one CTA each.  What decides is whether every cluster of the
// launch finds room while the projection in front still runs, one CTA per SM: seven clusters of 16 do, 8 of 12, 15 of 8, 16 of 7, 33 of 4.  The
// eighth of 16 waited for the projection's SMs, and its CTAs asked for their keys when the others were half through.  us per step:
// batch 1 in 8 / 12 / 16 pieces at 400 positions 384 / 389 / 401, 800 400 / 393 / 403, 2000 435 / 419 / 421, 4096 515 / 468 / 487, 8000 657 / 566
// / 565 (10 pieces: 391 at 800, 478 at 4096; 14: 481 and, at 8000, 560); batch 2 in 4 / 7 / 8 at 60 402 / 396 / 400, 800 442 / 419 / 422, 4000
// 669 / 544 / 554, 8000 869 / 700 / 694.  Few positions need no split (batch 1, 30: 425, else 428-443, with the kernels as they were then).  The
// longest caches at batch 8 want two CTAs per SM (8100: 4 pieces 1577, 2 1623; 500: 604 and 592, likewise).  Batch 4 is cut in four at every
// length, which below 48 positions was not the best (30: 471, uncut 442, in two 465).
// A sequence's pieces follow from its OWN length, so that its sums are taken in the same order whatever the others of the
// batch hold; the clusters of a launch have the size that the longest needs (the rule does not fall with `len`), and in those of
// a shorter sequence the ranks past its pieces add exact zeros.
constexpr int kPieces[] = {1, 2, 4, 7, 8, 12};             // cluster sizes, in the order of Plan::exec
__host__ __device__ constexpr int pieces(int batch, int len) {
    if (batch == 4) return 4;
    if (len <= 48) return 1;
    if (batch == 1) return len <= 400 ? 8 : 12;
    if (batch == 2) return len <= 6000 ? 7 : 8;
    return len <= 700 ? 2 : 4;
}

// Whether gate/up takes two of its three tiles into registers while the activations travel (the same sums either way).  It pays while its
// weights are there by then; beside long caches they arrive late, and a tile held then only comes between the wait and the sums.  us per
// step without / with: batch 1 at 60 / 4096 / 6000 / 8000 positions 377 / 372, 460 / 457, 506 / 508, 559 / 564; batch 2 at 500 / 8000 404 / 400,
// 702 / 709; batch 4 at 300 / 2000 433 / 430, 561 / 565; batch 8 at 500 / 2000 548 / 545, 748 / 752.  All three tiles spill: 409 at 60.
__host__ __device__ constexpr bool hold_tiles(int batch, int len) { return batch * len <= 5000; }

template <int CS>
__global__ void __launch_bounds__(kAttnThreads, 2) attn_kernel(const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_v, const AttnChainArgs a) {
    extern __shared__ __align__(1024) unsigned char ring_raw[];
    unsigned char* ring = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(ring_raw) + 1023) & ~(uintptr_t)1023);
    constexpr int kMergers = CS >= 8 ? 8 : CS >= 4 ? 4 : CS, NE = 2 * HD / kMergers;      // the first ranks merge NE outputs each
    __shared__ unsigned long long full[kRing], empty[kRing], arrived;
    __shared__ __align__(16) uint32_t q_s[2][4][20];            // [head][t]: the 16 words that lane t of a quad holds as MMA operand
    __shared__ __align__(16) bf16 k_s[HD];
    __shared__ __align__(8) float2 pml[2][kAttnWarps + 1];      // reference and sum of the warps' partials and of the new position
    __shared__ __align__(16) float po[kAttnWarps + 1][2][HD];
    __shared__ __align__(8) bf16 rot_s[4][HD];                  // q gain, k gain, cos | sin of the new position
    __shared__ __align__(8) float rv[CS][CS == 1 ? 2 : NE];     // partials of all ranks for this rank's outputs, which are of one head
    __shared__ __align__(8) float2 rml[CS];
    __shared__ volatile uint32_t failed;
    const int tid = threadIdx.x, warp = warp_index(), lane = tid & 31;
    const int rank = CS == 1 ? 0 : (int)(blockIdx.x % CS), item = blockIdx.x / CS, b = item / NKV, kvh = item % NKV;
    const size_t head_row = (size_t)(a.layer * a.batch + b) * NKV + kvh;          // in units of kv_cap rows of the whole cache
    if (tid == 0) {
        for (int s = 0; s < kRing; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 2); }
        failed = 0;
        mbar_init(&arrived, 1);
        fence_mbar_init();
        if (CS > 1 && blockIdx.x % CS < kMergers) mbar_expect_tx(&arrived, CS * (NE * 4 + 8));
    }
    __syncthreads();
    // another CTA's shared memory may be written only once that CTA runs: every thread arrives here, waits before the merge
    if constexpr (CS > 1) asm volatile("barrier.cluster.arrive.release;" ::: "memory");
    pdl_trigger();
    // Positions and older cache rows are complete before the first kernel of this token lets its successors start
    // (late_trigger), so they may be read ahead of the wait.
    const int pos = (int)ld_relaxed(reinterpret_cast<const uint32_t*>(&a.st->cur_pos[b]));
    const int n_old = pos < 0 ? 0 : pos;
    const int own = pieces(a.batch, n_old), cut = own < CS ? own : CS;
    const int chunk = ((n_old + cut - 1) / cut + 15) & ~15;
    const int p0 = rank * chunk < n_old ? rank * chunk : n_old, p1 = p0 + chunk < n_old ? p0 + chunk : n_old;
    const int n_tiles = (p1 - p0 + kTilePos - 1) / kTilePos;
    const int row_base = (int)(head_row * (size_t)a.kv_cap) + p0;
    uint64_t policy = 0;
    auto issue = [&](int it) {
        const int s = ring_slot(it);
        unsigned char* t = ring + s * kTileBytes;
        mbar_expect_tx(&full[s], kTileBytes);
        const int y = row_base + it * kTilePos;
        tma_load_2d_hint(t, &tm_k, 0, y, &full[s], policy);
        tma_load_2d_hint(t + kHalfTile, &tm_k, 64, y, &full[s], policy);
        tma_load_2d_hint(t + 2 * kHalfTile, &tm_v, 0, y, &full[s], policy);
        tma_load_2d_hint(t + 3 * kHalfTile, &tm_v, 64, y, &full[s], policy);
    };
    if (warp == kAttnWarps) {
        if (lane == 0) {
            asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(policy));
#pragma unroll 1
            for (int it = 0; it < n_tiles; ++it) {
                if (it >= kRing && !mbar_wait_bounded(&empty[ring_slot(it)], ring_parity(it) ^ 1, a.limit_parked)) { failed = 1; break; }
                issue(it);
            }
        }
        __syncwarp();
    } else {
        // rotary row and gains do not depend on the token's vectors: in shared memory before the wait
        const bool is_q = warp < 2;
        const int hi_half = lane >> 4, ei = 4 * (lane & 15), g = lane >> 2, t = lane & 3;
        if (warp < 3) {
            const bf16* src = warp == 0 ? a.qn : warp == 1 ? a.kn : a.rope + (size_t)n_old * HD;
            *reinterpret_cast<uint2*>(&rot_s[warp][4 * lane]) = *reinterpret_cast<const uint2*>(src + 4 * lane);
        }
        compute_sync();
        const int e0 = is_q ? (2 * kvh + warp) * HD : (warp == 2 ? DQ : DQ + NKV * HD) + kvh * HD;
        const bf16* src_row = a.qkv + (size_t)b * DQKV + e0 + 4 * lane;
        const size_t cache_row = ((size_t)(b * NKV + kvh) * a.kv_cap + n_old) * HD + 4 * lane;
        const int mat = lane >> 3, r8 = lane & 7;
        const int group = warp >> 1, w4 = warp & 1;              // the warp's 16 rows of its group's tiles
        const int krow = 16 * w4 + (mat & 1) * 8 + r8, kchunk = mat >> 1;       // keys: rows +8 in matrix bit 0, columns +8 in bit 1
        const int vrow = 16 * w4 + (mat >> 1) * 8 + r8, vchunk = mat & 1;       // values: the other way round
        const uint32_t k_off = swz(0u, krow, kchunk), v_off = swz(0u, vrow, vchunk);
        pdl_wait();
        const bool owner = rank == 0 && pos >= 0;             // of the new position
        uint2 r = make_uint2(0u, 0u);
        {
            uint2 u = make_uint2(0u, 0u);
            if (warp < 4) asm volatile("ld.global.cg.v2.u32 {%0,%1}, [%2];" : "=r"(u.x), "=r"(u.y) : "l"(src_row));
            const float x[4] = {bf_lo(u.x), bf_hi(u.x), bf_lo(u.y), bf_hi(u.y)};
            if (warp == 3) {
                if (owner) {
                    *reinterpret_cast<uint2*>(a.vcache + cache_row) = u;
                    *reinterpret_cast<float4*>(&po[kAttnWarps][0][4 * lane]) = make_float4(x[0], x[1], x[2], x[3]);
                    *reinterpret_cast<float4*>(&po[kAttnWarps][1][4 * lane]) = make_float4(x[0], x[1], x[2], x[3]);
                }
            } else if (is_q || (warp == 2 && owner)) {
                // the rounding steps of qk_rope_scatter_kernel on packed pairs: a product or a sum of two bf16 values, rounded once
                const float ss = warp_sum(x[0] * x[0] + x[1] * x[1] + x[2] * x[2] + x[3] * x[3]);
                const float rstd = rsqrt_full(ss * (1.0f / HD) + a.eps);
                const uint2 gq = *reinterpret_cast<const uint2*>(&rot_s[is_q ? 0 : 1][4 * lane]);
                const uint2 cq = *reinterpret_cast<const uint2*>(&rot_s[2][ei]), sq = *reinterpret_cast<const uint2*>(&rot_s[2][HD / 2 + ei]);
                const uint32_t n0 = mul_bf16x2(pack_bf16x2(x[0] * rstd, x[1] * rstd), gq.x), n1 = mul_bf16x2(pack_bf16x2(x[2] * rstd, x[3] * rstd), gq.y);
                const uint32_t neg = hi_half ? 0u : 0x80008000u;
                const uint32_t y0 = __shfl_xor_sync(0xffffffffu, n0, 16) ^ neg, y1 = __shfl_xor_sync(0xffffffffu, n1, 16) ^ neg;      // elements j +- 64
                r.x = add_bf16x2(mul_bf16x2(n0, cq.x), mul_bf16x2(y0, sq.x));
                r.y = add_bf16x2(mul_bf16x2(n1, cq.y), mul_bf16x2(y1, sq.y));
                if (is_q) {                        // words 2 lane and 2 lane + 1: k-step lane / 4, half (lane / 2) % 2, t = 2 (lane % 2) and the next
                    uint32_t* w = &q_s[warp][2 * (lane & 1)][2 * (lane >> 2) + ((lane >> 1) & 1)];
                    w[0] = r.x; w[20] = r.y;
                } else {
                    *reinterpret_cast<uint2*>(k_s + 4 * lane) = r;
                    *reinterpret_cast<uint2*>(a.kcache + cache_row) = r;
                }
            }
        }
        compute_sync();
        if (warp < 2) {
            if (owner) {                           // the new position's score for this head
                const uint2 k2 = *reinterpret_cast<const uint2*>(k_s + 4 * lane);
                const float s = warp_sum(bf_lo(r.x) * bf_lo(k2.x) + bf_hi(r.x) * bf_hi(k2.x) + bf_lo(r.y) * bf_lo(k2.y) + bf_hi(r.y) * bf_hi(k2.y));
                if (lane == 0) pml[warp][kAttnWarps] = make_float2(s * kScoreScale, 1.f);
            } else {
                if (lane == 0) pml[warp][kAttnWarps] = make_float2(-INFINITY, 0.f);
                *reinterpret_cast<float4*>(&po[kAttnWarps][warp][4 * lane]) = make_float4(0.f, 0.f, 0.f, 0.f);
            }
        }
        uint32_t qb[8][2];                                     // N columns: heads 0, 1, 0, 1, ...
#pragma unroll
        for (int k = 0; k < 8; k += 2) {
            const uint4 q = *reinterpret_cast<const uint4*>(&q_s[g & 1][t][2 * k]);
            qb[k][0] = q.x; qb[k][1] = q.y; qb[k + 1][0] = q.z; qb[k + 1][1] = q.w;
        }
        float m0 = -INFINITY, m1 = -INFINITY, l0 = 0.f, l1 = 0.f;
        float o[8][4];
#pragma unroll
        for (int i = 0; i < 8; ++i) { o[i][0] = 0.f; o[i][1] = 0.f; o[i][2] = 0.f; o[i][3] = 0.f; }
#pragma unroll 1
        for (int it = group; it < n_tiles; it += kGroups) {
            const int s = ring_slot(it);
            bool ok = true;
            uint32_t spins = 0;
            while (!mbar_try_wait(&full[s], ring_parity(it))) { if (++spins >= a.limit || failed) { ok = false; break; } }
            if (!__all_sync(0xffffffffu, ok)) { failed = 1; break; }          // one answer for the warp
            const int nv = p1 - p0 - it * kTilePos - 16 * w4;  // valid positions of this warp's sixteen
            if (nv > 0) {
                const uint32_t tk = smem_u32(ring + s * kTileBytes), tv = tk + 2 * kHalfTile;
                const uint32_t ak = tk + k_off, av = tv + v_off;               // chunk 0 of this lane's row; chunk 2 c: that ^ (c << 5)
                if (nv < 16) {
                    // rows past the sequence: whatever the cache holds there (it may be NaN) must not reach P V
#pragma unroll 1
                    for (int i = lane; i < (16 - nv) * 16; i += 32) {
                        const int row = 16 * w4 + nv + (i >> 4), c = i & 15;
                        asm volatile("st.shared.v4.u32 [%0], {%1, %1, %1, %1};" ::"r"(swz(tv + (c >> 3) * kHalfTile, row, c & 7)), "r"(0u) : "memory");
                    }
                    __syncwarp();
                }
                float sa[4] = {0.f, 0.f, 0.f, 0.f}, sb[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                for (int k = 0; k < 8; k += 2) {
                    uint32_t f[4];
                    ldsm4(f, (ak ^ ((k & 3) << 5)) + (k >> 2) * kHalfTile);
                    mma16816(sa, f[0], f[1], f[2], f[3], qb[k][0], qb[k][1]);
                    ldsm4(f, (ak ^ (((k + 1) & 3) << 5)) + (k >> 2) * kHalfTile);
                    mma16816(sb, f[0], f[1], f[2], f[3], qb[k + 1][0], qb[k + 1][1]);
                }
                // every lane holds (position g, heads 0 and 1) and (position g + 8, ...)
                float s0 = (sa[0] + sb[0]) * kScoreScale, s1 = (sa[1] + sb[1]) * kScoreScale;
                float s2 = (sa[2] + sb[2]) * kScoreScale, s3 = (sa[3] + sb[3]) * kScoreScale;
                if (g >= nv) { s0 = -INFINITY; s1 = -INFINITY; }
                if (g + 8 >= nv) { s2 = -INFINITY; s3 = -INFINITY; }
                // The reference may lag behind the maximum: sums and probabilities are floating point, so nothing is lost
                // until a score passes it by 2^60.  It starts as the maximum of the warp's first positions.
                const bool over = fmaxf(s0, s2) > m0 + 60.f || fmaxf(s1, s3) > m1 + 60.f;
                if (__any_sync(0xffffffffu, over)) {
                    float x0 = fmaxf(s0, s2), x1 = fmaxf(s1, s3);
#pragma unroll
                    for (int of = 4; of < 32; of <<= 1) {
                        x0 = fmaxf(x0, __shfl_xor_sync(0xffffffffu, x0, of));
                        x1 = fmaxf(x1, __shfl_xor_sync(0xffffffffu, x1, of));
                    }
                    const float n0 = fmaxf(m0, x0), n1 = fmaxf(m1, x1);
                    const float c0 = ex2f(m0 - n0), c1 = ex2f(m1 - n1);
                    m0 = n0; m1 = n1; l0 *= c0; l1 *= c1;
#pragma unroll
                    for (int i = 0; i < 8; ++i) { o[i][0] *= c0; o[i][1] *= c1; o[i][2] *= c0; o[i][3] *= c1; }
                }
                const float e0 = ex2f(s0 - m0), e1 = ex2f(s1 - m1), e2 = ex2f(s2 - m0), e3 = ex2f(s3 - m1);
                l0 += e0 + e2; l1 += e1 + e3;
                const uint32_t h01 = pack_bf16x2(e0, e1), h23 = pack_bf16x2(e2, e3);
                // Lane t = 2 supplies the high part, 0 the middle one, 1 the low one (both differences are exact), 3 nothing.
                const float r0 = e0 - bf_lo(h01), r1 = e1 - bf_hi(h01), r2 = e2 - bf_lo(h23), r3 = e3 - bf_hi(h23);
                const uint32_t m01 = pack_bf16x2(r0, r1), m23 = pack_bf16x2(r2, r3);
                uint32_t u = t == 2 ? h01 : m01, v = t == 2 ? h23 : m23;
                if (t == 1) { u = pack_bf16x2(r0 - bf_lo(m01), r1 - bf_hi(m01)); v = pack_bf16x2(r2 - bf_lo(m23), r3 - bf_hi(m23)); }
                if (t == 3) { u = 0u; v = 0u; }
                const uint32_t b0 = movm_t(u), b1 = movm_t(v);
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    uint32_t f[4];
                    ldsm4_t(f, (av ^ ((i & 3) << 5)) + (i >> 2) * kHalfTile);
                    mma16816(o[i], f[0], f[1], f[2], f[3], b0, b1);
                }
            }
            __syncwarp();
            if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&empty[s])) : "memory");
        }
#pragma unroll
        for (int of = 4; of < 32; of <<= 1) { l0 += __shfl_xor_sync(0xffffffffu, l0, of); l1 += __shfl_xor_sync(0xffffffffu, l1, of); }
        if (lane == 0) { pml[0][warp] = make_float2(m0, l0); pml[1][warp] = make_float2(m1, l1); }
        // The three parts of an output lie in lanes t = 0, 1, 2: added up (middle + low, then high) in two exchanges that leave each
        // lane a quarter of the sums, lane t the rows with bit 3 = t & 1 and bit 4 = t >> 1, so that the 32 lanes of a store hit
        // 32 banks.
        const bool t0 = (t & 1) != 0, t1 = (t & 2) != 0;
        float w[8][2];
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int j = 0; j < 2; ++j) w[i][j] = (t0 ? o[i][j + 2] : o[i][j]) + __shfl_xor_sync(0xffffffffu, t0 ? o[i][j] : o[i][j + 2], 1);
#pragma unroll
        for (int i = 0; i < 8; i += 2)
#pragma unroll
            for (int j = 0; j < 2; ++j)
                po[warp][j][16 * (i + (t >> 1)) + 8 * (t & 1) + g] = (t1 ? w[i + 1][j] : w[i][j]) + __shfl_xor_sync(0xffffffffu, t1 ? w[i][j] : w[i + 1][j], 2);
        compute_sync();
        bf16* out = a.attn + (size_t)b * DQ + 2 * kvh * HD;
        if constexpr (CS > 1) asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
        // two outputs a thread; with more than one rank the partials go to the rank that owns them (st.async: the receiver waits for
        // the bytes on a barrier of its own, one way, where stores and a cluster barrier took a round trip more)
        if (tid < HD) {
            const int e = 2 * tid, h = tid >> 6, d = e % HD;
            float m = -1e30f, l = 0.f;
            float2 acc = make_float2(0.f, 0.f);
#pragma unroll
            for (int w = 0; w <= kAttnWarps; ++w) m = fmaxf(m, pml[h][w].x);
#pragma unroll
            for (int w = 0; w <= kAttnWarps; ++w) {
                const float2 ml = pml[h][w], p = *reinterpret_cast<const float2*>(&po[w][h][d]);
                const float c = ex2f(ml.x - m);
                l = fmaf(ml.y, c, l); acc.x = fmaf(p.x, c, acc.x); acc.y = fmaf(p.y, c, acc.y);
            }
            if constexpr (CS == 1) {
                *reinterpret_cast<uint32_t*>(out + e) = l > 0.f ? pack_bf16x2(acc.x / l, acc.y / l) : 0u;
            } else {
                st_async_f32x2(&rv[rank][e % NE], e / NE, acc.x, acc.y, &arrived);
                if (e % NE == 0) st_async_f32x2(&rml[rank], e / NE, m, l, &arrived);
            }
        }
        if constexpr (CS > 1) {
            if (rank < kMergers && tid < NE / 2) {
                uint32_t spins = 0;
                while (!mbar_try_wait_cluster(&arrived, 0)) { if (++spins >= a.limit) { failed = 1; break; } }
                float m = -1e30f, l = 0.f;
                float2 acc = make_float2(0.f, 0.f);
#pragma unroll
                for (int q = 0; q < CS; ++q) m = fmaxf(m, rml[q].x);
#pragma unroll
                for (int q = 0; q < CS; ++q) {
                    const float2 ml = rml[q], p = *reinterpret_cast<const float2*>(&rv[q][2 * tid]);
                    const float c = ex2f(ml.x - m);
                    l = fmaf(ml.y, c, l); acc.x = fmaf(p.x, c, acc.x); acc.y = fmaf(p.y, c, acc.y);
                }
                *reinterpret_cast<uint32_t*>(out + rank * NE + 2 * tid) = l > 0.f ? pack_bf16x2(acc.x / l, acc.y / l) : 0u;
            }
        }
    }
    if constexpr (CS > 1) {
        if (warp == kAttnWarps) {                                // the feeding warp's share of the barrier
            asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
        }
    }
    __syncthreads();
    if (failed) {
        // A CTA that gave up may be ahead of ranks that have yet to write here, and must not leave before they have.  All send, also where
        // their waits ran out, so the bytes come; should one take longer than this wait, the barrier holds this CTA until the others have left
        // (threads that have exited count as arrived).  Only here: an arrival by everyone behind the sends costs a step 15 us.
        if constexpr (CS > 1) {
            bool all = rank >= kMergers;                       // nobody sends there
            for (uint32_t spins = 0; !all && spins < kSpin; ++spins) all = mbar_try_wait_cluster(&arrived, 0);
            if (!__syncthreads_and(all)) {
                asm volatile("barrier.cluster.arrive.release;" ::: "memory");
                asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
            }
        }
        if (tid == 0) {
            if (atomicCAS(&a.status[0], 0u, (uint32_t)ITTAI_ST_STREAM_TIMEOUT) == 0u) { a.status[1] = (uint32_t)n_tiles; a.status[2] = blockIdx.x; }
            const long long t0 = clock64();                    // copies still in flight land before the shared memory is handed back
            while (clock64() - t0 < 2000000) {}
        }
        __syncthreads();
    }
}

// ---- host side --------------------------------------------------------------------------------------------------------------
struct Plan {
    IttaiQwen3Decode p;
    Buffers w;
    CUtensorMap tm_k, tm_v;
    int n_sms = 0;
    bool bound = false;
    cudaStream_t side = nullptr;
    cudaEvent_t last = nullptr;
    cudaGraphExec_t exec[sizeof(kPieces) / sizeof(int)][2][2] = {};   // by cluster size, whether gate/up holds tiles and whether the head runs
    cudaGraphExec_t several[sizeof(kPieces) / sizeof(int)][2] = {};   // kSeveral tokens with the head
    int queued[sizeof(kPieces) / sizeof(int)][2] = {};                // tokens of that kind queued one by one
    std::mutex mu;
};
// Tokens of a kind in one graph.  Between the kernels of a graph a launch overlaps its predecessor's tail, and the first projection's weights come
// while the last kernel of the token before runs; between graphs neither.  us per step with 1 / 2 / 4 / 8 / 16 tokens a graph: batch 1 at 60
// 374.8 / 373.5 / 371.9 / 371.3 / 370.8, at 4096 460 / 458.2 / 456.7 / 456.6 / 456, batch 4 at 300 434 / 430.4 / 429.4 / 429.2 / 428.2, batch 8 at 1000
// 615.8 / 613 / 611.6 / 610.9 / 610.  Capturing four takes the host 2.4 to 3.3 ms: it is done while the GPU has work of the call, behind the 16th token
// of a long one, or behind the last of a call of eight or more once 64 have been queued one by one (the request loop's).
constexpr int kSeveral = 4, kSeveralInCall = 16, kSeveralAfter = 64, kSeveralBehind = 8;

template <typename F>
static cudaError_t prefer_shared(F* fn, int dynamic = 0) {
    // every kernel of the chain asks for the same carve-out: CTAs of two kernels share an SM only under one L1 / shared split
    cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
    if (e == cudaSuccess && dynamic > 0) e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, dynamic);
    return e;
}
template <int NB>
static cudaError_t set_attributes_nb() {
    cudaError_t e = prefer_shared(gemv_kernel<NB, D, 32, kPlain>, gemv_smem<D, 32>());
    if (e == cudaSuccess) e = prefer_shared(gemv_kernel<NB, D, 48, kSwiglu>, gemv_smem<D, 48>());
    if (e == cudaSuccess) e = prefer_shared(gemv_kernel<NB, D, 48, kSwiglu, 2>, gemv_smem<D, 48>());
    if (e == cudaSuccess) e = prefer_shared(gemv_kernel<NB, DQ, 8, kResidual>, gemv_smem<DQ, 8>());
    if (e == cudaSuccess) e = prefer_shared(gemv_kernel<NB, FF, 8, kResidual>, gemv_smem<FF, 8>());
    if (e == cudaSuccess) e = prefer_shared(head_kernel<NB>, kHeadSmem);
    if (e == cudaSuccess) e = prefer_shared(finish_kernel<NB, true>);
    if (e == cudaSuccess) e = prefer_shared(finish_kernel<NB, false>);
    return e;
}
static cudaError_t set_attributes() {
    static thread_local int attr_dev = -1;
    int dev = 0;
    cudaGetDevice(&dev);
    if (attr_dev == dev) return cudaSuccess;
    cudaError_t e = set_attributes_nb<1>();
    if (e == cudaSuccess) e = set_attributes_nb<2>();
    if (e == cudaSuccess) e = set_attributes_nb<4>();
    if (e == cudaSuccess) e = set_attributes_nb<8>();
    if (e == cudaSuccess) e = prefer_shared(attn_kernel<1>, kAttnSmem);
    if (e == cudaSuccess) e = prefer_shared(attn_kernel<2>, kAttnSmem);
    if (e == cudaSuccess) e = prefer_shared(attn_kernel<4>, kAttnSmem);
    if (e == cudaSuccess) e = prefer_shared(attn_kernel<7>, kAttnSmem);
    if (e == cudaSuccess) e = prefer_shared(attn_kernel<8>, kAttnSmem);
    if (e == cudaSuccess) e = prefer_shared(attn_kernel<12>, kAttnSmem);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(attn_kernel<12>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e == cudaSuccess) attr_dev = dev;
    return e;
}

template <int CS>
static cudaError_t launch_attn(const Plan& pl, const AttnChainArgs& a, cudaStream_t st) {
    return launch_pdl(attn_kernel<CS>, dim3(a.batch * NKV * CS), dim3(kAttnThreads), kAttnSmem, st, CS, pl.tm_k, pl.tm_v, a);
}

// The kernels of one token, in order, on `st` (captured into a graph, or launched as they are).
template <int NB>
static cudaError_t enqueue_token(const Plan& pl, int cs, bool held, bool head, cudaStream_t st) {
    const IttaiQwen3Decode& p = pl.p;
    const Buffers& w = pl.w;
    auto bp = [](const void* q, size_t off = 0) { return reinterpret_cast<const bf16*>(q) + off; };
    const uint32_t limit = p.spin_limit > 0 ? (uint32_t)p.spin_limit : kSpin, limit_parked = p.spin_limit > 0 ? (uint32_t)p.spin_limit : kSpinParked;
    const int drop = (p.flags & ITTAI_F_TEST_DROP_CTA) != 0;
    cudaError_t e = cudaSuccess;
    for (int l = 0; l < p.n_layers && e == cudaSuccess; ++l) {
        const size_t kv = (size_t)l * NB * NKV * p.kv_cap * HD;
        GemvArgs q{bp(p.wqkv, (size_t)l * DQKV * D), w.h, bp(p.ln1, (size_t)l * D), nullptr, w.qkv, DQKV, p.eps, p.status, nullptr, nullptr, nullptr, 0, nullptr, 0, l == 0, drop, limit_parked};
        e = launch_pdl(gemv_kernel<NB, D, 32, kPlain>, dim3(DQKV / 32), dim3(kGemvThreads), gemv_smem<D, 32>(), st, 1, q);
        if (e != cudaSuccess) break;
        AttnChainArgs a{w.st, w.qkv, bp(p.qn, (size_t)l * HD), bp(p.kn, (size_t)l * HD), bp(p.rope), reinterpret_cast<bf16*>(p.kcache) + kv,
                        reinterpret_cast<bf16*>(p.vcache) + kv, w.attn, p.status, l, NB, p.kv_cap, p.eps, limit, limit_parked};
        switch (cs) {
            case 1: e = launch_attn<1>(pl, a, st); break;
            case 2: e = launch_attn<2>(pl, a, st); break;
            case 4: e = launch_attn<4>(pl, a, st); break;
            case 7: e = launch_attn<7>(pl, a, st); break;
            case 8: e = launch_attn<8>(pl, a, st); break;
            default: e = launch_attn<12>(pl, a, st); break;
        }
        if (e != cudaSuccess) break;
        // gate/up finds no room on an SM while attention is there: its weights come as far as L2
        GemvArgs o{bp(p.wo, (size_t)l * D * DQ), w.attn, nullptr, w.h, w.hmid, D, p.eps, p.status, nullptr, nullptr, nullptr, 0,
                   reinterpret_cast<const unsigned char*>(bp(p.wgu, (size_t)l * DGU * D)), DGU * D * 2 / (D / 8) / 8, 0, drop, limit_parked};
        e = launch_pdl(gemv_kernel<NB, DQ, 8, kResidual>, dim3(D / 8), dim3(kGemvThreads), gemv_smem<DQ, 8>(), st, 1, o);
        if (e != cudaSuccess) break;
        const size_t kv1 = kv + (size_t)NB * NKV * p.kv_cap * HD;
        const bf16 *k1 = l + 1 < p.n_layers ? reinterpret_cast<const bf16*>(p.kcache) + kv1 : nullptr, *v1 = reinterpret_cast<const bf16*>(p.vcache) + kv1;
        GemvArgs gu{bp(p.wgu, (size_t)l * DGU * D), w.hmid, bp(p.ln2, (size_t)l * D), nullptr, w.act, FF, p.eps, p.status, w.st,
                    NB > 1 ? k1 : nullptr, v1, p.kv_cap, nullptr, 0, 0, drop, limit_parked};
        e = launch_pdl(held ? gemv_kernel<NB, D, 48, kSwiglu, 2> : gemv_kernel<NB, D, 48, kSwiglu>, dim3(DGU / 48), dim3(kGemvThreads), gemv_smem<D, 48>(), st, 1, gu);
        if (e != cudaSuccess) break;
        GemvArgs dn{bp(p.wd, (size_t)l * D * FF), w.act, nullptr, w.hmid, w.h, D, p.eps, p.status, w.st,
                    NB == 1 ? k1 : nullptr, v1, p.kv_cap, nullptr, 0, 0, drop, limit_parked};
        e = launch_pdl(gemv_kernel<NB, FF, 8, kResidual>, dim3(D / 8), dim3(kGemvThreads), gemv_smem<FF, 8>(), st, 1, dn);
    }
    if (e != cudaSuccess) return e;
    TokenArgs t{w.st, bp(p.embed), w.h, w.cand_val, w.cand_idx, pl.n_sms, p.pos, p.next_id, p.status, p.vocab, p.kv_cap};
    if (!head) return launch_pdl(finish_kernel<NB, false>, dim3(1), dim3(32 * NB), 0, st, 1, t);
    HeadArgs h{bp(p.embed), w.h, bp(p.fin_w), p.write_logits ? reinterpret_cast<bf16*>(p.logits) : nullptr, w.cand_val, w.cand_idx, p.status, p.vocab, p.eps, limit_parked};
    e = launch_pdl(head_kernel<NB>, dim3(pl.n_sms), dim3(kGemvThreads + 32), kHeadSmem, st, 1, h);
    if (e != cudaSuccess) return e;
    return launch_pdl(finish_kernel<NB, true>, dim3(1), dim3(32 * NB), 0, st, 1, t);
}
static cudaError_t enqueue_token(const Plan& pl, int cs, bool held, bool head, cudaStream_t st) {
    switch (pl.p.batch) {
        case 1: return enqueue_token<1>(pl, cs, held, head, st);
        case 2: return enqueue_token<2>(pl, cs, held, head, st);
        case 4: return enqueue_token<4>(pl, cs, held, head, st);
        default: return enqueue_token<8>(pl, cs, held, head, st);
    }
}
static void enqueue_begin(const Plan& pl, const IttaiQwen3Decode& c, cudaStream_t st) {
    const IttaiQwen3Decode& p = pl.p;
    TokenArgs t{pl.w.st, reinterpret_cast<const bf16*>(p.embed), pl.w.h, pl.w.cand_val, pl.w.cand_idx, pl.n_sms, p.pos, p.next_id, p.status, p.vocab, p.kv_cap};
    switch (p.batch) {
        case 1: begin_kernel<1><<<1, 32, 0, st>>>(t, c.out_ids, c.forced, c.step_ns, c.n_steps, c.n_forced); break;
        case 2: begin_kernel<2><<<1, 64, 0, st>>>(t, c.out_ids, c.forced, c.step_ns, c.n_steps, c.n_forced); break;
        case 4: begin_kernel<4><<<1, 128, 0, st>>>(t, c.out_ids, c.forced, c.step_ns, c.n_steps, c.n_forced); break;
        default: begin_kernel<8><<<1, 256, 0, st>>>(t, c.out_ids, c.forced, c.step_ns, c.n_steps, c.n_forced); break;
    }
}

static void drop_graphs(Plan* pl) {
    for (auto& size : pl->exec)
        for (auto& row : size)
            for (cudaGraphExec_t& x : row)
                if (x != nullptr) { cudaGraphExecDestroy(x); x = nullptr; }
    for (auto& size : pl->several)
        for (cudaGraphExec_t& x : size)
            if (x != nullptr) { cudaGraphExecDestroy(x); x = nullptr; }
    for (auto& size : pl->queued)
        for (int& n : size) n = 0;
}

}  // namespace chain

void set_error(const char* fmt, ...);
int cuda_fail(cudaError_t e, const char* what);
int decode_check_args(const IttaiQwen3Decode* p);      // qwen3_decode.cu

namespace chain {

static int bind(Plan* pl, const IttaiQwen3Decode* p) {
    pl->p = *p;
    layout(p->batch, reinterpret_cast<char*>(p->workspace), &pl->w);
    const long long rows = (long long)p->n_layers * p->batch * NKV * p->kv_cap;
    if (rows >= (1ll << 31)) { set_error("the cache has %lld rows; at most 2^31 - 1 are supported", rows); return ITTAI_E_ARG; }
    int rc = make_tmap_bf16(&pl->tm_k, p->kcache, rows, HD, HD, kTilePos);
    if (rc == ITTAI_OK) rc = make_tmap_bf16(&pl->tm_v, p->vcache, rows, HD, HD, kTilePos);
    return rc;
}
// Whether a graph captured for `a` also serves `b`: everything but the per-call parameters, which travel in State.
static bool same_binding(const IttaiQwen3Decode& a, const IttaiQwen3Decode& b) {
    return a.n_layers == b.n_layers && a.vocab == b.vocab && a.kv_cap == b.kv_cap && a.batch == b.batch && a.eps == b.eps && a.write_logits == b.write_logits &&
           a.flags == b.flags && a.spin_limit == b.spin_limit &&
           a.wqkv == b.wqkv && a.wo == b.wo && a.wgu == b.wgu && a.wd == b.wd && a.ln1 == b.ln1 && a.ln2 == b.ln2 && a.qn == b.qn && a.kn == b.kn &&
           a.fin_w == b.fin_w && a.embed == b.embed && a.rope == b.rope && a.kcache == b.kcache && a.vcache == b.vcache && a.pos == b.pos &&
           a.next_id == b.next_id && a.logits == b.logits && a.workspace == b.workspace && a.status == b.status;
}

static int capture(Plan* pl, int cs, bool held, bool head, int tokens, cudaGraphExec_t* out) {
    if (pl->side == nullptr) {
        const cudaError_t e = cudaStreamCreateWithFlags(&pl->side, cudaStreamNonBlocking);
        if (e != cudaSuccess) return cuda_fail(e, "cudaStreamCreateWithFlags");
    }
    cudaGraph_t g = nullptr;
    cudaError_t e = cudaStreamBeginCapture(pl->side, cudaStreamCaptureModeThreadLocal);
    if (e != cudaSuccess) return cuda_fail(e, "cudaStreamBeginCapture");
    cudaError_t el = cudaSuccess;
    for (int i = 0; i < tokens && el == cudaSuccess; ++i) el = enqueue_token(*pl, cs, held, head, pl->side);
    e = cudaStreamEndCapture(pl->side, &g);
    if (el != cudaSuccess || e != cudaSuccess) {
        if (g != nullptr) cudaGraphDestroy(g);
        cudaGetLastError();
        return cuda_fail(el != cudaSuccess ? el : e, "capture of a decode step");
    }
    e = cudaGraphInstantiate(out, g, 0);
    cudaGraphDestroy(g);
    if (e != cudaSuccess) return cuda_fail(e, "cudaGraphInstantiate");
    return ITTAI_OK;
}

// Everything one call queues on `st`.
static int enqueue_call(Plan* pl, const IttaiQwen3Decode& p, int max_len, bool captured, cudaStream_t st) {
    enqueue_begin(*pl, p, st);
    bool refused = false;                              // a graph of several tokens could not be had in this call: it goes on with those of one
    for (int i = 0; i < p.n_steps; ++i) {
        const bool head = i >= p.n_forced - 1;
        const int cs = pieces(p.batch, max_len + i);
        const bool held = hold_tiles(p.batch, max_len + i);
        int slot = 0;
        while (kPieces[slot] != cs) ++slot;
        cudaError_t e;
        if (captured) {                                // a graph launch cannot be captured: the kernels themselves can
            e = enqueue_token(*pl, cs, held, head, st);
        } else {
            const int last = i + kSeveral - 1, len = max_len + last;
            const bool same = head && last < p.n_steps && pieces(p.batch, len) == cs && hold_tiles(p.batch, len) == held;
            cudaGraphExec_t& s = pl->several[slot][held ? 1 : 0];
            int& queued = pl->queued[slot][held ? 1 : 0];
            if (same && s == nullptr && i >= kSeveralInCall && !refused && capture(pl, cs, held, head, kSeveral, &s) != ITTAI_OK) { cudaGetLastError(); refused = true; }
            const bool several = same && s != nullptr;
            cudaGraphExec_t& x = several ? s : pl->exec[slot][held ? 1 : 0][head ? 1 : 0];
            if (x == nullptr) {
                const int rc = capture(pl, cs, held, head, 1, &x);
                if (rc != ITTAI_OK) return rc;
            }
            e = cudaGraphLaunch(x, st);
            if (several) i = last;
            else if (head && queued < kSeveralAfter) ++queued;
            if (i + 1 >= p.n_steps && i + 1 >= kSeveralBehind && head && queued >= kSeveralAfter && s == nullptr && !refused && e == cudaSuccess) {
                // the call's work is queued: without this graph the next calls go on one by one, and it is tried again 64 tokens later
                if (capture(pl, cs, held, true, kSeveral, &s) != ITTAI_OK) { cudaGetLastError(); queued = 0; }
            }
        }
        if (e != cudaSuccess) return cuda_fail(e, "launch of a decode step");
    }
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? ITTAI_OK : cuda_fail(e, "decode chain");
}

}  // namespace chain
}  // namespace ittai

using namespace ittai;

extern "C" int ittai_qwen3_chain_create(void** plan) {
    if (!plan) { set_error("null plan"); return ITTAI_E_ARG; }
    *plan = new (std::nothrow) chain::Plan();
    if (*plan == nullptr) { set_error("chain_create: out of host memory"); return ITTAI_E_ARG; }
    return ITTAI_OK;
}

extern "C" int ittai_qwen3_chain_destroy(void* plan) {
    chain::Plan* pl = reinterpret_cast<chain::Plan*>(plan);
    if (pl == nullptr) return ITTAI_OK;
    if (pl->last != nullptr) { cudaEventSynchronize(pl->last); cudaEventDestroy(pl->last); }
    chain::drop_graphs(pl);
    if (pl->side != nullptr) cudaStreamDestroy(pl->side);
    delete pl;
    return ITTAI_OK;
}

extern "C" int ittai_qwen3_chain_run(void* plan, const IttaiQwen3Decode* p, int32_t max_len, void* stream) {
    chain::Plan* pl = reinterpret_cast<chain::Plan*>(plan);
    if (!pl || max_len < 0) { set_error("chain_run: null plan or negative length"); return ITTAI_E_ARG; }
    int rc = decode_check_args(p);
    if (rc != ITTAI_OK) return rc;
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    std::lock_guard<std::mutex> lock(pl->mu);
    cudaError_t e = chain::set_attributes();
    if (e != cudaSuccess) return cuda_fail(e, "cudaFuncSetAttribute(decode chain)");
    if (pl->n_sms == 0) {
        int dev = 0;
        cudaGetDevice(&dev);
        e = cudaDeviceGetAttribute(&pl->n_sms, cudaDevAttrMultiProcessorCount, dev);
        if (e != cudaSuccess) return cuda_fail(e, "cudaDeviceGetAttribute(sm count)");
        if (pl->n_sms > chain::kMaxHeadCtas) pl->n_sms = chain::kMaxHeadCtas;
        e = cudaEventCreateWithFlags(&pl->last, cudaEventDisableTiming);
        if (e != cudaSuccess) return cuda_fail(e, "cudaEventCreateWithFlags");
    }
    if (!pl->bound || !chain::same_binding(pl->p, *p)) {
        if (pl->bound) { cudaEventSynchronize(pl->last); chain::drop_graphs(pl); }
        pl->bound = false;
        rc = chain::bind(pl, p);
        if (rc != ITTAI_OK) return rc;
        pl->bound = true;
    }
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    e = cudaStreamIsCapturing(st, &cap);
    if (e != cudaSuccess) return cuda_fail(e, "cudaStreamIsCapturing");
    const bool captured = cap != cudaStreamCaptureStatusNone;
    if (!captured) {                                   // the call before may be on another stream; both use one state record
        e = cudaStreamWaitEvent(st, pl->last, 0);      // (no wait before the first call has recorded it)
        if (e != cudaSuccess) return cuda_fail(e, "cudaStreamWaitEvent");
    }
    rc = chain::enqueue_call(pl, *p, max_len, captured, st);
    if (!captured) {                                   // also where the call failed half way: what it has queued still runs
        e = cudaEventRecord(pl->last, st);
        if (rc == ITTAI_OK && e != cudaSuccess) return cuda_fail(e, "cudaEventRecord");
    }
    return rc;
}
