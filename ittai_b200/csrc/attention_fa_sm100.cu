// Flash attention with a key loop on tcgen05, head_dim 128: the Qwen3 prefill (causal, grouped-query, keys and values in
// the cache layout, optionally behind a prefix).  Replaces the mma.sync attention task of the reference
// (src/ittai/qwen3/sm80.py:274-403) with tensor-memory MMAs: per CTA one tile of 128 query rows of one (sequence, head),
// walking the visible keys 128 at a time.
//
//   warp 0, one lane: TMA loads (Q once; K and V blocks single-buffered, each refilled as soon as the MMA that read it
//     has completed) and every MMA: S = Q K^T (M128 N128, 8 k-steps over the 128 dims), then O += P V as one
//     M128 N128 series whose A operand P is read from tensor memory and whose B operand V is used as loaded (MN-major:
//     the two 64-dim swizzle atoms of the tile are one operand, 16 KB apart in the descriptor's leading-dimension field).
//   warps 1-8: two threads per query row, one for the first 64 keys of a block and one for the others, ONE pass over the scores:
//     P = 2^(s*scale - ref) packed to bf16 over the consumed scores of the same half, and the half's running sum.  ref is the maximum
//     of the row's first block, raised only when 16 neighbouring P add up to more than 2^8: P, sums and O are floating point, so a
//     reference that lags behind the maximum costs little, and after that block there is no maximum to find ahead of the exponentials.  Raising is rare: the thread
//     rescales what it has written, and a vote of the quarter's two warps, which ends every block, brings the other half and O
//     to the same reference.  The halves' sums meet in the epilogue.
//     (One thread a row, two passes, a maximum kept within 2^8: 175 us a layer at 8 x 2048 tokens, 135 at 64 x 512, 53 for 55 texts of
//     16 to 512, 188 dense at 4 x 2048; this way 156, 128, 48 and 158.  Of the difference, a third came with the elected issuing lane.
//     Without any softmax, the two CTAs' MMAs and hand-offs alone: 115 at 8 x 2048.)
//     The error against 64 bits is that of two passes for scores without an order (0.994 to 1.011 of it at 256 to 3000 keys and scores up
//     to 30 log2 units wide).  What a raise finds already written is rounded to bf16 a second time, which two passes did not do: where the
//     scores keep rising along the keys the result stays within 2^-7 of the largest value, as tested, but is not as exact.
// TMEM (256 columns, two CTAs per SM): S / P in columns 0..127, O in 128..255.  Shared memory: Q, K, V tiles of 32 KB each
// (two 128-byte-swizzled atoms of 64 dims); the V tile doubles as the output staging area.
//
// A CTA does not end with its tile: it takes over the next tile that no CTA has begun (clusterlaunchcontrol.try_cancel: the
// hardware hands the CTAs out in index order as before, so the balance stays dynamic and the longest tiles first) and works
// across the seam: the next Q and first K block travel from the moment the last S of this tile is complete, and the next
// tile's first S is computed while this one's output is stored.  Launch, barrier set-up, tensor-memory allocation, the first
// loads and the first S were 7 us of a tile's 13 at 512 tokens (2.3 us per key block).  Every wait is a bounded mbarrier
// wait; on expiry the abort flag routes all roles to the common exit, where TMEM is freed.
#include "launch.h"
#include "tcgen05.cuh"
#include "tmap.h"

namespace ittai {

constexpr int kFaThreads = 288;               // the issuing warp and eight softmax warps
constexpr int kFaBlk = 128;                  // keys per block = query rows per tile = head_dim
constexpr uint32_t kFaCols = 256, kFaOCol = 128;
constexpr uint32_t kFaSpin = 1u << 22;
constexpr uint32_t kFaQ = 0, kFaK = 32768, kFaV = 65536, kFaBar = 98304;
constexpr uint32_t kFaX = kFaBar + 256;      // float [2 halves][128 rows]: what the two threads of a row tell each other
constexpr int kFaListSeqs = 256, kFaListSteps = 64;
// Ragged sequences: the non-empty (sequence, step of 128 rows) pairs in the order in which they are handed out, the last steps first.
// order: sequences by their number of steps, descending; those that have step z are its first start[j + 1] - start[j], j = steps - 1 - z.
struct FaList {
    int total;
    int start[kFaListSteps + 1];
    unsigned short order[kFaListSeqs], steps[kFaListSeqs];
};
constexpr uint32_t kFaList = kFaX + 1024;
constexpr uint32_t kFaSmem = kFaList + 1024, kFaSmemList = kFaSmem + ((sizeof(FaList) + 15) & ~15);
constexpr float kFaRaise = 256.f;            // the reference is raised once sixteen neighbouring keys' P add up to more

struct AttnFaArgs {
    const int4* seqs;
    bf16* o;
    long long o_row, o_head;
    int group, causal, seqs_ready;
    int k_seq_rows, k_head_rows;             // cache layout: strides in rows of 128 elements
    int n_seqs, n_steps;                     // of a list
    int k_head_cols;                         // packed layout (heads side by side in a row, sequences by their row offsets): HDIM, else 0
    float scale_log2;
    uint32_t* status;
};

__device__ __forceinline__ void fa_arrive(void* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool fa_wait(void* bar, uint32_t parity, volatile uint32_t* abort_flag) {
    uint32_t spins = 0;
    while (!mbar_try_wait_parked(bar, parity)) {
        if (((++spins) & 255u) == 0u && (*abort_flag || spins >= kFaSpin)) { *abort_flag = 1; return false; }
    }
    return true;
}
// The same for a whole warp: one answer for all lanes, which go on with warp-wide steps.
__device__ __forceinline__ bool fa_wait_warp(void* bar, uint32_t parity, volatile uint32_t* abort_flag) {
    return __all_sync(0xffffffffu, fa_wait(bar, parity, abort_flag)) != 0;
}
__device__ __forceinline__ float fa_ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// Asks for a CTA of this grid that has not begun; the 16-byte answer is counted on `bar`.
__device__ __forceinline__ void fa_try_cancel(void* answer, void* bar) {
    asm volatile("clusterlaunchcontrol.try_cancel.async.shared::cta.mbarrier::complete_tx::bytes.b128 [%0], [%1];" ::"r"(smem_u32(answer)), "r"(smem_u32(bar)) : "memory");
}
// (x, y, z) of the CTA taken over and 1, or w = 0: none was left.
__device__ __forceinline__ int4 fa_answer(const void* answer) {
    int4 id = make_int4(0, 0, 0, 0);
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        ".reg .b128 r;\n"
        "ld.shared.b128 r, [%4];\n"
        "clusterlaunchcontrol.query_cancel.is_canceled.pred.b128 p, r;\n"
        "selp.s32 %3, 1, 0, p;\n"
        "@p clusterlaunchcontrol.query_cancel.get_first_ctaid.v4.b32.b128 {%0, %1, %2, _}, r;\n"
        "}\n"
        : "+r"(id.x), "+r"(id.y), "+r"(id.z), "=r"(id.w) : "r"(smem_u32(answer)) : "memory");
    return id;
}
// The two warps of a lane quarter (64 threads) meet; true in both if either passes true.
__device__ __forceinline__ bool fa_vote(int q4, bool v) {
    uint32_t r;
    asm volatile("{\n.reg .pred p, o;\nsetp.ne.u32 p, %1, 0;\nbarrier.cta.red.or.pred o, %2, 64, p;\nselp.u32 %0, 1, 0, o;\n}\n" : "=r"(r) : "r"((uint32_t)v), "r"(1 + q4) : "memory");
    return r != 0;
}
// The first `cols` keys of this thread's P (bf16 pairs in tensor memory) times f.  Warp-wide; rare.
__device__ __noinline__ void fa_rescale_p(uint32_t t_half, int cols, float f) {
    tmem_st_wait();
#pragma unroll 1
    for (int cp = 0; cp < cols; cp += 16) {
        uint32_t u[8];
        tmem_ld_32x8(t_half + (uint32_t)(cp >> 1), u);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 8; ++i) { asm volatile("" : "+r"(u[i])); u[i] = pack_bf16x2(__uint_as_float(u[i] << 16) * f, __uint_as_float(u[i] & 0xFFFF0000u) * f); }
        tmem_st_32x8(t_half + (uint32_t)(cp >> 1), u);
    }
    tmem_st_wait();
}
// Largest of this thread's 64 scores, unscaled, of those 0..lim unless ALL are visible.  Warp-wide.
template <bool ALL>
__device__ __forceinline__ float fa_half_max(uint32_t t_half, int lim) {
    float m0 = -INFINITY, m1 = -INFINITY;
#pragma unroll
    for (int c0 = 0; c0 < 64; c0 += 32) {
        uint32_t v[16], u[16];
        tmem_ld_32x16(t_half + (uint32_t)c0, v);
        tmem_ld_32x16(t_half + (uint32_t)(c0 + 16), u);
        tmem_ld_wait16(v);
        tmem_ld_tie16(u);
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            m0 = fmaxf(m0, ALL || c0 + i <= lim ? __uint_as_float(v[i]) : -INFINITY);
            m1 = fmaxf(m1, ALL || c0 + 16 + i <= lim ? __uint_as_float(u[i]) : -INFINITY);
        }
    }
    return fmaxf(m0, m1);
}
// One query tile: where it lies and how many key blocks it sees.
struct FaTile { int head, r0, q_len, kv_len, n_blk, q_row, q_col, kv_row, kv_col; };
template <int HDIM, bool PAIR, bool LIST>
__device__ __forceinline__ FaTile fa_tile(const AttnFaArgs& a, const FaList* list, int x, int y, int z) {
    constexpr int kRows = PAIR ? kFaBlk / 2 : kFaBlk;        // query rows of a tile
    FaTile t;
    int step = (int)gridDim.z - 1 - z;
    if constexpr (LIST) {
        if (y >= list->total) { t = FaTile{}; return t; }      // no rows: passed over like the tiles of a sequence that is too short
        int lo = 0, hi = a.n_steps - 1;                        // the last j with start[j] <= y
        while (lo < hi) { const int m = (lo + hi + 1) >> 1; if (list->start[m] <= y) lo = m; else hi = m - 1; }
        step = a.n_steps - 1 - lo;
        y = list->order[y - list->start[lo]];
    }
    const int4 sinfo = a.seqs[y];
    // PAIR: x is two times the key/value head and which 64 rows of a step of 128, the later ones first.  (With steps of 64 in z the tiles that
    // share keys and values lie a whole layer of tiles apart: 64 texts of 512 tokens, whose keys and values exceed L2, 142 us instead of 126.)
    t.head = PAIR ? x & ~1 : x; t.r0 = step * kFaBlk + (PAIR && (x & 1) == 0 ? kRows : 0); t.q_len = sinfo.y; t.kv_len = sinfo.w;
    // causal: query r sees keys <= r + (kv_len - q_len)
    const int last_key = a.causal ? min(t.kv_len - 1, t.r0 + kRows - 1 + t.kv_len - t.q_len) : t.kv_len - 1;
    t.n_blk = last_key < 0 ? 0 : last_key / kFaBlk + 1;
    const int kvh = PAIR ? x >> 1 : x / a.group;
    t.q_row = sinfo.x + t.r0; t.q_col = t.head * HDIM;
    t.kv_row = y * a.k_seq_rows + kvh * a.k_head_rows + sinfo.z; t.kv_col = kvh * a.k_head_cols;
    return t;
}
template <int HDIM, bool PAIR, bool LIST>
__device__ __forceinline__ FaTile fa_tile(const AttnFaArgs& a, const FaList* list, int index) {
    const int yz = index / (int)gridDim.x;
    return fa_tile<HDIM, PAIR, LIST>(a, list, index - yz * (int)gridDim.x, yz % (int)gridDim.y, yz / (int)gridDim.y);
}
template <int HDIM, bool PAIR>
__device__ __forceinline__ void fa_zero_rows(const AttnFaArgs& a, const FaTile& t, int tid, int threads) {
    for (int i = tid; i < kFaBlk * 16; i += threads) {
        const int r = i >> 4, row = PAIR ? r & 63 : r, head = t.head + (PAIR ? r >> 6 : 0);
        if (t.r0 + row < t.q_len && (i & 15) < HDIM / 8)
            *reinterpret_cast<uint4*>(a.o + (long long)(t.q_row + row) * a.o_row + (long long)head * a.o_head + (i & 15) * 8) = make_uint4(0, 0, 0, 0);
    }
}
// Whole CTA.  A sequence takes part with the steps it has; ranks by counting (at most 256 x 256 comparisons, 55 texts 0.5 us, ahead of the wait
// for the kernel in front).
__device__ __forceinline__ void fa_build_list(const AttnFaArgs& a, FaList* list) {
    for (int i = threadIdx.x; i < a.n_seqs; i += kFaThreads) list->steps[i] = (unsigned short)min(max(a.seqs[i].y + kFaBlk - 1, 0) / kFaBlk, a.n_steps);
    __syncthreads();
    for (int i = threadIdx.x; i < a.n_seqs; i += kFaThreads) {
        const int mine = list->steps[i];
        int rank = 0;
        for (int u = 0; u < a.n_seqs; ++u) { const int s = list->steps[u]; rank += s > mine || (s == mine && u < i); }
        list->order[rank] = (unsigned short)i;
    }
    // thread j: everything in front of step n_steps - 1 - j, all sequences' steps above it
    for (int j = threadIdx.x; j <= a.n_steps; j += kFaThreads) {
        int before = 0;
        for (int u = 0; u < a.n_seqs; ++u) before += max((int)list->steps[u] - (a.n_steps - j), 0);
        list->start[j] = before;
        if (j == a.n_steps) list->total = before;
    }
    __syncthreads();
}
// Both 64-column atoms of a tile of 128 rows.
__device__ __forceinline__ void fa_load(unsigned char* dst, const CUtensorMap* tm, int col, int row, void* bar) {
    mbar_expect_tx(bar, 32768);
    tma_load_2d(dst, tm, col, row, bar);
    tma_load_2d(dst + 16384, tm, col + 64, row, bar);
}

// The query rows of a tile: 128 of one head, or with PAIR (boxes of 64 rows) 64 of each of two neighbouring heads.
template <bool PAIR>
__device__ __forceinline__ void fa_load_q(unsigned char* dst, const CUtensorMap* tm, const FaTile& t, void* bar) {
    if constexpr (!PAIR) {
        fa_load(dst, tm, t.q_col, t.q_row, bar);
    } else {
        mbar_expect_tx(bar, 32768);
#pragma unroll
        for (int i = 0; i < 4; ++i) tma_load_2d(dst + (i & 1) * 16384 + (i >> 1) * 8192, tm, t.q_col + 64 * i, t.q_row, bar);
    }
}

// HDIM: 128, or 80 for heads packed 80 columns apart (a head_dim of 72, zero-padded to whole k-steps of 16): S then takes five
// k-steps instead of eight and the projections around the kernel are 80/128 as wide.  The loads still fetch 128 columns (the
// next head's, or zeros past the last one) and P V still computes 128: an MN-major operand comes in whole 64-column atoms.
// The surplus columns of O are never read.
// PAIR, where two query heads share a key/value head (HDIM 128): a tile is 64 query rows of both, rows 0..63 of the first and 64..127 of
// the second.  The same keys and values serve both, and sequences are cut every 64 rows instead of 128: as many key blocks where the
// lengths are multiples of 128, fewer otherwise (a text of 142 tokens: four per pair of heads instead of six, one of 30: one instead of two).
// LIST: the tiles come from a list (see FaList).  A form of its own: with both ways in one kernel (53 -> 67 KB of code) the plain one took up to
// 30 % longer (16 texts of 512 tokens 45 us instead of 35).
template <int HDIM, bool PAIR, bool LIST>
__global__ void __launch_bounds__(kFaThreads, 2)
attn_fa_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
               const __grid_constant__ CUtensorMap tm_v, const AttnFaArgs a) {
    pdl_trigger();
    // The first tile's record is read here, ahead of the kernels that may still be running, only where the caller says that
    // none of them writes it.  A kernel of the same run of dependent launches may (position rows of variable-resolution
    // images): every launch in between lets its successors start on entry, so nothing but the wait orders the two.
    if (!a.seqs_ready) pdl_wait();
    extern __shared__ __align__(1024) unsigned char fa_raw[];
    unsigned char* sm = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(fa_raw) + 1023) & ~(uintptr_t)1023);
    FaList* list = reinterpret_cast<FaList*>(sm + kFaList);
    if constexpr (LIST) {
        fa_build_list(a, list);
        // Records that share rows have more tiles than the grid, whose length the host takes from the rows: the surplus is not computed.
        if (threadIdx.x == 0 && list->total > (int)gridDim.y && atomicCAS(&a.status[0], 0u, (uint32_t)ITTAI_ST_BAD_SEQS) == 0u) {
            a.status[1] = (uint32_t)list->total; a.status[2] = gridDim.y;
        }
    }
    // Grid (heads, sequences, query tiles) with the tiles in descending order: CTAs are handed out in index order, so the
    // causal tiles that walk the most key blocks start first and the last ones are short.
    const FaTile first = fa_tile<HDIM, PAIR, LIST>(a, list, blockIdx.x, blockIdx.y, blockIdx.z);
    if (first.r0 >= first.q_len) return;                   // the whole CTA: nothing allocated yet
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (first.n_blk == 0) {                                // no visible key: zero rows
        pdl_wait();
        fa_zero_rows<HDIM, PAIR>(a, first, threadIdx.x, kFaThreads);
        return;
    }

    unsigned long long* bars = reinterpret_cast<unsigned long long*>(sm + kFaBar);
    unsigned long long* bar_q = bars;             // Q landed
    unsigned long long* bar_k = bars + 1;         // K block landed (one phase per block)
    unsigned long long* bar_v = bars + 2;         // V block landed
    unsigned long long* bar_s = bars + 3;         // S of the block ready (also: K buffer free)
    unsigned long long* bar_p = bars + 4;         // P written, O rescaled (one arrival per softmax warp)
    unsigned long long* bar_o = bars + 5;         // PV of the block done (also: V buffer free)
    unsigned long long* bar_e = bars + 6;         // output stored: V buffer and O free (one arrival per softmax warp, one phase per tile)
    unsigned long long* bar_t = bars + 7;         // [2] next tile published, tile n in slot n % 2
    unsigned long long* bar_c = bars + 9;         // answer to try_cancel landed
    unsigned char* answer = reinterpret_cast<unsigned char*>(bars + 10);     // 16 bytes
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 12);
    volatile uint32_t* abort_flag = tmem_slot + 1;
    volatile int* next_tile = reinterpret_cast<volatile int*>(tmem_slot + 2);    // [2] CTA index, -1: none

    if (threadIdx.x == 0) {
        mbar_init(bar_q, 1); mbar_init(bar_k, 1); mbar_init(bar_v, 1); mbar_init(bar_s, 1); mbar_init(bar_p, 8); mbar_init(bar_o, 1);
        mbar_init(bar_e, 8); mbar_init(bar_t, 1); mbar_init(bar_t + 1, 1); mbar_init(bar_c, 1);
        *abort_flag = 0;
        fence_mbar_init();
        pdl_wait();                                        // q, k, v come from the kernels before this one
        fa_load_q<PAIR>(sm + kFaQ, &tm_q, first, bar_q);
        fa_load(sm + kFaK, &tm_k, first.kv_col, first.kv_row, bar_k);
        fa_load(sm + kFaV, &tm_v, first.kv_col, first.kv_row, bar_v);
    }
    if (warp == 0) { __syncwarp(); tmem_alloc(tmem_slot, kFaCols); }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    pdl_wait();
    const uint32_t tmem_base = *tmem_slot;

    if (warp == 0) {
        if (elect_one()) {
            constexpr uint32_t idesc_s = umma_idesc_bf16(128, 128), idesc_o = umma_idesc_bf16(128, 128) | umma_idesc_b_mn;
            FaTile cur = first, nt = first;
            uint32_t c = 0, asked = 0, nq = 0;               // key blocks before this tile, questions answered, Q tiles before this one
            int next;                                        // CTA index taken over, -1: none left, -2: not known yet
            bool ok = true;
            auto ask = [&]() {
                fence_proxy_async_smem();                    // the last answer has been read
                mbar_expect_tx(bar_c, 16);
                fa_try_cancel(answer, bar_c);
            };
            // Takes the answer if it is there (or waits for it); an empty tile is passed over.
            auto resolve = [&](bool wait) {
                while (next == -2) {
                    if (!mbar_test(bar_c, asked & 1)) {
                        if (!wait) return;
                        if (!fa_wait(bar_c, asked & 1, abort_flag)) { ok = false; return; }
                    }
                    ++asked;
                    const int4 id = fa_answer(answer);
                    if (id.w == 0) { next = -1; return; }
                    nt = fa_tile<HDIM, PAIR, LIST>(a, list, id.x, id.y, id.z);
                    if (nt.r0 >= nt.q_len) ask();
                    else next = (id.z * (int)gridDim.y + id.y) * (int)gridDim.x + id.x;
                }
            };
            auto load_next = [&]() {                         // Q and K are free once the last S of this tile is complete
                if (nt.n_blk == 0) return;
                fa_load_q<PAIR>(sm + kFaQ, &tm_q, nt, bar_q);
                fa_load(sm + kFaK, &tm_k, nt.kv_col, nt.kv_row, bar_k);
            };
            for (int t = 0; ok; ++t) {
                const int n_blk = cur.n_blk;
                bool loaded = false;
                next = -2;
                if (n_blk == 0) ask();
                else ok = fa_wait(bar_q, nq & 1, abort_flag);
                for (int j = 0; j < n_blk && ok; ++j) {
                    const uint32_t ph = (c + j) & 1;
                    ok = fa_wait(bar_k, ph, abort_flag);
                    if (!ok) break;
                    tc_fence_after();
                    if (j == n_blk - 1) ask();
                    // ---- S = Q K^T over the head's dims: atoms of 64 dims, 4 k-steps each
#pragma unroll
                    for (int k = 0; k < HDIM / 16; ++k)
                        umma_bf16(tmem_base, umma_desc_sw128(sm + kFaQ + (k >> 2) * 16384) + 2 * (k & 3),
                                  umma_desc_sw128(sm + kFaK + (k >> 2) * 16384) + 2 * (k & 3), idesc_s, k > 0 ? 1u : 0u);
                    umma_commit(bar_s);
                    if (j > 0 || t > 0) {
                        // the previous PV has finished reading the V buffer, or the tile before has left it: refill it (waiting
                        // for bar_e twice, after a tile without keys, passes at once)
                        ok = j > 0 ? fa_wait(bar_o, (c + j - 1) & 1, abort_flag) : fa_wait(bar_e, (t - 1) & 1, abort_flag);
                        if (!ok) break;
                        tc_fence_after();
                        fa_load(sm + kFaV, &tm_v, cur.kv_col, cur.kv_row + j * kFaBlk, bar_v);
                    }
                    ok = fa_wait(bar_s, ph, abort_flag);
                    if (!ok) break;
                    if (j + 1 < n_blk) {
                        // S is complete, so the K buffer is free: the next block's keys travel during this block's softmax
                        fa_load(sm + kFaK, &tm_k, cur.kv_col, cur.kv_row + (j + 1) * kFaBlk, bar_k);
                    } else {
                        // the same for the next tile, if it is known before the softmax is through
                        for (uint32_t spins = 0; next == -2 && spins < kFaSpin && !mbar_test(bar_p, ph); ++spins) resolve(false);
                        if (next >= 0) { load_next(); loaded = true; }
                    }
                    ok = fa_wait(bar_p, ph, abort_flag) && fa_wait(bar_v, ph, abort_flag);
                    if (!ok) break;
                    tc_fence_after();
                    // ---- O += P V: P from tensor memory (8 columns per 16 keys, a half of the keys over its own scores), V rows 16 at a time
                    {
                        const uint64_t dv = umma_desc_sw128_mn(sm + kFaV, 16384);      // both 64-dim atoms of the V tile: N = 128
#pragma unroll
                        for (int ks = 0; ks < 8; ++ks)
                            umma_bf16_tmem_a(tmem_base + kFaOCol, tmem_base + (ks < 4 ? 8 * ks : 64 + 8 * (ks - 4)), dv + (uint64_t)ks * (2048 >> 4), idesc_o,
                                             (j > 0 || ks > 0) ? 1u : 0u);
                    }
                    umma_commit(bar_o);
                }
                if (!ok) break;
                resolve(true);
                if (!ok) break;
                if (next >= 0 && !loaded) load_next();
                // a tile without keys passes through no MMA: bar_e would get a phase ahead of this thread
                if (next >= 0 && nt.n_blk == 0 && !fa_wait(bar_e, t & 1, abort_flag)) break;
                // slot (t + 1) % 2 was read before tile t - 1 ended, which bar_e has shown
                next_tile[(t + 1) & 1] = next;
                fa_arrive(bar_t + ((t + 1) & 1));
                if (next < 0) break;
                c += n_blk;
                nq += n_blk > 0 ? 1 : 0;
                cur = nt;
            }
        }
    } else {
      int index = ((int)blockIdx.z * (int)gridDim.y + (int)blockIdx.y) * (int)gridDim.x + (int)blockIdx.x;
      uint32_t c = 0;                                        // key blocks before this tile
      for (int t = 0;; ++t) {
        const int q4 = warp & 3, half = (warp - 1) >> 2, r = q4 * 32 + lane;   // TMEM lane quarter; keys 64 half .. + 63 of a block; query row inside the tile
        const FaTile tile = fa_tile<HDIM, PAIR, LIST>(a, list, index);
        const int n_blk = tile.n_blk, kv_len = tile.kv_len;
        const uint32_t t_row = tmem_base + ((uint32_t)(q4 * 32) << 16), t_half = t_row + 64 * half;
        const int row_limit = a.causal ? min(kv_len - 1, tile.r0 + (PAIR ? r & 63 : r) + kv_len - tile.q_len) : kv_len - 1;   // last key this row sees
        float* xrow = reinterpret_cast<float*>(sm + kFaX) + r;       // [2 halves], 128 floats apart
        float ref = 0.f;                                     // P = 2^(s * scale - ref); between blocks the same for both threads of a row
        float2 l2 = make_float2(0.f, 0.f);                   // this half's sum of P, even / odd keys
        bool ok = true;
        for (int j = 0; j < n_blk; ++j) {
            const uint32_t ph = (c + j) & 1;
            ok = fa_wait_warp(bar_s, ph, abort_flag);
            tc_fence_after();
            if (j == 0) {
                // the first block's exact maximum: where a few keys dominate a row, their P is then close to 1 and nearly free of rounding
                float m = -INFINITY;
                if (ok) {
                    const int lim = row_limit - 64 * half;
                    m = __all_sync(0xffffffffu, lim >= 63) ? fa_half_max<true>(t_half, lim) : fa_half_max<false>(t_half, lim);
                    xrow[128 * half] = m;
                }
                if (fa_vote(q4, !ok)) { ok = false; break; }
                m = fmaxf(m, xrow[128 * (half ^ 1)]);
                ref = m == -INFINITY ? 0.f : m * a.scale_log2;
            }
            const float ref0 = ref;
            if (ok) {
                const int lim = row_limit - j * kFaBlk - 64 * half;  // columns 0..lim of this half are visible to this row
                const bool full = __all_sync(0xffffffffu, lim >= 63);
                auto emit_p = [&](uint32_t (&v)[16], uint32_t (&flight)[16], int c0) {      // flight: the next sixteen scores, requested (c0 < 48)
                    uint32_t w[8];
                    if (!full && !__any_sync(0xffffffffu, c0 <= lim)) {      // no row of the warp sees these keys
#pragma unroll
                        for (int i = 0; i < 8; ++i) w[i] = 0u;
                        tmem_st_32x8(t_half + (uint32_t)(c0 >> 1), w);
                        return;
                    }
                    float2 p[8], cs;
                    auto exps = [&]() {
                        const float2 nr = make_float2(-ref, -ref), sc2 = make_float2(a.scale_log2, a.scale_log2);
#pragma unroll
                        for (int i = 0; i < 8; ++i) {
                            const float2 t = __ffma2_rn(make_float2(__uint_as_float(v[2 * i]), __uint_as_float(v[2 * i + 1])), sc2, nr);
                            p[i] = make_float2(fa_ex2(t.x), fa_ex2(t.y));
                        }
                        if (!full) {
#pragma unroll
                            for (int i = 0; i < 8; ++i) { if (c0 + 2 * i > lim) p[i].x = 0.f; if (c0 + 2 * i + 1 > lim) p[i].y = 0.f; }
                        }
                        cs = __fadd2_rn(__fadd2_rn(__fadd2_rn(p[0], p[1]), __fadd2_rn(p[2], p[3])), __fadd2_rn(__fadd2_rn(p[4], p[5]), __fadd2_rn(p[6], p[7])));
                    };
                    auto store_p = [&]() {
#pragma unroll
                        for (int i = 0; i < 8; ++i) w[i] = pack_bf16x2(p[i].x, p[i].y);
                        tmem_st_32x8(t_half + (uint32_t)(c0 >> 1), w);
                    };
                    exps();
                    store_p();
                    // The reference lags behind the maximum: sums and P are floating point, so little is lost by it.  Where it
                    // falls far behind, this thread's reference is raised to the chunk's maximum, what it has written of this
                    // block is rescaled, and the chunk written again; the other half and O follow after the block.
                    const bool raise = cs.x + cs.y > kFaRaise;
                    if (__any_sync(0xffffffffu, raise)) {
                        // a call follows, around which registers may be moved: none of them may still be waiting for tensor memory
                        if (c0 < 48) tmem_ld_wait16(flight);
                        float m = -INFINITY;
#pragma unroll
                        for (int i = 0; i < 16; ++i) if (c0 + i <= lim) m = fmaxf(m, __uint_as_float(v[i]));
                        const float nref = raise ? fmaxf(m * a.scale_log2, ref) : ref, f = fa_ex2(ref - nref);
                        l2.x *= f; l2.y *= f;
                        fa_rescale_p(t_half, c0, f);
                        ref = nref;
                        exps();
                        store_p();
                    }
                    l2 = __fadd2_rn(l2, cs);
                };
                // sixteen scores at a time, the next sixteen on their way
                uint32_t va[16], vb[16];
                tmem_ld_32x16(t_half, va);
#pragma unroll
                for (int c0 = 0; c0 < 64; c0 += 32) {
                    tmem_ld_wait16(va);
                    tmem_ld_32x16(t_half + (uint32_t)(c0 + 16), vb);
                    emit_p(va, vb, c0);
                    tmem_ld_wait16(vb);
                    if (c0 == 0) tmem_ld_32x16(t_half + 32, va);
                    emit_p(vb, va, c0 + 16);
                }
                tmem_st_wait();
            }
            if (j == n_blk - 1 && (kv_len & (kFaBlk - 1)) != 0 && kv_len < (j + 1) * kFaBlk) {
                // rows of the V tile past the sequence belong to a neighbour (or are unwritten cache): zero them, so that
                // 0 * V stays 0 whatever they hold
                if (ok) ok = fa_wait_warp(bar_v, ph, abort_flag);
                const int first = kv_len - j * kFaBlk;       // first row to clear
                if (ok) {
                    for (int i = threadIdx.x - 32; i < (kFaBlk - first) * 16; i += 256) {
                        const int row = first + (i >> 4), piece = i & 15;
                        *reinterpret_cast<uint4*>(sm + kFaV + (piece >> 3) * 16384 + row * 128 + (piece & 7) * 16) = make_uint4(0, 0, 0, 0);
                    }
                    fence_proxy_async_smem();
                }
            }
            // Both warps of a quarter leave together, so that no meeting waits for a warp that has gone: a wait that ran out is part of
            // the vote.  A raised reference is too: it has to be the same for both halves and O before P is used.
            if (fa_vote(q4, !ok || __any_sync(0xffffffffu, ref != ref0))) {
                xrow[128 * half] = ref;
                if (fa_vote(q4, !ok)) { ok = false; break; }
                const float m = fmaxf(ref, xrow[128 * (half ^ 1)]), f = fa_ex2(ref - m);
                l2.x *= f; l2.y *= f;
                fa_rescale_p(t_half, 64, f);
                ref = m;
                if (j > 0) {
                    ok = fa_wait_warp(bar_o, (c + j - 1) & 1, abort_flag);        // O must be complete before it is rewritten
                    tc_fence_after();
                    const float fo = fa_ex2(ref0 - m);
                    for (int c0 = 16 * half; ok && c0 < HDIM; c0 += 32) {
                        uint32_t v[16];
                        tmem_ld_32x16(t_row + kFaOCol + c0, v);
                        tmem_ld_wait16(v);
#pragma unroll
                        for (int i = 0; i < 16; i += 8) {
                            uint32_t w[8];
#pragma unroll
                            for (int k = 0; k < 8; ++k) w[k] = __float_as_uint(__uint_as_float(v[i + k]) * fo);
                            tmem_st_32x8(t_row + kFaOCol + c0 + i, w);
                        }
                    }
                    tmem_st_wait();
                }
                if (fa_vote(q4, !ok)) { ok = false; break; }
            }
            // one arrival per warp: 32 lanes arriving on one barrier word are 32 shared-memory atomics one after the other
            tc_fence_before();
            __syncwarp();
            if (lane == 0) fa_arrive(bar_p);
        }
        if (!ok) break;
        if (n_blk > 0) {
        // ---- epilogue: O / rowsum -> bf16 -> staging tile (the V tile is dead) -> whole rows; the warps of a quarter take every
        //      other 16 columns, then 16 rows each
        ok = fa_wait_warp(bar_o, (c + n_blk - 1) & 1, abort_flag);
        tc_fence_after();
        xrow[128 * half] = l2.x + l2.y;
        if (fa_vote(q4, !ok)) break;
        const float l = xrow[0] + xrow[128];
        const float inv = l > 0.f ? 1.0f / l : 0.f;
        unsigned char* stage = sm + kFaV;
#pragma unroll 1
        for (int c0 = 16 * half; c0 < HDIM; c0 += 32) {
            uint32_t v[16];
            tmem_ld_32x16(t_row + kFaOCol + c0, v);
            tmem_ld_wait16(v);
#pragma unroll
            for (int jj = 0; jj < 2; ++jj)
                *reinterpret_cast<uint4*>(stage + r * 256 + ((((c0 >> 3) + jj) ^ (r & 15)) << 4)) =
                    make_uint4(pack_bf16x2(__uint_as_float(v[8 * jj]) * inv, __uint_as_float(v[8 * jj + 1]) * inv),
                               pack_bf16x2(__uint_as_float(v[8 * jj + 2]) * inv, __uint_as_float(v[8 * jj + 3]) * inv),
                               pack_bf16x2(__uint_as_float(v[8 * jj + 4]) * inv, __uint_as_float(v[8 * jj + 5]) * inv),
                               pack_bf16x2(__uint_as_float(v[8 * jj + 6]) * inv, __uint_as_float(v[8 * jj + 7]) * inv));
        }
        fa_vote(q4, false);
        const int sub = lane & 15;
        const FaTile out = fa_tile<HDIM, PAIR, LIST>(a, list, index);          // once more: kept across the key loop it would cost registers there
#pragma unroll 4
        for (int it = 0; it < 8; ++it) {
            const int rr = q4 * 32 + half * 16 + it * 2 + (lane >> 4), tr = PAIR ? rr & 63 : rr, row = out.r0 + tr, head = out.head + (PAIR ? rr >> 6 : 0);
            const uint4 val = *reinterpret_cast<const uint4*>(stage + rr * 256 + ((sub ^ (rr & 15)) << 4));
            if (row < out.q_len && sub < HDIM / 8) *reinterpret_cast<uint4*>(a.o + (long long)(out.q_row + tr) * a.o_row + (long long)head * a.o_head + 8 * sub) = val;
        }
        } else fa_zero_rows<HDIM, PAIR>(a, tile, threadIdx.x - 32, 256);
        fence_proxy_async_smem();                            // the next V block is written through the async proxy
        tc_fence_before();
        __syncwarp();
        if (lane == 0) fa_arrive(bar_e);
        c += n_blk;
        if (fa_vote(q4, !fa_wait_warp(bar_t + ((t + 1) & 1), (t >> 1) & 1, abort_flag))) break;
        index = next_tile[(t + 1) & 1];
        if (index < 0) break;
      }
    }
    tc_fence_before();
    __syncthreads();
    if (*abort_flag) {
        if (threadIdx.x == 0) {
            if (atomicCAS(&a.status[0], 0u, (uint32_t)ITTAI_ST_GEMM_TIMEOUT) == 0u) { a.status[1] = blockIdx.x; a.status[2] = blockIdx.y; }
            const long long t0 = clock64();
            while (clock64() - t0 < 2000000) {}
        }
        __syncthreads();
    }
    if (warp == 0) { __syncwarp(); tmem_dealloc(tmem_base, kFaCols); }
}

int cuda_fail(cudaError_t e, const char* what);

// Whether the key-loop kernel covers this call: head_dim 128, heads adjacent in the q rows, keys and values as dense rows
// of 128 elements (the cache layout), identical strides for k and v, more than 64 query rows in some sequence.
// Keys and values either in the cache layout (rows of 128 elements; heads and sequences whole numbers of rows apart) or
// packed like the queries (the heads of a token side by side in one row, sequences told apart by their row offsets).
static bool fa_packed_kv(const IttaiAttention* p) { return p->k_seq == 0 && p->v_seq == 0 && p->k_head == p->head_dim && p->v_head == p->head_dim && p->k_row == p->v_row && p->k_row > 128; }
bool attn_fa_supported(const IttaiAttention* p) {
    const bool cache = p->head_dim == 128 && p->k_row == 128 && p->v_row == 128 && p->k_head % 128 == 0 && p->k_seq % 128 == 0;
    return (p->head_dim == 128 || p->head_dim == 80) && p->status != nullptr && p->max_q_len > 64 && p->q_head == p->head_dim && (cache || fa_packed_kv(p)) &&
           p->v_head == p->k_head && p->v_seq == p->k_seq && p->q_rows_total > 0 &&
           p->kv_rows_total > 0 && ((uintptr_t)p->q & 15) == 0 && ((uintptr_t)p->k & 15) == 0 && ((uintptr_t)p->v & 15) == 0 &&
           ((uintptr_t)p->o & 15) == 0 && p->o_row % 8 == 0 && p->o_head % 8 == 0;
}

static int fa_steps(const IttaiAttention* p) { return (p->max_q_len + kFaBlk - 1) / kFaBlk; }
static int fa_list_bound(const IttaiAttention* p) { return p->q_rows_total / kFaBlk + p->n_seqs; }
// A list of the non-empty tiles where the grid of all of them would be longer (sequences of different lengths): empty CTAs and answers that
// name an empty tile cost more than the list.  55 texts of 16 to 512 tokens, us a layer: tiles of one head 51, of head pairs 47, from a list 39;
// 200 texts of 16 to 80 56, 37 and 39 (one step each: no list).  Its length has a bound on the host only if the sequences' rows are
// disjoint, which the prefill vouches for.
static bool fa_list_pays(const IttaiAttention* p) {
    return p->seqs_ready && p->n_seqs <= kFaListSeqs && fa_steps(p) <= kFaListSteps && (long long)fa_steps(p) * p->n_seqs > fa_list_bound(p);
}
template <int HDIM, bool PAIR, bool LIST>
static int attn_fa_launch_t(const IttaiAttention* p, cudaStream_t st) {
    CUtensorMap tq, tk, tv;
    int rc = make_tmap_bf16(&tq, p->q, p->q_rows_total, (long long)p->n_heads * HDIM, p->q_row, PAIR ? 64 : 128);
    const bool packed = fa_packed_kv(p);
    const long long kv_cols = packed ? (long long)(p->n_heads / p->group) * HDIM : 128, kv_ld = packed ? p->k_row : 128;
    if (rc == ITTAI_OK) rc = make_tmap_bf16(&tk, p->k, p->kv_rows_total, kv_cols, kv_ld, 128);
    if (rc == ITTAI_OK) rc = make_tmap_bf16(&tv, p->v, p->kv_rows_total, kv_cols, kv_ld, 128);
    if (rc != ITTAI_OK) return rc;
    static thread_local int attr_dev = -1;
    int dev = 0;
    cudaGetDevice(&dev);
    if (attr_dev != dev) {
        const cudaError_t e = cudaFuncSetAttribute(attn_fa_kernel<HDIM, PAIR, LIST>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(LIST ? kFaSmemList : kFaSmem));
        if (e != cudaSuccess) return cuda_fail(e, "cudaFuncSetAttribute(attn_fa_kernel)");
        attr_dev = dev;
    }
    AttnFaArgs a;
    a.seqs = reinterpret_cast<const int4*>(p->seqs);
    a.o = reinterpret_cast<bf16*>(p->o);
    a.o_row = p->o_row; a.o_head = p->o_head;
    a.group = p->group; a.causal = p->causal; a.seqs_ready = p->seqs_ready;
    a.k_seq_rows = packed ? 0 : (int)(p->k_seq / 128); a.k_head_rows = packed ? 0 : (int)(p->k_head / 128);
    a.k_head_cols = packed ? HDIM : 0;
    a.scale_log2 = 1.4426950408889634f / sqrtf((float)HDIM);
    a.status = p->status;
    a.n_seqs = p->n_seqs; a.n_steps = fa_steps(p);
    // a list's grid is the bound on its length
    const dim3 grid = LIST ? dim3(p->n_heads, fa_list_bound(p), 1) : dim3(p->n_heads, p->n_seqs, fa_steps(p));
    const cudaError_t e = launch_pdl(attn_fa_kernel<HDIM, PAIR, LIST>, grid, dim3(kFaThreads), LIST ? kFaSmemList : kFaSmem, st, 1, tq, tk, tv, a);
    return e == cudaSuccess ? ITTAI_OK : cuda_fail(e, "launch attn_fa_kernel");
}

// `disjoint`: no two sequences share a query row.
int attn_fa_launch(const IttaiAttention* p, bool disjoint, cudaStream_t st) {
    if (p->head_dim == 80) return attn_fa_launch_t<80, false, false>(p, st);
    if (p->group != 2 || p->n_heads % 2 != 0) return attn_fa_launch_t<128, false, false>(p, st);
    return disjoint && fa_list_pays(p) ? attn_fa_launch_t<128, true, true>(p, st) : attn_fa_launch_t<128, true, false>(p, st);
}

}  // namespace ittai
