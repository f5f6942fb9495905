// Attention column mean for B200 (sm_100a): kernels and their C ABI.
//
// out[b, k] = 1/(H * R) * sum_h sum_{q < R} softmax_k(scale * Q[b,h,q,:] . K[b,h,k,:])
//
// Two streaming kernels share one warp-specialised skeleton (TMA -> shared
// memory -> tcgen05 MMA -> tensor memory -> consumer warps):
//
//   statistics pass  S  = Q K^T : tensor-memory lane = query row, so the running
//                    row maximum and sum of exp2 stay inside one thread.  It
//                    writes -(log2-sum-exp + log2(H*R)) per query row.
//   column pass      S^T = K Q^T: tensor-memory lane = key, so the reduction
//                    down the query axis stays inside one thread as well.  It
//                    adds exp2(c*s - lse) into a per-key fp32 accumulator and
//                    flushes that with one atomic add per (key tile, CTA range).
//                    -lse/c reaches the accumulator through 16 extra contraction
//                    columns (MODE_COLSUM_EXT); for tiny scales it is staged
//                    through shared memory instead (MODE_COLSUM).  A query axis of
//                    one or two 256-row blocks over sixteen or more key tiles swaps
//                    the roles (MODE_COLSUM_EXT_SHORT / _SHORT2): the head's query
//                    blocks stay in shared memory, the key tiles stream through a
//                    deep ring, and with at most 128 queries two key tiles share
//                    one accumulator buffer.
//
// Both operands are row tiles with the head dimension contiguous, so the same
// shared-memory layout serves as A (128 resident rows) or B (256 streamed rows)
// of the MMA; one step is a 128 x 256 x D MMA into one of two accumulator
// buffers of 256 tensor-memory columns.  Calls with at most four query rows
// take the matrix-vector kernel of colsum_small_q.cuh instead; short non-causal
// key axes at head dimension 64 take the single-pass cluster kernel of
// colsum_single_pass.cuh; a query axis of at most 128 rows over a few thousand keys
// takes the one-kernel cluster form of colsum_fused_short.cuh; select_topk.cuh holds
// the pruning step that callers run on the result.
#include "sm100_ptx.cuh"
#include "schedule.h"
#include "colsum_small_q.cuh"
#include "colsum_few_rows.cuh"
#include "colsum_math.cuh"
#include "round_fp32.cuh"

#include <math.h>
#include <stdarg.h>
#include <stdio.h>
#include <string.h>

#include <mutex>
#include <vector>

#include "../../include/flash_colsum_b200.h"
#include "host_api.h"

#include "colsum_single_pass.cuh"
#include "select_topk.cuh"

namespace fcs {

constexpr int NUM_TBUF = 2;        // accumulator buffers of 256 tensor-memory columns
constexpr int TMEM_COLS = 512;
constexpr int NUM_LSE = 4;         // per-query-block log-sum-exp vectors in flight (column pass)
// Consumer warps come in groups of four (a group covers the 128 tensor-memory
// lanes); every group takes an equal run of the columns of each accumulator.
constexpr int CONSUMER_GROUPS = 4;
constexpr int GROUP_COLS = BLOCK / CONSUMER_GROUPS;
constexpr int CONSUMER_WARPS = 4 * CONSUMER_GROUPS;
constexpr int CONSUMER_THREADS = 32 * CONSUMER_WARPS;
constexpr int PRODUCER_WARP = CONSUMER_WARPS;
constexpr int MMA_WARP = CONSUMER_WARPS + 1;
constexpr int THREADS = 32 * (CONSUMER_WARPS + 2);
static_assert(GROUP_COLS == 64, "a group consumes one 64-column block per step");

// Item-end partials of the statistics pass wait in one of these slots until a group
// combines them; consumer groups are never more than two steps apart, so four
// slots cannot be overrun.
constexpr int MERGE_SLOTS = 4;
constexpr int EXT_K = 16;                        // extra contraction columns that carry -(lse)/c
constexpr int EXT_ROW_BYTES = EXT_K * 2;
constexpr int EXT_A_BYTES = TILE * EXT_ROW_BYTES;    // the constant key-side columns
constexpr int EXT_B_BYTES = BLOCK * EXT_ROW_BYTES;   // the query-side columns of one block

template <int D, int MODE>
struct Layout {
    static constexpr bool COMBINE = (MODE == MODE_COLSUM_EXT_SHORT_COMBINE) || (MODE == MODE_COLSUM_EXT_SHORT2_COMBINE);
    static constexpr bool SHORT2 = (MODE == MODE_COLSUM_EXT_SHORT2) || (MODE == MODE_COLSUM_EXT_SHORT2_COMBINE);
    static constexpr bool SHORT = (MODE == MODE_COLSUM_EXT_SHORT) || (MODE == MODE_COLSUM_EXT_SHORT_COMBINE) || SHORT2;
    static constexpr int NB = SHORT2 ? 2 : 1;   // (short modes) resident query blocks
    static constexpr bool EXT = (MODE == MODE_COLSUM_EXT) || SHORT;
    static constexpr int SLABS = D / 64;              // 64-element (128-byte) column slabs
    static constexpr int A_SLAB_BYTES = TILE * 128;
    static constexpr int B_SLAB_BYTES = BLOCK * 128;
    static constexpr int A_BYTES = SLABS * A_SLAB_BYTES;
    static constexpr int B_BYTES = SLABS * B_SLAB_BYTES;
    static constexpr int B_STAGE_BYTES = B_BYTES + (EXT ? EXT_B_BYTES : 0);   // block, then its extension
    static constexpr int NS = SHORT ? NB : (D == 64) ? 4 : 2;     // streamed-operand stages
    // resident-operand buffers: two; in the short modes they are what streams -- 128 KiB of them,
    // or what two 128-wide query blocks leave
    static constexpr int NA = !SHORT ? 2 : (NB == 2 && D == 128) ? 2 : 256 / SLABS / 32;
    static constexpr int A_OFF = 0;
    static constexpr int B_OFF = NA * A_BYTES;
    static constexpr int EXTA_OFF = B_OFF + NS * B_STAGE_BYTES;             // 128 rows of the constant
    static constexpr int LSE_OFF = EXTA_OFF + (EXT ? EXT_A_BYTES : 0);      // NUM_LSE slots of 256 floats
    static constexpr int BAR_OFF = LSE_OFF + (MODE == MODE_COLSUM ? NUM_LSE * BLOCK * 4 : 0);
    // barriers: a_full[NA] a_empty[NA] b_full[NS] b_empty[NS] t_full[2] t_empty[2] merge[MERGE_SLOTS]
    //           l_full[NUM_LSE] l_empty[NUM_LSE]
    static constexpr int NUM_BARS = 2 * NA + 2 * NS + 2 * NUM_TBUF + MERGE_SLOTS + 2 * NUM_LSE;
    static constexpr int MISC_OFF = BAR_OFF + NUM_BARS * 8;        // tmem address, abort flag
    static constexpr int META_OFF = (MISC_OFF + 16 + 15) / 16 * 16;   // int4[MERGE_SLOTS]: (b, h, query tile, key range) of an item
    static constexpr int MERGE_OFF = META_OFF + (MODE == MODE_STATS ? MERGE_SLOTS * 16 : 0);  // float2[MERGE_SLOTS][groups][128]
    // (short column modes: float[MERGE_SLOTS][groups][128], the groups' sums of an item before the one add)
    static constexpr int PROB_OFF = MERGE_OFF + (MODE == MODE_STATS ? MERGE_SLOTS * CONSUMER_GROUPS * TILE * 8
                                                                    : COMBINE ? MERGE_SLOTS * CONSUMER_GROUPS * TILE * 4 : 0);
    // a copy of the call's parameters: what is read once per item (the item iterators) is read from
    // here -- in the constant bank those words are cold by the next item, a miss each
    static constexpr int TOTAL = PROB_OFF + (int)((sizeof(Problem) + 15) / 16 * 16);
    static constexpr int DYN_BYTES = TOTAL + 1024;    // slack to align the base to 1024
    static_assert(DYN_BYTES <= 227 * 1024, "shared memory budget");
};

// A group's 64 columns of one accumulator, all of them visible: `taddr` and `nl` are relative to its first column.
__device__ __forceinline__ void stats_tile_full(uint32_t taddr, float c, float& m, float& l) {
    uint32_t r[32];
    tmem_ld_x32(taddr, r);
    tmem_ld_wait(r);
    stats_block32<BLOCK_FULL>(r, 32, c, m, l);
    tmem_ld_x32(taddr + 32, r);
    tmem_ld_wait(r);
    stats_block32<BLOCK_FULL>(r, 32, c, m, l);
}
__device__ __forceinline__ void colsum_tile_ext_full(uint32_t taddr, float c, float (&acc)[4]) {
    // 16 columns at a time, the next 16 in flight from tensor memory while these are in the exp pipes
    uint32_t ra[16], rb[16];
    tmem_ld_16cols(taddr, ra);
    tmem_wait_16cols(ra);
    tmem_ld_16cols(taddr + 16, rb);
    colsum_chunk16_ext<0>(ra, c, acc);
    tmem_wait_16cols(rb);
    tmem_ld_16cols(taddr + 32, ra);
    colsum_chunk16_ext<8>(rb, c, acc);
    tmem_wait_16cols(ra);
    tmem_ld_16cols(taddr + 48, rb);
    colsum_chunk16_ext<0>(ra, c, acc);
    tmem_wait_16cols(rb);
    colsum_chunk16_ext<8>(rb, c, acc);
}
// The same where some elements are hidden, in runs of 32 columns: what no row of the warp sees is not read, only the runs
// that the diagonal or the ragged end goes through are masked, and the four groups share what is visible.  (Before, a
// group masked its fixed quarter as a whole.)  Its exps are all the special-function unit's, in a run that all rows see
// too: the polynomial is for whole tiles and whole quarters of one.
//
// Statistics: columns 0 .. lim of this row are visible; lim_first / lim_last: the same of the warp's first and
// last row (the least and the most any of its rows sees).
__device__ __forceinline__ void stats_tile(uint32_t taddr, int cols, int lim, int lim_first, int lim_last, float c, float& m,
                                           float& l) {
    if (lim_last < cols - 1) cols = lim_last + 1;
#pragma unroll 1
    for (int j = 0; j < cols; j += 32) {
        uint32_t r[32];
        tmem_ld_x32(taddr + j, r);
        tmem_ld_wait(r);
        if (lim_first >= j + 31) stats_block32<BLOCK_EXACT>(r, 32, c, m, l);
        else stats_block32<BLOCK_MASKED>(r, lim - j, c, m, l);
    }
}
// Columns thr <= j < end of this row are visible; thr_first / thr_last: thr of the warp's first and last row.
__device__ __forceinline__ void colsum_tile_ext(uint32_t taddr, int cols, int thr, int thr_first, int thr_last, int end, float c,
                                                float (&acc)[4]) {
    if (end < cols) cols = end;
#pragma unroll 1
    for (int j = thr_first > 0 ? thr_first & ~31 : 0; j < cols; j += 32) {
        uint32_t r[32];
        tmem_ld_x32(taddr + j, r);
        tmem_ld_wait(r);
        if (thr_last <= j && j + 32 <= end) colsum_chunk_ext<BLOCK_EXACT>(r, 0, 32, c, acc);
        else colsum_chunk_ext<BLOCK_MASKED>(r, thr - j, end - j, c, acc);
    }
}
template <bool MASKED>
__device__ __forceinline__ void colsum_tile(uint32_t taddr, const float4* nl, int thr, int end, float c,
                                            float (&acc)[4]) {
    uint32_t r[32];
#pragma unroll
    for (int ch = 0; ch < GROUP_COLS / 32; ++ch) {
        tmem_ld_x32(taddr + 32 * ch, r);
        tmem_ld_wait(r);
        colsum_chunk<MASKED>(r, nl + 8 * ch, thr - 32 * ch, end - 32 * ch, c, acc);
    }
}

// The key-side constant of the extension: every 16-byte piece is (k, k, k, 0, 0, 0, 0, 0), which reads
// the same under any swizzle of the pieces.
__device__ __forceinline__ void fill_ext_constant(uint8_t* dst, bool bf16) {
    const uint32_t k16 = bf16 ? 0x3F80u : 0x5C00u;   // bf16 1.0 / fp16 256.0
    uint4* ones = reinterpret_cast<uint4*>(dst);
    for (int i = threadIdx.x; i < EXT_A_BYTES / 16; i += THREADS) ones[i] = make_uint4(k16 | (k16 << 16), k16, 0u, 0u);
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// Release stores at system scope, kept out of line: with a system-scope fence or release store
// in its own body the streaming kernel's adds into another GPU's memory run markedly slower
// (measured on the long-context shape: 0.363 against 0.289 ms for the column pass of a rank that
// adds over NVLink, whether or not the store is ever executed).
__device__ __noinline__ void release_store_system(int* const* flags, int n, int value) {
    __threadfence_system();
    for (int i = 0; i < n; ++i)
        asm volatile("st.release.sys.global.s32 [%0], %1;" ::"l"(flags[i]), "r"(value) : "memory");
}
__device__ __noinline__ void release_store_system_one(int* flag, int value) {
    __threadfence_system();
    asm volatile("st.release.sys.global.s32 [%0], %1;" ::"l"(flag), "r"(value) : "memory");
}

// ---------------------------------------------------------------------------
// The streaming kernel.  tm_a: resident operand (box of 128 rows), tm_b:
// streamed operand (box of 256 rows), tm_ext: the 16 extension columns of the
// query blocks (MODE_COLSUM_EXT only).
// ---------------------------------------------------------------------------
template <int D, int MODE>
__global__ void __launch_bounds__(THREADS, 1)
colsum_stream_kernel(const __grid_constant__ CUtensorMap tm_a, const __grid_constant__ CUtensorMap tm_b,
                     const __grid_constant__ CUtensorMap tm_ext, const Problem p) {
    using L = Layout<D, MODE>;
    constexpr bool EXT = L::EXT;
    constexpr int NA = L::NA;
    using Items = typename ItemsOf<MODE>::type;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                               ~static_cast<uintptr_t>(1023));
    const uint32_t smem_base = smem_u32(smem);
    const uint32_t a_smem = smem_base + L::A_OFF;
    const uint32_t b_smem = smem_base + L::B_OFF;
    const uint32_t lse_smem = smem_base + L::LSE_OFF;
    const uint32_t bars = smem_base + L::BAR_OFF;
    auto a_full = [&](int i) { return bars + 8u * i; };
    auto a_empty = [&](int i) { return bars + 8u * (NA + i); };
    auto b_full = [&](int i) { return bars + 8u * (2 * NA + i); };
    auto b_empty = [&](int i) { return bars + 8u * (2 * NA + L::NS + i); };
    auto t_full = [&](int i) { return bars + 8u * (2 * NA + 2 * L::NS + i); };
    auto t_empty = [&](int i) { return bars + 8u * (2 * NA + 2 * L::NS + NUM_TBUF + i); };
    auto merge_bar = [&](int i) { return bars + 8u * (2 * NA + 2 * L::NS + 2 * NUM_TBUF + i); };
    auto l_full = [&](int i) { return bars + 8u * (2 * NA + MERGE_SLOTS + 2 * L::NS + 2 * NUM_TBUF + i); };
    auto l_empty = [&](int i) { return bars + 8u * (2 * NA + MERGE_SLOTS + 2 * L::NS + 2 * NUM_TBUF + NUM_LSE + i); };
    volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(smem + L::MISC_OFF);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + L::MISC_OFF + 4);
    float2* merge_buf = reinterpret_cast<float2*>(smem + L::MERGE_OFF);
    // The item iterators take the parameters by reference; taken from the kernel's parameter block
    // that is a copy in local memory, whose lines are cold -- a miss each, 450 cycles per item in all --
    // by the time the next item is decoded.  They read this copy in shared memory instead.  (The mask
    // rules, evaluated every step, keep the local copy: its lines stay in L1, and the long-context
    // column pass was 2 % slower with them on the shared copy.)
    Problem& ps = *reinterpret_cast<Problem*>(smem + L::PROB_OFF);

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;

    if (threadIdx.x == 32) ps = p;
    if (threadIdx.x == 0) {
        for (int i = 0; i < NA; ++i) { mbar_init(a_full(i), 1); mbar_init(a_empty(i), 1); }
        for (int i = 0; i < L::NS; ++i) { mbar_init(b_full(i), 1); mbar_init(b_empty(i), 1); }
        for (int i = 0; i < NUM_TBUF; ++i) { mbar_init(t_full(i), 1); mbar_init(t_empty(i), CONSUMER_THREADS); }
        for (int i = 0; i < MERGE_SLOTS; ++i) mbar_init(merge_bar(i), CONSUMER_THREADS);
        for (int i = 0; i < NUM_LSE; ++i) { mbar_init(l_full(i), 1); mbar_init(l_empty(i), CONSUMER_THREADS); }
        *abort_flag = 0;
        mbar_fence_init();
    }
    if constexpr (EXT) fill_ext_constant(smem + L::EXTA_OFF, p.ext_bf16 != 0);
    if (warp == PRODUCER_WARP && lane == 0) {
        prefetch_tensormap(&tm_a);
        prefetch_tensormap(&tm_b);
        if constexpr (EXT) prefetch_tensormap(&tm_ext);
    }
    if (warp == MMA_WARP) {
        tmem_alloc(smem_u32(const_cast<uint32_t*>(tmem_slot)), TMEM_COLS);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    // everything above touched only this CTA's shared and tensor memory; from here on the
    // results of the kernels before this one in the stream are read
    grid_dependency_wait();
    grid_launch_dependents();   // (behind the wait: 200 queries over 8 x 45613 keys, 88.2 us a call with it at the top, 86.0 here)
    if (p.fmt) {
        // the element type was decided by a kernel of this call
        const int bf16 = *p.fmt;
        if constexpr (EXT) fill_ext_constant(smem + L::EXTA_OFF, bf16 != 0);
        if (threadIdx.x == 0 && bf16) { ps.ext_bf16 = 1; ps.idesc |= IDESC_BF16; }
        __syncthreads();
    }
    if (MODE != MODE_STATS && (p.sig_wait || p.sig_post_n > 0)) {
        // head shards on several GPUs adding into one buffer: nothing is added before the owner of
        // the buffer has said that it is clear (a flag in this GPU's memory, written over NVLink;
        // the wait is bounded), and the owner says so for the buffer of the next call once the
        // kernels before this one (its statistics pass cleared that buffer) have completed
        if (threadIdx.x == 0) {
            if (p.sig_wait) {
                const long long t0 = clock64();
                unsigned spins = 0;
                while (true) {
                    int v;
                    asm volatile("ld.acquire.sys.global.s32 %0, [%1];" : "=r"(v) : "l"(p.sig_wait) : "memory");
                    if (v >= p.sig_wait_value) break;
                    if ((++spins & 63u) == 0u && clock64() - t0 > g_wait_limit_cycles) {
                        if (p.status) atomicCAS(p.status, 0, FCS_STATUS_WAIT_PEER);
                        break;
                    }
                    __nanosleep(200);
                }
            }
            if (blockIdx.x == 0 && p.sig_post_n > 0) {
                // (In the generic modes the flag pointers come from the shared copy, and with that the
                // compiler keeps no copy of the parameter block in local memory at all: the headline
                // shape's column pass is 5 % faster without it.  The short-query modes measured 2.5 %
                // slower without that copy, so there its address is still taken.)
                if constexpr (L::SHORT) release_store_system(p.sig_post, p.sig_post_n, p.sig_post_value);
                else release_store_system(ps.sig_post, p.sig_post_n, p.sig_post_value);
            }
        }
        __syncthreads();
    }

    // The producer and MMA warps run their loops with all 32 lanes converged (so
    // that addresses, descriptors and counters stay in uniform registers) and
    // elect one lane only around the instructions that must be issued once.
    auto wait_all = [&](uint32_t bar, uint32_t parity, int code) -> bool {
        const bool ok = mbar_wait(bar, parity, abort_flag, p.status, code);
        return __all_sync(0xffffffffu, ok);
    };

    if (warp >= CONSUMER_WARPS) {
        if (warp == PRODUCER_WARP) {
            // -------------------------------------------- TMA producer
            Items it;
            it.init(ps, blockIdx.x, gridDim.x);
            int a_cnt = 0, stage = 0, n = 0;
            uint32_t phase = 0;
            bool ok = p.withhold_loads == 0;   // (self-test: nothing is loaded, every wait for data runs out)
            // which streamed block every stage holds: when a (batch, head) has no more blocks
            // than there are stages (short query axes in the column pass, short key axes in the
            // statistics pass), the next item finds its blocks still in shared memory and the
            // stage is handed to the MMA warp again without a copy
            long long held[L::NS];
#pragma unroll
            for (int i = 0; i < L::NS; ++i) held[i] = -1;
            if constexpr (L::SHORT) {
                // Short query axis: an item is one or two key tiles against the head's only query
                // block.  The key tiles run ahead as far as their ring is deep; the query block
                // is loaded when the head changes.
                int cur_bh = -1, b_cnt = 0;
                for (; ok && !it.done; it.next(ps)) {
                    for (int t = 0; t < it.nt; ++t, ++a_cnt) {
                        const int ab = a_cnt % NA;
                        if (!wait_all(a_empty(ab), ((a_cnt / NA) & 1) ^ 1, FCS_STATUS_WAIT_PRODUCER)) { ok = false; break; }
                        if (elect_one_sync()) {
                            mbar_arrive_expect_tx(a_full(ab), L::A_BYTES);
#pragma unroll
                            for (int sl = 0; sl < L::SLABS; ++sl)
                                tma_load_4d(a_smem + ab * L::A_BYTES + sl * L::A_SLAB_BYTES, &tm_a, a_full(ab),
                                            sl * 64, it.a_row() + t * TILE, it.h, it.b);
                        }
                    }
                    if (!ok) break;
                    const int bh = it.b * p.H + it.h;
                    if (bh != cur_bh) {
                        if (!wait_all(b_empty(0), (b_cnt & 1) ^ 1, FCS_STATUS_WAIT_PRODUCER)) break;
                        if (elect_one_sync()) {
                            mbar_arrive_expect_tx(b_full(0), (uint32_t)p.NQB * L::B_STAGE_BYTES);
                            for (int qb = 0; qb < p.NQB; ++qb) {
#pragma unroll
                                for (int sl = 0; sl < L::SLABS; ++sl)
                                    tma_load_4d(b_smem + qb * L::B_STAGE_BYTES + sl * L::B_SLAB_BYTES, &tm_b, b_full(0),
                                                sl * 64, qb * BLOCK, it.h, it.b);
                                tma_load_3d(b_smem + qb * L::B_STAGE_BYTES + L::B_BYTES, &tm_ext, b_full(0), 0,
                                            qb * BLOCK, bh);
                            }
                        }
                        __syncwarp();
                        ++b_cnt;
                        cur_bh = bh;
                    }
                }
            } else {
            for (; ok && !it.done; it.next(ps), ++a_cnt) {
                const int ab = a_cnt & 1;
                if (!wait_all(a_empty(ab), ((a_cnt >> 1) & 1) ^ 1, FCS_STATUS_WAIT_PRODUCER)) break;
                if (elect_one_sync()) {
                    mbar_arrive_expect_tx(a_full(ab), L::A_BYTES);
#pragma unroll
                    for (int sl = 0; sl < L::SLABS; ++sl)
                        tma_load_4d(a_smem + ab * L::A_BYTES + sl * L::A_SLAB_BYTES, &tm_a, a_full(ab),
                                    sl * 64, it.a_row(), it.h, it.b);
                }
                const float* lse_src = nullptr;
                if constexpr (MODE == MODE_COLSUM)
                    lse_src = p.neg_lse + ((long long)it.b * p.H + it.h) * p.lse_rows;
                const int bh = it.b * p.H + it.h;
                for (int st = it.s0; st < it.s1; ++st, ++n) {
                    if (!wait_all(b_empty(stage), phase ^ 1, FCS_STATUS_WAIT_PRODUCER)) { ok = false; break; }
                    const long long block_id = ((long long)bh << 32) | (unsigned)st;
                    bool reuse = false;
#pragma unroll
                    for (int i = 0; i < L::NS; ++i)
                        if (i == stage) { reuse = held[i] == block_id; held[i] = block_id; }
                    if (reuse) {
                        if (elect_one_sync()) mbar_arrive(b_full(stage));
                    } else if (elect_one_sync()) {
                        mbar_arrive_expect_tx(b_full(stage), L::B_STAGE_BYTES);
#pragma unroll
                        for (int sl = 0; sl < L::SLABS; ++sl)
                            tma_load_4d(b_smem + stage * L::B_STAGE_BYTES + sl * L::B_SLAB_BYTES, &tm_b,
                                        b_full(stage), sl * 64, it.b_row(st), it.h, it.b);
                        if constexpr (EXT)
                            tma_load_3d(b_smem + stage * L::B_STAGE_BYTES + L::B_BYTES, &tm_ext, b_full(stage),
                                        0, it.b_row(st), bh);
                    }
                    if constexpr (MODE == MODE_COLSUM) {
                        // -(lse) of the 256 queries of this block, for the consumers
                        const int ls = n & (NUM_LSE - 1);
                        if (!wait_all(l_empty(ls), ((n / NUM_LSE) & 1) ^ 1, FCS_STATUS_WAIT_PRODUCER)) {
                            ok = false; break;
                        }
                        if (elect_one_sync()) {
                            mbar_arrive_expect_tx(l_full(ls), BLOCK * 4);
                            bulk_load(lse_smem + ls * BLOCK * 4, lse_src + (long long)st * BLOCK, BLOCK * 4,
                                      l_full(ls));
                        }
                    }
                    __syncwarp();
                    if (++stage == L::NS) { stage = 0; phase ^= 1; }
                }
            }
            }
        } else if (warp == MMA_WARP) {
            // -------------------------------------------- MMA issuer
            Items it;
            it.init(ps, blockIdx.x, gridDim.x);
            const uint32_t idesc = ps.idesc;
            int a_cnt = 0, stage = 0, n = 0;
            uint32_t phase = 0;
            bool ok = true;
            if constexpr (L::SHORT) {
                int cur_bh = -1, b_cnt = 0;
                for (; ok && !it.done; it.next(ps)) {
                    const int bh = it.b * p.H + it.h;
                    if (bh != cur_bh) {
                        // the MMAs of the head before this one have read its query block: hand
                        // the buffer back, then wait for this head's block
                        if (cur_bh >= 0 && elect_one_sync()) umma_commit(b_empty(0));
                        __syncwarp();
                        if (!wait_all(b_full(0), b_cnt & 1, FCS_STATUS_WAIT_MMA)) break;
                        ++b_cnt;
                        cur_bh = bh;
                    }
                    if constexpr (L::SHORT2) {
                        // one key tile against the head's resident query blocks, a step each
                        const int ab = a_cnt % NA;
                        if (!wait_all(a_full(ab), (a_cnt / NA) & 1, FCS_STATUS_WAIT_MMA)) break;
                        const uint64_t da = umma_desc_k_sw128(a_smem + ab * L::A_BYTES);
                        for (int st = it.s0; st < it.s1; ++st, ++n) {
                            const int buf = n & (NUM_TBUF - 1);
                            if (!wait_all(t_empty(buf), ((n >> 1) & 1) ^ 1, FCS_STATUS_WAIT_MMA)) { ok = false; break; }
                            tc_fence_after();
                            const uint64_t db = umma_desc_k_sw128(b_smem + st * L::B_STAGE_BYTES);
                            const uint32_t d_tmem = tmem_base + buf * BLOCK;
                            if (elect_one_sync()) {
#pragma unroll
                                for (int ks = 0; ks < D / 16; ++ks) {
                                    const uint64_t oa = (uint64_t)(((ks >> 2) * L::A_SLAB_BYTES + (ks & 3) * 32) >> 4);
                                    const uint64_t ob = (uint64_t)(((ks >> 2) * L::B_SLAB_BYTES + (ks & 3) * 32) >> 4);
                                    umma_f16(d_tmem, da + oa, db + ob, idesc, ks > 0 ? 1u : 0u);
                                }
                                umma_f16(d_tmem, umma_desc_k_sw32(smem_base + L::EXTA_OFF),
                                         umma_desc_k_sw32(b_smem + st * L::B_STAGE_BYTES + L::B_BYTES), idesc, 1u);
                                umma_commit(t_full(buf));
                                if (st + 1 == it.s1) umma_commit(a_empty(ab));
                            }
                            __syncwarp();
                        }
                        ++a_cnt;
                        continue;
                    }
                    // one step: the item's key tiles side by side in one accumulator buffer
                    const int buf = n & (NUM_TBUF - 1);
                    if (!wait_all(t_empty(buf), ((n >> 1) & 1) ^ 1, FCS_STATUS_WAIT_MMA)) break;
                    const uint64_t db = umma_desc_k_sw128(b_smem);
                    for (int t = 0; t < it.nt; ++t, ++a_cnt) {
                        const int ab = a_cnt % NA;
                        if (!wait_all(a_full(ab), (a_cnt / NA) & 1, FCS_STATUS_WAIT_MMA)) { ok = false; break; }
                        tc_fence_after();
                        const uint64_t da = umma_desc_k_sw128(a_smem + ab * L::A_BYTES);
                        const uint32_t d_tmem = tmem_base + buf * BLOCK + t * (BLOCK / 2);
                        if (elect_one_sync()) {
#pragma unroll
                            for (int ks = 0; ks < D / 16; ++ks) {
                                const uint64_t oa = (uint64_t)(((ks >> 2) * L::A_SLAB_BYTES + (ks & 3) * 32) >> 4);
                                const uint64_t ob = (uint64_t)(((ks >> 2) * L::B_SLAB_BYTES + (ks & 3) * 32) >> 4);
                                umma_f16(d_tmem, da + oa, db + ob, idesc, ks > 0 ? 1u : 0u);
                            }
                            umma_f16(d_tmem, umma_desc_k_sw32(smem_base + L::EXTA_OFF),
                                     umma_desc_k_sw32(b_smem + L::B_BYTES), idesc, 1u);
                            umma_commit(a_empty(ab));
                            if (t + 1 == it.nt) umma_commit(t_full(buf));
                        }
                        __syncwarp();
                    }
                    ++n;
                }
            } else {
            for (; ok && !it.done; it.next(ps), ++a_cnt) {
                const int ab = a_cnt & 1;
                if (!wait_all(a_full(ab), (a_cnt >> 1) & 1, FCS_STATUS_WAIT_MMA)) break;
                const uint64_t da = umma_desc_k_sw128(a_smem + ab * L::A_BYTES);
                for (int st = it.s0; st < it.s1; ++st, ++n) {
                    if (!wait_all(b_full(stage), phase, FCS_STATUS_WAIT_MMA)) { ok = false; break; }
                    const int buf = n & (NUM_TBUF - 1);
                    if (!wait_all(t_empty(buf), ((n >> 1) & 1) ^ 1, FCS_STATUS_WAIT_MMA)) { ok = false; break; }
                    tc_fence_after();
                    const uint64_t db = umma_desc_k_sw128(b_smem + stage * L::B_STAGE_BYTES);
                    const uint32_t d_tmem = tmem_base + buf * BLOCK;
                    if (elect_one_sync()) {
#pragma unroll
                        for (int ks = 0; ks < D / 16; ++ks) {
                            // 32 bytes per 16-element step inside a slab
                            const uint64_t oa = (uint64_t)(((ks >> 2) * L::A_SLAB_BYTES + (ks & 3) * 32) >> 4);
                            const uint64_t ob = (uint64_t)(((ks >> 2) * L::B_SLAB_BYTES + (ks & 3) * 32) >> 4);
                            umma_f16(d_tmem, da + oa, db + ob, idesc, ks > 0 ? 1u : 0u);
                        }
                        if constexpr (EXT)   // + (key-side constant) x (-(lse)/c parts of the queries)
                            umma_f16(d_tmem, umma_desc_k_sw32(smem_base + L::EXTA_OFF),
                                     umma_desc_k_sw32(b_smem + stage * L::B_STAGE_BYTES + L::B_BYTES), idesc, 1u);
                        umma_commit(b_empty(stage));
                        umma_commit(t_full(buf));
                        if (st + 1 == it.s1) umma_commit(a_empty(ab));
                    }
                    __syncwarp();
                    if (++stage == L::NS) { stage = 0; phase ^= 1; }
                }
            }
            }
        }
    } else {
        // ------------------------------------------------ consumers
        const int wg = warp >> 2;                  // consumer group
        const int col0 = wg * GROUP_COLS;          // its first column of every accumulator
        const int row = ((warp & 3) << 5) | lane;  // tensor-memory lane of this thread
        const uint32_t lane_addr = tmem_base + ((uint32_t)((warp & 3) << 5) << 16) + col0;
        const float c = p.c;
        bool ok = true;

        if (MODE == MODE_STATS && p.clear_out) {
            // the output is accumulated by the column pass: clear it here
            const long long n_out = (long long)p.B * p.Sk;
            for (long long idx = (long long)blockIdx.x * CONSUMER_THREADS + threadIdx.x; idx < n_out;
                 idx += (long long)gridDim.x * CONSUMER_THREADS) {
                const long long bb = idx / p.Sk;
                p.out[bb * p.out_ld + (idx - bb * p.Sk)] = 0.f;
            }
        }

        if (MODE == MODE_STATS && p.clear_extra) {
            // a buffer the caller wants zeroed alongside this call (the target of its next call)
            for (long long idx = (long long)blockIdx.x * CONSUMER_THREADS + threadIdx.x; idx < p.clear_extra_n;
                 idx += (long long)gridDim.x * CONSUMER_THREADS)
                p.clear_extra[idx] = 0.f;
        }

        Items it;
        it.init(ps, blockIdx.x, gridDim.x);
        float m_run = ROW_MAX_START, l_run = 0.f;      // statistics pass state
        float acc[4] = {0.f, 0.f, 0.f, 0.f};       // column pass state
        int item_cnt = 0, n = 0;
        // statistics pass: the item whose partials this group still has to combine
        // (its count; which item that is waits in shared memory, not in four registers.  Item n + 4 is this group's next, in
        // the same place: every item has a step, and the step of item n + 4 comes into an accumulator that all threads have
        // released in item n + 2 or later, after they have finished item n.)
        static_assert(MERGE_SLOTS == CONSUMER_GROUPS && NUM_TBUF == 2, "a slot is one group's, and free when it comes round");
        int pend_cnt = -1;
        int4* meta = reinterpret_cast<int4*>(smem + L::META_OFF);
        auto finish_item = [&]() -> bool {
            const int slot = pend_cnt & (MERGE_SLOTS - 1);
            bool good = mbar_wait(merge_bar(slot), (pend_cnt / MERGE_SLOTS) & 1, abort_flag, p.status,
                                  FCS_STATUS_WAIT_CONSUMER);
            good = __all_sync(0xffffffffu, good);
            pend_cnt = -1;
            if (!good) return false;
            const int4 item = meta[slot];
            const float2* mb = merge_buf + slot * CONSUMER_GROUPS * TILE;
            float mm = -INFINITY;
#pragma unroll
            for (int g = 0; g < CONSUMER_GROUPS; ++g) mm = fmaxf(mm, mb[g * TILE + row].x);
            const float ms = (mm == -INFINITY) ? 0.f : mm;
            float ll = 0.f;
#pragma unroll
            for (int g = 0; g < CONSUMER_GROUPS; ++g) {
                const float2 o = mb[g * TILE + row];
                ll += o.y * exp2f(o.x - ms);
            }
            const long long bh = (long long)item.x * p.H + item.y;
            const int q_abs = item.z * TILE + row;
            if (p.nsplit == 1) {
                const float nlv = (q_abs < p.Sq) ? negative_lse(mm, ll, p.log2_norm) : -INFINITY;
                p.neg_lse[bh * p.lse_rows + q_abs] = nlv;
                uint4 e0, e1;
                make_ext_row(nlv, p.inv_c, ps.ext_bf16 != 0, e0, e1);
                uint4* er = reinterpret_cast<uint4*>(p.ext) + (bh * p.lse_rows + q_abs) * 2;
                er[0] = e0;
                er[1] = e1;
            } else {
                const long long rows = (long long)p.NQ * TILE;
                reinterpret_cast<float2*>(p.part)[((long long)item.w * p.B * p.H + bh) * rows + q_abs] =
                    make_float2(mm, ll);
            }
            return true;
        };
        // short column modes: every item ends a key tile, and its sums sit in four groups.  When
        // `out` may be another GPU's memory (the _COMBINE modes) they meet in shared memory and one group,
        // a different one every item, adds them into the output after its next step -- one add per
        // key over NVLink instead of four, nobody waits.  (With a local `out` the four adds are
        // cheaper than the meeting: measured +2 % on the long-context shape.)
        float* colbuf = reinterpret_cast<float*>(smem + L::MERGE_OFF);
        bool cpend = false;
        int cp_cnt = 0, cp_b = 0, cp_kt = 0, cp_nt = 0;
        auto finish_cols = [&]() -> bool {
            const int slot = cp_cnt & (MERGE_SLOTS - 1);
            bool good = mbar_wait(merge_bar(slot), (cp_cnt / MERGE_SLOTS) & 1, abort_flag, p.status,
                                  FCS_STATUS_WAIT_CONSUMER);
            good = __all_sync(0xffffffffu, good);
            cpend = false;
            if (!good) return false;
            const float* cb = colbuf + slot * CONSUMER_GROUPS * TILE + row;
            // system scope: `out` may live on another GPU and take adds from several
            float* dst = p.out + (long long)cp_b * p.out_ld;
            const int k0 = cp_kt * TILE + row;
            if (p.col_pack == 2) {   // groups 0, 1 hold the first key tile, groups 2, 3 the second
                if (k0 < p.Sk) atomicAdd_system(dst + k0, cb[0] + cb[TILE]);
                if (cp_nt == 2 && k0 + TILE < p.Sk) atomicAdd_system(dst + k0 + TILE, cb[2 * TILE] + cb[3 * TILE]);
            } else if (k0 < p.Sk) {
                atomicAdd_system(dst + k0, (cb[0] + cb[TILE]) + (cb[2 * TILE] + cb[3 * TILE]));
            }
            return true;
        };
        for (; ok && !it.done; it.next(ps), ++item_cnt) {
            // steps f_lo <= st < f_hi need no masks: their per-step work is kept minimal
            int f_lo, f_hi;
            if constexpr (MODE == MODE_STATS) stats_full_range(ps, it.qt, f_lo, f_hi);
            else colsum_full_range(ps, it.kt, f_lo, f_hi);
            for (int st = it.s0; st < it.s1; ++st, ++n) {
                const int buf = n & (NUM_TBUF - 1);
                ok = mbar_wait(t_full(buf), (n >> 1) & 1, abort_flag, p.status, FCS_STATUS_WAIT_CONSUMER);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
                tc_fence_after();
                const uint32_t taddr = lane_addr + buf * BLOCK;
                const bool full = (st >= f_lo) && (st < f_hi);
                if constexpr (MODE == MODE_STATS) {
                    bool whole = full;
                    int cols = GROUP_COLS, first = col0, lim = 0, lim_first = 0, lim_last = 0;
                    if (!full) {
                        // the columns that some row of the tile sees, in four runs of whole 32
                        int seen = stats_last_visible(p, it.qt, st, TILE - 1) + 1;
                        seen = seen < BLOCK ? seen : BLOCK;
                        cols = ((seen + 127) >> 7) << 5;
                        first = wg * cols;
                        lim = stats_last_visible(p, it.qt, st, row) - first;
                        lim_first = __shfl_sync(0xffffffffu, lim, 0);
                        lim_last = __shfl_sync(0xffffffffu, lim, 31);
                        whole = cols == GROUP_COLS && lim_first >= GROUP_COLS - 1;
                    }
                    if (whole) stats_tile_full(taddr, c, m_run, l_run);
                    else stats_tile(taddr - col0 + first, cols, lim, lim_first, lim_last, c, m_run, l_run);
                } else if constexpr (EXT) {
                    // the accumulator already holds s - lse/c
                    if (full) {
                        colsum_tile_ext_full(taddr, c, acc);
                    } else {
                        if constexpr (L::SHORT) {
                            // Partly visible here are the blocks at the end of the query axis -- every item has one -- and
                            // a few key tiles on the diagonal: fixed shares, decided with the fewest instructions.
                            // Two key tiles in this accumulator buffer, 128 query columns each: groups 0, 1 take the
                            // halves of the first tile's columns, groups 2, 3 the second's.  At most 128 query
                            // columns otherwise: 32 for each group, not 64 for two of them.
                            const bool packed = p.col_pack == 2, narrow = !packed && colsum_end_visible(p, st) <= BLOCK / 2;
                            const int tg = packed ? wg >> 1 : 0;
                            const int q0 = packed ? (wg & 1) * GROUP_COLS : narrow ? wg * (GROUP_COLS / 2) : col0;
                            if (tg < it.nt) {
                                const int end = colsum_end_visible(p, st) - q0;
                                const int thr = colsum_first_visible(p, it.kt + tg, st, row) - q0;
                                const int thr_first = __shfl_sync(0xffffffffu, thr, 0), thr_last = __shfl_sync(0xffffffffu, thr, 31);
                                if (narrow) {
                                    if (end > 0 && thr_first < GROUP_COLS / 2) {
                                        uint32_t r[32];
                                        tmem_ld_x32(taddr - col0 + q0, r);
                                        tmem_ld_wait(r);
                                        if (end >= GROUP_COLS / 2 && thr_last <= 0) colsum_chunk_ext<BLOCK_FULL>(r, 0, 32, c, acc);
                                        else colsum_chunk_ext<BLOCK_MASKED>(r, thr, end, c, acc);
                                    }
                                } else if (end > 0 && thr_first < GROUP_COLS) {
                                    if (end >= GROUP_COLS && thr_last <= 0) colsum_tile_ext_full(taddr, c, acc);
                                    else colsum_tile_ext(taddr, GROUP_COLS, thr, thr_first, thr_last, end, c, acc);
                                }
                            }
                        } else {
                            // the columns that some row of the tile sees, in four runs of whole 32
                            const int from = colsum_first_visible(p, it.kt, st, 0) & ~31;
                            const int cols = ((colsum_end_visible(p, st) - from + 127) >> 7) << 5, q0 = from + wg * cols;
                            const int end = colsum_end_visible(p, st) - q0;
                            const int thr = colsum_first_visible(p, it.kt, st, row) - q0;
                            // what the block's queries see of this warp's keys: nothing, everything, or some
                            const int thr_first = __shfl_sync(0xffffffffu, thr, 0), thr_last = __shfl_sync(0xffffffffu, thr, 31);
                            const uint32_t at = taddr - col0 + q0;
                            if (cols == GROUP_COLS && from % GROUP_COLS == 0 && end >= GROUP_COLS && thr_last <= 0)
                                colsum_tile_ext_full(at, c, acc);
                            else colsum_tile_ext(at, cols, thr, thr_first, thr_last, end, c, acc);
                        }
                    }
                } else {
                    const int ls = n & (NUM_LSE - 1);
                    ok = mbar_wait(l_full(ls), (n / NUM_LSE) & 1, abort_flag, p.status, FCS_STATUS_WAIT_CONSUMER);
                    ok = __all_sync(0xffffffffu, ok);
                    if (!ok) break;
                    const float4* nl = reinterpret_cast<const float4*>(smem + L::LSE_OFF + ls * BLOCK * 4) + col0 / 4;
                    if (full) {
                        colsum_tile<false>(taddr, nl, 0, GROUP_COLS, c, acc);
                    } else {
                        const int thr = colsum_first_visible(p, it.kt, st, row) - col0;
                        const int end = colsum_end_visible(p, st) - col0;
                        // skip the block when no key of the tile is seen by any of its queries
                        const int thr_first_row = __shfl_sync(0xffffffffu, thr, 0);
                        if (end > 0 && thr_first_row < GROUP_COLS) colsum_tile<true>(taddr, nl, thr, end, c, acc);
                    }
                    mbar_arrive(l_empty(ls));
                }
                tc_fence_before();
                mbar_arrive(t_empty(buf));
                if constexpr (MODE == MODE_STATS) {
                    if (pend_cnt >= 0) { ok = finish_item(); if (!ok) break; }
                }
                if constexpr (L::COMBINE) {
                    if (cpend) { ok = finish_cols(); if (!ok) break; }
                }
            }
            if (!ok) break;
            if constexpr (MODE == MODE_STATS) {
                // post this group's partial (max, sum); one group, a different one every
                // item, combines the four partials after its next step, when the others
                // have long since posted -- nobody stands waiting at the end of an item
                if (pend_cnt >= 0) { ok = finish_item(); if (!ok) break; }
                const int slot = item_cnt & (MERGE_SLOTS - 1);
                merge_buf[(slot * CONSUMER_GROUPS + wg) * TILE + row] = make_float2(m_run, l_run);
                if ((item_cnt % CONSUMER_GROUPS) == wg) {
                    pend_cnt = item_cnt;
                    if (row == 0) meta[slot] = make_int4(it.b, it.h, it.qt, it.sp);
                }
                mbar_arrive(merge_bar(slot));
                m_run = ROW_MAX_START; l_run = 0.f;
            } else if constexpr (L::SHORT) {
                if constexpr (!L::COMBINE) {
                    // four adds per key, straight from the groups: cheapest when `out` is local
                    int tg = 0;
                    bool mine = true;
                    if (p.col_pack == 2) { tg = wg >> 1; mine = tg < it.nt; }
                    const int k_abs = (it.kt + tg) * TILE + row;
                    if (k_abs < p.Sk && mine)
                        atomicAdd_system(p.out + (long long)it.b * p.out_ld + k_abs, column_sum(acc));
                    acc[0] = acc[1] = acc[2] = acc[3] = 0.f;
                } else {
                    if (cpend) { ok = finish_cols(); if (!ok) break; }
                    const int slot = item_cnt & (MERGE_SLOTS - 1);
                    colbuf[(slot * CONSUMER_GROUPS + wg) * TILE + row] = column_sum(acc);
                    mbar_arrive(merge_bar(slot));
                    if ((item_cnt % CONSUMER_GROUPS) == wg) {
                        cpend = true;
                        cp_cnt = item_cnt; cp_b = it.b; cp_kt = it.kt; cp_nt = it.nt;
                    }
                    acc[0] = acc[1] = acc[2] = acc[3] = 0.f;
                }
            } else {
                if (it.flush()) {
                    const int k_abs = it.kt * TILE + row;
                    if (k_abs < p.Sk)
                        // system scope: `out` may live on another GPU and take adds from several
                        atomicAdd_system(p.out + (long long)it.b * p.out_ld + k_abs, column_sum(acc));
                    acc[0] = acc[1] = acc[2] = acc[3] = 0.f;
                }
            }
        }
        if constexpr (MODE == MODE_STATS) {
            if (ok && pend_cnt >= 0) finish_item();
        }
        if constexpr (L::COMBINE) {
            if (ok && cpend) finish_cols();
        }
    }

    // ---------------------------------------------------- teardown
    tc_fence_before();
    __syncthreads();
    if (MODE != MODE_STATS && p.sig_done && threadIdx.x == 0) {
        // every add of this CTA was issued before the barrier above; the last CTA to get here tells
        // the owner of the output (release, system scope) that this GPU's share of the call is in.
        // One system-scope fence per grid, by that last CTA: a system-scope fence in every CTA cost
        // 67 us on the long-context shape (they are served one after the other); the CTAs hand
        // their writes on to it through device-scope fences and the counter.
        __threadfence();
        const int arrived = atomicAdd(p.sig_counter, 1);
        if (arrived == (int)gridDim.x - 1) {
            *p.sig_counter = 0;
            release_store_system_one(p.sig_done, p.sig_done_value);
        }
    }
    if (warp == MMA_WARP) {
        if (*abort_flag) __nanosleep(1000000);   // let copies and MMAs in flight land
        tc_fence_after();
        tmem_dealloc(tmem_base, TMEM_COLS);
    }
}

// Combine the key-range partials of the statistics pass into the per-row value
// the column pass subtracts.
__global__ void merge_stats_kernel(const Problem p) {
    grid_dependency_wait();
    grid_launch_dependents();
    const long long rows = (long long)p.NQ * TILE;
    const long long n = (long long)p.B * p.H * rows;
    const float2* part = reinterpret_cast<const float2*>(p.part);
    for (long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x; idx < n;
         idx += (long long)gridDim.x * blockDim.x) {
        const long long bh = idx / rows;
        const int q_abs = (int)(idx - bh * rows);
        float v = -INFINITY;
        if (q_abs < p.Sq) {
            float mm = -INFINITY;
            for (int s = 0; s < p.nsplit; ++s) mm = fmaxf(mm, part[s * n + idx].x);
            float ll = 0.f;
            for (int s = 0; s < p.nsplit; ++s) {
                const float2 t = part[s * n + idx];
                ll += t.y * exp2f(t.x - mm);
            }
            v = negative_lse(mm, ll, p.log2_norm);
        }
        p.neg_lse[bh * p.lse_rows + q_abs] = v;
        uint4 e0, e1;
        make_ext_row(v, p.inv_c, p.fmt ? *p.fmt != 0 : p.ext_bf16 != 0, e0, e1);
        uint4* er = reinterpret_cast<uint4*>(p.ext) + (bh * p.lse_rows + q_abs) * 2;
        er[0] = e0;
        er[1] = e1;
    }
}

// ---------------------------------------------------------------------------
// Flags between the GPUs of a node (peer-mapped memory), for callers that order their
// kernels across ranks without a collective: a release store per flag, and a bounded wait
// until every flag has reached a value.
// ---------------------------------------------------------------------------
}  // namespace fcs

#include "colsum_fused_short.cuh"

namespace fcs {

constexpr int PEER_FLAGS_MAX = 16;
struct PeerFlagPointers { int* p[PEER_FLAGS_MAX]; };

__global__ void peer_post_kernel(const PeerFlagPointers flags, int n, int value) {
    if ((int)threadIdx.x < n) {
        // everything the kernels before this one in the stream wrote (to any GPU) is visible to
        // whoever reads this value with an acquire load
        __threadfence_system();
        asm volatile("st.release.sys.global.s32 [%0], %1;" ::"l"(flags.p[threadIdx.x]), "r"(value) : "memory");
    }
}

__global__ void peer_wait_kernel(const int* flags, int n, int value, int* status) {
    if ((int)threadIdx.x < n) {
        const long long t0 = clock64();
        unsigned spins = 0;
        while (true) {
            int v;
            asm volatile("ld.acquire.sys.global.s32 %0, [%1];" : "=r"(v) : "l"(flags + threadIdx.x) : "memory");
            if (v >= value) break;
            if ((++spins & 63u) == 0u && clock64() - t0 > g_wait_limit_cycles) {
                if (status) atomicCAS(status, 0, FCS_STATUS_WAIT_PEER);
                break;
            }
            __nanosleep(100);
        }
    }
}

// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------
static thread_local char g_err[512] = "";

static int fail(int code, const char* fmt, ...) {
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(g_err, sizeof(g_err), fmt, ap);
    va_end(ap);
    return code;
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*,
                                  CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
                                  CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_tiled_fn() {
    static EncodeTiledFn fn = nullptr;
    if (!fn) {
        void* sym = nullptr;
        cudaDriverEntryPointQueryResult qres;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &qres) == cudaSuccess &&
            qres == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(sym);
    }
    return fn;
}

static int num_sms() {
    static int cached[64] = {0};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 148;
    if (cached[dev] == 0) {
        int n = 0;
        if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
        cached[dev] = n;
    }
    return cached[dev];
}

// (D, S, H, B) view of a [B, H, S, D] tensor, boxes of `box_rows` rows x 64
// elements, 128-byte swizzle, out-of-range rows read as zero -- and so do the columns
// from D on when D is not a multiple of 64: the kernels contract 64 or 128 columns, the
// padding adds nothing to a score.
static int make_tensor_map(CUtensorMap* m, const void* base, int dtype, int B, int H, int S, int D,
                           int64_t sb, int64_t sh, int64_t ss, int box_rows) {
    EncodeTiledFn enc = encode_tiled_fn();
    if (!enc) return fail(FCS_ERR_CUDA, "cuTensorMapEncodeTiled is not available from the driver");
    cuuint64_t dims[4] = {(cuuint64_t)D, (cuuint64_t)S, (cuuint64_t)H, (cuuint64_t)B};
    cuuint64_t strides[3] = {(cuuint64_t)ss * 2, (cuuint64_t)sh * 2, (cuuint64_t)sb * 2};
    cuuint32_t box[4] = {64, (cuuint32_t)box_rows, 1, 1};
    cuuint32_t estr[4] = {1, 1, 1, 1};
    CUresult r = enc(m, dtype == FCS_DTYPE_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16,
                     4, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                     CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                     CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail(FCS_ERR_CUDA, "cuTensorMapEncodeTiled failed with CUresult %d", (int)r);
    return FCS_OK;
}

// The same view in boxes of `box_rows` whole rows, not swizzled: rows of D elements one after the
// other in shared memory.
static int make_plain_tensor_map(CUtensorMap* m, const void* base, int dtype, int B, int H, int S, int D,
                                 int64_t sb, int64_t sh, int64_t ss, int box_rows) {
    EncodeTiledFn enc = encode_tiled_fn();
    if (!enc) return fail(FCS_ERR_CUDA, "cuTensorMapEncodeTiled is not available from the driver");
    cuuint64_t dims[4] = {(cuuint64_t)D, (cuuint64_t)S, (cuuint64_t)H, (cuuint64_t)B};
    const int es = dtype == FCS_DTYPE_FP32 ? 4 : 2;
    cuuint64_t strides[3] = {(cuuint64_t)ss * es, (cuuint64_t)sh * es, (cuuint64_t)sb * es};
    cuuint32_t box[4] = {(cuuint32_t)D, (cuuint32_t)box_rows, 1, 1};
    cuuint32_t estr[4] = {1, 1, 1, 1};
    const CUresult r = enc(m, dtype == FCS_DTYPE_FP32   ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32
                              : dtype == FCS_DTYPE_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16
                                                        : CU_TENSOR_MAP_DATA_TYPE_FLOAT16,
                           4, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                           CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                           CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail(FCS_ERR_CUDA, "cuTensorMapEncodeTiled failed with CUresult %d", (int)r);
    return FCS_OK;
}

// Optional per-pass timing: when enabled, events are recorded on the caller's
// stream around each kernel of a call.
struct PassTimers {
    bool ready = false;
    bool recorded = false;
    cudaEvent_t ev[4];
};
static bool g_profiling = false;
static PassTimers g_timers[64];

static PassTimers* timers_for_current_device() {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return nullptr;
    PassTimers& t = g_timers[dev];
    if (!t.ready) {
        for (int i = 0; i < 4; ++i)
            if (cudaEventCreate(&t.ev[i]) != cudaSuccess) return nullptr;
        t.ready = true;
    }
    return &t;
}

// (16, rows, planes) view of the [planes][rows][16] extension columns: boxes of 256
// rows x 16 elements (32 bytes), 32-byte swizzle.
static int make_ext_tensor_map(CUtensorMap* m, const void* base, int dtype, long long planes, long long rows) {
    EncodeTiledFn enc = encode_tiled_fn();
    if (!enc) return fail(FCS_ERR_CUDA, "cuTensorMapEncodeTiled is not available from the driver");
    cuuint64_t dims[3] = {(cuuint64_t)EXT_K, (cuuint64_t)rows, (cuuint64_t)planes};
    cuuint64_t strides[2] = {(cuuint64_t)EXT_ROW_BYTES, (cuuint64_t)rows * EXT_ROW_BYTES};
    cuuint32_t box[3] = {(cuuint32_t)EXT_K, (cuuint32_t)BLOCK, 1};
    cuuint32_t estr[3] = {1, 1, 1};
    CUresult r = enc(m, dtype == FCS_DTYPE_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16,
                     3, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                     CU_TENSOR_MAP_SWIZZLE_32B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                     CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail(FCS_ERR_CUDA, "cuTensorMapEncodeTiled (extension) failed with CUresult %d", (int)r);
    return FCS_OK;
}

template <int D, int MODE>
static cudaError_t launch_stream(const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& text,
                                 const Problem& p, int grid, cudaStream_t stream, bool overlap) {
    using LayoutT = Layout<D, MODE>;
    static bool configured[64] = {false};
    int dev = 0;
    cudaGetDevice(&dev);
    auto kern = colsum_stream_kernel<D, MODE>;
    if (dev >= 0 && dev < 64 && !configured[dev]) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             LayoutT::DYN_BYTES);
        if (e != cudaSuccess) return e;
        configured[dev] = true;
    }
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = LayoutT::DYN_BYTES;
    cfg.stream = stream;
    // (see overlap_previous below)
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = overlap ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kern, ta, tb, text, p);
}

// Every kernel of the operator is launched as a programmatic dependent of whatever is before it in
// the stream, lets its own dependents start early, and waits for everything before it
// (grid_dependency_wait) when its set-up -- barriers, tensor memory, descriptors -- is done and before
// its first access to global memory.  Between two kernels of a call, and between two calls, only
// the wake-up is left of a launch.  Back to back, us per call: 8 pairs of 256 keys 14.3 -> 8.2, a CLS
// row over 32 x 16 x 577 14.3 -> 12.1, 128 queries over 32 x 4096 keys 20.5 -> 19.0.  With per-pass
// timing on, the kernels run one after the other.
static bool overlap_previous() { return !g_profiling; }

// Zeroes the B x S valid entries of `out`.
static int launch_clear(float* out, long long out_ld, long long B, long long S, cudaStream_t stream) {
    if (B <= 0 || S <= 0) return FCS_OK;
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof(cfg));
    const long long per_row = (S + 1023) / 1024;
    cfg.gridDim = dim3((unsigned)(per_row < 1024 ? per_row : 1024), (unsigned)(B < 1024 ? B : 1024));
    cfg.blockDim = dim3(256);
    cfg.stream = stream;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = overlap_previous() ? 1 : 0;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, clear_rows_kernel, out, out_ld, B, S);
    if (e != cudaSuccess) return fail(FCS_ERR_CUDA, "clearing the output failed: %s", cudaGetErrorString(e));
    return FCS_OK;
}

// Rows of 16-byte multiples (what a tensor map and a bulk copy can address), at most two
// 64-column slabs.
static bool head_dim_ok(int D) { return D >= 8 && D <= 128 && D % 8 == 0; }

static int check_operand(const char* name, const void* ptr, int64_t sb, int64_t sh, int64_t ss, int granule = 8) {
    if (!ptr) return fail(FCS_ERR_INVALID_ARGUMENT, "%s is NULL", name);
    if (reinterpret_cast<uintptr_t>(ptr) % 16)
        return fail(FCS_ERR_INVALID_ARGUMENT, "%s must be 16-byte aligned", name);
    if (sb <= 0 || sh <= 0 || ss <= 0 || sb % granule || sh % granule || ss % granule)
        return fail(FCS_ERR_INVALID_ARGUMENT,
                    "%s strides must be positive multiples of %d elements (got b=%lld h=%lld s=%lld)", name, granule,
                    (long long)sb, (long long)sh, (long long)ss);
    return FCS_OK;
}

// Few query rows: the matrix-vector kernel (a kernel that clears the output, then the
// clustered kernel as its programmatic dependent).
template <int D, bool BF16, int RMAX, int W>
static cudaError_t launch_small_q_w(const SmallQParams& sp, int grid, size_t smem, cudaStream_t stream) {
    static bool configured[64] = {false};
    int dev = 0;
    cudaGetDevice(&dev);
    auto kern = colsum_small_q_kernel<D, BF16, RMAX, W>;
    if (dev >= 0 && dev < 64 && !configured[dev]) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMALLQ_MAX_SMEM);
        if (e != cudaSuccess) return e;
        configured[dev] = true;
    }
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3(32 * (W + 1));
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    // The cluster attribute is given for clusters of one as well: the kernel's cluster instructions
    // (barrier.cluster, mapa, st.async) are illegal in a launch without it.
    cudaLaunchAttribute attrs[2];
    attrs[0].id = cudaLaunchAttributeClusterDimension;
    attrs[0].val.clusterDim.x = (unsigned)sp.CL;
    attrs[0].val.clusterDim.y = 1;
    attrs[0].val.clusterDim.z = 1;
    // behind the clearing kernel: start at once, wait for it only before the adds
    attrs[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attrs[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attrs;
    cfg.numAttrs = overlap_previous() ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, kern, sp);
}

template <int D, bool BF16, int RMAX>
static cudaError_t launch_small_q_r(const SmallQParams& sp, int grid, size_t smem, cudaStream_t stream) {
    if (sp.wide) return launch_small_q_w<D, BF16, RMAX, SMALLQ_WIDE_WARPS>(sp, grid, smem, stream);
    return launch_small_q_w<D, BF16, RMAX, SMALLQ_CONSUMER_WARPS>(sp, grid, smem, stream);
}

template <int D, bool BF16>
static cudaError_t launch_small_q_t(const SmallQParams& sp, int grid, size_t smem, cudaStream_t stream) {
    if (sp.R == 1) return launch_small_q_r<D, BF16, 1>(sp, grid, smem, stream);
    if (sp.R == 2) return launch_small_q_r<D, BF16, 2>(sp, grid, smem, stream);
    return launch_small_q_r<D, BF16, 4>(sp, grid, smem, stream);
}

static int launch_small_q(const void* q, const void* k, float* out, int64_t out_ld, int B, int H, int R, int Sk,
                          int D, int dtype, int64_t qsb, int64_t qsh, int64_t qss, int64_t ksb, int64_t ksh,
                          int64_t kss, float scale, int causal, int k_past, int h_norm, bool clear_out,
                          int* status, cudaStream_t stream) {
    const int sms = num_sms();
    if (clear_out) {
        const int rc = launch_clear(out, (long long)out_ld, B, Sk, stream);
        if (rc != FCS_OK) return rc;
    }
    SmallQParams sp;
    memset(&sp, 0, sizeof(sp));
    sp.q = q; sp.k = k; sp.out = out; sp.out_ld = out_ld;
    sp.H = H; sp.R = R; sp.Sk = Sk;
    sp.qsb = qsb; sp.qsh = qsh; sp.qss = qss; sp.ksb = ksb; sp.ksh = ksh; sp.kss = kss;
    sp.c = scale * 1.4426950408889634f;
    sp.causal = causal; sp.k_past = causal ? k_past : 0;
    sp.inv_norm = 1.0f / ((float)h_norm * (float)R);
    sp.status = status;
    // keys past the last query's horizon are seen by no row: not read, their columns stay zero
    long long keys = Sk;
    if (causal && (long long)k_past + R < keys) keys = (long long)k_past + R;
    sp.keys = (int)keys;
    size_t smem = 0;
    sp.units = B * H;
    if (!smallq_plan(sp.units, R, sp.keys, D, sms, &sp.CL, &sp.clusters, &sp.range_rows, &sp.stages, &sp.bufs, &sp.wide, &smem))
        return fail(FCS_ERR_UNSUPPORTED, "few-row kernel: %d keys do not fit", Sk);
    const int grid = sp.clusters * sp.CL;
    const bool bf16 = dtype == FCS_DTYPE_BF16;
    const cudaError_t e =
        (D == 64) ? (bf16 ? launch_small_q_t<64, true>(sp, grid, smem, stream)
                          : launch_small_q_t<64, false>(sp, grid, smem, stream))
                  : (bf16 ? launch_small_q_t<128, true>(sp, grid, smem, stream)
                          : launch_small_q_t<128, false>(sp, grid, smem, stream));
    if (e != cudaSuccess) return fail(FCS_ERR_CUDA, "few-row kernel launch failed: %s", cudaGetErrorString(e));
    return FCS_OK;
}

// At most four query rows with scratch to be had: the scores kernel and the columns kernel.
template <int DK, int T, int R>
static cudaError_t launch_few_rows_t(const CUtensorMap& tk, const few::Params& fp, int grid, cudaStream_t stream) {
    static bool configured[64] = {false};
    int dev = 0;
    cudaGetDevice(&dev);
    auto kern = few::few_rows_scores_kernel<DK, T, R>;
    if (dev >= 0 && dev < 64 && !configured[dev]) {
        const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, few::SMEM_BYTES);
        if (e != cudaSuccess) return e;
        configured[dev] = true;
    }
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3(few::THREADS);
    cfg.dynamicSmemBytes = few::SMEM_BYTES;
    cfg.stream = stream;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = overlap_previous() ? 1 : 0;
    cudaError_t e = cudaLaunchKernelEx(&cfg, kern, tk, fp);
    if (e != cudaSuccess) return e;
    const int B = fp.units / fp.H;
    cfg.gridDim = dim3((unsigned)((fp.Sk + few::COLUMN_KEYS - 1) / few::COLUMN_KEYS), (unsigned)(B < 65535 ? B : 65535));
    cfg.blockDim = dim3(few::COLUMN_THREADS);
    cfg.dynamicSmemBytes = 0;
    return cudaLaunchKernelEx(&cfg, few::few_rows_columns_kernel, fp);
}
template <int DK, int T, int R, int W>
static cudaError_t launch_few_rows_cluster_w(const CUtensorMap& tk, const few::Params& fp, cudaStream_t stream) {
    static bool configured[64] = {false};
    int dev = 0;
    cudaGetDevice(&dev);
    auto kern = few::few_rows_cluster_kernel<DK, T, R, W>;
    if (dev >= 0 && dev < 64 && !configured[dev]) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, few::CLUSTER_SMEM_LIMIT);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
        if (e != cudaSuccess) return e;
        configured[dev] = true;
    }
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = dim3((unsigned)fp.units);
    cfg.blockDim = dim3(32 * (W + 1));
    cfg.dynamicSmemBytes = (size_t)few::cluster_smem<DK, T, W>(fp.R, fp.keys);
    cfg.stream = stream;
    cudaLaunchAttribute attrs[2];
    attrs[0].id = cudaLaunchAttributeClusterDimension;
    attrs[0].val.clusterDim.x = (unsigned)fp.H;
    attrs[0].val.clusterDim.y = 1;
    attrs[0].val.clusterDim.z = 1;
    attrs[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attrs[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attrs;
    cfg.numAttrs = overlap_previous() ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, kern, tk, fp);
}

template <int DK, int T, int R>
static cudaError_t launch_few_rows_cluster_t(const CUtensorMap& tk, const few::Params& fp, bool narrow, cudaStream_t stream) {
    return narrow ? launch_few_rows_cluster_w<DK, T, R, 4>(tk, fp, stream) : launch_few_rows_cluster_w<DK, T, R, 8>(tk, fp, stream);
}

// Which form takes a call with at most four query rows.  Measured back to back on a B200, us per call in
// clusters per batch entry / in two kernels / in clusters over key ranges (colsum_small_q.cuh; "-": it
// does not take the call or is far behind), one CLS row over B x H x keys of 64 columns unless said:
//     2 x 4 x 128            4.3 /  6.6 /  6.1       38 x 4 x 185           5.3 /  8.3 /  -
//     8 x 12 x 577 strided   7.7 /  7.9 / 34         32 x 12 x 257 of 128   8.1 / 12.0 /  9.5
//     32 x 16 x 577         18.7 / 15.2 / 12.1       64 x 12 x 197         12.0 / 12.8 /  9.9
//     16 x 16 x 700 of 80   14.8 / 12.6 /  -         8 x 16 x 2048, 3 rows 20.7 / 16.6 / 18.0
//     8 x 2000 of 128          - /  8.1 /  6.7       32 x 4096 of 128         - / 12.0 / 12.2
//     32 x 32768 of 128        - / 50.4 / 60.4       the same, 4 rows         - / 64.6 / 98.6
// and in clusters with four CTAs per SM: 25 x 16 x 577, 4 rows 10.2 (two kernels 17.9), 40 x 12 x 300 of 80
// 7.0 (12.7), 32 x 12 x 257 of 128 7.4 (key ranges 9.5), 64 x 8 x 577 11.5 (12.3), but 32 x 16 x 577 16.5 (12.1).
enum : int { FEW_CLUSTER = 0, FEW_CLUSTER_NARROW = 3, FEW_TWO_KERNELS = 1, FEW_KEY_RANGES = 2 };
static int few_rows_form(int B, int H, int R, int keys, int D, int row_bytes, bool dense, bool fp32, int smem, int smem_narrow, int sms) {
    const long long units = (long long)B * H, unit_bytes = (long long)keys * row_bytes;
    // many short units keep four CTAs on every SM busy; few bytes in all are over before two launches are
    const bool ranges_ok = !fp32 && dense && (D == 64 || D == 128);
    const bool many_short = units >= 2 * sms && unit_bytes <= 80 * 1024;
    if (H <= few::CLUSTER_MAX && unit_bytes <= 80 * 1024) {
        if (units <= 2 * sms && smem <= few::CLUSTER_SMEM_LIMIT) return FEW_CLUSTER;
        // four CTAs of four consumer warps per SM, as long as all clusters run at once (large ones do not fill
        // every SM); where the alternative is two kernels, in two rounds as well
        const long long at_once = H <= 8 ? 4ll * sms : 13ll * sms / 4;
        if (smem_narrow <= 55 * 1024 && units <= (ranges_ok ? at_once : 6ll * sms)) return FEW_CLUSTER_NARROW;
    }
    if (ranges_ok && R <= 2 && (many_short || units * unit_bytes <= (6ll << 20))) return FEW_KEY_RANGES;
    return FEW_TWO_KERNELS;
}

static int launch_few_rows(const void* q, const void* k, float* out, int64_t out_ld, int B, int H, int R, int Sk, int D,
                           int dtype, int64_t qsb, int64_t qsh, int64_t qss, int64_t ksb, int64_t ksh, int64_t kss,
                           float scale, int causal, int k_past, int h_norm, int* status, cudaStream_t stream,
                           void* (*alloc)(void*, size_t), void* alloc_ctx) {
    few::Params fp;
    memset(&fp, 0, sizeof(fp));
    fp.q = q; fp.out = out; fp.out_ld = out_ld;
    fp.H = H; fp.R = R; fp.D = D; fp.Sk = Sk;
    fp.units = B * H;
    // keys past the last query's horizon are seen by no row: not read, their columns are zero
    fp.keys = causal && (long long)k_past + R < Sk ? k_past + R : Sk;
    fp.qsb = qsb; fp.qsh = qsh; fp.qss = qss;
    fp.c = scale * 1.4426950408889634f;
    fp.causal = causal;
    fp.k_past = causal ? k_past : 0;
    fp.inv_norm = 1.0f / ((float)h_norm * (float)R);
    fp.status = status;
    const int sms = num_sms();
    const bool bf16 = dtype == FCS_DTYPE_BF16, fp32 = dtype == FCS_DTYPE_FP32;
    CUtensorMap tk;
    memset(&tk, 0, sizeof(tk));
    int rc;
    cudaError_t e;
    auto cluster_bytes = [&](int w) {
        const int stages = w * (fp32 ? 32 * (D <= 64 ? 64 : 128) * 4 : 8192);
        return stages + few::cluster_smem<64, few::T_FP16, 1>(R, fp.keys) - few::ClusterStage<64, few::T_FP16>::BYTES + w * 48;
    };
    const int form = few_rows_form(B, H, R, fp.keys, D, D * (fp32 ? 4 : 2), kss == D, fp32, cluster_bytes(8), cluster_bytes(4), sms);
    if (form == FEW_KEY_RANGES)
        return launch_small_q(q, k, out, out_ld, B, H, R, Sk, D, dtype, qsb, qsh, qss, ksb, ksh, kss, scale, causal,
                              k_past, h_norm, true, status, stream);
    if (form == FEW_CLUSTER || form == FEW_CLUSTER_NARROW) {
        const int rows = fp32      ? few::ClusterStage<64, few::T_FP32>::ROWS
                         : D <= 64 ? few::ClusterStage<64, few::T_FP16>::ROWS
                                   : few::ClusterStage<128, few::T_FP16>::ROWS;
        if ((rc = make_plain_tensor_map(&tk, k, dtype, B, H, Sk, D, ksb, ksh, kss, rows)) != FCS_OK) return rc;
        if (fp32)   // (more than 64 columns never come here: the stages alone are over both limits)
            e = R == 1 ? launch_few_rows_cluster_t<64, few::T_FP32, 1>(tk, fp, form == FEW_CLUSTER_NARROW, stream)
                       : launch_few_rows_cluster_t<64, few::T_FP32, 4>(tk, fp, form == FEW_CLUSTER_NARROW, stream);
        else
            e = D <= 64 ? (bf16 ? launch_few_rows_cluster_t<64, few::T_BF16, 4>(tk, fp, form == FEW_CLUSTER_NARROW, stream)
                            : launch_few_rows_cluster_t<64, few::T_FP16, 4>(tk, fp, form == FEW_CLUSTER_NARROW, stream))
                    : (bf16 ? launch_few_rows_cluster_t<128, few::T_BF16, 4>(tk, fp, form == FEW_CLUSTER_NARROW, stream)
                            : launch_few_rows_cluster_t<128, few::T_FP16, 4>(tk, fp, form == FEW_CLUSTER_NARROW, stream));
        if (e != cudaSuccess) return fail(FCS_ERR_CUDA, "few-row cluster form launch failed: %s", cudaGetErrorString(e));
        return FCS_OK;
    }
    const long long total = (long long)fp.units * fp.keys;
    long long share = (total + sms - 1) / sms;
    if (share < few::MIN_SHARE) share = few::MIN_SHARE;
    share = (share + 31) / 32 * 32;
    fp.share = (int)share;
    fp.slots = (int)((fp.keys + share - 2) / share) + 1;
    fp.score_ld = (fp.keys + 3) / 4 * 4;
    const size_t part_bytes = align_up((size_t)fp.units * fp.slots * few::CONSUMER_WARPS * few::MAX_ROWS * sizeof(float2), 256);
    uint8_t* ws = static_cast<uint8_t*>(alloc(alloc_ctx, part_bytes + (size_t)fp.units * R * fp.score_ld * sizeof(float)));
    if (!ws) return fail(FCS_ERR_WORKSPACE, "no scratch memory for the few-row form");
    fp.part = reinterpret_cast<float2*>(ws);
    fp.scores = reinterpret_cast<float*>(ws + part_bytes);
    const int rows = fp32      ? few::Stage<64, few::T_FP32>::ROWS
                     : D <= 64 ? few::Stage<64, few::T_FP16>::ROWS
                               : few::Stage<128, few::T_FP16>::ROWS;
    if ((rc = make_plain_tensor_map(&tk, k, dtype, B, H, Sk, D, ksb, ksh, kss, rows)) != FCS_OK) return rc;
    const int grid = (int)((total + share - 1) / share);
    if (fp32)
        e = D <= 64 ? (R == 1 ? launch_few_rows_t<64, few::T_FP32, 1>(tk, fp, grid, stream)
                              : launch_few_rows_t<64, few::T_FP32, 4>(tk, fp, grid, stream))
                    : (R == 1 ? launch_few_rows_t<128, few::T_FP32, 1>(tk, fp, grid, stream)
                              : launch_few_rows_t<128, few::T_FP32, 4>(tk, fp, grid, stream));
    else
        e = D <= 64 ? (bf16 ? launch_few_rows_t<64, few::T_BF16, 4>(tk, fp, grid, stream)
                        : launch_few_rows_t<64, few::T_FP16, 4>(tk, fp, grid, stream))
                : (bf16 ? launch_few_rows_t<128, few::T_BF16, 4>(tk, fp, grid, stream)
                        : launch_few_rows_t<128, few::T_FP16, 4>(tk, fp, grid, stream));
    if (e != cudaSuccess) return fail(FCS_ERR_CUDA, "few-row form launch failed: %s", cudaGetErrorString(e));
    return FCS_OK;
}

// Short key axes (non-causal, head dimension 64, S_k <= 2048): the single-pass
// cluster kernel.  g_single_pass: 0 = as single_pass_applies says, 1 = never, 2 = whenever
// the shape allows.
static int g_single_pass = 0;

static int single_pass_cluster_size(int Sk) {
    return (Sk + 255) / 256;   // one CTA per 256 keys; any size up to eight is a legal cluster
}

static bool single_pass_applies(int B, int H, int Sq, int Sk, int D, int causal) {
    if (g_single_pass == 1 || causal || D > 64 || Sk > 256 * sp::MAX_CL) return false;   // (D < 64: zero-filled columns)
    if (g_single_pass == 2) return true;
    const int cl = single_pass_cluster_size(Sk);
    // us per call, this form / the two passes, at 32 x 16 pairs and at 2 x 8: 96 keys 16/20 7/8, 150 21/30 7/12,
    // 300 48/56 9/15, 320 44/54 10/15, 520 101/119 12/20, 640 95/141 12/21, 1030 293/358 19/22, 1400 416/556 22/37,
    // 1700 760/805 34/46, 2048 847/1077 37/49.  The line lies where this form won when it was drawn, before it took the
    // last 10 to 20 %: at any fill of one slice, from a fill of 60 % up to six (the time goes by whole slices of 256
    // keys), and with clusters of 7 and 8, which fit only 15 at a time (105 / 120 of 148 SMs), on small calls only.  It is
    // the faster one beyond the line, too, by now; the line stays because calls past it have their exps summed in
    // 32 bits, and here they are rounded to fp16.
    if (cl == 1) return true;
    if (cl <= 6) return (long long)Sk * 100 >= (long long)cl * 256 * 60;
    if ((long long)Sk * 100 < (long long)cl * 256 * 85) return false;
    const long long tiles = (long long)B * H * ((Sq + TILE - 1) / TILE);
    return tiles <= 512;
}

// Clusters of `cl` CTAs of `kern` that the current device runs at once; 0 where it holds none, or does not say.  Asked
// once per device; `answers` holds one more than the answer.
static int resident_clusters(const void* kern, int cl, int threads, int smem, int (&answers)[64]) {
    int dev = 0, n = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
    if (answers[dev]) return answers[dev] - 1;
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = dim3((unsigned)(cl * 64));
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = (size_t)smem;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = (unsigned)cl;
    attr.val.clusterDim.y = 1;
    attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess ||
        cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess || n < 0) {
        cudaGetLastError();
        n = 0;
    }
    answers[dev] = n + 1;
    return n;
}

// The instance for clusters of `cl` CTAs.
typedef void (*SinglePassKernel)(const CUtensorMap, const CUtensorMap, const SinglePassParams);
template <bool PADDED>
static SinglePassKernel single_pass_kernel(int cl) {
    if (cl <= 1) return colsum_single_pass_kernel<PADDED, 1>;
    if (cl == 2) return colsum_single_pass_kernel<PADDED, 2>;
    if (cl <= 4) return colsum_single_pass_kernel<PADDED, 4>;
    return colsum_single_pass_kernel<PADDED, 8>;
}

// Clusters of `cl` CTAs that can be resident at once (0 if the query fails).
static int single_pass_max_clusters(int cl) {
    static int cached[64][sp::MAX_CL + 1] = {{0}};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64 || cl < 1 || cl > sp::MAX_CL) return 0;
    const int idx = cl;
    if (cached[dev][idx] == 0) {
        // (both instances for this size: the same block, shared memory and registers)
        if (cudaFuncSetAttribute(single_pass_kernel<true>(cl), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 sp::DYN_BYTES) != cudaSuccess ||
            cudaFuncSetAttribute(single_pass_kernel<false>(cl), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 sp::DYN_BYTES) != cudaSuccess)
            return 0;
        if (cl == 1) return cached[dev][idx] = num_sms();    // (no clusters: a CTA fills an SM)
        cudaLaunchConfig_t cfg;
        memset(&cfg, 0, sizeof(cfg));
        cfg.gridDim = dim3((unsigned)(cl * 64));
        cfg.blockDim = dim3(sp::THREADS);
        cfg.dynamicSmemBytes = sp::DYN_BYTES;
        cudaLaunchAttribute attr;
        attr.id = cudaLaunchAttributeClusterDimension;
        attr.val.clusterDim.x = (unsigned)cl;
        attr.val.clusterDim.y = 1;
        attr.val.clusterDim.z = 1;
        cfg.attrs = &attr;
        cfg.numAttrs = 1;
        int n = 0;
        if (cudaOccupancyMaxActiveClusters(&n, single_pass_kernel<false>(cl), &cfg) != cudaSuccess || n <= 0) {
            cudaGetLastError();
            return 0;
        }
        cached[dev][idx] = n;
    }
    return cached[dev][idx];
}

static int launch_single_pass(const CUtensorMap& tq, const CUtensorMap& tk, float* out, int64_t out_ld, int B,
                              int H, int Sq, int Sk, float scale, int h_norm, int dtype, bool clear_out,
                              int max_clusters, int* status, const int* fmt_word, cudaStream_t stream) {
    if (clear_out) {
        const int rc = launch_clear(out, out_ld, B, Sk, stream);
        if (rc != FCS_OK) return rc;
    }
    SinglePassParams sp_;
    memset(&sp_, 0, sizeof(sp_));
    sp_.B = B; sp_.H = H; sp_.Sq = Sq; sp_.Sk = Sk;
    sp_.NQ = (Sq + TILE - 1) / TILE;
    sp_.CL = single_pass_cluster_size(Sk);
    sp_.units = B * H;
    // the (batch, head, query tile) list is cut evenly over the clusters, through pairs if need be
    {
        const long long tiles = (long long)sp_.units * sp_.NQ;
        sp_.clusters = tiles < max_clusters ? (int)tiles : max_clusters;
    }
    // at most 1024 accumulations (16 query rows each) per flush: NQ is 16 at most, since every entry point that comes
    // here has as many keys as queries (or fewer rows that enter the mean)
    sp_.flush_units = 128 / sp_.NQ > 1 ? 128 / sp_.NQ : 1;
    // (a scale of zero under a ragged end as the smallest number there is: every fp32 score times it is below 5e-7
    // in size, and the -inf of a column of padding stays -inf)
    sp_.c = fmaxf(fabsf(scale) * 1.4426950408889634f, Sk % 64 ? 1.4e-45f : 0.f);
    sp_.out_scale = 1.0f / ((float)h_norm * (float)Sq * 1024.0f);
    sp_.out = out;
    sp_.out_ld = out_ld;
    sp_.status = status;
    sp_.fmt = fmt_word;
    const uint32_t fmt = dtype == FCS_DTYPE_BF16 ? 1u : 0u;
    // a score MMA covers half the 256 keys of the slice: M = 128, N = 128
    sp_.idesc_scores = (1u << 4) | (fmt << 7) | (fmt << 10) | ((scale < 0.f ? 1u : 0u) << 13) |
                       ((uint32_t)((BLOCK / 2) >> 3) << 17) | ((uint32_t)(TILE >> 4) << 24);
    // fp16 x fp16 -> fp32, A and B stored with the M and N index contiguous, M = 128, N = 16
    sp_.idesc_colsum = (1u << 4) | (1u << 15) | (1u << 16) | ((uint32_t)(sp::W_N >> 3) << 17) | ((uint32_t)(TILE >> 4) << 24);
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = dim3((unsigned)(sp_.clusters * sp_.CL));
    cfg.blockDim = dim3(sp::THREADS);
    cfg.dynamicSmemBytes = sp::DYN_BYTES;
    cfg.stream = stream;
    cudaLaunchAttribute attrs[2];
    attrs[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attrs[0].val.programmaticStreamSerializationAllowed = overlap_previous() ? 1 : 0;
    attrs[1].id = cudaLaunchAttributeClusterDimension;
    attrs[1].val.clusterDim.x = (unsigned)sp_.CL;
    attrs[1].val.clusterDim.y = 1;
    attrs[1].val.clusterDim.z = 1;
    cfg.attrs = attrs;
    cfg.numAttrs = sp_.CL > 1 ? 2 : 1;      // (the instance for one CTA has no cluster instruction)
    const SinglePassKernel kern = Sk % 64 ? single_pass_kernel<true>(sp_.CL) : single_pass_kernel<false>(sp_.CL);
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, tq, tk, sp_);
    if (e != cudaSuccess) return fail(FCS_ERR_CUDA, "single-pass kernel launch failed: %s", cudaGetErrorString(e));
    return FCS_OK;
}

// Short query axis over a short key axis: the one-kernel cluster form.
// g_short_fused: 0 = where fused_short_plan says so, 1 = never, 2 = whenever the query
// rows fit one tile.
static int g_short_fused = 0;

// Clusters of 1..8 CTAs of the one-kernel form that the current device runs at once
// (table[c]; fewer than SMs / c: a cluster stays inside one GPC).  Without a device to ask,
// seven eighths of SMs / c, which is what a B200 answers for clusters of four and of eight.
template <int D>
static const int* fused_short_max_clusters() {
    static int cached[64][fused::MAX_CL + 1] = {{0}};
    static int fallback[fused::MAX_CL + 1];
    int dev = 0;
    const bool have_dev = cudaGetDevice(&dev) == cudaSuccess && dev >= 0 && dev < 64;
    if (!have_dev) cudaGetLastError();
    const int sms = num_sms();
    int* table = have_dev ? cached[dev] : fallback;
    if (have_dev && table[1] != 0) return table;
    auto kern = fused::colsum_fused_short_kernel<D>;
    bool ask = have_dev && cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                fused::FLayout<D>::DYN_BYTES) == cudaSuccess;
    for (int cl = 1; cl <= fused::MAX_CL; ++cl) {
        int n = 0;
        if (ask) {
            cudaLaunchConfig_t cfg;
            memset(&cfg, 0, sizeof(cfg));
            cfg.gridDim = dim3((unsigned)(cl * 64));
            cfg.blockDim = dim3(THREADS);
            cfg.dynamicSmemBytes = fused::FLayout<D>::DYN_BYTES;
            cudaLaunchAttribute attr;
            attr.id = cudaLaunchAttributeClusterDimension;
            attr.val.clusterDim.x = (unsigned)cl;
            attr.val.clusterDim.y = 1;
            attr.val.clusterDim.z = 1;
            cfg.attrs = &attr;
            cfg.numAttrs = 1;
            if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess || n <= 0) {
                cudaGetLastError();
                n = 0;
            }
        }
        if (n <= 0) n = cl == 1 ? sms : (sms / cl) * 7 / 8;
        table[cl] = n > 0 ? n : 1;
    }
    return table;
}

static bool short_fused_applies(int B, int H, int Sq, int Sk, int D, int causal, int k_past, int* cl_out,
                                int* nkb_out, int* bpc_out) {
    if (g_short_fused == 1) return false;
    if (causal && k_past < 0) k_past = Sk > Sq ? Sk - Sq : 0;
    const int* table = D <= 64 ? fused_short_max_clusters<64>() : fused_short_max_clusters<128>();
    return fused_short_plan(B, H, Sq, Sk, causal, causal ? k_past : 0, num_sms(), table, g_short_fused == 2, cl_out,
                            nkb_out, bpc_out);
}

// Whether all (batch, head) pairs of a call the one-kernel form takes run at once: such a call
// goes there even where the single-pass kernel would take it (B=4 H=16, 100 CLS rows over 577
// keys: 11.9 against 12.6 us, 20 rows 10.5 / 11.9, 8 x 16 x 577 a tie at 14); with several waves of CTAs the
// single-pass kernel keeps it (B=32: 31 against 51 us).  (8 x 16 x 256, 64 rows: 8.4 here, 7.3 there; as with
// the line above, this form's exps keep 32 bits.)
static bool short_fused_one_wave(int B, int H, int D, int cl) {
    const int* table = D <= 64 ? fused_short_max_clusters<64>() : fused_short_max_clusters<128>();
    return (long long)B * H <= (cl > 1 ? table[cl] : num_sms());
}

template <int D>
static cudaError_t launch_fused_short_d(const CUtensorMap& tq, const CUtensorMap& tk, const fused::Params& fp,
                                        cudaStream_t stream) {
    using LayoutT = fused::FLayout<D>;
    static bool configured[64] = {false};
    int dev = 0;
    cudaGetDevice(&dev);
    auto kern = fused::colsum_fused_short_kernel<D>;
    if (dev >= 0 && dev < 64 && !configured[dev]) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, LayoutT::DYN_BYTES);
        if (e != cudaSuccess) return e;
        configured[dev] = true;
    }
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = dim3((unsigned)((long long)fp.p.B * fp.p.H * fp.CL));
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = LayoutT::DYN_BYTES;
    cfg.stream = stream;
    // (the cluster attribute also for clusters of one: the kernel uses cluster instructions)
    cudaLaunchAttribute attrs[2];
    attrs[0].id = cudaLaunchAttributeClusterDimension;
    attrs[0].val.clusterDim.x = (unsigned)fp.CL;
    attrs[0].val.clusterDim.y = 1;
    attrs[0].val.clusterDim.z = 1;
    attrs[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attrs[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attrs;
    cfg.numAttrs = overlap_previous() ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, kern, tq, tk, fp);
}

// `p` carries the sizes, the mask rule, the scale and the output; tq: boxes of 128 query rows,
// tk: boxes of 256 key rows.
static int launch_fused_short(const CUtensorMap& tq, const CUtensorMap& tk, const Problem& p, int DK, float scale,
                              bool use_ext, int cl, int nkb, int bpc, bool clear_out, float* clear_extra,
                              long long clear_extra_n, cudaStream_t stream) {
    int rc;
    if (clear_extra && (rc = launch_clear(clear_extra, clear_extra_n, 1, clear_extra_n, stream)) != FCS_OK) return rc;
    if (clear_out && (rc = launch_clear(p.out, p.out_ld, p.B, p.Sk, stream)) != FCS_OK) return rc;
    fused::Params fp;
    memset(&fp, 0, sizeof(fp));
    fp.p = p;
    fp.CL = cl;
    fp.nkb = nkb;
    fp.blocks_per_cta = bpc;
    fp.use_ext = use_ext ? 1 : 0;
    const uint32_t fmt = p.ext_bf16 ? 1u : 0u;
    const uint32_t common = (1u << 4) | (fmt << 7) | (fmt << 10) | ((scale < 0.f ? 1u : 0u) << 13) |
                            ((uint32_t)(TILE >> 4) << 24);
    fp.idesc_scores = common | ((uint32_t)(BLOCK >> 3) << 17);
    fp.idesc_cols = common | ((uint32_t)((BLOCK / 2) >> 3) << 17);
    const cudaError_t e = (DK == 64) ? launch_fused_short_d<64>(tq, tk, fp, stream)
                                     : launch_fused_short_d<128>(tq, tk, fp, stream);
    if (e != cudaSuccess) return fail(FCS_ERR_CUDA, "one-kernel short form launch failed: %s", cudaGetErrorString(e));
    return FCS_OK;
}

// fp32 operands rounded into `q16` / `k16` (dense [B][H][rows][D]); `fmt` receives the type.  `out` (or NULL): B rows
// of Sk values, out_ld apart, that are zeroed alongside.  `one_kernel_follows`: the call's kernels behind it are one.
static int launch_round_fp32(const float* q, const float* k, void* q16, void* k16, int* notes, int n_notes, int* fmt, float* out,
                             int64_t out_ld, bool one_kernel_follows, int B,
                             int H, int Sq, int Sk, int D, int64_t qsb, int64_t qsh, int64_t qss, int64_t ksb, int64_t ksh,
                             int64_t kss, cudaStream_t stream) {
    rnd::Params rp;
    memset(&rp, 0, sizeof(rp));
    auto operand = [&](rnd::Operand& o, const float* src, void* dst, int rows, int64_t sb, int64_t sh, int64_t ss) {
        o.src = src;
        o.dst = static_cast<uint16_t*>(dst);
        o.rows = (unsigned)rows;
        o.H = (unsigned)H;
        o.d8 = (unsigned)(D / 8);
        o.pieces = (unsigned)((long long)B * H * rows * (D / 8));
        o.sb = sb; o.sh = sh; o.ss = ss;
        o.dense = ss == D && sh == (int64_t)rows * D && sb == (int64_t)H * rows * D;
        return (long long)B * H * rows * (D / 8) <= 0xffffffffll;
    };
    if (!operand(rp.op[0], q, q16, Sq, qsb, qsh, qss) || !operand(rp.op[1], k, k16, Sk, ksb, ksh, kss))
        return fail(FCS_ERR_UNSUPPORTED, "fp32 operands of more than 2^35 elements are not supported");
    rp.notes = notes;
    rp.n_notes = n_notes;
    rp.fmt = fmt;
    rp.out = out;
    rp.out_ld = out_ld;
    rp.out_rows = (unsigned)B;
    rp.out_cols = (unsigned)Sk;
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof(cfg));
    cfg.stream = stream;
    cudaLaunchAttribute attrs[2];
    attrs[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attrs[0].val.programmaticStreamSerializationAllowed = 1;
    attrs[1].id = cudaLaunchAttributeClusterDimension;
    attrs[1].val.clusterDim.x = rnd::SMALL_CTAS;
    attrs[1].val.clusterDim.y = 1;
    attrs[1].val.clusterDim.z = 1;
    cudaError_t e;
    static int resident[64] = {0};
    if (round_in_one_kernel((long long)rp.op[0].pieces + rp.op[1].pieces, one_kernel_follows,
                            resident_clusters(reinterpret_cast<const void*>(rnd::round_small_kernel), rnd::SMALL_CTAS,
                                              rnd::SMALL_THREADS, 0, resident))) {
        cfg.gridDim = dim3(rnd::SMALL_CTAS);
        cfg.blockDim = dim3(rnd::SMALL_THREADS);
        cfg.attrs = overlap_previous() ? attrs : attrs + 1;
        cfg.numAttrs = overlap_previous() ? 2 : 1;
        e = cudaLaunchKernelEx(&cfg, rnd::round_small_kernel, rp);
    } else {
        cfg.gridDim = dim3((unsigned)n_notes);
        cfg.blockDim = dim3(rnd::THREADS);
        cfg.attrs = attrs;
        cfg.numAttrs = overlap_previous() ? 1 : 0;
        e = cudaLaunchKernelEx(&cfg, rnd::round_kernel, rp);
        if (e == cudaSuccess) e = cudaLaunchKernelEx(&cfg, rnd::settle_kernel, rp);
    }
    if (e != cudaSuccess) return fail(FCS_ERR_CUDA, "rounding fp32 operands failed: %s", cudaGetErrorString(e));
    return FCS_OK;
}

enum : int { PASSES_BOTH = 0, PASSES_STATS = 1, PASSES_COLUMNS = 2 };

// -(log-sum-exp) per query row -> the 16 extension columns the column pass contracts with.
__global__ void ext_from_lse_kernel(const Problem p) {
    const long long n = (long long)p.B * p.H * p.lse_rows;
    for (long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x; idx < n;
         idx += (long long)gridDim.x * blockDim.x) {
        uint4 e0, e1;
        make_ext_row(p.neg_lse[idx], p.inv_c, p.ext_bf16 != 0, e0, e1);
        uint4* er = reinterpret_cast<uint4*>(p.ext) + idx * 2;
        er[0] = e0;
        er[1] = e1;
    }
}

// The one implementation behind the three entry points.
static int colsum_impl(const void* q, const void* k, float* out, int64_t out_ld, int B, int H, int Sq_full,
                       int Sk, int D, int dtype, int64_t qsb, int64_t qsh, int64_t qss, int64_t ksb,
                       int64_t ksh, int64_t kss, float scale, int causal, int k_past, int cls_n, int h_norm,
                       void* workspace, size_t workspace_bytes, int* status, void* stream_v,
                       bool clear_out = true, int passes = PASSES_BOTH, float* shared_lse = nullptr,
                       long long norm_rows = 0, float* clear_extra = nullptr, long long clear_extra_n = 0,
                       const FcsPeerSignals* sig = nullptr, void* (*alloc)(void*, size_t) = nullptr,
                       void* alloc_ctx = nullptr) {
    // passes: both, or one of the two for work split over devices (non-causal only) --
    // PASSES_STATS writes -(log-sum-exp + log2(h_norm * norm_rows)) of the given query rows to
    // `shared_lse`; PASSES_COLUMNS takes that vector for ALL query rows and the given keys.
    // Scratch is `workspace`, or without one what `alloc` returns for the bytes the call needs.
    g_err[0] = 0;
    if (B <= 0 || H <= 0 || Sq_full <= 0 || Sk <= 0)
        return fail(FCS_ERR_INVALID_ARGUMENT, "sizes must be positive (B=%d H=%d Sq=%d Sk=%d)", B, H, Sq_full, Sk);
    if (!head_dim_ok(D))
        return fail(FCS_ERR_UNSUPPORTED, "head dimension must be a multiple of 8 from 8 to 128, got %d", D);
    if (dtype != FCS_DTYPE_FP16 && dtype != FCS_DTYPE_BF16 && !(dtype == FCS_DTYPE_FP32 && alloc))
        return fail(FCS_ERR_UNSUPPORTED, "dtype must be FCS_DTYPE_FP16 or FCS_DTYPE_BF16, got %d", dtype);
    const int DK = D <= 64 ? 64 : 128;   // columns the streaming kernels contract (zero-filled beyond D)
    if (passes != PASSES_STATS) {
        if (!out) return fail(FCS_ERR_INVALID_ARGUMENT, "out is NULL");
        if (out_ld < Sk)
            return fail(FCS_ERR_INVALID_ARGUMENT, "out_ld (%lld) is smaller than the key length", (long long)out_ld);
    }
    if (passes != PASSES_BOTH) {
        if (causal) return fail(FCS_ERR_UNSUPPORTED, "the passes can be run apart for non-causal calls only");
        if (!shared_lse || reinterpret_cast<uintptr_t>(shared_lse) % 16)
            return fail(FCS_ERR_INVALID_ARGUMENT, "the statistics vector must be a 16-byte aligned device pointer");
    }
    if (!isfinite(scale)) return fail(FCS_ERR_INVALID_ARGUMENT, "scale must be finite");
    if (!causal && cls_n != -1 && cls_n <= 0)
        return fail(FCS_ERR_INVALID_ARGUMENT, "cls_n must be -1 or positive, got %d", cls_n);
    int rc;
    const int granule = dtype == FCS_DTYPE_FP32 ? 4 : 8;   // 16 bytes
    if ((rc = check_operand("q", q, qsb, qsh, qss, granule)) != FCS_OK) return rc;
    if ((rc = check_operand("k", k, ksb, ksh, kss, granule)) != FCS_OK) return rc;
    if (h_norm <= 0) h_norm = H;

    int Sq = Sq_full;                       // rows that enter the mean
    if (!causal && cls_n > 0 && cls_n < Sq_full) Sq = cls_n;
    if (causal && k_past < 0) k_past = Sk > Sq ? Sk - Sq : 0;
    if (causal && k_past > Sk) k_past = Sk;   // (every row sees every key; the kernels add the row index in 32 bits)

    cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_v);
    if (passes == PASSES_BOTH && !sig && alloc && clear_out && Sq <= few::MAX_ROWS) {
        // reported as a call whose statistics and merge passes take no time
        PassTimers* tms = g_profiling ? timers_for_current_device() : nullptr;
        if (tms) {
            tms->recorded = false;
            for (int i = 0; i < 3; ++i) cudaEventRecord(tms->ev[i], stream);
        }
        rc = launch_few_rows(q, k, out, out_ld, B, H, Sq, Sk, D, dtype, qsb, qsh, qss, ksb, ksh, kss, scale, causal,
                             k_past, h_norm, status, stream, alloc, alloc_ctx);
        if (rc == FCS_OK && tms) { cudaEventRecord(tms->ev[3], stream); tms->recorded = true; }
        return rc;
    }
    const int* fmt_word = nullptr;
    bool to_clear = clear_out;     // the output still has to be zeroed
    if (dtype == FCS_DTYPE_FP32) {
        // one allocation: the type, the notes, both operands
        const long long pieces = (long long)B * H * ((long long)Sq + Sk) * (D / 8);
        long long notes = (pieces + rnd::THREADS - 1) / rnd::THREADS;
        if (notes > 8ll * num_sms()) notes = 8ll * num_sms();
        const size_t head = align_up((size_t)(notes + 1) * sizeof(int), 256);
        const size_t q_bytes = align_up((size_t)B * H * Sq * D * 2, 256), k_bytes = (size_t)B * H * Sk * D * 2;
        uint8_t* ws = static_cast<uint8_t*>(alloc(alloc_ctx, head + q_bytes + k_bytes));
        if (!ws) return fail(FCS_ERR_WORKSPACE, "no scratch memory for the rounded fp32 operands");
        int* words = reinterpret_cast<int*>(ws);
        const bool one_kernel = passes == PASSES_BOTH &&
                                (single_pass_applies(B, H, Sq, Sk, D, causal) ||
                                 (!sig && short_fused_applies(B, H, Sq, Sk, D, causal, k_past, nullptr, nullptr, nullptr)));
        rc = launch_round_fp32(static_cast<const float*>(q), static_cast<const float*>(k), ws + head, ws + head + q_bytes,
                               words + 1, (int)notes, words, passes == PASSES_BOTH && clear_out ? out : nullptr, out_ld,
                               one_kernel, B, H, Sq, Sk, D, qsb, qsh, qss, ksb, ksh, kss, stream);
        if (rc != FCS_OK) return rc;
        to_clear = false;
        q = ws + head;
        k = ws + head + q_bytes;
        qss = kss = D;
        qsh = (int64_t)Sq * D; qsb = qsh * H;
        ksh = (int64_t)Sk * D; ksb = ksh * H;
        dtype = FCS_DTYPE_FP16;
        fmt_word = words;
    }
    if (sig && passes == PASSES_BOTH && smallq_fits(Sq, Sk, D, B * H, num_sms()))
        return fail(FCS_ERR_UNSUPPORTED, "calls with at most four query rows take the few-row kernel, which does not "
                                         "signal other GPUs; order them with a barrier");
    // (a type that is decided on the device is known to the kernels below this one only)
    if (passes == PASSES_BOTH && !fmt_word && smallq_fits(Sq, Sk, D, B * H, num_sms())) {
        // reported as a call whose statistics and merge passes take no time
        PassTimers* tms = g_profiling ? timers_for_current_device() : nullptr;
        if (tms) {
            tms->recorded = false;
            for (int i = 0; i < 3; ++i) cudaEventRecord(tms->ev[i], stream);
        }
        if (clear_extra && (rc = launch_clear(clear_extra, clear_extra_n, 1, clear_extra_n, stream)) != FCS_OK) return rc;
        rc = launch_small_q(q, k, out, out_ld, B, H, Sq, Sk, D, dtype, qsb, qsh, qss, ksb, ksh, kss, scale,
                            causal, k_past, h_norm, clear_out, status, stream);
        if (rc == FCS_OK && tms) { cudaEventRecord(tms->ev[3], stream); tms->recorded = true; }
        return rc;
    }

    const int sms = num_sms();
    // -(lse) rides in the MMA of the column pass unless the scale is so small that
    // -(lse)/c leaves the range of its 16-bit parts
    const bool use_ext = fabsf(scale) * 1.4426950408889634f >= 1e-4f;
    Problem p;
    memset(&p, 0, sizeof(p));
    plan(p, B, H, Sq, Sk, causal, k_past, sms, COL_INTERLEAVE_MIN_ROWS, /*head_major_ok=*/use_ext);
    p.ext_bf16 = dtype == FCS_DTYPE_BF16 ? 1 : 0;
    p.fmt = fmt_word;
    p.out = out;
    p.out_ld = out_ld;
    p.clear_out = (to_clear && passes == PASSES_BOTH) ? 1 : 0;   // (the statistics pass does the clearing)
    p.col_combine = clear_out ? 0 : 1;   // accumulating into a caller's buffer: it may be peer-mapped
    p.clear_extra = clear_extra_n > 0 ? clear_extra : nullptr;
    p.clear_extra_n = clear_extra_n;
    p.status = status;
    p.c = fabsf(scale) * 1.4426950408889634f;
    p.inv_c = use_ext ? (scale < 0.f ? -1.0f : 1.0f) / p.c : 0.f;
    p.log2_norm = log2f((float)h_norm * (float)(norm_rows > 0 ? norm_rows : Sq));
    const uint32_t fmt = dtype == FCS_DTYPE_BF16 ? 1u : 0u;
    // fp32 accumulate, K-major A and B, M = 128, N = 256; a negative scale negates A
    p.idesc = (1u << 4) | (fmt << 7) | (fmt << 10) | ((scale < 0.f ? 1u : 0u) << 13) |
              ((uint32_t)(BLOCK >> 3) << 17) | ((uint32_t)(TILE >> 4) << 24);

    // each tensor is the resident operand (128-row boxes) of one pass and the
    // streamed operand (256-row boxes) of the other
    // (the two cluster kernels take queries in 128-row and keys in 256-row boxes only: the other two
    // maps are encoded once it is known that the streaming passes run -- an encode is a microsecond
    // of host time, and the calls the cluster kernels take are bound by the host when issued back to back)
    CUtensorMap tq_a, tq_b, tk_a, tk_b;
    if ((rc = make_tensor_map(&tq_a, q, dtype, B, H, Sq, D, qsb, qsh, qss, TILE)) != FCS_OK) return rc;
    if ((rc = make_tensor_map(&tk_b, k, dtype, B, H, Sk, D, ksb, ksh, kss, BLOCK)) != FCS_OK) return rc;
    int fcl = 0, fnkb = 0, fbpc = 0;
    const bool fused_ok = passes == PASSES_BOTH && !sig && short_fused_applies(B, H, Sq, Sk, D, causal, k_past, &fcl, &fnkb, &fbpc);
    const bool fused_first = fused_ok && short_fused_one_wave(B, H, D, fcl);
    if (passes == PASSES_BOTH && !fused_first && single_pass_applies(B, H, Sq, Sk, D, causal)) {
        const int max_clusters = single_pass_max_clusters(single_pass_cluster_size(Sk));
        if (max_clusters > 0) {
            // reported as a call whose statistics and merge passes take no time
            PassTimers* tms = g_profiling ? timers_for_current_device() : nullptr;
            if (tms) {
                tms->recorded = false;
                for (int i = 0; i < 3; ++i) cudaEventRecord(tms->ev[i], stream);
            }
            rc = launch_single_pass(tq_a, tk_b, out, out_ld, B, H, Sq, Sk, scale, h_norm, dtype, to_clear,
                                    max_clusters, status, fmt_word, stream);
            if (rc == FCS_OK && tms) { cudaEventRecord(tms->ev[3], stream); tms->recorded = true; }
            return rc;
        }
    }
    {
        if (fused_ok) {
            // reported as a call whose statistics and merge passes take no time
            PassTimers* tms = g_profiling ? timers_for_current_device() : nullptr;
            if (tms) {
                tms->recorded = false;
                for (int i = 0; i < 3; ++i) cudaEventRecord(tms->ev[i], stream);
            }
            rc = launch_fused_short(tq_a, tk_b, p, DK, scale, use_ext, fcl, fnkb, fbpc, to_clear, clear_extra,
                                    clear_extra_n, stream);
            if (rc == FCS_OK && tms) { cudaEventRecord(tms->ev[3], stream); tms->recorded = true; }
            return rc;
        }
    }
    if ((rc = make_tensor_map(&tq_b, q, dtype, B, H, Sq, D, qsb, qsh, qss, BLOCK)) != FCS_OK) return rc;
    if ((rc = make_tensor_map(&tk_a, k, dtype, B, H, Sk, D, ksb, ksh, kss, TILE)) != FCS_OK) return rc;
    // the two streaming passes are the only kernels that use scratch memory
    size_t part_off = 0, ext_off = 0;
    const size_t need = workspace_layout(p, &part_off, &ext_off);
    if (!workspace && alloc) {
        workspace = alloc(alloc_ctx, need);
        workspace_bytes = workspace ? need : 0;
    }
    if (!workspace || workspace_bytes < need)
        return fail(FCS_ERR_WORKSPACE, "workspace too small: need %zu bytes, got %zu", need, workspace_bytes);
    if (reinterpret_cast<uintptr_t>(workspace) % 256)
        return fail(FCS_ERR_WORKSPACE, "workspace must be 256-byte aligned");
    p.neg_lse = passes == PASSES_BOTH ? reinterpret_cast<float*>(workspace) : shared_lse;
    p.part = reinterpret_cast<uint8_t*>(workspace) + part_off;
    p.ext = reinterpret_cast<uint8_t*>(workspace) + ext_off;
    CUtensorMap text = tq_b;   // placeholder when the extension is not used
    if (use_ext && (rc = make_ext_tensor_map(&text, p.ext, dtype, (long long)B * H, p.lse_rows)) != FCS_OK) return rc;

    const int grid1 = (int)(p.stats_items < sms ? p.stats_items : sms);
    stats_set_grid(p, grid1);
    long long col_items = p.steps_total;
    if (p.col_interleave == COL_HEAD_MAJOR) col_items = (long long)B * H * ceil_div(p.NKC, p.col_pack);
    const int grid2 = (int)(col_items < sms ? col_items : sms);
    PassTimers* tm = g_profiling ? timers_for_current_device() : nullptr;
    if (tm) { tm->recorded = false; cudaEventRecord(tm->ev[0], stream); }
    cudaError_t e = cudaSuccess;
    if (passes == PASSES_COLUMNS) {
        // the caller's statistics -> the column pass's operand form; the output starts from zero
        int blocks = (int)(((long long)B * H * p.lse_rows + 255) / 256);
        if (blocks > sms * 8) blocks = sms * 8;
        ext_from_lse_kernel<<<blocks, 256, 0, stream>>>(p);
        e = cudaGetLastError();
        if (e == cudaSuccess && clear_out)
            e = cudaMemset2DAsync(out, (size_t)out_ld * sizeof(float), 0, (size_t)Sk * sizeof(float), (size_t)B, stream);
        if (e != cudaSuccess) return fail(FCS_ERR_CUDA, "preparing the column pass failed: %s", cudaGetErrorString(e));
    } else {
        e = (DK == 64) ? launch_stream<64, MODE_STATS>(tq_a, tk_b, text, p, grid1, stream, !tm)
                      : launch_stream<128, MODE_STATS>(tq_a, tk_b, text, p, grid1, stream, !tm);
    }
    if (e != cudaSuccess) return fail(FCS_ERR_CUDA, "statistics pass launch failed: %s", cudaGetErrorString(e));
    if (tm) cudaEventRecord(tm->ev[1], stream);
    if (p.nsplit > 1 && passes != PASSES_COLUMNS) {
        const long long n = (long long)B * H * p.NQ * TILE;
        int blocks = (int)((n + 255) / 256);
        if (blocks > sms * 8) blocks = sms * 8;
        cudaLaunchConfig_t cfg;
        memset(&cfg, 0, sizeof(cfg));
        cfg.gridDim = dim3((unsigned)blocks);
        cfg.blockDim = dim3(256);
        cfg.stream = stream;
        cudaLaunchAttribute attr;
        attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr.val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = &attr;
        cfg.numAttrs = tm ? 0 : 1;   // (event records between the kernels when timing is on)
        e = cudaLaunchKernelEx(&cfg, merge_stats_kernel, p);
        if (e != cudaSuccess) return fail(FCS_ERR_CUDA, "statistics merge launch failed: %s", cudaGetErrorString(e));
    }
    if (tm) cudaEventRecord(tm->ev[2], stream);
    if (passes == PASSES_STATS) {
        if (tm) { cudaEventRecord(tm->ev[3], stream); tm->recorded = true; }
        return FCS_OK;
    }
    const bool chained = !tm;
    // a query axis of at most 128 rows fills half a streamed block: the MMAs need N = 128 only
    if (Sq <= BLOCK / 2)
        p.idesc = (p.idesc & ~(0x3Fu << 17)) | ((uint32_t)((BLOCK / 2) >> 3) << 17);
    if (sig) {   // the column pass orders itself against the other GPUs of a head-sharded call
        p.sig_wait = sig->wait_flag;
        p.sig_wait_value = sig->wait_value;
        p.sig_post_n = sig->post_n;
        p.sig_post_value = sig->post_value;
        for (int i = 0; i < sig->post_n; ++i) p.sig_post[i] = sig->post[i];
        p.sig_counter = sig->counter;
        p.sig_done = sig->done_flag;
        p.sig_done_value = sig->done_value;
    }
    const bool head_major = use_ext && p.col_interleave == COL_HEAD_MAJOR;
    if (head_major && p.col_combine && p.NQB == 2)
        e = (DK == 64) ? launch_stream<64, MODE_COLSUM_EXT_SHORT2_COMBINE>(tk_a, tq_b, text, p, grid2, stream, chained)
                      : launch_stream<128, MODE_COLSUM_EXT_SHORT2_COMBINE>(tk_a, tq_b, text, p, grid2, stream, chained);
    else if (head_major && p.col_combine)
        e = (DK == 64) ? launch_stream<64, MODE_COLSUM_EXT_SHORT_COMBINE>(tk_a, tq_b, text, p, grid2, stream, chained)
                      : launch_stream<128, MODE_COLSUM_EXT_SHORT_COMBINE>(tk_a, tq_b, text, p, grid2, stream, chained);
    else if (head_major && p.NQB == 2)   // two resident query blocks per head
        e = (DK == 64) ? launch_stream<64, MODE_COLSUM_EXT_SHORT2>(tk_a, tq_b, text, p, grid2, stream, chained)
                      : launch_stream<128, MODE_COLSUM_EXT_SHORT2>(tk_a, tq_b, text, p, grid2, stream, chained);
    else if (head_major)   // one query block per head, many key tiles: the key tiles stream
        e = (DK == 64) ? launch_stream<64, MODE_COLSUM_EXT_SHORT>(tk_a, tq_b, text, p, grid2, stream, chained)
                      : launch_stream<128, MODE_COLSUM_EXT_SHORT>(tk_a, tq_b, text, p, grid2, stream, chained);
    else if (use_ext)
        e = (DK == 64) ? launch_stream<64, MODE_COLSUM_EXT>(tk_a, tq_b, text, p, grid2, stream, chained)
                      : launch_stream<128, MODE_COLSUM_EXT>(tk_a, tq_b, text, p, grid2, stream, chained);
    else
        e = (DK == 64) ? launch_stream<64, MODE_COLSUM>(tk_a, tq_b, text, p, grid2, stream, chained)
                      : launch_stream<128, MODE_COLSUM>(tk_a, tq_b, text, p, grid2, stream, chained);
    if (e != cudaSuccess) return fail(FCS_ERR_CUDA, "column pass launch failed: %s", cudaGetErrorString(e));
    if (tm) { cudaEventRecord(tm->ev[3], stream); tm->recorded = true; }
    return FCS_OK;
}

// ---------------------------------------------------------------------------
// Pruning step (select_topk.cuh): rows of at most 1024 elements take CTAs of 256 threads with
// four elements each and 8-bit digits, longer ones 1024 threads with as few of 4, 8 or 16 elements
// as hold a CTA's slice (a thread's elements are consecutive: with more, whole warps would have none).
// ---------------------------------------------------------------------------
template <typename... Params, typename... Args>
static cudaError_t launch_row_clusters(void (*kern)(Params...), int smem, bool (&configured)[64], int B, int cl,
                                       int threads, cudaStream_t stream, Args... args) {
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 0 && dev < 64 && !configured[dev]) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
        if (e != cudaSuccess) return e;
        configured[dev] = true;
    }
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = dim3((unsigned)((long long)B * cl));
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = (size_t)smem;
    cfg.stream = stream;
    cudaLaunchAttribute attrs[2];
    attrs[0].id = cudaLaunchAttributeClusterDimension;
    attrs[0].val.clusterDim.x = (unsigned)cl;
    attrs[0].val.clusterDim.y = 1;
    attrs[0].val.clusterDim.z = 1;
    // the set-up may overlap the end of the kernel that produced the means; it is waited for inside
    attrs[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attrs[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attrs;
    cfg.numAttrs = 2;
    return cudaLaunchKernelEx(&cfg, kern, Params(args)...);
}

template <int NT, int E, int BITS, int CL>
static cudaError_t launch_topk_t(const float* colsum, long long ld, int B, int S, int k, int* indices, float* values,
                                 cudaStream_t stream) {
    static bool configured[64] = {false};
    return launch_row_clusters(sel::topk_kernel<NT, E, BITS, CL>, sel::topk_smem<NT, E, BITS, CL>(), configured, B, CL, NT,
                               stream, colsum, ld, S, k, indices, values);
}
static cudaError_t launch_topk(const float* colsum, long long ld, int B, int S, int k, int* indices, float* values,
                               cudaStream_t stream) {
    const int cl = sel::cluster_size(S);
    static int resident[64] = {0};
    const bool wide = topk_on_sixteen(S, B, 16) &&
                      topk_on_sixteen(S, B, resident_clusters(reinterpret_cast<const void*>(sel::topk_kernel<1024, 8, 11, 16>),
                                                              16, 1024, sel::topk_smem<1024, 8, 11, 16>(), resident));
#define FCS_TOPK(NT, E, BITS, CL) return launch_topk_t<NT, E, BITS, CL>(colsum, ld, B, S, k, indices, values, stream)
    if (S <= 1024) FCS_TOPK(256, 4, 8, 1);
    if (cl == 1) FCS_TOPK(1024, 4, 11, 1);
    if (cl == 2) FCS_TOPK(1024, 4, 11, 2);
    if (cl == 4) FCS_TOPK(1024, 4, 11, 4);
    if (cl == 8 && S <= 8 * 4096) FCS_TOPK(1024, 4, 11, 8);
    if (cl == 8 && S <= 8 * 8192) FCS_TOPK(1024, 8, 11, 8);
    if (wide) FCS_TOPK(1024, 8, 11, 16);
    if (cl == 8) FCS_TOPK(1024, 16, 11, 8);
    FCS_TOPK(1024, 16, 11, 16);
#undef FCS_TOPK
}

template <int NT, int E, int CL>
static cudaError_t launch_threshold_t(const float* colsum, long long ld, int B, int S, float threshold, int relative,
                                      int* indices, int* counts, cudaStream_t stream) {
    static bool configured[64] = {false};
    return launch_row_clusters(sel::threshold_kernel<NT, E, CL>, sel::stage_bytes<NT, E>(), configured, B, CL, NT, stream,
                               colsum, ld, S, threshold, relative, indices, counts);
}
static cudaError_t launch_threshold(const float* colsum, long long ld, int B, int S, float threshold, int relative,
                                    int* indices, int* counts, cudaStream_t stream) {
    const int cl = sel::cluster_size(S);
#define FCS_THRESHOLD(NT, E, CL) \
    return launch_threshold_t<NT, E, CL>(colsum, ld, B, S, threshold, relative, indices, counts, stream)
    if (S <= 1024) FCS_THRESHOLD(256, 4, 1);
    if (cl == 1) FCS_THRESHOLD(1024, 4, 1);
    if (cl == 2) FCS_THRESHOLD(1024, 4, 2);
    if (cl == 4) FCS_THRESHOLD(1024, 4, 4);
    if (cl == 8 && S <= 8 * 4096) FCS_THRESHOLD(1024, 4, 8);
    if (cl == 8 && S <= 8 * 8192) FCS_THRESHOLD(1024, 8, 8);
    if (cl == 8) FCS_THRESHOLD(1024, 16, 8);
    FCS_THRESHOLD(1024, 16, 16);
#undef FCS_THRESHOLD
}

// ---------------------------------------------------------------------------
// Host-memory calls: the operands are copied in chunks on a stream of their own while the chunk before is
// computed.  The copies bound the call (64 MiB at 54 GB/s: 1.23 ms, against 0.27 ms of kernels), so that the
// chunks are few and large at first and small at the end: three quarters of the batch entries that are left,
// and the last entry by heads (whose sums are added up on the device), down to chunks of 2 MiB (40 us; 1 MiB
// and 4 MiB: the 8 x 16 x 2048 call 1335 and 1304 us against 1303, 64 x 16 x 512 2518 and 2523 against 2509).
// ---------------------------------------------------------------------------
constexpr size_t HOST_CHUNK_MIN_BYTES = 2u << 20;

static cudaStream_t host_copy_stream() {
    static cudaStream_t streams[64] = {nullptr};
    static std::mutex mutex;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return nullptr;
    std::lock_guard<std::mutex> lock(mutex);
    if (!streams[dev] && cudaStreamCreateWithFlags(&streams[dev], cudaStreamNonBlocking) != cudaSuccess) streams[dev] = nullptr;
    return streams[dev];
}

struct HostChunk { int b0, nb, h0, nh; };

// (`whole`: no entry is cut -- calls with at most four query rows, whose kernels take a hundredth of the copies'
// time and write the columns instead of adding to them)
static std::vector<HostChunk> host_chunks(int B, int H, size_t pair_bytes, int batch_chunk, bool whole) {
    std::vector<HostChunk> out;
    if (batch_chunk > 0) {
        for (int b = 0; b < B; b += batch_chunk) out.push_back({b, B - b < batch_chunk ? B - b : batch_chunk, 0, H});
        return out;
    }
    int b = 0;
    while (b < B - 1) {
        const int left = B - b;
        if ((size_t)left * H * pair_bytes <= HOST_CHUNK_MIN_BYTES) { out.push_back({b, left, 0, H}); return out; }
        const int n = left - (left / 4 > 1 ? left / 4 : 1);
        out.push_back({b, n, 0, H});
        b += n;
    }
    if (whole) {
        out.push_back({b, 1, 0, H});
        return out;
    }
    for (int h = 0; h < H;) {
        const int left = H - h;
        const bool last = left == 1 || (size_t)left * pair_bytes <= HOST_CHUNK_MIN_BYTES;
        const int n = last ? left : left - (left / 4 > 1 ? left / 4 : 1);
        out.push_back({b, 1, h, n});
        h += n;
    }
    return out;
}

static int run_host_call(const FcsHostCall* hc) {
    const FcsCall& c = hc->call;
    const size_t es = c.dtype == FCS_DTYPE_FP32 ? 4 : 2;
    const size_t q_pair = (size_t)c.Sq * c.D * es, k_pair = (size_t)c.Sk * c.D * es;
    cudaStream_t main = reinterpret_cast<cudaStream_t>(c.stream);
    const int rows = !c.causal && c.cls_n > 0 && c.cls_n < c.Sq ? c.cls_n : c.Sq;
    const std::vector<HostChunk> chunks = host_chunks(c.B, c.H, q_pair + k_pair, hc->batch_chunk, rows <= few::MAX_ROWS);
    // (one chunk: nothing to overlap, everything goes on the caller's stream)
    const bool overlap = chunks.size() > 1;
    cudaStream_t copy = overlap ? host_copy_stream() : main;
    if (overlap && !copy) return fail(FCS_ERR_CUDA, "no stream for the copies");
    std::vector<cudaEvent_t> events(overlap ? chunks.size() + 1 : 0, nullptr);
    cudaError_t e = cudaSuccess;
    for (auto& ev : events)
        if (e == cudaSuccess) e = cudaEventCreateWithFlags(&ev, cudaEventDisableTiming);
    // the device buffers may still be in use by earlier work of the caller's stream
    if (overlap && e == cudaSuccess) e = cudaEventRecord(events.back(), main);
    if (overlap && e == cudaSuccess) e = cudaStreamWaitEvent(copy, events.back(), 0);
    auto copy_in = [&](size_t i) {
        const HostChunk& ch = chunks[i];
        const size_t first = (size_t)ch.b0 * c.H + ch.h0, n = (size_t)ch.nb * ch.nh;
        auto bytes = [](const void* p, size_t off) { return static_cast<const uint8_t*>(p) + off; };
        if (e == cudaSuccess)
            e = cudaMemcpyAsync(const_cast<uint8_t*>(bytes(c.q, first * q_pair)), bytes(hc->host_q, first * q_pair), n * q_pair,
                                cudaMemcpyHostToDevice, copy);
        if (e == cudaSuccess)
            e = cudaMemcpyAsync(const_cast<uint8_t*>(bytes(c.k, first * k_pair)), bytes(hc->host_k, first * k_pair), n * k_pair,
                                cudaMemcpyHostToDevice, copy);
        if (overlap && e == cudaSuccess) e = cudaEventRecord(events[i], copy);
    };
    int rc = FCS_OK;
    if (e == cudaSuccess) copy_in(0);
    for (size_t i = 0; i < chunks.size() && e == cudaSuccess && rc == FCS_OK; ++i) {
        if (i + 1 < chunks.size()) copy_in(i + 1);     // (queued before the kernels of this chunk are)
        if (overlap && e == cudaSuccess) e = cudaStreamWaitEvent(main, events[i], 0);
        if (e != cudaSuccess) break;
        const HostChunk& ch = chunks[i];
        const size_t first = (size_t)ch.b0 * c.H + ch.h0;
        rc = colsum_impl(static_cast<const uint8_t*>(c.q) + first * q_pair, static_cast<const uint8_t*>(c.k) + first * k_pair,
                         c.out + (size_t)ch.b0 * c.out_ld, c.out_ld, ch.nb, ch.nh, c.Sq, c.Sk, c.D, c.dtype, c.q_stride[0],
                         c.q_stride[1], c.q_stride[2], c.k_stride[0], c.k_stride[1], c.k_stride[2], c.scale, c.causal, c.k_past,
                         c.cls_n, c.H, nullptr, 0, c.status, c.stream, /*clear_out=*/ch.h0 == 0, PASSES_BOTH, nullptr, 0, nullptr,
                         0, nullptr, c.alloc, c.alloc_ctx);
    }
    if (e == cudaSuccess && rc == FCS_OK)
        e = cudaMemcpyAsync(hc->host_out, c.out, (size_t)c.B * c.Sk * sizeof(float), cudaMemcpyDeviceToHost, main);
    // (also on the way out of an error: nothing of this call is left in flight over the caller's buffers)
    const cudaError_t e2 = overlap ? cudaStreamSynchronize(copy) : cudaSuccess, e3 = cudaStreamSynchronize(main);
    for (auto ev : events)
        if (ev) cudaEventDestroy(ev);
    if (rc != FCS_OK) return rc;
    if (e == cudaSuccess) e = e2 != cudaSuccess ? e2 : e3;
    if (e != cudaSuccess) return fail(FCS_ERR_CUDA, "host-memory call failed: %s", cudaGetErrorString(e));
    return FCS_OK;
}

// ---------------------------------------------------------------------------
// Built-in scratch for callers that have no device allocator to draw from.
// One copy lives in every device that loads this library, for the life of the
// process.  The name below is a host-side handle in host code, not a device
// address: the address is looked up per device with cudaGetSymbolAddress.
// ---------------------------------------------------------------------------
static __device__ __align__(256) unsigned char g_static_scratch[FCS_STATIC_SCRATCH_BYTES];

static int static_scratch_address(void** out_ptr) {
    static void* cached[64] = {nullptr};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return fail(FCS_ERR_CUDA, "cudaGetDevice failed: %s", cudaGetErrorString(e));
    if (dev < 0 || dev >= 64) return fail(FCS_ERR_UNSUPPORTED, "device ordinal %d is out of range", dev);
    if (!cached[dev]) {
        void* ptr = nullptr;
        e = cudaGetSymbolAddress(&ptr, g_static_scratch);
        if (e != cudaSuccess || !ptr)
            return fail(FCS_ERR_CUDA, "cudaGetSymbolAddress(static scratch) failed: %s", cudaGetErrorString(e));
        cached[dev] = ptr;
    }
    *out_ptr = cached[dev];
    return FCS_OK;
}

}  // namespace fcs

// ---------------------------------------------------------------------------
// C ABI
// ---------------------------------------------------------------------------
extern "C" {

int fcs_version(void) { return 202; }

const char* fcs_last_error(void) { return fcs::g_err; }

int fcs_set_profiling(int enabled) {
    fcs::g_profiling = enabled != 0;
    return FCS_OK;
}

int fcs_set_single_pass(int mode) {
    if (mode < 0 || mode > 2) return FCS_ERR_INVALID_ARGUMENT;
    fcs::g_single_pass = mode;
    return FCS_OK;
}

int fcs_set_short_fused(int mode) {
    if (mode < 0 || mode > 2) return FCS_ERR_INVALID_ARGUMENT;
    fcs::g_short_fused = mode;
    return FCS_OK;
}

int fcs_short_fused_applies(int B, int H, int sq_rows, int Sk, int D, int is_causal, int k_past, int* cluster_size,
                            int* blocks_per_cta) {
    if (B <= 0 || H <= 0 || sq_rows <= 0 || Sk <= 0 || !fcs::head_dim_ok(D)) return 0;
    int cl = 0, nkb = 0, bpc = 0;
    if (!fcs::short_fused_applies(B, H, sq_rows, Sk, D, is_causal ? 1 : 0, k_past, &cl, &nkb, &bpc)) return 0;
    if (cluster_size) *cluster_size = cl;
    if (blocks_per_cta) *blocks_per_cta = bpc;
    return 1;
}

int fcs_single_pass_applies(int B, int H, int sq_rows, int Sk, int D, int is_causal) {
    if (B <= 0 || H <= 0 || sq_rows <= 0 || Sk <= 0) return 0;
    return fcs::single_pass_applies(B, H, sq_rows, Sk, D, is_causal ? 1 : 0) ? 1 : 0;
}

int fcs_single_pass_info(int Sk, int* cluster_size, int* max_clusters) {
    if (Sk <= 0 || Sk > 256 * fcs::sp::MAX_CL) return FCS_ERR_UNSUPPORTED;
    const int cl = fcs::single_pass_cluster_size(Sk);
    if (cluster_size) *cluster_size = cl;
    if (max_clusters) *max_clusters = fcs::single_pass_max_clusters(cl);
    return FCS_OK;
}

int fcs_last_pass_ms(float* stats_ms, float* merge_ms, float* colsum_ms) {
    fcs::g_err[0] = 0;
    fcs::PassTimers* tm = fcs::timers_for_current_device();
    if (!tm || !tm->recorded)
        return fcs::fail(FCS_ERR_INVALID_ARGUMENT, "no profiled call has been made on this device");
    cudaError_t e = cudaEventSynchronize(tm->ev[3]);
    if (e != cudaSuccess) return fcs::fail(FCS_ERR_CUDA, "event synchronize failed: %s", cudaGetErrorString(e));
    float a = 0.f, b = 0.f, c = 0.f;
    cudaEventElapsedTime(&a, tm->ev[0], tm->ev[1]);
    cudaEventElapsedTime(&b, tm->ev[1], tm->ev[2]);
    cudaEventElapsedTime(&c, tm->ev[2], tm->ev[3]);
    if (stats_ms) *stats_ms = a;
    if (merge_ms) *merge_ms = b;
    if (colsum_ms) *colsum_ms = c;
    return FCS_OK;
}

int fcs_plan_info(int B, int H, int sq_rows, int Sk, int is_causal, int* nsplit, long long* stats_items,
                  long long* colsum_steps, int* sms) {
    if (B <= 0 || H <= 0 || sq_rows <= 0 || Sk <= 0) return FCS_ERR_INVALID_ARGUMENT;
    fcs::Problem p;
    memset(&p, 0, sizeof(p));
    const int k_past = Sk > sq_rows ? Sk - sq_rows : 0;
    const int n_sm = fcs::num_sms();
    fcs::plan(p, B, H, sq_rows, Sk, is_causal ? 1 : 0, k_past, n_sm);
    if (nsplit) *nsplit = p.nsplit;
    if (stats_items) *stats_items = p.stats_items;
    if (colsum_steps) *colsum_steps = p.steps_total;
    if (sms) *sms = n_sm;
    return FCS_OK;
}

size_t fcs_workspace_bytes(int B, int H, int sq_rows, int Sk, int D, int is_causal) {
    if (B <= 0 || H <= 0 || sq_rows <= 0 || Sk <= 0 || !fcs::head_dim_ok(D)) return 0;
    // An upper bound for every k_past and every kernel choice: the layout of the two streaming
    // passes with the key range of the statistics pass split as far as any k_past allows (the
    // split grows with the keys the first query tile sees, and k_past = Sk shows it all of them).
    fcs::Problem p;
    memset(&p, 0, sizeof(p));
    fcs::plan(p, B, H, sq_rows, Sk, is_causal ? 1 : 0, is_causal ? Sk : 0, fcs::num_sms());
    return fcs::workspace_layout(p, nullptr);
}

int fcs_call_workspace_bytes(int B, int H, int sq_rows, int Sk, int D, int is_causal, int k_past,
                             size_t* bytes) {
    fcs::g_err[0] = 0;
    if (!bytes) return fcs::fail(FCS_ERR_INVALID_ARGUMENT, "bytes is NULL");
    *bytes = 0;
    if (B <= 0 || H <= 0 || sq_rows <= 0 || Sk <= 0)
        return fcs::fail(FCS_ERR_INVALID_ARGUMENT, "sizes must be positive (B=%d H=%d Sq=%d Sk=%d)", B, H, sq_rows, Sk);
    if (!fcs::head_dim_ok(D))
        return fcs::fail(FCS_ERR_UNSUPPORTED, "head dimension must be a multiple of 8 from 8 to 128, got %d", D);
    const int causal = is_causal ? 1 : 0;
    // the same decisions, in the same order, as the call itself
    if (fcs::smallq_fits(sq_rows, Sk, D, B * H, fcs::num_sms()))
        return FCS_OK;   // few-row kernel: no scratch
    if (fcs::single_pass_applies(B, H, sq_rows, Sk, D, causal) &&
        fcs::single_pass_max_clusters(fcs::single_pass_cluster_size(Sk)) > 0)
        return FCS_OK;   // single-pass kernel: no scratch
    if (causal && k_past < 0) k_past = Sk > sq_rows ? Sk - sq_rows : 0;
    if (fcs::short_fused_applies(B, H, sq_rows, Sk, D, causal, k_past, nullptr, nullptr, nullptr))
        return FCS_OK;   // one-kernel short form: no scratch
    fcs::Problem p;
    memset(&p, 0, sizeof(p));
    fcs::plan(p, B, H, sq_rows, Sk, causal, causal ? k_past : 0, fcs::num_sms());
    *bytes = fcs::workspace_layout(p, nullptr);
    return FCS_OK;
}

int fcs_colsum_batched(const void* q, const void* k, float* out, int64_t out_ld, int B, int H, int S, int D,
                       int dtype, int64_t q_stride_b, int64_t q_stride_h, int64_t q_stride_s,
                       int64_t k_stride_b, int64_t k_stride_h, int64_t k_stride_s, float scale, int cls_n,
                       int h_norm, void* workspace, size_t workspace_bytes, int* status, void* stream) {
    return fcs::colsum_impl(q, k, out, out_ld, B, H, S, S, D, dtype, q_stride_b, q_stride_h, q_stride_s,
                            k_stride_b, k_stride_h, k_stride_s, scale, 0, 0, cls_n, h_norm, workspace,
                            workspace_bytes, status, stream);
}

int fcs_colsum_non_batched(const void* q, const void* k, float* out, int H, int S, int D, int dtype,
                           int64_t q_stride_h, int64_t q_stride_s, int64_t k_stride_h, int64_t k_stride_s,
                           float scale, int cls_n, int h_norm, void* workspace, size_t workspace_bytes,
                           int* status, void* stream) {
    return fcs::colsum_impl(q, k, out, S, 1, H, S, S, D, dtype, q_stride_h * H, q_stride_h, q_stride_s,
                            k_stride_h * H, k_stride_h, k_stride_s, scale, 0, 0, cls_n, h_norm, workspace,
                            workspace_bytes, status, stream);
}

int fcs_colsum_causal(const void* q, const void* k, float* out, int H, int q_len, int k_len, int D, int dtype,
                      int64_t q_stride_h, int64_t q_stride_s, int64_t k_stride_h, int64_t k_stride_s,
                      float scale, int k_past, int h_norm, void* workspace, size_t workspace_bytes,
                      int* status, void* stream) {
    return fcs::colsum_impl(q, k, out, k_len, 1, H, q_len, k_len, D, dtype, q_stride_h * H, q_stride_h,
                            q_stride_s, k_stride_h * H, k_stride_h, k_stride_s, scale, 1, k_past, -1, h_norm,
                            workspace, workspace_bytes, status, stream);
}

int fcs_colsum_causal_batched(const void* q, const void* k, float* out, int64_t out_ld, int B, int H, int q_len,
                              int k_len, int D, int dtype, int64_t q_stride_b, int64_t q_stride_h,
                              int64_t q_stride_s, int64_t k_stride_b, int64_t k_stride_h, int64_t k_stride_s,
                              float scale, int k_past, int h_norm, void* workspace, size_t workspace_bytes,
                              int* status, void* stream) {
    return fcs::colsum_impl(q, k, out, out_ld, B, H, q_len, k_len, D, dtype, q_stride_b, q_stride_h, q_stride_s,
                            k_stride_b, k_stride_h, k_stride_s, scale, 1, k_past, -1, h_norm, workspace,
                            workspace_bytes, status, stream);
}

int fcs_run_call(const FcsCall* c) {
    return fcs::colsum_impl(c->q, c->k, c->out, c->out_ld, c->B, c->H, c->Sq, c->Sk, c->D, c->dtype, c->q_stride[0],
                            c->q_stride[1], c->q_stride[2], c->k_stride[0], c->k_stride[1], c->k_stride[2], c->scale,
                            c->causal, c->k_past, c->cls_n, c->h_norm, nullptr, 0, c->status, c->stream, true,
                            fcs::PASSES_BOTH, nullptr, 0, nullptr, 0, nullptr, c->alloc, c->alloc_ctx);
}

int fcs_run_host_call(const FcsHostCall* call) { return fcs::run_host_call(call); }

size_t fcs_statistics_rows(int q_rows) {
    return q_rows > 0 ? (size_t)fcs::ceil_div(q_rows, fcs::BLOCK) * fcs::BLOCK : 0;
}

int fcs_colsum_statistics(const void* q, const void* k, float* neg_lse, int B, int H, int q_rows, int Sk, int D,
                          int dtype, int64_t q_stride_b, int64_t q_stride_h, int64_t q_stride_s,
                          int64_t k_stride_b, int64_t k_stride_h, int64_t k_stride_s, float scale,
                          int64_t norm_rows, int h_norm, void* workspace, size_t workspace_bytes, int* status,
                          void* stream) {
    if (norm_rows < q_rows) {
        fcs::g_err[0] = 0;
        return fcs::fail(FCS_ERR_INVALID_ARGUMENT, "norm_rows (%lld) is smaller than the rows given (%d)",
                         (long long)norm_rows, q_rows);
    }
    return fcs::colsum_impl(q, k, nullptr, 0, B, H, q_rows, Sk, D, dtype, q_stride_b, q_stride_h, q_stride_s,
                            k_stride_b, k_stride_h, k_stride_s, scale, 0, 0, -1, h_norm, workspace,
                            workspace_bytes, status, stream, false, fcs::PASSES_STATS, neg_lse, norm_rows);
}

int fcs_colsum_columns(const void* q, const void* k, const float* neg_lse, float* out, int64_t out_ld, int B, int H,
                       int q_rows, int k_rows, int D, int dtype, int64_t q_stride_b, int64_t q_stride_h,
                       int64_t q_stride_s, int64_t k_stride_b, int64_t k_stride_h, int64_t k_stride_s,
                       float scale, void* workspace, size_t workspace_bytes, int* status, void* stream) {
    return fcs::colsum_impl(q, k, out, out_ld, B, H, q_rows, k_rows, D, dtype, q_stride_b, q_stride_h, q_stride_s,
                            k_stride_b, k_stride_h, k_stride_s, scale, 0, 0, -1, 0, workspace, workspace_bytes,
                            status, stream, true, fcs::PASSES_COLUMNS, const_cast<float*>(neg_lse), 0);
}

int fcs_select_topk(const float* colsum, int64_t ld, int B, int S, int k, int* indices, float* values,
                    void* stream) {
    fcs::g_err[0] = 0;
    if (!colsum || !indices) return fcs::fail(FCS_ERR_INVALID_ARGUMENT, "colsum and indices must not be NULL");
    if (B <= 0 || S <= 0 || ld < S)
        return fcs::fail(FCS_ERR_INVALID_ARGUMENT, "bad sizes (B=%d S=%d ld=%lld)", B, S, (long long)ld);
    if (k <= 0 || k > S) return fcs::fail(FCS_ERR_INVALID_ARGUMENT, "k must be in 1..S, got %d (S=%d)", k, S);
    const cudaError_t e = fcs::launch_topk(colsum, (long long)ld, B, S, k, indices, values, reinterpret_cast<cudaStream_t>(stream));
    if (e != cudaSuccess) return fcs::fail(FCS_ERR_CUDA, "top-k selection launch failed: %s", cudaGetErrorString(e));
    return FCS_OK;
}

int fcs_peer_post(int* const* flags, int n_flags, int value, void* stream) {
    fcs::g_err[0] = 0;
    if (!flags || n_flags <= 0 || n_flags > fcs::PEER_FLAGS_MAX)
        return fcs::fail(FCS_ERR_INVALID_ARGUMENT, "1 to %d flag pointers are expected, got %d", fcs::PEER_FLAGS_MAX, n_flags);
    fcs::PeerFlagPointers fp;
    memset(&fp, 0, sizeof(fp));
    for (int i = 0; i < n_flags; ++i) {
        if (!flags[i] || reinterpret_cast<uintptr_t>(flags[i]) % 4)
            return fcs::fail(FCS_ERR_INVALID_ARGUMENT, "flag %d is NULL or misaligned", i);
        fp.p[i] = flags[i];
    }
    fcs::peer_post_kernel<<<1, 32, 0, reinterpret_cast<cudaStream_t>(stream)>>>(fp, n_flags, value);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return fcs::fail(FCS_ERR_CUDA, "flag post launch failed: %s", cudaGetErrorString(e));
    return FCS_OK;
}

int fcs_peer_wait(const int* flags, int n_flags, int value, int* status, void* stream) {
    fcs::g_err[0] = 0;
    if (!flags || n_flags <= 0 || n_flags > 32 || reinterpret_cast<uintptr_t>(flags) % 4)
        return fcs::fail(FCS_ERR_INVALID_ARGUMENT, "1 to 32 consecutive, aligned flags are expected, got %d", n_flags);
    fcs::peer_wait_kernel<<<1, 32, 0, reinterpret_cast<cudaStream_t>(stream)>>>(flags, n_flags, value, status);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return fcs::fail(FCS_ERR_CUDA, "flag wait launch failed: %s", cudaGetErrorString(e));
    return FCS_OK;
}

int fcs_selftest_wait_expiry(const void* q, const void* k, void* workspace, size_t workspace_bytes, int* status,
                              double limit_seconds, void* stream_v) {
    fcs::g_err[0] = 0;
    using namespace fcs;
    if (!q || !k || !workspace || !status)
        return fail(FCS_ERR_INVALID_ARGUMENT, "q, k, workspace and status must not be NULL");
    if (!(limit_seconds > 0.0) || limit_seconds > 2.0)
        return fail(FCS_ERR_INVALID_ARGUMENT, "limit_seconds must be in (0, 2]");
    cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_v);
    // a statistics pass over one 128 x 256 tile of fp16 inputs with D = 64
    const int B = 1, H = 1, Sq = TILE, Sk = BLOCK, D = 64;
    Problem p;
    memset(&p, 0, sizeof(p));
    plan(p, B, H, Sq, Sk, 0, 0, num_sms());
    size_t part_off = 0, ext_off = 0;
    const size_t need = workspace_layout(p, &part_off, &ext_off);
    if (workspace_bytes < need || reinterpret_cast<uintptr_t>(workspace) % 256)
        return fail(FCS_ERR_WORKSPACE, "workspace too small or misaligned: need %zu bytes", need);
    p.neg_lse = reinterpret_cast<float*>(workspace);
    p.part = reinterpret_cast<uint8_t*>(workspace) + part_off;
    p.ext = reinterpret_cast<uint8_t*>(workspace) + ext_off;
    p.status = status;
    p.c = 0.125f * 1.4426950408889634f;
    p.inv_c = 1.0f / p.c;
    p.log2_norm = log2f((float)Sq);
    p.idesc = (1u << 4) | ((uint32_t)(BLOCK >> 3) << 17) | ((uint32_t)(TILE >> 4) << 24);
    p.withhold_loads = 1;
    CUtensorMap tq, tk;
    int rc;
    if ((rc = make_tensor_map(&tq, q, FCS_DTYPE_FP16, B, H, Sq, D, (int64_t)Sq * D, (int64_t)Sq * D, D, TILE)) != FCS_OK) return rc;
    if ((rc = make_tensor_map(&tk, k, FCS_DTYPE_FP16, B, H, Sk, D, (int64_t)Sk * D, (int64_t)Sk * D, D, BLOCK)) != FCS_OK) return rc;
    static long long short_limit, full_limit = kWaitLimitCycles;
    short_limit = (long long)(limit_seconds * 1.9e9);
    cudaError_t e = cudaMemcpyToSymbolAsync(g_wait_limit_cycles, &short_limit, sizeof(long long), 0,
                                            cudaMemcpyHostToDevice, stream);
    if (e == cudaSuccess) e = launch_stream<64, MODE_STATS>(tq, tk, tq, p, 1, stream, false);
    const cudaError_t e2 = cudaMemcpyToSymbolAsync(g_wait_limit_cycles, &full_limit, sizeof(long long), 0,
                                                   cudaMemcpyHostToDevice, stream);
    if (e != cudaSuccess || e2 != cudaSuccess)
        return fail(FCS_ERR_CUDA, "wait-expiry self-test failed to launch: %s",
                    cudaGetErrorString(e != cudaSuccess ? e : e2));
    return FCS_OK;
}

int fcs_selftest_wait_expiry_cluster(const void* q, const void* k, float* out, int* status, double limit_seconds,
                                     void* stream_v) {
    fcs::g_err[0] = 0;
    using namespace fcs;
    if (!q || !k || !out || !status)
        return fail(FCS_ERR_INVALID_ARGUMENT, "q, k, out and status must not be NULL");
    if (!(limit_seconds > 0.0) || limit_seconds > 2.0)
        return fail(FCS_ERR_INVALID_ARGUMENT, "limit_seconds must be in (0, 2]");
    cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_v);
    // the one-kernel form on one head: 128 queries, two blocks of 256 keys, a cluster of two CTAs
    const int B = 1, H = 1, Sq = TILE, Sk = 2 * BLOCK, D = 64;
    Problem p;
    memset(&p, 0, sizeof(p));
    p.B = B; p.H = H; p.Sq = Sq; p.Sk = Sk;
    p.out = out;
    p.out_ld = Sk;
    p.status = status;
    p.c = 0.125f * 1.4426950408889634f;
    p.inv_c = 1.0f / p.c;
    p.log2_norm = log2f((float)Sq);
    p.withhold_loads = 1;
    CUtensorMap tq, tk;
    int rc;
    if ((rc = make_tensor_map(&tq, q, FCS_DTYPE_FP16, B, H, Sq, D, (int64_t)Sq * D, (int64_t)Sq * D, D, TILE)) != FCS_OK) return rc;
    if ((rc = make_tensor_map(&tk, k, FCS_DTYPE_FP16, B, H, Sk, D, (int64_t)Sk * D, (int64_t)Sk * D, D, BLOCK)) != FCS_OK) return rc;
    static long long short_limit, full_limit = kWaitLimitCycles;
    short_limit = (long long)(limit_seconds * 1.9e9);
    cudaError_t e = cudaMemcpyToSymbolAsync(g_wait_limit_cycles, &short_limit, sizeof(long long), 0,
                                            cudaMemcpyHostToDevice, stream);
    if (e == cudaSuccess)
        rc = launch_fused_short(tq, tk, p, 64, 0.125f, true, /*cl=*/2, /*nkb=*/2, /*bpc=*/1, /*clear_out=*/true, nullptr, 0,
                                stream);
    const cudaError_t e2 = cudaMemcpyToSymbolAsync(g_wait_limit_cycles, &full_limit, sizeof(long long), 0,
                                                   cudaMemcpyHostToDevice, stream);
    if (e != cudaSuccess || e2 != cudaSuccess)
        return fail(FCS_ERR_CUDA, "wait-expiry self-test failed to launch: %s",
                    cudaGetErrorString(e != cudaSuccess ? e : e2));
    return rc;
}

int fcs_select_threshold(const float* colsum, int64_t ld, int B, int S, float threshold, int relative, int* indices,
                         int* counts, void* stream) {
    fcs::g_err[0] = 0;
    if (!colsum || !indices || !counts)
        return fcs::fail(FCS_ERR_INVALID_ARGUMENT, "colsum, indices and counts must not be NULL");
    if (B <= 0 || S <= 0 || ld < S)
        return fcs::fail(FCS_ERR_INVALID_ARGUMENT, "bad sizes (B=%d S=%d ld=%lld)", B, S, (long long)ld);
    if (!(threshold == threshold)) return fcs::fail(FCS_ERR_INVALID_ARGUMENT, "threshold is not a number");
    const cudaError_t e = fcs::launch_threshold(colsum, (long long)ld, B, S, threshold, relative ? 1 : 0, indices, counts,
                                                reinterpret_cast<cudaStream_t>(stream));
    if (e != cudaSuccess) return fcs::fail(FCS_ERR_CUDA, "threshold selection launch failed: %s", cudaGetErrorString(e));
    return FCS_OK;
}

int fcs_colsum_batched_static_scratch(const void* q, const void* k, float* out, int64_t out_ld, int B, int H,
                                      int S, int D, int dtype, int64_t q_stride_b, int64_t q_stride_h,
                                      int64_t q_stride_s, int64_t k_stride_b, int64_t k_stride_h,
                                      int64_t k_stride_s, float scale, int cls_n, int h_norm, int* status,
                                      void* stream) {
    fcs::g_err[0] = 0;
    if (B <= 0 || H <= 0 || S <= 0 || !fcs::head_dim_ok(D))
        return fcs::fail(FCS_ERR_INVALID_ARGUMENT, "bad sizes (B=%d H=%d S=%d D=%d)", B, H, S, D);
    const int rows = (cls_n > 0 && cls_n < S) ? cls_n : S;
    // what this call will really use: nothing when it takes the few-row or the single-pass kernel
    size_t need = 0;
    const int qrc = fcs_call_workspace_bytes(B, H, rows, S, D, 0, 0, &need);
    if (qrc != FCS_OK) return qrc;
    if (need > (size_t)FCS_STATIC_SCRATCH_BYTES)
        return fcs::fail(FCS_ERR_WORKSPACE,
                         "this call needs %zu bytes of scratch but the built-in scratch holds %zu; "
                         "use fcs_colsum_batched with a caller-provided workspace",
                         need, (size_t)FCS_STATIC_SCRATCH_BYTES);
    void* scratch = nullptr;
    const int rc = fcs::static_scratch_address(&scratch);
    if (rc != FCS_OK) return rc;
    return fcs::colsum_impl(q, k, out, out_ld, B, H, S, S, D, dtype, q_stride_b, q_stride_h, q_stride_s,
                            k_stride_b, k_stride_h, k_stride_s, scale, 0, 0, cls_n, h_norm, scratch,
                            (size_t)FCS_STATIC_SCRATCH_BYTES, status, stream);
}

int fcs_colsum_causal_accumulate(const void* q, const void* k, float* out, int H, int q_len, int k_len, int D,
                                 int dtype, int64_t q_stride_h, int64_t q_stride_s, int64_t k_stride_h,
                                 int64_t k_stride_s, float scale, int k_past, int h_norm, void* workspace,
                                 size_t workspace_bytes, int* status, void* stream) {
    return fcs::colsum_impl(q, k, out, k_len, 1, H, q_len, k_len, D, dtype, q_stride_h * H, q_stride_h,
                            q_stride_s, k_stride_h * H, k_stride_h, k_stride_s, scale, 1, k_past, -1, h_norm,
                            workspace, workspace_bytes, status, stream, /*clear_out=*/false);
}

int fcs_colsum_causal_accumulate_and_clear(const void* q, const void* k, float* out, float* clear_buf, int H,
                                           int q_len, int k_len, int D, int dtype, int64_t q_stride_h,
                                           int64_t q_stride_s, int64_t k_stride_h, int64_t k_stride_s, float scale,
                                           int k_past, int h_norm, void* workspace, size_t workspace_bytes,
                                           int* status, void* stream) {
    return fcs::colsum_impl(q, k, out, k_len, 1, H, q_len, k_len, D, dtype, q_stride_h * H, q_stride_h,
                            q_stride_s, k_stride_h * H, k_stride_h, k_stride_s, scale, 1, k_past, -1, h_norm,
                            workspace, workspace_bytes, status, stream, /*clear_out=*/false, fcs::PASSES_BOTH, nullptr,
                            0, clear_buf, clear_buf ? (long long)k_len : 0);
}

int fcs_colsum_causal_accumulate_signalled(const void* q, const void* k, float* out, float* clear_buf, int H,
                                           int q_len, int k_len, int D, int dtype, int64_t q_stride_h,
                                           int64_t q_stride_s, int64_t k_stride_h, int64_t k_stride_s, float scale,
                                           int k_past, int h_norm, void* workspace, size_t workspace_bytes,
                                           int* status, void* stream, const FcsPeerSignals* signals) {
    fcs::g_err[0] = 0;
    if (!signals) return fcs::fail(FCS_ERR_INVALID_ARGUMENT, "signals is NULL");
    if (signals->post_n < 0 || signals->post_n > 15)
        return fcs::fail(FCS_ERR_INVALID_ARGUMENT, "at most 15 flags can be posted, got %d", signals->post_n);
    if (signals->done_flag && !signals->counter)
        return fcs::fail(FCS_ERR_INVALID_ARGUMENT, "a done flag needs a counter");
    return fcs::colsum_impl(q, k, out, k_len, 1, H, q_len, k_len, D, dtype, q_stride_h * H, q_stride_h,
                            q_stride_s, k_stride_h * H, k_stride_h, k_stride_s, scale, 1, k_past, -1, h_norm,
                            workspace, workspace_bytes, status, stream, /*clear_out=*/false, fcs::PASSES_BOTH, nullptr,
                            0, clear_buf, clear_buf ? (long long)k_len : 0, signals);
}

}  // extern "C"
