// Single-pass attention column mean for short key axes (S_k <= 2048, head
// dimension 64, non-causal), one thread-block cluster per stream of (batch, head)
// pairs.
//
// The two-pass kernels evaluate every score and every exp twice.  When the whole
// key axis fits a cluster of up to eight CTAs (256 keys each), one pass is enough:
//
//   S      = Q_tile K_slice^T            tcgen05 MMA, 128 queries x 256 keys, fp32 in tensor memory
//   P~     = exp2(c*S - m_g)             per thread (= query row) and 64-key group g, fp16 -> shared memory
//   (m, l) exchange                      per row: 4 groups in the CTA, then all CTAs of the cluster
//                                        through distributed shared memory (st.async + mbarrier
//                                        byte counts: nobody waits for a store to land)
//   w_g    = exp2(m_g - M) / L           the factor that turns P~ into softmax probabilities
//   D2    += P~^T W                      second MMA: contraction over the 128 query rows; W holds
//                                        w_g of the four groups as two fp16 parts (hi in columns
//                                        0..3, lo in 4..7 of a 16-wide operand), so D2[key][g] and
//                                        D2[key][4 + g] are the column sums of a key of group g
//
// D2 lives in tensor memory across all query tiles and heads of a batch entry and
// is added to the output once per (cluster, batch entry).  P~ is double-buffered:
// the column-sum MMA of tile i runs while the consumers work on tiles i+1 and i+2,
// which is the time the statistics of tile i have to go around the cluster.
//
// A tile takes a CTA the same time whatever the number of real keys in its slice; keys past S_k are
// overwritten in tensor memory (masked in registers, 400 keys took 71 us instead of 63, 577 137 instead of 117,
// B = 32, H = 16, when that was measured; 56 and 101 now).  The rule for which calls come here is with the launcher.
#pragma once

#include <float.h>

#include "colsum_math.cuh"
#include "schedule.h"
#include "sm100_ptx.cuh"

namespace fcs {

struct SinglePassParams {
    int B, H, Sq, Sk;
    int NQ;                 // 128-row query tiles
    int CL;                 // CTAs per cluster = 256-key slices (1 .. 8)
    int units;              // B * H
    int clusters;           // gridDim.x / CL
    int flush_units;        // most (batch, head) pairs accumulated in tensor memory before a flush
    float c;                // |scale| * log2(e); not zero where the key axis ends inside a group of 64
    float out_scale;        // 1 / (h_norm * R * 2^10): the weights are stored times 2^10
    float* out;
    long long out_ld;
    int* status;
    uint32_t idesc_scores;  // 128 x 128 x 16, K-major operands
    const int* fmt;         // NULL, or where a kernel of this call has written the operands' type (1: bf16)
    uint32_t idesc_colsum;  // 128 x 16 x 16, A = P~ (M-major), B = W (N-major), fp16
};

namespace sp {

constexpr int CONSUMER_GROUPS = 4;
constexpr int CONSUMER_WARPS = 16;
constexpr int CONSUMER_THREADS = 512;
constexpr int HALF_THREADS = 256;          // consumers of one half (two groups)
constexpr int SCORES_WARP = 16;
constexpr int COLSUM_WARP = 17;
constexpr int XCHG_WARP = 18;
constexpr int XCHG_WARPS = 2;
constexpr int XCHG_ROWS_PER_WARP = 128 / XCHG_WARPS;
static_assert(XCHG_ROWS_PER_WARP == 64, "a lane of an exchange warp has two neighbouring rows");
constexpr int THREADS = 32 * (XCHG_WARP + XCHG_WARPS);
constexpr int MAX_CL = 8;
constexpr int TMEM_COLS = 512;
constexpr int S_BUFS = 3;              // score accumulators of 128 columns (one half of a tile) in tensor memory
constexpr int D2_COL = 128 * S_BUFS;   // tensor-memory column of the column-sum accumulators
constexpr int W_N = 16;                // columns of the weight operand (eight of them used: hi and lo of four groups)
constexpr float W_SCALE_LOG2 = 10.f;   // weights are stored times 2^10 to stay in the fp16 normal range

// shared memory (head dimension 64)
constexpr int K_BYTES = 256 * 128;                 // key slice: 256 rows of 128 bytes, 128-byte swizzle
constexpr int Q_BYTES = 128 * 128;                 // query tile
constexpr int P_TILE_BYTES = 128 * 128 * 2;        // P~ of one key tile: 128 keys x 128 query rows fp16
constexpr int P_BYTES = 2 * P_TILE_BYTES;          // both key tiles of the slice
constexpr int P_ATOM_COL_BYTES = 16 * 1024;        // 64 keys x 128 query rows
constexpr int W_BYTES = 128 * 2 * W_N;             // 128 query rows of 16 columns: rows of 32 bytes, 32-byte swizzle
constexpr int K_OFF = 0;
constexpr int Q_OFF = K_OFF + K_BYTES;             // two buffers
constexpr int P_OFF = Q_OFF + 2 * Q_BYTES;         // two buffers
constexpr int W_OFF = P_OFF + 2 * P_BYTES;         // two buffers
constexpr int XCHG_OFF = W_OFF + 2 * W_BYTES;      // float2 [2][MAX_CL][128]: every CTA's (max, sum) per row
constexpr int LST_OFF = XCHG_OFF + 2 * MAX_CL * 128 * 8;   // float2 [2][groups][128]
constexpr int BAR_OFF = LST_OFF + 2 * CONSUMER_GROUPS * 128 * 8;
constexpr int NUM_BARS = 28;
constexpr int MISC_OFF = BAR_OFF + NUM_BARS * 8;
constexpr int TOTAL = MISC_OFF + 16;               // tensor-memory address, abort flag
constexpr int DYN_BYTES = TOTAL + 1024;
static_assert(DYN_BYTES <= 227 * 1024, "shared memory budget");

// ---------------------------------------------------------------- cluster helpers
__device__ __forceinline__ uint32_t cluster_ctarank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
// The shared::cluster address of `addr` (a shared::cta address) in CTA `rank`.
__device__ __forceinline__ uint32_t map_to_cta(uint32_t addr, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
// Asynchronous store of four floats (16-byte aligned) into another CTA's shared memory; its 16 bytes are
// counted on that CTA's barrier `mbar` when they have landed, so the sender neither
// waits nor fences.
__device__ __forceinline__ void st_async_f32x4(uint32_t addr, float a, float b, float c, float d, uint32_t mbar) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%1, %2, %3, %4}, [%5];"
                 ::"r"(addr), "f"(a), "f"(b), "f"(c), "f"(d), "r"(mbar)
                 : "memory");
}
__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ bool mbar_try_wait_cluster(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t"
        ".reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2, %3;\n\t"
        "selp.b32 %0, 1, 0, p;\n\t"
        "}\n"
        : "=r"(ok)
        : "r"(bar), "r"(parity), "r"(kSuspendHintNs)
        : "memory");
    return ok != 0;
}
// Bounded wait on a barrier that other CTAs of the cluster arrive on.
__device__ __forceinline__ bool mbar_wait_cluster(uint32_t bar, uint32_t parity, volatile int* abort_flag,
                                                  int* status, int code) {
    if (mbar_try_wait_cluster(bar, parity)) return true;
    const long long t0 = clock64();
    unsigned spins = 0;
    while (true) {
        if (mbar_try_wait_cluster(bar, parity)) return true;
        if ((++spins & 15u) == 0u) {
            if (*abort_flag) return false;
            if (clock64() - t0 > kWaitLimitCycles) {
                *abort_flag = 1;
                if (status) atomicCAS(status, 0, code);
                return false;
            }
        }
    }
}

// 32 lanes x 16 consecutive fp32 columns.
__device__ __forceinline__ void tmem_ld_x16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void tmem_ld_wait16(uint32_t (&r)[16]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]),
                   "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]),
                   "+r"(r[15])
                 :
                 : "memory");
}

// Shared-memory descriptor of an M-major operand tile (the M index is contiguous in
// memory) with the 128-byte swizzle: atoms of 64 M-elements (128 bytes) x 8 K-rows
// (1024 bytes); the next 64 M-elements are `P_ATOM_COL_BYTES` further (leading
// offset), the next 8 K-rows 1024 bytes further (stride offset).
__device__ __forceinline__ uint64_t umma_desc_mn_sw128(uint32_t smem_addr) {
    const uint32_t lo = ((smem_addr >> 4) & 0x3FFFu) | ((uint32_t)(P_ATOM_COL_BYTES >> 4) << 16);
    const uint32_t hi = 64u | (1u << 14) | (2u << 29);
    return (static_cast<uint64_t>(hi) << 32) | lo;
}

// The same for the weights: rows of 16 N-elements (32 bytes) with the 32-byte swizzle, the next 8 K-rows 256
// bytes further (stride offset; there is no second run of N-elements).
__device__ __forceinline__ uint64_t umma_desc_mn_sw32(uint32_t smem_addr) { return umma_desc_k_sw32(smem_addr); }

__device__ __forceinline__ void st_shared_v4(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d)
                 : "memory");
}
__device__ __forceinline__ uint32_t pack_half2(float lo, float hi) {
    const __half2 h = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&h);
}

__device__ __forceinline__ float max_of_32(const uint32_t (&r)[32]) {
    float m0 = max3(__uint_as_float(r[0]), __uint_as_float(r[1]), __uint_as_float(r[2]));
    float m1 = max3(__uint_as_float(r[3]), __uint_as_float(r[4]), __uint_as_float(r[5]));
    float m2 = max3(__uint_as_float(r[6]), __uint_as_float(r[7]), __uint_as_float(r[8]));
    float m3 = max3(__uint_as_float(r[9]), __uint_as_float(r[10]), __uint_as_float(r[11]));
#pragma unroll
    for (int j = 12; j < 28; j += 8) {
        m0 = max3(m0, __uint_as_float(r[j]), __uint_as_float(r[j + 1]));
        m1 = max3(m1, __uint_as_float(r[j + 2]), __uint_as_float(r[j + 3]));
        m2 = max3(m2, __uint_as_float(r[j + 4]), __uint_as_float(r[j + 5]));
        m3 = max3(m3, __uint_as_float(r[j + 6]), __uint_as_float(r[j + 7]));
    }
    m0 = max3(m0, __uint_as_float(r[28]), __uint_as_float(r[29]));
    m1 = max3(m1, __uint_as_float(r[30]), __uint_as_float(r[31]));
    return max_or_nan(max_or_nan(m0, m1), max_or_nan(m2, m3));
}

// exp2(c*s - m) of 8 scores -> four packed fp16 pairs; adds the fp32 values to `sum`.
// `pair0` is the index (mod 16) of the first pair in the exp-unit / polynomial pattern.
// POLY: pairs of 16 that the polynomial takes.
template <int POLY>
__device__ __forceinline__ void exp8_packed(int pair0, const uint32_t* s, f32x2 c2, f32x2 nm2, f32x2& sum0,
                                            f32x2& sum1, uint32_t* h) {
#pragma unroll
    for (int pr = 0; pr < 4; ++pr) {
        const f32x2 t = fma2(pack2(__uint_as_float(s[2 * pr]), __uint_as_float(s[2 * pr + 1])), c2, nm2);
        f32x2 e;
        float e0, e1;
        if (pair_uses_polynomial((pair0 + pr) & 15, POLY)) {
            e = ex2_poly2(t);
            unpack2(e, e0, e1);
        } else {
            unpack2(t, e0, e1);
            e0 = ex2_approx(e0);
            e1 = ex2_approx(e1);
            e = pack2(e0, e1);
        }
        if (pr & 1) sum1 = add2(sum1, e); else sum0 = add2(sum0, e);
        h[pr] = pack_half2(e0, e1);
    }
}

// Writes `value` into `n` columns of this warp's 32 tensor-memory lanes.
__device__ __forceinline__ void tmem_fill(uint32_t taddr, int n, uint32_t value) {
    for (; n >= 8; n -= 8, taddr += 8)
        asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %1, %1, %1, %1, %1, %1, %1};" ::"r"(taddr), "r"(value) : "memory");
    for (; n > 0; --n, ++taddr)
        asm volatile("tcgen05.st.sync.aligned.32x32b.x1.b32 [%0], {%1};" ::"r"(taddr), "r"(value) : "memory");
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}
template <bool V> struct Flag { static constexpr bool value = V; };

}  // namespace sp

// ---------------------------------------------------------------------------
// tm_q: boxes of 128 query rows, tm_k: boxes of 256 key rows (both 64 elements
// wide, 128-byte swizzle).  Grid = clusters * CL CTAs, launched with cluster
// dimension CL; CTA `rank` of a cluster owns keys [256*rank, 256*rank + 256).
//
// Roles in a CTA (20 warps):
//   16 consumer warps  four groups of 128 threads (thread = query row of the tile, group =
//                      64 key columns).  Groups 0,1 and groups 2,3 form two "halves" (the two
//                      128-key tiles of the slice), each with its own P~ buffers and column-sum
//                      accumulator.  The scores of half h of tile i are accumulator (2 i + h) % 3: a half need
//                      not wait for the other one's loads, and the two drift apart, so that one's loads and
//                      stores fall into the other's exps.
//   1 scores warp      key slice per (batch, head), query tile per step (a step ahead), scores(i) as soon
//                      as the consumers have read scores(i-1) out of tensor memory.
//   1 column-sum warp  column sums(i) of both halves when the weights of tile i are there.
//   2 exchange warps   64 rows each, two neighbouring ones per lane: combine the four groups' (max, sum) of
//                      a row, post the result to every CTA of the cluster, and when all CTAs' values are in,
//                      write the weights W of the four groups.
// What bounds it: the chain of these warps' instructions, 6 to 11 cycles apart next to 16 busy consumer
// warps.  With one warp for both products (scores(i), column sums(i-2), scores(i+1), ...) a tile's scores waited
// for the weights of the tile before last, the consumers for the scores -- all groups at once, so that their
// loads, exps and stores never overlapped -- and the exchange warps were busy for 2 700 of a tile's 3 200 cycles.
// Apart, with the exchange unrolled for the cluster's size, two rows to a load and a store, and the weights in
// one 16-byte store per row: us per call, 32 x 16 pairs, back to back, 577 keys 112.4 -> 100.9, 1024 keys 230.4 -> 198.5.
// What is left of a tile's 2 900 cycles: 1 400 in the exps, the rest the latencies around them (tensor-memory loads
// 270, stores 330, barriers and loop 600), and a half that runs ahead waits for the other one's statistics.
// ---------------------------------------------------------------------------
// PADDED: the key axis ends inside a group of 64 keys.  (An instance of its own: the test for it in the
// loop costs 4 % at 512 and 1024 keys.)  CLMAX: most CTAs of a cluster (1, 2, 4 or 8): the exchange is unrolled
// for as many.  The instance for one CTA has no cluster instruction and is launched without a cluster.
template <bool PADDED, int CLMAX>
__global__ void __launch_bounds__(sp::THREADS, 1)
colsum_single_pass_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                          const SinglePassParams p) {
    using namespace sp;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                               ~static_cast<uintptr_t>(1023));
    const uint32_t smem_base = smem_u32(smem);
    const uint32_t k_smem = smem_base + K_OFF;
    const uint32_t q_smem = smem_base + Q_OFF;
    const uint32_t p_smem = smem_base + P_OFF;
    const uint32_t w_smem = smem_base + W_OFF;
    const uint32_t xchg_smem = smem_base + XCHG_OFF;
    const uint32_t bars = smem_base + BAR_OFF;
    // barriers; `hf` is the half (key tile of the slice), `s` a P~ / statistics slot
    const uint32_t k_full = bars, k_empty = bars + 8;
    auto q_full = [&](int s) { return bars + 8u * (2 + s); };
    auto q_empty = [&](int s) { return bars + 8u * (4 + s); };
    auto s_empty = [&](int b) { return bars + 8u * (6 + b); };
    auto s_full = [&](int b) { return bars + 8u * (16 + b); };
    auto stats_bar = [&](int s) { return bars + 8u * (10 + s); };
    auto xchg_bar = [&](int s) { return bars + 8u * (12 + s); };
    auto w_ready = [&](int s) { return bars + 8u * (14 + s); };
    auto pw_free = [&](int s, int hf) { return bars + 8u * (20 + 2 * s + hf); };
    auto d2_full = [&](int hf) { return bars + 8u * (24 + hf); };
    auto d2_empty = [&](int hf) { return bars + 8u * (26 + hf); };
    volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(smem + MISC_OFF);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + MISC_OFF + 4);
    float2* lstats = reinterpret_cast<float2*>(smem + LST_OFF);
    const float2* xchg = reinterpret_cast<const float2*>(smem + XCHG_OFF);

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const uint32_t rank = CLMAX > 1 ? cluster_ctarank() : 0u;
    const int CL = CLMAX > 1 ? p.CL : 1;
    const int cluster_id = blockIdx.x / CL;
    const int NQ = p.NQ;
    // this cluster's share of the (batch, head, query tile) list
    TileRange range;
    range.init(p.units, NQ, cluster_id, p.clusters);
    const int u0 = range.u0, u1 = range.u1;
    auto t_lo = [&](int u) { return range.t_lo(u); };
    auto t_hi = [&](int u) { return range.t_hi(u); };

    if (threadIdx.x == 0) {
        mbar_init(k_full, 1); mbar_init(k_empty, 1);
        for (int i = 0; i < S_BUFS; ++i) { mbar_init(s_full(i), 1); mbar_init(s_empty(i), HALF_THREADS); }
        for (int i = 0; i < 2; ++i) {
            mbar_init(q_full(i), 1); mbar_init(q_empty(i), 1);
            mbar_init(stats_bar(i), CONSUMER_THREADS);
            mbar_init(xchg_bar(i), XCHG_WARPS);   // this CTA's exchange warps; the data counts as bytes
            mbar_init(w_ready(i), XCHG_WARPS * 32);
            for (int hf = 0; hf < 2; ++hf) mbar_init(pw_free(i, hf), 1);
            mbar_init(d2_full(i), 1); mbar_init(d2_empty(i), HALF_THREADS);
        }
        *abort_flag = 0;
        mbar_fence_init();
    }
    {   // the weight operand: only columns 0..7 are ever written, the rest stays zero
        uint4* w = reinterpret_cast<uint4*>(smem + W_OFF);
        for (int i = threadIdx.x; i < 2 * W_BYTES / 16; i += THREADS) w[i] = make_uint4(0u, 0u, 0u, 0u);
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == SCORES_WARP && lane == 0) {
        prefetch_tensormap(&tm_q);
        prefetch_tensormap(&tm_k);
    }
    if (warp == COLSUM_WARP) {
        tmem_alloc(smem_u32(const_cast<uint32_t*>(tmem_slot)), TMEM_COLS);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    if constexpr (CLMAX > 1) cluster_sync_all();   // every CTA's barriers exist before a peer signals them
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    if (CLMAX == 1 || clusters_pack(p.CL)) grid_launch_dependents();   // (not before this CTA has its tensor memory)
    grid_dependency_wait();   // the set-up is done; what follows reads the inputs and adds into the cleared output

    auto wait_all = [&](uint32_t bar, uint32_t parity, int code) -> bool {
        const bool ok = mbar_wait(bar, parity, abort_flag, p.status, code);
        return __all_sync(0xffffffffu, ok);
    };
    // The column sums leave tensor memory at the end of a batch entry, of this cluster's range,
    // and every `flush_units` pairs: the tensor core truncates when it adds into its fp32
    // accumulator (about half a unit in the last place lost per accumulation), and the bound
    // keeps that bias below ~1e-4 of a column sum however many heads there are.  (A pair has at most 16 query
    // tiles: these calls have no more queries than keys.)
    auto last_of_batch = [&](int u) { return range.flush_after(u, p.H, p.flush_units); };

    if (warp == SCORES_WARP) {
        // ------------------------------------------------ loads and scores
        const uint32_t idesc_scores = p.idesc_scores | (p.fmt && *p.fmt ? IDESC_BF16 : 0u);
        const uint64_t dk = umma_desc_k_sw128(k_smem);
        const int total = range.tiles();
        int lu = u0, lt = t_lo(u0), li = 0;      // the next query tile to fetch
        bool ok = true;
        auto fetch_query_tile = [&]() -> bool {
            if (li >= total) return true;
            const int qs = li & 1;
            if (!wait_all(q_empty(qs), ((li >> 1) & 1) ^ 1, FCS_STATUS_WAIT_PRODUCER)) return false;
            const int b = lu / p.H, h = lu - b * p.H;
            if (elect_one_sync()) {
                mbar_arrive_expect_tx(q_full(qs), Q_BYTES);
                tma_load_4d(q_smem + qs * Q_BYTES, &tm_q, q_full(qs), 0, lt * 128, h, b);
            }
            __syncwarp();
            ++li;
            if (++lt >= NQ) { lt = 0; ++lu; }
            return true;
        };
        int i = 0, uc = 0, sb = 0, sph = 1;      // sb, sph: the next score accumulator, the phase it is free in
        for (int u = u0; ok && u < u1; ++u, ++uc) {
            const int b = u / p.H, h = u - b * p.H;
            // (the slice is free once the last scores of the pair before it are formed)
            if (!wait_all(k_empty, (uc & 1) ^ 1, FCS_STATUS_WAIT_PRODUCER)) break;
            if (elect_one_sync()) {
                mbar_arrive_expect_tx(k_full, K_BYTES);
                tma_load_4d(k_smem, &tm_k, k_full, 0, 256 * (int)rank, h, b);
            }
            __syncwarp();
            if (u == u0 && !fetch_query_tile()) break;
            if (!wait_all(k_full, uc & 1, FCS_STATUS_WAIT_MMA)) break;
            const int t_end = t_hi(u);
            for (int t = t_lo(u); t < t_end; ++t, ++i) {
                const int qs = i & 1;
                if (!wait_all(q_full(qs), (i >> 1) & 1, FCS_STATUS_WAIT_MMA)) { ok = false; break; }
                const uint64_t dq = umma_desc_k_sw128(q_smem + qs * Q_BYTES);
#pragma unroll
                for (int hf = 0; hf < 2; ++hf) {
                    if (ok && !wait_all(s_empty(sb), sph, FCS_STATUS_WAIT_MMA)) ok = false;
                    if (!ok) break;
                    tc_fence_after();
                    if (elect_one_sync()) {
                        if (256 * (int)rank + 128 * hf < p.Sk) {    // (a half without keys has no scores)
#pragma unroll
                            for (int ks = 0; ks < 4; ++ks)
                                umma_f16(tmem_base + 128 * sb, dq + (uint64_t)((ks * 32) >> 4),
                                         dk + (uint64_t)((hf * 128 * 128 + ks * 32) >> 4), idesc_scores, ks > 0 ? 1u : 0u);
                        }
                        umma_commit(s_full(sb));
                        if (hf == 1) {
                            umma_commit(q_empty(qs));
                            if (t + 1 == t_end) umma_commit(k_empty);
                        }
                    }
                    __syncwarp();
                    if (++sb == S_BUFS) { sb = 0; sph ^= 1; }
                    // The next query tile: its buffer is free since scores(i-1), and fetched only behind both halves of
                    // scores(i) it came 1 100 cycles after them, with an accumulator free (1024 keys 222.6 -> 211.2 us)
                    if (hf == 0) ok = fetch_query_tile();
                }
                if (!ok) break;
            }
        }
    } else if (warp >= XCHG_WARP) {
        // ------------------------------------------------ statistics exchange and weights
        const int row = (warp - XCHG_WARP) * XCHG_ROWS_PER_WARP + 2 * lane;   // this lane's rows: row, row + 1
        const int total = range.tiles();
        // where this CTA's pairs go in every CTA of the cluster, and the barrier that counts them there
        uint32_t post[CLMAX], post_bar[CLMAX];
        if constexpr (CLMAX > 1) {
#pragma unroll
            for (int r = 0; r < CLMAX; ++r) {
                post[r] = r < CL ? map_to_cta(xchg_smem + (uint32_t)(((int)rank * 128 + row) * 8), (uint32_t)r) : 0u;
                post_bar[r] = r < CL ? map_to_cta(xchg_bar(0), (uint32_t)r) : 0u;
            }
        }
        const uint32_t w_row = w_smem + row * (2 * W_N) + (((uint32_t)row >> 2) & 1u) * 16u;   // (32-byte swizzle)
        // (the query tile of the share's i-th tile, kept by counting: decoding it is a 64-bit
        // modulo, a hundred instructions in the warp every tile's exchange waits for)
        int t = total > 0 ? range.tile_of(0) : 0;
        for (int i = 0; i < total; ++i, t = (t + 1 == p.NQ) ? 0 : t + 1) {
            const int slot = i & 1;
            // (1) the four groups' (max, sum) of this CTA -> one pair per row, posted to every CTA
            if (!wait_all(stats_bar(slot), (i >> 1) & 1, FCS_STATUS_WAIT_CONSUMER)) break;
            const float4* ls = reinterpret_cast<const float4*>(lstats + slot * CONSUMER_GROUPS * 128 + row);
            float4 o[CONSUMER_GROUPS];      // (max, sum) of row, (max, sum) of row + 1
#pragma unroll
            for (int g = 0; g < CONSUMER_GROUPS; ++g) o[g] = ls[g * 64];
            float M0 = fmaxf(fmaxf(o[0].x, o[1].x), fmaxf(o[2].x, o[3].x));
            float M1 = fmaxf(fmaxf(o[0].z, o[1].z), fmaxf(o[2].z, o[3].z));
            const float ms0 = (M0 == -INFINITY) ? 0.f : M0, ms1 = (M1 == -INFINITY) ? 0.f : M1;
            float L0 = 0.f, L1 = 0.f;
#pragma unroll
            for (int g = 0; g < CONSUMER_GROUPS; ++g) {
                L0 = fmaf(o[g].y, ex2_approx(o[g].x - ms0), L0);
                L1 = fmaf(o[g].w, ex2_approx(o[g].z - ms1), L1);
            }
            if constexpr (CLMAX > 1) {
                const uint32_t slot_off = (uint32_t)slot * (MAX_CL * 128 * 8);
#pragma unroll
                for (int r = 0; r < CLMAX; ++r)
                    if (r < CL) st_async_f32x4(post[r] + slot_off, M0, L0, M1, L1, post_bar[r] + 8u * slot);
                // what this CTA's own barrier will receive for this warp's rows: 8 bytes per row and CTA
                if (lane == 0) mbar_arrive_expect_tx(xchg_bar(slot), (uint32_t)(CL * XCHG_ROWS_PER_WARP * 8));

                // (2) every CTA's pair of the row -> the weights of this CTA's four groups
                const bool good = mbar_wait_cluster(xchg_bar(slot), (i >> 1) & 1, abort_flag, p.status,
                                                    FCS_STATUS_WAIT_CONSUMER);
                if (!__all_sync(0xffffffffu, good)) break;
                const float4* xs = reinterpret_cast<const float4*>(xchg + slot * MAX_CL * 128 + row);
                float4 v[CLMAX];
#pragma unroll
                for (int r = 0; r < CLMAX; ++r) v[r] = (r < CL) ? xs[r * 64] : make_float4(-INFINITY, 0.f, -INFINITY, 0.f);
                M0 = v[0].x; M1 = v[0].z;
#pragma unroll
                for (int r = 1; r < CLMAX; ++r) { M0 = fmaxf(M0, v[r].x); M1 = fmaxf(M1, v[r].z); }
                L0 = 0.f; L1 = 0.f;
#pragma unroll
                for (int r = 0; r < CLMAX; ++r) {
                    L0 = fmaf(v[r].y, ex2_approx(v[r].x - M0), L0);
                    L1 = fmaf(v[r].w, ex2_approx(v[r].z - M1), L1);
                }
            } else {
                // (a row without a key to see: NaN, as -inf - -inf makes it in the exchange)
                L0 = M0 == -INFINITY ? nanf("") : L0;
                L1 = M1 == -INFINITY ? nanf("") : L1;
            }
            const float base0 = !PADDED || M0 > -FLT_MAX ? W_SCALE_LOG2 - M0 - __log2f(L0) : nanf("");
            const float base1 = !PADDED || M1 > -FLT_MAX ? W_SCALE_LOG2 - M1 - __log2f(L1) : nanf("");
            const int live = p.Sq - (t * 128 + row);   // rows past the end of the query axis weigh nothing
            // columns 0..3: the groups' weights as fp16, columns 4..7: what that leaves of them.  (The MMAs that
            // read this buffer, two tiles ago, are done: every consumer waited for them before it posted.)
            uint32_t w0[4], w1[4];
#pragma unroll
            for (int a = 0; a < 2; ++a) {
                const float w00 = live > 0 ? ex2_approx(o[2 * a].x + base0) : 0.f, w01 = live > 0 ? ex2_approx(o[2 * a + 1].x + base0) : 0.f;
                const float w10 = live > 1 ? ex2_approx(o[2 * a].z + base1) : 0.f, w11 = live > 1 ? ex2_approx(o[2 * a + 1].z + base1) : 0.f;
                const __half2 h0 = __floats2half2_rn(w00, w01), h1 = __floats2half2_rn(w10, w11);
                const float2 f0 = __half22float2(h0), f1 = __half22float2(h1);
                w0[a] = *reinterpret_cast<const uint32_t*>(&h0);
                w1[a] = *reinterpret_cast<const uint32_t*>(&h1);
                w0[2 + a] = pack_half2(w00 - f0.x, w01 - f0.y);
                w1[2 + a] = pack_half2(w10 - f1.x, w11 - f1.y);
            }
            st_shared_v4(w_row + slot * W_BYTES, w0[0], w0[1], w0[2], w0[3]);
            st_shared_v4(w_row + slot * W_BYTES + 2 * W_N, w1[0], w1[1], w1[2], w1[3]);
            mbar_arrive(w_ready(slot));   // (the column-sum warp fences before the tensor core reads W)
        }
    } else if (warp == COLSUM_WARP) {
        // ------------------------------------------------ column sums: D2_hf (+)= P~_hf(i)^T W(i)
        int i = 0, fc = 0;
        bool ok = true, fresh = true;   // fresh: the next MMAs start a new accumulation
        for (int u = u0; ok && u < u1; ++u) {
            const bool flush = last_of_batch(u);
            const int t_end = t_hi(u);
            for (int t = t_lo(u); ok && t < t_end; ++t, ++i) {
                const int slot = i & 1;
                const bool last = flush && t + 1 == t_end;
                if (!wait_all(w_ready(slot), (i >> 1) & 1, FCS_STATUS_WAIT_MMA)) { ok = false; break; }
                if (fresh && fc > 0) {   // the previous sums have been read out
                    if (!wait_all(d2_empty(0), (fc - 1) & 1, FCS_STATUS_WAIT_MMA) ||
                        !wait_all(d2_empty(1), (fc - 1) & 1, FCS_STATUS_WAIT_MMA)) { ok = false; break; }
                }
                // P~ and W were written with ordinary stores by threads this warp has synchronised with (for P~ by way
                // of the exchange warps: its stores come before the statistics are posted); the fence orders
                // them before the tensor core's reads
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                tc_fence_after();
                const uint64_t da = umma_desc_mn_sw128(p_smem + slot * P_BYTES);
                const uint64_t db = umma_desc_mn_sw32(w_smem + slot * W_BYTES);
                if (elect_one_sync()) {
#pragma unroll
                    for (int hf = 0; hf < 2; ++hf) {
#pragma unroll
                        for (int ks = 0; ks < 8; ++ks)   // 16 query rows per instruction
                            umma_f16(tmem_base + D2_COL + W_N * hf, da + (uint64_t)((hf * P_TILE_BYTES + ks * 2048) >> 4),
                                     db + (uint64_t)((ks * 32 * W_N) >> 4), p.idesc_colsum, (fresh && ks == 0) ? 0u : 1u);
                        umma_commit(pw_free(slot, hf));
                        if (last) umma_commit(d2_full(hf));
                    }
                }
                __syncwarp();
                fresh = last;
                fc += last ? 1 : 0;
            }
        }
    } else {
        // ------------------------------------------------ consumers
        const int wg = warp >> 2;                  // group: columns 64*wg .. 64*wg+63 of the scores
        const int hf = wg >> 1;                    // half = key tile of the slice
        const int half64 = wg & 1;                 // 64-key half of that key tile
        const int w4 = warp & 3;                   // 32-row block of the tile
        const int row = (w4 << 5) | lane;          // tensor-memory lane = query row of the tile
        const uint32_t lane_base = tmem_base + ((uint32_t)(w4 << 5) << 16);
        const float c = p.c;
        const int keys_valid = p.Sk - (256 * (int)rank + 64 * wg);   // >= 64: the whole group is real keys
        // this thread's 128-byte line of P~ (one line per query row and 64-key group)
        const uint32_t p_line = (uint32_t)(hf * P_TILE_BYTES + half64 * P_ATOM_COL_BYTES + (row >> 3) * 1024 +
                                           (row & 7) * 128);
        const uint32_t sw = (uint32_t)(row & 7);
        // columns of the group past S_k (zero rows of the TMA box): their scores are overwritten in tensor
        // memory, so that the loop knows no masks -- in registers they cost it spills (12 % at 1024 keys), and a
        // second copy of it for the ragged group does not fit the instruction cache next to the first
        // (385-447 keys: 89 us a call against 62)
        const int padding = keys_valid < 64 ? 64 - keys_valid : 0;
        // Pairs of 16 on the FMA pipe, us per call with 2 / 3 / 4 / 5: padded, 32 x 16 x 577 keys 104.0 / 100.9 / 102.4 / 98.4,
        // 8 x 12 x 900 47.6 / 46.1 / 47.9 / 46.9, 16 x 16 x 1000 110.0 / 106.2 / 109.4 / 106.9, 8 x 16 x 1500 122.0 / 119.5 /
        // 122.3 / 120.2; in the other instance 32 x 16 x 512 keys 55.5 / 56.1 / 53.2 / 52.1, 1024 214.9 / 215.6 / 205.9 / 198.5.
        constexpr int POLY = PADDED ? 3 : FCS_POLY_PAIRS;
        // Whether the wait for tile i-2's buffers is asked early, so that the answer is there when it is needed.  Measured, not
        // derived: the two instances have their registers differently full, and each has the form that leaves it the
        // better schedule.  (us per call, 32 x 16 pairs, asked early / not: 577 keys 100.9 / 107.8; 512 keys 56.2 /
        // 52.1, 1024 keys 211.4 / 198.5.)  Another compiler may turn it over.
        constexpr bool ASK_EARLY = PADDED;
        auto consume = [&](auto keys) {
        constexpr bool KEYS = decltype(keys)::value;     // false: nothing but padding
        int i = 0, fc = 0, sb = hf, sph = 0;             // sb, sph: this half's score accumulator and its phase
        // column sums of a batch entry -> output, two tiles after its last one: the wait for that tile's
        // buffers covers the accumulators then, and nobody stands waiting for its statistics to go around
        int flush_at = 0x7fffffff;
        auto flush_sums = [&]() -> bool {
            bool good = mbar_wait(d2_full(hf), fc & 1, abort_flag, p.status, FCS_STATUS_WAIT_CONSUMER);
            good = __all_sync(0xffffffffu, good);
            if (!good) return false;
            tc_fence_after();
            if (half64 == 0) {
                uint32_t d[16];
                tmem_ld_x16(lane_base + D2_COL + W_N * hf, d);
                tmem_ld_wait16(d);
                // lanes 0..63 hold keys of the half's first group, the rest its second's: hi in column g, lo in 4 + g
                const float v0 = hf ? __uint_as_float(d[2]) + __uint_as_float(d[6]) : __uint_as_float(d[0]) + __uint_as_float(d[4]);
                const float v1 = hf ? __uint_as_float(d[3]) + __uint_as_float(d[7]) : __uint_as_float(d[1]) + __uint_as_float(d[5]);
                const int key = 256 * (int)rank + 128 * hf + row;
                const long long b = (range.g0 + (flush_at - 2)) / NQ / p.H;   // (rare enough to decode it; a register less)
                if (key < p.Sk) atomicAdd_system(p.out + b * p.out_ld + key, ((row >> 6) ? v1 : v0) * p.out_scale);
            }
            tc_fence_before();
            mbar_arrive(d2_empty(hf));
            ++fc;
            flush_at = 0x7fffffff;
            return true;
        };
        bool ok = true, ready = false;
        const int total = range.tiles();
        for (int u = u0, left = t_hi(u0) - t_lo(u0); i < total; ++i) {      // left: tiles of pair u from here on
            const int slot = i & 1;
            // ---- scores of this thread's row and group (asked for before the stores of the tile before)
            if (!__all_sync(0xffffffffu, ready)) {
                ok = mbar_wait(s_full(sb), sph, abort_flag, p.status, FCS_STATUS_WAIT_CONSUMER);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
            }
            tc_fence_after();
            uint32_t sa[32], sb_[32];   // columns 0..31 and 32..63 of the group
            if constexpr (KEYS) {
                const uint32_t scores = lane_base + 128 * sb + 64 * half64;
                if (PADDED && padding > 0) tmem_fill(scores + keys_valid, padding, __float_as_uint(-INFINITY));
                tmem_ld_x32(scores, sa);
                tmem_ld_x32(scores + 32, sb_);
                tmem_ld_wait(sa);
                tmem_ld_wait(sb_);
            }
            tc_fence_before();
            mbar_arrive(s_empty(sb));
            sb += 2;                                   // (accumulators 2 i + hf, mod 3)
            if (sb >= S_BUFS) { sb -= S_BUFS; sph ^= 1; }
            const bool freed = ASK_EARLY && mbar_test_wait(pw_free(slot, hf), ((i >> 1) & 1) ^ 1);

            // ---- P~ = exp2(c*s - m_g) as packed fp16
            uint32_t h[32];
            float m_g = -INFINITY, l_g = 0.f;
            if constexpr (KEYS) {
                // A group of nothing but -inf (masked keys) has exps of zero and no part in its row; a row of such
                // groups is NaN.  The maximum that is passed on is -inf then, and the exchange comes to NaN by
                // -inf - -inf; in the padded instance it is the floor itself, and the exchange asks for it.  (us per
                // call, 32 x 16 pairs: 1024 keys 229.6 in this form, 237.5 in the padded instance's; 577 keys 113.1
                // in the other's, 112.0 in this one; 400 60.9 / 60.1.)
                m_g = PADDED ? max3(max_of_32(sa) * c, max_of_32(sb_) * c, -FLT_MAX)
                             : max_or_nan(max_of_32(sa), max_of_32(sb_)) * c;
                const float m_safe = PADDED ? m_g : max_or_nan(m_g, -FLT_MAX);
                const f32x2 c2 = pack2(c, c), nm2 = pack2(-m_safe, -m_safe);
                f32x2 sum0 = pack2(0.f, 0.f), sum1 = sum0;
#pragma unroll
                for (int j8 = 0; j8 < 4; ++j8) exp8_packed<POLY>(j8 * 4, &sa[8 * j8], c2, nm2, sum0, sum1, &h[4 * j8]);
#pragma unroll
                for (int j8 = 0; j8 < 4; ++j8)
                    exp8_packed<POLY>(j8 * 4, &sb_[8 * j8], c2, nm2, sum0, sum1, &h[16 + 4 * j8]);
                float x0, x1;
                unpack2(add2(sum0, sum1), x0, x1);
                l_g = x0 + x1;
            }
            // ---- tile i-2 is through: its column-sum MMA has read P~(i-2), and (before that)
            // the exchange warps have read its statistics -- both slots are free
            if (!ASK_EARLY || !__all_sync(0xffffffffu, freed)) {
                ok = mbar_wait(pw_free(slot, hf), ((i >> 1) & 1) ^ 1, abort_flag, p.status, FCS_STATUS_WAIT_CONSUMER);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
            }
            if (i == flush_at) { ok = flush_sums(); if (!ok) break; }
            ready = i + 1 < total && mbar_test_wait(s_full(sb), sph);
            // ---- this group's (max, sum), for the exchange warps, and P~ for the tensor core
            lstats[(slot * sp::CONSUMER_GROUPS + wg) * 128 + row] = make_float2(m_g, l_g);
            const uint32_t line = p_smem + slot * P_BYTES + p_line;
            if constexpr (KEYS) {
                if (m_g != m_g) {   // (a NaN row: one past the query axis -- zero times a masked key -- weighs zero,
                                    // and adds nothing then; any other is NaN by its weights)
#pragma unroll
                    for (int j = 0; j < 32; ++j) h[j] = 0u;
                }
#pragma unroll
                for (int j8 = 0; j8 < 8; ++j8)
                    st_shared_v4(line + ((((uint32_t)j8) ^ sw) << 4), h[4 * j8], h[4 * j8 + 1], h[4 * j8 + 2],
                                 h[4 * j8 + 3]);
            } else if (i < 2) {      // a group without keys: its exps are zero in both buffers, for good
                for (int j8 = 0; j8 < 8; ++j8) st_shared_v4(line + 16 * j8, 0u, 0u, 0u, 0u);
            }
            // (the column-sum warp makes these stores visible to the tensor core: it fences after its wait)
            mbar_arrive(stats_bar(slot));
            if (--left == 0) {
                if (last_of_batch(u)) {
                    // (a batch entry of one tile: the one before it is still to be written out)
                    if (flush_at != 0x7fffffff) { ok = flush_sums(); if (!ok) break; }
                    flush_at = i + 2;
                }
                ++u;
                left = u < u1 ? t_hi(u) - t_lo(u) : 0;
            }
        }
        if (ok && flush_at != 0x7fffffff) flush_sums();
        };
        if (keys_valid > 0) consume(Flag<true>{});
        else consume(Flag<false>{});
    }

    // ---------------------------------------------------- teardown
    tc_fence_before();
    __syncthreads();
    if constexpr (CLMAX > 1) cluster_sync_all();   // nobody leaves while a peer may still write into its shared memory
    if (warp == COLSUM_WARP) {
        if (*abort_flag) __nanosleep(1000000);   // let copies and MMAs in flight land
        tc_fence_after();
        tmem_dealloc(tmem_base, TMEM_COLS);
    }
}

}  // namespace fcs
