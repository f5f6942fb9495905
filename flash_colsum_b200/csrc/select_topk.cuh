// Token pruning on top of the column means, on the stream that produced the means: per batch
// row the k key positions with the largest mean, or those that reach a threshold, in ascending
// position order (top-k ties go to the lower position).
//
// A row belongs to one thread-block cluster of 1, 2, 4, 8 or 16 CTAs, each of which holds a
// contiguous slice of it: the row is read once, through shared memory into registers (a thread
// holds `E` consecutive elements), and everything after that is on chip.  Only slices of more
// than 16384 elements (rows past 262144) are read again, from L2, by every pass.
//
//   top-k      exact radix selection, 11 bits at a time from the top (8 for rows of at most
//              1024, where scanning 2048 bins costs more than a fourth pass): every CTA
//              counts its elements that still match the prefix chosen so far, sums its bins in
//              groups of 32 and stores the group sums into every CTA of the cluster; after the pass's only
//              cluster barrier one warp of every CTA finds the group the k-th largest falls into,
//              reads that group's bins of all CTAs through distributed shared memory and finds the
//              bin -- every CTA for itself.  What it adds up for the CTAs before its own, in
//              the bins passed over and in the bin chosen, says where its elements go: there is nothing to
//              exchange at the end.  A bin that is wanted whole ends the selection early.
//   threshold  (with `relative`: against a share of the row's average) a comparison per element; the counts
//              of the CTAs are exchanged once.
//   both       one scan over the block of the kept elements per thread, and every kept element
//              knows its place in the output.
//
// What bounds it: a dozen dependent steps of half a microsecond to one (launch of the cluster,
// load, cluster barriers, scans), not bytes.  Back to back on a B200, one CTA per row going over
// it from L2 with an element per thread and step (the form before) against this one: the 16384
// largest of 131072 216 -> 14.6 us, 2048 of 16384 32 -> 7.5, 32 rows of 65536 118 -> 31; values
// above the mean, 131072 122 -> 11.6 us, 32 rows of 65536 64 -> 13.6.  Rows of a few thousand are
// bound by the host (4.4 us a call).  Since then the group sums are stored into the peers and nothing is exchanged at
// the end, and rows of 131072 go to sixteen CTAs where they can: 11.1 or 14.0 us a call, 12.5 or 15.0 on eight -- a call of
// this kernel takes one of two times, 2 to 3 us apart, and keeps to it for a while; why is not known.  Four copies of the first pass's bins, against lanes meeting
// on one bin, were no faster (14.9 us): the hardware adds equal addresses of a warp in one go.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "colsum_small_q.cuh"
#include "sm100_ptx.cuh"

namespace fcs {
namespace sel {

constexpr int MAX_CL = 16;         // (above eight: an opt-in of the launch)

// Order-reversing map from float to unsigned (larger float -> smaller key), and its inverse.
__device__ __forceinline__ uint32_t key_of(uint32_t bits) {
    return (bits & 0x80000000u) ? bits : ~(bits | 0x80000000u);
}
__device__ __forceinline__ uint32_t bits_of(uint32_t key) {
    return (key & 0x80000000u) ? key : ~key & 0x7fffffffu;
}
__device__ __forceinline__ uint32_t ld_peer_u32(uint32_t local_addr, uint32_t rank) {
    uint32_t addr, v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(addr) : "r"(local_addr), "r"(rank));
    asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ void st_peer_u32(uint32_t local_addr, uint32_t rank, uint32_t v) {
    uint32_t addr;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(addr) : "r"(local_addr), "r"(rank));
    asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}
// The sum over the first `n` of the cluster's CL CTAs of the word at `local_addr` in each, all loads in
// flight at once (a loop over a runtime count waits for each: half a microsecond more per pass).
template <int CL>
__device__ __forceinline__ uint32_t sum_over_cluster(uint32_t local_addr, uint32_t n = CL) {
    uint32_t v[CL], sum = 0;
#pragma unroll
    for (int r = 0; r < CL; ++r) v[r] = (uint32_t)r < n ? ld_peer_u32(local_addr, (uint32_t)r) : 0u;
#pragma unroll
    for (int r = 0; r < CL; ++r) sum += v[r];
    return sum;
}
__device__ __forceinline__ void cluster_sync() {
    smallq_cluster_arrive();
    smallq_cluster_wait();
}
__device__ __forceinline__ uint32_t warp_scan(uint32_t v, int lane) {   // inclusive
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += t;
    }
    return v;
}

// One CTA's part of a row: elements [lo, hi), in tiles of NT * E.
template <int NT, int E>
struct Slice {
    static constexpr int TILE_ELEMS = NT * E;
    static constexpr int PITCH = E + 1;             // a thread's run in shared memory, conflict-free
    const uint32_t* row;
    uint32_t* stage;                                // [NT * PITCH]
    uint32_t lo, hi;
    int tiles;

    __device__ void init(const float* row_, uint32_t* stage_, int S, int cl, uint32_t rank) {
        row = reinterpret_cast<const uint32_t*>(row_);
        stage = stage_;
        const uint32_t n = (uint32_t)S, per = (n + cl - 1) / cl;
        lo = rank * per < n ? rank * per : n;
        hi = n - lo < per ? n : lo + per;
        tiles = (int)((per + TILE_ELEMS - 1) / TILE_ELEMS);
    }
    __device__ uint32_t first(int tile) const { return lo + (uint32_t)tile * TILE_ELEMS + threadIdx.x * E; }
    // This thread's E consecutive elements of a tile, as bits.  (Elements at hi and past it are undefined.)
    __device__ void load(int tile, uint32_t (&v)[E]) const {
        const uint32_t base = lo + (uint32_t)tile * TILE_ELEMS;
        uint32_t t[E];
#pragma unroll
        for (int j = 0; j < E; ++j) {
            const uint32_t i = base + j * NT + threadIdx.x;
            t[j] = i < hi ? row[i] : 0u;
        }
        if (tile > 0) __syncthreads();              // (the tile before has been taken out of the stage)
#pragma unroll
        for (int j = 0; j < E; ++j) {
            const int at = j * NT + (int)threadIdx.x;
            stage[at + at / E] = t[j];
        }
        __syncthreads();
#pragma unroll
        for (int j = 0; j < E; ++j) v[j] = stage[(int)threadIdx.x * PITCH + j];
    }
};

// Exclusive scan over the block of one packed count per thread; `total` is the block's sum.
template <int NT>
__device__ __forceinline__ uint32_t block_scan(uint32_t v, uint32_t* warp_sums, uint32_t& total) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const uint32_t inc = warp_scan(v, lane);
    __syncthreads();                                // (warp_sums of the scan before have been read)
    if (lane == 31) warp_sums[wid] = inc;
    __syncthreads();
    const uint32_t w = lane < NT / 32 ? warp_sums[lane] : 0u;
    const uint32_t ws = warp_scan(w, lane);
    total = __shfl_sync(0xffffffffu, ws, 31);
    const uint32_t before = __shfl_sync(0xffffffffu, ws, wid == 0 ? 0 : wid - 1);
    return inc - v + (wid == 0 ? 0u : before);
}

template <int NT, int E>
constexpr int stage_bytes() { return NT * (E + 1) * 4; }
template <int BITS>
struct Digits {
    static constexpr int BINS = 1 << BITS, GROUPS = BINS / 32, PASSES = (32 + BITS - 1) / BITS;
};
template <int NT, int E, int BITS, int CL>
constexpr int topk_smem() {
    return stage_bytes<NT, E>() + Digits<BITS>::PASSES * (Digits<BITS>::BINS + CL * Digits<BITS>::GROUPS) * 4;
}

template <int NT, int E, int BITS, int CL>
__global__ void __launch_bounds__(NT)
topk_kernel(const float* __restrict__ colsum, long long ld, int S, int k, int* __restrict__ indices,
            float* __restrict__ values) {
    constexpr int BINS = Digits<BITS>::BINS, GROUPS = Digits<BITS>::GROUPS, PASSES = Digits<BITS>::PASSES;
    constexpr int GPL = (GROUPS + 31) / 32;         // groups per lane of the choosing warp
    extern __shared__ __align__(16) uint32_t sel_smem[];
    uint32_t* stage = sel_smem;
    uint32_t* hist = sel_smem + NT * (E + 1);       // [PASSES][BINS]: a fresh one per pass, cleared once
    uint32_t* gsum = hist + PASSES * BINS;          // [PASSES][CL][GROUPS]: of every CTA
    __shared__ uint32_t warp_sums[32];
    __shared__ uint32_t choice[5];                  // digit, elements before its bin, in it, and both of the CTAs before this
    const uint32_t rank = smallq_cluster_rank();
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const long long b = blockIdx.x / CL;

    for (int i = threadIdx.x; i < PASSES * BINS; i += NT) hist[i] = 0u;
    if constexpr (CL > 1) smallq_cluster_arrive();  // (waited for before the first store into a peer)
    grid_dependency_wait();
    grid_launch_dependents();
    Slice<NT, E> sl;
    sl.init(colsum + b * ld, stage, S, CL, rank);
    uint32_t key[E];
    auto fetch = [&](int tile) {
        sl.load(tile, key);
#pragma unroll
        for (int j = 0; j < E; ++j) key[j] = key_of(key[j]);
    };
    const bool resident = sl.tiles == 1;
    if (resident) fetch(0);
    else __syncthreads();                           // (the bins are clear)
    if constexpr (CL > 1) smallq_cluster_wait();

    // ---- the k-th smallest key, BITS bits at a time
    uint32_t prefix = 0, mask = 0, need = (uint32_t)k;   // `need`: still to take among the elements matching `prefix`
    uint32_t lt0 = 0, eq0 = 0;                           // elements of the CTAs before this one: below the prefix, matching it
    for (int pass = 0; pass < PASSES; ++pass) {
        const int shift = 32 - BITS * (pass + 1) > 0 ? 32 - BITS * (pass + 1) : 0;
        const uint32_t digits = pass == PASSES - 1 ? (1u << (32 - BITS * pass)) - 1u : (uint32_t)(BINS - 1);
        uint32_t* h = hist + pass * BINS;
        uint32_t* gs = gsum + pass * CL * GROUPS;
        for (int tile = 0; tile < sl.tiles; ++tile) {
            if (!resident) fetch(tile);
            const uint32_t i0 = sl.first(tile);
#pragma unroll
            for (int j = 0; j < E; ++j)
                if (i0 + j < sl.hi && (key[j] & mask) == prefix) atomicAdd(&h[(key[j] >> shift) & digits], 1u);
        }
        __syncthreads();
        for (int g = wid; g < GROUPS; g += NT / 32) {
            uint32_t v = h[g * 32 + lane];
            v = __reduce_add_sync(0xffffffffu, v);
            if constexpr (CL > 1) {
                if (lane < CL) st_peer_u32(smem_u32(gs + rank * GROUPS + g), (uint32_t)lane, v);
            } else {
                if (lane == 0) gs[g] = v;
            }
        }
        if constexpr (CL > 1) cluster_sync(); else __syncthreads();
        if (wid == 0) {
            uint32_t gv[GPL], gl[GPL], sum = 0, low = 0;    // of all CTAs, and of those before this one
#pragma unroll
            for (int i = 0; i < GPL; ++i) {
                const int g = lane * GPL + i;
                gv[i] = gl[i] = 0u;
#pragma unroll
                for (int r = 0; r < CL; ++r) {
                    const uint32_t x = g < GROUPS ? gs[r * GROUPS + g] : 0u;
                    gv[i] += x;
                    gl[i] += (uint32_t)r < rank ? x : 0u;
                }
                sum += gv[i];
                low += gl[i];
            }
            const uint32_t inc = warp_scan(sum, lane);
            const int f = __ffs(__ballot_sync(0xffffffffu, inc >= need)) - 1;
            uint32_t before = inc - sum, low_before = CL > 1 ? warp_scan(low, lane) - low : 0u;    // (of lane f, below)
            int g = lane * GPL;
#pragma unroll
            for (int i = 0; i + 1 < GPL; ++i)
                if (before + gv[i] < need && g == lane * GPL + i) { before += gv[i]; low_before += gl[i]; ++g; }
            g = __shfl_sync(0xffffffffu, g, f);
            before = __shfl_sync(0xffffffffu, before, f);
            low_before = __shfl_sync(0xffffffffu, low_before, f);
            uint32_t bins[CL], v = 0, lv = 0;
#pragma unroll
            for (int r = 0; r < CL; ++r)             // (all loads in flight at once)
                bins[r] = CL > 1 ? ld_peer_u32(smem_u32(h + g * 32 + lane), (uint32_t)r) : h[g * 32 + lane];
#pragma unroll
            for (int r = 0; r < CL; ++r) { v += bins[r]; lv += (uint32_t)r < rank ? bins[r] : 0u; }
            const uint32_t vi = before + warp_scan(v, lane);
            const uint32_t li = low_before + (CL > 1 ? warp_scan(lv, lane) - lv : 0u);
            const int d = __ffs(__ballot_sync(0xffffffffu, vi >= need)) - 1;
            if (lane == d) { choice[0] = (uint32_t)(g * 32 + d); choice[1] = vi - v; choice[2] = v; choice[3] = li; choice[4] = lv; }
        }
        __syncthreads();
        prefix |= choice[0] << shift;
        mask |= digits << shift;
        need -= choice[1];
        lt0 += choice[3];
        eq0 = choice[4];
        const bool whole = choice[2] == need;       // every element of the bin is wanted
        if (whole) break;
    }

    // ---- every element's place: the elements of its CTA before it, below the prefix and matching it
    auto counts = [&](int tile) {
        uint32_t c = 0;
        const uint32_t i0 = sl.first(tile);
#pragma unroll
        for (int j = 0; j < E; ++j) {
            const uint32_t m = key[j] & mask;
            if (i0 + j < sl.hi) c += m < prefix ? 1u : m == prefix ? 0x10000u : 0u;
        }
        return c;
    };
    uint32_t scan = 0, tile_total = 0;              // (counts of a tile fit 16 bits each: at most NT * E = 16384)
    if constexpr (CL > 1) smallq_cluster_arrive();  // nobody leaves before its peers have read its bins
    int* out_idx = indices + b * k;
    float* out_val = values ? values + b * k : nullptr;
    for (int tile = 0; tile < sl.tiles; ++tile) {
        if (!resident) fetch(tile);
        scan = block_scan<NT>(counts(tile), warp_sums, tile_total);
        uint32_t lt = lt0 + (scan & 0xffffu), eq = eq0 + (scan >> 16);
        const uint32_t i0 = sl.first(tile);
#pragma unroll
        for (int j = 0; j < E; ++j) {
            const uint32_t m = key[j] & mask;
            const bool in = i0 + j < sl.hi, below = in && m < prefix, equal = in && m == prefix;
            if (below || (equal && eq < need)) {
                const uint32_t pos = lt + (eq < need ? eq : need);
                out_idx[pos] = (int)(i0 + j);
                if (out_val) out_val[pos] = __uint_as_float(bits_of(key[j]));
            }
            lt += below ? 1u : 0u;
            eq += equal ? 1u : 0u;
        }
        lt0 += tile_total & 0xffffu;
        eq0 += tile_total >> 16;
    }
    if constexpr (CL > 1) smallq_cluster_wait();
}

// The threshold form: positions whose column mean is at least `threshold` (relative = 0) or at
// least `threshold` times the row's mean value (relative = 1; the means of a row sum to one, so
// that is threshold / S), ascending, in indices[row][0 .. counts[row]); the rest of the row of
// `indices` is filled with -1.
//
// The row sum is added up in one fixed order whatever the cluster size -- 1024 strided partial
// sums, each in index order, then a tree over 32 and a run over 32 -- so that a value that ties
// with the threshold to the last bit is kept or not by the same arithmetic everywhere.
constexpr int SUM_LANES = 1024;

template <int NT, int E, int CL>
__global__ void __launch_bounds__(NT)
threshold_kernel(const float* __restrict__ colsum, long long ld, int S, float threshold, int relative,
                 int* __restrict__ indices, int* __restrict__ counts_out) {
    extern __shared__ __align__(16) uint32_t sel_smem[];
    __shared__ uint32_t warp_sums[32];
    __shared__ uint32_t totals[1];
    __shared__ uint32_t part_sums[32];              // (bits) sums over 32 strided partial sums each
    __shared__ float row_thr;
    const uint32_t rank = smallq_cluster_rank();
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const long long b = blockIdx.x / CL;
    grid_dependency_wait();
    grid_launch_dependents();
    const float* row = colsum + b * ld;
    Slice<NT, E> sl;
    sl.init(row, sel_smem, S, CL, rank);
    uint32_t v[E];
    const bool resident = sl.tiles == 1;
    if (resident) sl.load(0, v);
    float thr = threshold;
    if (relative) {
        // this CTA's share of the strided partial sums
        const int lanes = SUM_LANES / CL, t0 = (int)rank * lanes;
        for (int t = threadIdx.x; t < lanes; t += NT) {
            float part = 0.f;
            int i = t0 + t;
            for (; i + 15 * SUM_LANES < S; i += 16 * SUM_LANES) {
                float x[16];
#pragma unroll
                for (int j = 0; j < 16; ++j) x[j] = row[i + j * SUM_LANES];
#pragma unroll
                for (int j = 0; j < 16; ++j) part += x[j];
            }
            for (; i < S; i += SUM_LANES) part += row[i];
            for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
            if (lane == 0) part_sums[t >> 5] = __float_as_uint(part);
        }
        if constexpr (CL > 1) cluster_sync(); else __syncthreads();
        if (wid == 0) {
            const int per = lanes / 32;             // part_sums per CTA
            const float mine = __uint_as_float(ld_peer_u32(smem_u32(&part_sums[lane % per]), (uint32_t)(lane / per)));
            float total = 0.f;
            for (int w = 0; w < 32; ++w) total += __shfl_sync(0xffffffffu, mine, w);
            if (lane == 0) row_thr = threshold * total / (float)S;
        }
        __syncthreads();
        thr = row_thr;
    }
    auto counts = [&](int tile) {
        uint32_t c = 0;
        const uint32_t i0 = sl.first(tile);
#pragma unroll
        for (int j = 0; j < E; ++j) c += (i0 + j < sl.hi && __uint_as_float(v[j]) >= thr) ? 1u : 0u;
        return c;
    };
    uint32_t scan = 0, tile_total = 0, n = 0;
    for (int tile = 0; tile < sl.tiles; ++tile) {
        if (!resident) sl.load(tile, v);
        scan = block_scan<NT>(counts(tile), warp_sums, tile_total);
        n += tile_total;
    }
    uint32_t before = 0, all = n;
    if constexpr (CL > 1) {
        if (threadIdx.x == 0) totals[0] = n;
        cluster_sync();
        before = sum_over_cluster<CL>(smem_u32(&totals[0]), rank);
        all = sum_over_cluster<CL>(smem_u32(&totals[0]));
        smallq_cluster_arrive();                    // nobody leaves before its peers have read its count
    }
    int* out_idx = indices + b * S;
    for (int tile = 0; tile < sl.tiles; ++tile) {
        if (!resident) {
            sl.load(tile, v);
            scan = block_scan<NT>(counts(tile), warp_sums, tile_total);
        }
        uint32_t pos = before + scan;
        const uint32_t i0 = sl.first(tile);
#pragma unroll
        for (int j = 0; j < E; ++j)
            if (i0 + j < sl.hi && __uint_as_float(v[j]) >= thr) out_idx[pos++] = (int)(i0 + j);
        before += tile_total;
    }
    for (long long i = (long long)all + (long long)rank * NT + threadIdx.x; i < S; i += (long long)CL * NT) out_idx[i] = -1;
    if (rank == 0 && threadIdx.x == 0) counts_out[b] = (int)all;
    if constexpr (CL > 1) smallq_cluster_wait();
}

// CTAs per row: as many as it takes for 4096 elements each, at most eight -- or sixteen where that
// keeps the slices in registers (more than 131072 elements; one row of 262144: 17.7 us against 38).
// (Below that sixteen lose to eight in general: the cluster barriers and the launch grow with the cluster, and fewer
// of them run at once.  Top-k calls of few rows have a line of their own, topk_on_sixteen.)
inline int cluster_size(int S) {
    const int most = S > 8 * 16384 ? MAX_CL : 8;
    int cl = 1;
    while (cl < most && (long long)cl * 4096 < S) cl *= 2;
    return cl;
}

}  // namespace sel
}  // namespace fcs
