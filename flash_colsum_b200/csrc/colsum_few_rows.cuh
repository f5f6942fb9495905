// Column mean of at most four query rows (a CLS prefix, decode queries) in two kernels over
// scratch memory: R dot products per key, bound by reading every key once.
//
//   scores   The rows of all (batch, head) units' keys are one list, cut evenly over one
//            persistent CTA per SM -- through units where need be, so that every SM streams the same
//            number of bytes whatever the number of heads.  One warp fills a ring of 16 KiB
//            shared-memory stages (tensor-map tiles of whole rows, contiguous or strided alike;
//            untiled bulk copies were no faster, and 20 % slower in 8 KiB pieces) and runs
//            ahead of eight consumer warps across the unit boundaries.
//            A pair of consumer warps takes every fourth stage: the dot products are m16n8k16
//            matrix instructions, 16 keys by 8 query columns of which R are real -- a warp-wide
//            dot product spends its time on converting 16-bit values and on shuffles, an
//            order of magnitude more instructions, and with four query rows took longer than the memory.
//            (The fifth-generation matrix unit has nothing to win at 8 columns: the scores would have
//            to come back through tensor memory.)  Scores (log2 domain) go to scratch,
//            with one (maximum, sum of exp2) per row, warp and piece of a unit: the warps never
//            meet.
//   columns  Every key's exp2(score - maximum) / sum over the heads and rows, written once: no adds
//            into memory, nothing to clear, the same bits every time.
//
// Against the one-kernel form of colsum_small_q.cuh (whose clusters keep the scores on chip but
// can only use as many SMs as whole clusters per head come to: 128 of 148 for 32 heads) this
// reads and writes 4 bytes per key and row more, next to 2 D bytes of key.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "colsum_small_q.cuh"
#include "sm100_ptx.cuh"

namespace fcs {
namespace few {

constexpr int MAX_ROWS = 4;
constexpr int CONSUMER_WARPS = 8;
constexpr int GANGS = 4;                    // consumer warps come in pairs, a stage is a pair's
constexpr int GANG_WARPS = CONSUMER_WARPS / GANGS;
constexpr int CONSUMER_THREADS = 32 * CONSUMER_WARPS;
constexpr int THREADS = CONSUMER_THREADS + 32;
constexpr int RING_BYTES = 192 * 1024;
constexpr int MAX_STAGES = 12;
constexpr int MIN_SHARE = 128;              // key rows that are worth a CTA
// the columns kernel: COLUMN_KEYS keys by COLUMN_SLICES slices of the heads per CTA
constexpr int COLUMN_KEYS = 128;
constexpr int COLUMN_SLICES = 2;
constexpr int COLUMN_THREADS = COLUMN_KEYS * COLUMN_SLICES;
constexpr int COLUMN_PAIRS = 32;            // (head, row) pairs whose statistics are held at a time
constexpr int COLUMN_PER_SLICE = COLUMN_PAIRS / COLUMN_SLICES;
static_assert(COLUMN_PAIRS * CONSUMER_WARPS == COLUMN_THREADS, "eight threads merge a pair's statistics");

enum : int { T_FP16 = 0, T_BF16 = 1, T_FP32 = 2 };

struct Params {
    const void* q;
    float* out;
    long long out_ld;
    int H, R, D, Sk;
    int units;                // (batch, head) pairs
    int keys;                 // keys that some row sees; the columns past them are zero
    int share;                // key rows per CTA
    int slots;                // most pieces a unit is cut into
    long long qsb, qsh, qss;  // in elements
    float c;                  // scale * log2(e), sign included
    int causal, k_past;
    float inv_norm;           // 1 / (h_norm * R)
    float* scores;            // [units][R][score_ld]
    long long score_ld;
    float2* part;             // [units][slots][CONSUMER_WARPS][MAX_ROWS] (maximum, sum)
    int* status;
};

constexpr int SMEM_BYTES = RING_BYTES + 2 * MAX_STAGES * 8 + 16 + 1024;

// A ring stage: rows of one unit, one after the other.  Stage n of a CTA is gang n % 4's, in the
// (n / 4) % DEPTH-th of that gang's own slots: the parity of a slot's barrier is told apart by warps that
// use it in order and one phase from each other at most, whatever the other gangs are at.
template <int DK, int T>
struct Stage {
    static constexpr int ROWS = T == T_FP32 ? 64 : 128 * 64 / DK;
    static constexpr int WARP_ROWS = ROWS / GANG_WARPS;
    static constexpr int BYTES = ROWS * DK * (T == T_FP32 ? 4 : 2);
    static constexpr int DEPTH = RING_BYTES / BYTES / GANGS;
    static constexpr int COUNT = DEPTH * GANGS;
    static_assert(DEPTH >= 1 && COUNT <= MAX_STAGES, "a stage per gang");
};

// The unit that row `g` of the list belongs to (32-bit division where the list allows it: a 64-bit one
// is a hundred instructions).
__device__ __forceinline__ int unit_of(long long g, int keys) {
    return g <= 0xffffffffll ? (int)((unsigned)g / (unsigned)keys) : (int)(g / keys);
}
__device__ __forceinline__ int cta_of(long long g, int share) {
    return g <= 0xffffffffll ? (int)((unsigned)g / (unsigned)share) : (int)(g / share);
}

// d += a (16 x 16, row) * b (16 x 8, column), fp32 accumulators
template <bool BF16>
__device__ __forceinline__ void mma_16x8x16(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                            uint32_t b1) {
    if constexpr (BF16)
        asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                     : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                     : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
    else
        asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                     : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                     : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// A consumer warp's dot products of one stage: `run` leaves in v[i][j] the product of the key row
// `row_of(i)` of the stage and the query column `first_col() + j`; the lanes that differ in the bits
// from LANE_STEP up hold the same columns.
//
// 16-bit operands.  The order of the contraction is free as long as both operands have it: lane
// quarter t = lane % 4 reads 16 bytes -- elements 8 (4 j + t) .. + 7 of its rows -- at once, and they
// serve as the operands of two 16-wide steps.  (Rows a multiple of 128 bytes apart: these loads
// conflict two ways, which leaves them at three times the rate the keys arrive at.)
template <int DK, bool BF16>
struct MatrixDots {
    static constexpr int STEPS = DK / 32;            // pairs of 16-wide steps
    static constexpr int COLS = 2, LANE_STEP = 4;
    template <int ROWS> struct Values { static constexpr int N = ROWS / 8; };
    uint4 q[STEPS];                                  // of query column lane / 4

    __device__ static uint4 chunk(const uint8_t* row, int c, int D) {
        return c * 8 < D ? *reinterpret_cast<const uint4*>(row + c * 16) : make_uint4(0u, 0u, 0u, 0u);
    }
    __device__ void load_queries(const Params& p, int unit, int lane) {
        const int bb = unit / p.H, h = unit - bb * p.H, col = lane >> 2;
        const uint16_t* row = reinterpret_cast<const uint16_t*>(p.q) + (long long)bb * p.qsb + (long long)h * p.qsh +
                              (long long)col * p.qss;
#pragma unroll
        for (int j = 0; j < STEPS; ++j)
            q[j] = col < p.R ? chunk(reinterpret_cast<const uint8_t*>(row), 4 * j + (lane & 3), p.D) : make_uint4(0u, 0u, 0u, 0u);
    }
    __device__ static int first_col(int lane) { return (lane & 3) * 2; }
    __device__ static int row_of(int i, int lane) { return i * 8 + (lane >> 2); }

    template <int ROWS>
    __device__ void run(const uint8_t* rows, int lane, int D, float (&v)[ROWS / 8][COLS]) const {
        const int pitch = D * 2;
        const uint8_t* base = rows + (lane >> 2) * pitch;
#pragma unroll
        for (int t = 0; t < ROWS / 16; ++t) {
            float d[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int j = 0; j < STEPS; ++j) {
                const uint4 a = chunk(base + (t * 16) * pitch, 4 * j + (lane & 3), D);
                const uint4 b = chunk(base + (t * 16 + 8) * pitch, 4 * j + (lane & 3), D);
                mma_16x8x16<BF16>(d, a.x, b.x, a.y, b.y, q[j].x, q[j].y);
                mma_16x8x16<BF16>(d, a.z, b.z, a.w, b.w, q[j].z, q[j].w);
            }
            v[2 * t][0] = d[0]; v[2 * t][1] = d[1];
            v[2 * t + 1][0] = d[2]; v[2 * t + 1][1] = d[3];
        }
    }
};

// fp32 inputs count as rounded to fp16 (what the tensor-core forms do with them); values that do
// not fit that are taken as they are.
__device__ __forceinline__ float as_fp16(float x) {
    return fabsf(x) < 60000.f ? __half2float(__float2half_rn(x)) : x;
}

// fp32 operands: DK / 8 adjacent lanes to a key row, eight elements each (4 piece .. + 3 and
// DK / 2 + 4 piece .. + 3: adjacent lanes read adjacent 16 bytes), over DK / 8 passes for 32 rows; the
// partial products are transposed and summed with DK / 8 - 1 shuffles.
template <int DK, int R>
struct FloatDots {
    static constexpr int LPR = DK / 8, RPW = 32 / LPR;
    static constexpr int COLS = R, LANE_STEP = 1;
    template <int ROWS> struct Values { static constexpr int N = ROWS / 32; };
    float q[R][8];

    __device__ static void load_piece(const float* row, int piece, int D, float (&f)[8]) {
        float4 a = make_float4(0.f, 0.f, 0.f, 0.f), b = a;
        if (piece * 4 < D) a = *reinterpret_cast<const float4*>(row + piece * 4);
        if ((LPR + piece) * 4 < D) b = *reinterpret_cast<const float4*>(row + (LPR + piece) * 4);
        f[0] = as_fp16(a.x); f[1] = as_fp16(a.y); f[2] = as_fp16(a.z); f[3] = as_fp16(a.w);
        f[4] = as_fp16(b.x); f[5] = as_fp16(b.y); f[6] = as_fp16(b.z); f[7] = as_fp16(b.w);
    }
    __device__ void load_queries(const Params& p, int unit, int lane) {
        const int bb = unit / p.H, h = unit - bb * p.H;
        const float* qb = reinterpret_cast<const float*>(p.q) + (long long)bb * p.qsb + (long long)h * p.qsh;
#pragma unroll
        for (int r = 0; r < R; ++r) {
            if (r < p.R) load_piece(qb + (long long)r * p.qss, lane % LPR, p.D, q[r]);
            else
#pragma unroll
                for (int j = 0; j < 8; ++j) q[r][j] = 0.f;
        }
    }
    __device__ static int first_col(int) { return 0; }
    __device__ static int row_of(int i, int lane) { return i * 32 + (lane % LPR) * RPW + lane / LPR; }

    template <int ROWS>
    __device__ void run(const uint8_t* stage, int lane, int D, float (&v)[ROWS / 32][R]) const {
        const int piece = lane % LPR, sub = lane / LPR;
#pragma unroll
        for (int t = 0; t < ROWS / 32; ++t) {
            float part[R][LPR];
#pragma unroll
            for (int j = 0; j < LPR; ++j) {
                float f[8];
                load_piece(reinterpret_cast<const float*>(stage) + (t * 32 + j * RPW + sub) * D, piece, D, f);
#pragma unroll
                for (int r = 0; r < R; ++r)
                    part[r][j] = ((f[0] * q[r][0] + f[1] * q[r][1]) + (f[2] * q[r][2] + f[3] * q[r][3])) +
                                 ((f[4] * q[r][4] + f[5] * q[r][5]) + (f[6] * q[r][6] + f[7] * q[r][7]));
            }
#pragma unroll
            for (int half = LPR / 2; half >= 1; half >>= 1) {
                const bool up = (piece & half) != 0;
#pragma unroll
                for (int r = 0; r < R; ++r)
#pragma unroll
                    for (int x = 0; x < half; ++x) {
                        const float send = up ? part[r][x] : part[r][x + half];
                        const float keep = up ? part[r][x + half] : part[r][x];
                        part[r][x] = keep + __shfl_xor_sync(0xffffffffu, send, half);
                    }
            }
#pragma unroll
            for (int r = 0; r < R; ++r) v[t][r] = part[r][0];
        }
    }
};

template <int DK, int T, int R> struct DotsOf { typedef MatrixDots<DK, T == T_BF16> type; };
template <int DK, int R> struct DotsOf<DK, T_FP32, R> { typedef FloatDots<DK, R> type; };

// The scores of one query column of a stage: scaled, hidden ones -inf, kept at `dst`, and the lane's
// running (maximum, sum of exp2) with them.  lo: the piece's first key; r0: the stage's first row in the
// piece of `rows`.
template <typename Dots, int NV, int COLS>
__device__ __forceinline__ void keep_scores(const Params& p, const float (&v)[NV][COLS], int j, int col, int lo, int r0,
                                            int rows, int lane, float* dst, float& tm, float& tl) {
    float s[NV], m = tm;
#pragma unroll
    for (int x = 0; x < NV; ++x) {
        const int kl = r0 + Dots::row_of(x, lane);
        const bool seen = kl < rows && (!p.causal || lo + kl <= p.k_past + col);
        s[x] = seen ? v[x][j] * p.c : -INFINITY;
        if (kl < rows) dst[kl] = s[x];
        m = max_or_nan(m, s[x]);
    }
    if (m != -INFINITY) {
        float l = tl * ex2_approx(tm - m);
#pragma unroll
        for (int x = 0; x < NV; ++x) l += ex2_approx(s[x] - m);
        tl = l;
        tm = m;
    }
}
__device__ __forceinline__ float ld_peer_f32(uint32_t local_addr, uint32_t rank) {
    uint32_t addr;
    float v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(addr) : "r"(local_addr), "r"(rank));
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
    return v;
}

// DK: 64 or 128, a bound on the head dimension; R: a bound on the query rows (fp32 operands: 1 or 4;
// 16-bit operands: 4, the matrix instruction has eight columns anyway).
template <int DK, int T, int R>
__global__ void __launch_bounds__(THREADS, 1)
few_rows_scores_kernel(const __grid_constant__ CUtensorMap tm_k, const Params p) {
    using S = Stage<DK, T>;
    using Dots = typename DotsOf<DK, T, R>::type;
    extern __shared__ uint8_t few_smem[];
    uint8_t* ring = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(few_smem) + 1023) & ~static_cast<uintptr_t>(1023));
    uint8_t* fixed = ring + RING_BYTES;
    const uint32_t bars = smem_u32(fixed);
    auto full_bar = [&](int s) { return bars + 8u * s; };
    auto empty_bar = [&](int s) { return bars + 8u * (S::COUNT + s); };
    volatile int* abort_flag = reinterpret_cast<volatile int*>(fixed + 2 * MAX_STAGES * 8);

    grid_launch_dependents();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // this CTA's rows of the list, and the unit they start in
    const long long total = (long long)p.units * p.keys;
    long long g0 = (long long)blockIdx.x * p.share, g1 = g0 + p.share;
    if (g0 > total) g0 = total;
    if (g1 > total) g1 = total;
    const int u_first = unit_of(g0, p.keys);
    int lo = (int)(g0 - (long long)u_first * p.keys);
    long long left = g1 - g0;

    if (threadIdx.x == 0) {
        for (int s = 0; s < S::COUNT; ++s) { mbar_init(full_bar(s), 1); mbar_init(empty_bar(s), GANG_WARPS); }
        *abort_flag = 0;
        mbar_fence_init();
        prefetch_tensormap(&tm_k);
    }
    __syncthreads();
    grid_dependency_wait();

    if (warp == CONSUMER_WARPS) {
        // ------------------------------------------------ copies
        int n = 0;
        bool ok = true;
        for (int u = u_first; left > 0 && ok; ++u, lo = 0) {
            const int rows = p.keys - lo < left ? p.keys - lo : (int)left;
            const int b = u / p.H, h = u - b * p.H;
            for (int r = 0; r < rows; r += S::ROWS, ++n) {
                const int m = n / GANGS, slot = (n % GANGS) * S::DEPTH + m % S::DEPTH;
                if (n >= S::COUNT) {
                    ok = mbar_wait(empty_bar(slot), ((m / S::DEPTH) & 1) ^ 1, abort_flag, p.status, FCS_STATUS_WAIT_PRODUCER);
                    ok = __all_sync(0xffffffffu, ok);
                    if (!ok) break;
                }
                if (elect_one_sync()) {
                    // (a whole tile: rows past the unit's keys read as zero and cost no traffic, rows past this
                    // CTA's piece are not looked at)
                    mbar_arrive_expect_tx(full_bar(slot), (uint32_t)(S::ROWS * p.D * (T == T_FP32 ? 4 : 2)));
                    tma_load_4d(smem_u32(ring + slot * S::BYTES), &tm_k, full_bar(slot), 0, lo + r, h, b);
                }
                __syncwarp();
            }
            left -= rows;
        }
        return;
    }

    // ---------------------------------------------------- consumers: stage n is gang n % 4's, half of it this warp's
    constexpr int NV = Dots::template Values<S::WARP_ROWS>::N;
    constexpr int COLS = Dots::COLS;
    const int col0 = Dots::first_col(lane);
    const int gang = warp / GANG_WARPS, first_row = (warp % GANG_WARPS) * S::WARP_ROWS;
    bool ok = true;
    int n = 0;                                       // first stage of the current piece
    Dots dots, next;
    if (left > 0) dots.load_queries(p, u_first, lane);
    for (int u = u_first; left > 0; ++u, lo = 0) {
        const int rows = p.keys - lo < left ? p.keys - lo : (int)left;
        left -= rows;
        if (left > 0) next.load_queries(p, u + 1, lane);     // lands during this piece
        const int stages = (rows + S::ROWS - 1) / S::ROWS;
        float tm[COLS], tl[COLS];
#pragma unroll
        for (int j = 0; j < COLS; ++j) { tm[j] = -INFINITY; tl[j] = 0.f; }
        float* sc = p.scores + ((long long)u * p.R + col0) * p.score_ld + lo;
        for (int i = (gang - n) & (GANGS - 1); i < stages; i += GANGS) {
            const int m = (n + i) / GANGS, slot = gang * S::DEPTH + m % S::DEPTH;
            ok = ok && mbar_wait(full_bar(slot), (m / S::DEPTH) & 1, abort_flag, p.status, FCS_STATUS_WAIT_CONSUMER);
            ok = __all_sync(0xffffffffu, ok);
            float v[NV][COLS];
            dots.template run<S::WARP_ROWS>(ring + slot * S::BYTES + first_row * p.D * (T == T_FP32 ? 4 : 2), lane, p.D, v);
            __syncwarp();
            if (lane == 0) mbar_arrive(empty_bar(slot));     // the stage may be refilled
            const int r0 = i * S::ROWS + first_row;
#pragma unroll
            for (int j = 0; j < COLS; ++j)
                if (col0 + j < p.R)
                    keep_scores<Dots, NV, COLS>(p, v, j, col0 + j, lo, r0, rows, lane, sc + (long long)j * p.score_ld, tm[j], tl[j]);
        }
        n += stages;
        // this warp's (maximum, sum) of the piece
#pragma unroll
        for (int j = 0; j < COLS; ++j) {
#pragma unroll
            for (int o = Dots::LANE_STEP; o < 32; o <<= 1) {
                const float mo = __shfl_xor_sync(0xffffffffu, tm[j], o);
                const float lov = __shfl_xor_sync(0xffffffffu, tl[j], o);
                smallq_merge(tm[j], tl[j], mo, lov);
            }
            if (lane < Dots::LANE_STEP && col0 + j < p.R) {
                const int piece = (int)blockIdx.x - cta_of((long long)u * p.keys, p.share);   // its place among the unit's
                p.part[(((long long)u * p.slots + piece) * CONSUMER_WARPS + warp) * MAX_ROWS + col0 + j] =
                    make_float2(tm[j], ok ? tl[j] : INFINITY);
            }
        }
        dots = next;
    }
    if (*abort_flag) __nanosleep(1000000);   // let copies in flight land
}

// out[b, key] = inv_norm * sum over heads and rows of exp2(score - M) / L
__global__ void __launch_bounds__(COLUMN_THREADS)
few_rows_columns_kernel(const Params p) {
    __shared__ float2 mw[COLUMN_PAIRS];                // (maximum, weight) of a (head, row) pair
    __shared__ float sums[COLUMN_SLICES][COLUMN_KEYS];
    grid_launch_dependents();
    const int kx = threadIdx.x % COLUMN_KEYS, slice = threadIdx.x / COLUMN_KEYS;
    const int key = blockIdx.x * COLUMN_KEYS + kx;
    const int pairs = p.H * p.R;
    grid_dependency_wait();
    for (int b = blockIdx.y; b * p.H < p.units; b += gridDim.y) {
        float acc = 0.f;
        for (int i0 = 0; i0 < pairs; i0 += COLUMN_PAIRS) {
            // this thread's scores are under way while the statistics are merged
            float x[COLUMN_PER_SLICE];
#pragma unroll
            for (int j = 0; j < COLUMN_PER_SLICE; ++j) {
                const int i = i0 + slice * COLUMN_PER_SLICE + j;
                x[j] = i < pairs && key < p.keys ? p.scores[((long long)b * pairs + i) * p.score_ld + key] : -INFINITY;
            }
            {   // eight threads to a pair, one per consumer warp that wrote a piece of it
                const int i = i0 + (int)threadIdx.x / CONSUMER_WARPS, w = threadIdx.x % CONSUMER_WARPS;
                float mm = -INFINITY, ll = 0.f;
                if (i < pairs) {
                    const int u = b * p.H + i / p.R, r = i % p.R;
                    const int c0 = cta_of((long long)u * p.keys, p.share);
                    const int c1 = cta_of((long long)(u + 1) * p.keys - 1, p.share);
                    const float2* pt = p.part + ((long long)u * p.slots * CONSUMER_WARPS + w) * MAX_ROWS + r;
#pragma unroll 4
                    for (int s = 0; s <= c1 - c0; ++s) {
                        const float2 t = pt[s * (CONSUMER_WARPS * MAX_ROWS)];
                        smallq_merge(mm, ll, t.x, t.y);
                    }
                }
#pragma unroll
                for (int o = CONSUMER_WARPS / 2; o > 0; o >>= 1) {
                    const float mo = __shfl_xor_sync(0xffffffffu, mm, o);
                    const float lo = __shfl_xor_sync(0xffffffffu, ll, o);
                    smallq_merge(mm, ll, mo, lo);
                }
                if (w == 0 && i < pairs) mw[i - i0] = make_float2(mm, p.inv_norm / ll);
            }
            __syncthreads();
#pragma unroll
            for (int j = 0; j < COLUMN_PER_SLICE; ++j) {
                const int i = slice * COLUMN_PER_SLICE + j;
                if (i0 + i < pairs) acc += ex2_approx(x[j] - mw[i].x) * mw[i].y;
            }
            __syncthreads();
        }
        sums[slice][kx] = acc;     // (the reads of the batch entry before are two barriers back)
        __syncthreads();
        if (slice == 0 && key < p.Sk) {
            float v = 0.f;
#pragma unroll
            for (int s = 0; s < COLUMN_SLICES; ++s) v += sums[s][kx];
            p.out[(long long)b * p.out_ld + key] = v;
        }
    }
}

// ---------------------------------------------------------------------------
// Small calls: one thread-block cluster per batch entry instead of the two kernels, a CTA per head.  A
// head's scores stay in its CTA's shared memory and become its share of the columns there; the heads are
// summed through distributed shared memory and the columns written once.  Neither scratch, nor adds into
// memory, nor a second launch.
// ---------------------------------------------------------------------------
constexpr int CLUSTER_MAX = 16;                    // heads (above eight: an opt-in of the launch)
constexpr int CLUSTER_SMEM_LIMIT = 112 * 1024;     // two CTAs per SM

// A stage is one warp's: 8 KiB of 16-bit rows, 32 fp32 rows.
template <int DK, int T>
struct ClusterStage {
    static constexpr int ROWS = T == T_FP32 ? 32 : 64 * 64 / DK;
    static constexpr int BYTES = ROWS * DK * (T == T_FP32 ? 4 : 2);
};
// a stage per warp, [R][keys] scores, barriers and the warps' statistics
template <int DK, int T, int W>
constexpr int cluster_smem(int R, int keys) {
    return W * ClusterStage<DK, T>::BYTES + R * ((keys + 3) / 4 * 4) * 4 + 2 * W * 8 + 16 + W * MAX_ROWS * 8 + 128;
}

// W: consumer warps, eight with two CTAs per SM or four with four.
template <int DK, int T, int R, int W>
__global__ void __launch_bounds__(32 * (W + 1), 16 / W)
few_rows_cluster_kernel(const __grid_constant__ CUtensorMap tm_k, const Params p) {
    using S = ClusterStage<DK, T>;
    using Dots = typename DotsOf<DK, T, R>::type;
    extern __shared__ uint8_t few_smem[];
    uint8_t* ring = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(few_smem) + 127) & ~static_cast<uintptr_t>(127));
    const int pitch = (p.keys + 3) / 4 * 4;
    float* score = reinterpret_cast<float*>(ring + W * S::BYTES);        // [R][pitch]; row 0 becomes the head's columns
    uint8_t* fixed = reinterpret_cast<uint8_t*>(score + p.R * pitch);
    const uint32_t bars = smem_u32(fixed);
    auto full_bar = [&](int w) { return bars + 8u * w; };
    auto empty_bar = [&](int w) { return bars + 8u * (W + w); };
    volatile int* abort_flag = reinterpret_cast<volatile int*>(fixed + 2 * W * 8);
    float2* red = reinterpret_cast<float2*>(fixed + 2 * W * 8 + 16);     // [warps][MAX_ROWS]

    if (clusters_pack(p.H)) grid_launch_dependents();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int h = (int)smallq_cluster_rank(), b = (int)blockIdx.x / p.H;
    if (threadIdx.x == 0) {
        for (int w = 0; w < W; ++w) { mbar_init(full_bar(w), 1); mbar_init(empty_bar(w), 1); }
        *abort_flag = 0;
        mbar_fence_init();
        prefetch_tensormap(&tm_k);
    }
    __syncthreads();
    grid_dependency_wait();
    const int stages = (p.keys + S::ROWS - 1) / S::ROWS;
    bool ok = true;

    if (warp == W) {
        // ------------------------------------------------ copies (whole tiles: rows past the keys read as zero)
        for (int n = 0; n < stages && ok; ++n) {
            const int w = n % W, m = n / W;
            if (m > 0) {
                ok = mbar_wait(empty_bar(w), (m & 1) ^ 1, abort_flag, p.status, FCS_STATUS_WAIT_PRODUCER);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
            }
            if (elect_one_sync()) {
                mbar_arrive_expect_tx(full_bar(w), (uint32_t)(S::ROWS * p.D * (T == T_FP32 ? 4 : 2)));
                tma_load_4d(smem_u32(ring + w * S::BYTES), &tm_k, full_bar(w), 0, n * S::ROWS, h, b);
            }
            __syncwarp();
        }
    } else {
        constexpr int NV = Dots::template Values<S::ROWS>::N;
        constexpr int COLS = Dots::COLS;
        const int col0 = Dots::first_col(lane);
        Dots dots;
        dots.load_queries(p, b * p.H + h, lane);
        float tm[COLS], tl[COLS];
#pragma unroll
        for (int j = 0; j < COLS; ++j) { tm[j] = -INFINITY; tl[j] = 0.f; }
        for (int n = warp, m = 0; n < stages; n += W, ++m) {
            ok = ok && mbar_wait(full_bar(warp), m & 1, abort_flag, p.status, FCS_STATUS_WAIT_CONSUMER);
            ok = __all_sync(0xffffffffu, ok);
            float v[NV][COLS];
            dots.template run<S::ROWS>(ring + warp * S::BYTES, lane, p.D, v);
            __syncwarp();
            if (lane == 0) mbar_arrive(empty_bar(warp));     // the stage may be refilled
#pragma unroll
            for (int j = 0; j < COLS; ++j)
                if (col0 + j < p.R)
                    keep_scores<Dots, NV, COLS>(p, v, j, col0 + j, 0, n * S::ROWS, p.keys, lane,
                                                score + (col0 + j) * pitch, tm[j], tl[j]);
        }
#pragma unroll
        for (int j = 0; j < COLS; ++j) {
#pragma unroll
            for (int o = Dots::LANE_STEP; o < 32; o <<= 1) {
                const float mo = __shfl_xor_sync(0xffffffffu, tm[j], o);
                const float lo = __shfl_xor_sync(0xffffffffu, tl[j], o);
                smallq_merge(tm[j], tl[j], mo, lo);
            }
            if (lane < Dots::LANE_STEP && col0 + j < p.R) red[warp * MAX_ROWS + col0 + j] = make_float2(tm[j], tl[j]);
        }
        smallq_consumer_sync<W>();          // scores and statistics are in
        float M[R], weight[R];
#pragma unroll
        for (int r = 0; r < R; ++r) {
            M[r] = 0.f; weight[r] = 0.f;
            if (r < p.R) {
                float2 t[W];
                float mm = -INFINITY, ll = 0.f;
#pragma unroll
                for (int w = 0; w < W; ++w) { t[w] = red[w * MAX_ROWS + r]; mm = fmaxf(mm, t[w].x); }
#pragma unroll
                for (int w = 0; w < W; ++w) ll += t[w].y * ex2_approx(t[w].x - mm);
                M[r] = mm;
                weight[r] = ok ? p.inv_norm / ll : 0.f;
            }
        }
        for (int k = threadIdx.x; k < p.keys; k += 32 * W) {
            float v = 0.f;
#pragma unroll
            for (int r = 0; r < R; ++r)
                if (r < p.R) v += ex2_approx(score[r * pitch + k] - M[r]) * weight[r];
            score[k] = v;
        }
    }
    // ---------------------------------------------------- this CTA's share of the columns, over the heads
    __syncthreads();
    smallq_cluster_arrive();
    smallq_cluster_wait();
    const int per = (p.Sk + p.H - 1) / p.H, k1 = (h + 1) * per < p.Sk ? (h + 1) * per : p.Sk;
    for (int k = h * per + (int)threadIdx.x; k < k1; k += 32 * (W + 1)) {
        float v = 0.f;
        if (k < p.keys) {
            float x[CLUSTER_MAX];
#pragma unroll
            for (int r = 0; r < CLUSTER_MAX; ++r) x[r] = r < p.H ? ld_peer_f32(smem_u32(score + k), (uint32_t)r) : 0.f;
#pragma unroll
            for (int r = 0; r < CLUSTER_MAX; ++r) v += x[r];
        }
        p.out[(long long)b * p.out_ld + k] = v;
    }
    smallq_cluster_arrive();                         // nobody leaves before its peers have read its columns
    smallq_cluster_wait();
    if (*abort_flag) __nanosleep(1000000);           // let copies in flight land
}

}  // namespace few
}  // namespace fcs
