// fp32 inputs are rounded to 16 bits before the tensor cores see them: to fp16, whose ten mantissa
// bits are those of the TF32 format, or to bf16 when a value lies outside fp16's range.  Which of
// the two is decided on the device, so that the call neither synchronises nor waits:
//
//   round_kernel   both operands to fp16, and a note per CTA of values that do not fit
//   settle_kernel  reads the notes and says the type (`fmt`: 0 fp16, 1 bf16); where a value did not fit it
//                  rounds everything again, to bf16, else it is over in a microsecond
//
// and the kernels behind them take the element type from `fmt` (Problem::fmt).  Bound by memory: 6
// bytes per element.  (An abs / max / read-back per operand and two conversions by torch
// operators took 85 us for a call of a megabyte.)
//
// Small operands (round_in_one_kernel) are over before a launch is: there both steps are one kernel on one
// cluster of sixteen CTAs, which ask each other through shared memory instead of notes.  Either way the output of
// the call is zeroed on the side, which is a launch less for the kernels that add into it (2 x 4 x 256 x 64, a
// megabyte, back to back: four launches 11.45 us, two 10.24).
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "colsum_small_q.cuh"
#include "sm100_ptx.cuh"

namespace fcs {
namespace rnd {

constexpr int THREADS = 256;
constexpr int SMALL_CTAS = 16, SMALL_THREADS = 512;
constexpr float FP16_LIMIT = 60000.f;

struct Operand {
    const float* src;
    uint16_t* dst;                 // dense [B][H][rows][D]
    unsigned pieces;               // B * H * rows * D / 8: eight elements each
    unsigned rows, H, d8;
    long long sb, sh, ss;          // in elements
    int dense;                     // src has dst's layout
};
struct Params {
    Operand op[2];                 // query, key
    int* notes;                    // one per CTA of round_kernel
    int n_notes;
    int* fmt;
    float* out;                    // zeroed: `out_rows` rows of `out_cols`, out_ld apart (NULL: nothing)
    long long out_ld;
    unsigned out_rows, out_cols;
};

__device__ __forceinline__ void clear_output(const Params& p, unsigned thread, unsigned threads) {
    if (!p.out) return;
    const unsigned long long n = (unsigned long long)p.out_rows * p.out_cols;
    for (unsigned long long i = thread; i < n; i += threads) {
        const unsigned long long r = n <= 0xffffffffull ? (unsigned)i / p.out_cols : i / p.out_cols;
        p.out[(long long)r * p.out_ld + (long long)(i - r * p.out_cols)] = 0.f;
    }
}

__device__ __forceinline__ const float* piece_source(const Operand& o, unsigned i) {
    if (o.dense) return o.src + (size_t)i * 8;
    const unsigned row = i / o.d8, e = i - row * o.d8;
    const unsigned unit = row / o.rows, r = row - unit * o.rows;
    const unsigned b = unit / o.H, h = unit - b * o.H;
    return o.src + (long long)b * o.sb + (long long)h * o.sh + (long long)r * o.ss + e * 8;
}

// Piece `i` (a, b) as fp16; whether a value of it does not fit.
__device__ __forceinline__ bool to_fp16(const Operand& o, unsigned i, const float4& a, const float4& b) {
    const float m = fmaxf(fmaxf(fmaxf(fabsf(a.x), fabsf(a.y)), fmaxf(fabsf(a.z), fabsf(a.w))),
                          fmaxf(fmaxf(fabsf(b.x), fabsf(b.y)), fmaxf(fabsf(b.z), fabsf(b.w))));
    __half2 h[4] = {__floats2half2_rn(a.x, a.y), __floats2half2_rn(a.z, a.w), __floats2half2_rn(b.x, b.y),
                    __floats2half2_rn(b.z, b.w)};
    *reinterpret_cast<uint4*>(o.dst + (size_t)i * 8) = *reinterpret_cast<const uint4*>(h);
    return m >= FP16_LIMIT;
}
__device__ __forceinline__ void to_bf16(const Operand& o, unsigned i) {
    const float4* s = reinterpret_cast<const float4*>(piece_source(o, i));
    const float4 a = s[0], b = s[1];
    __nv_bfloat162 h[4] = {__floats2bfloat162_rn(a.x, a.y), __floats2bfloat162_rn(a.z, a.w),
                           __floats2bfloat162_rn(b.x, b.y), __floats2bfloat162_rn(b.z, b.w)};
    *reinterpret_cast<uint4*>(o.dst + (size_t)i * 8) = *reinterpret_cast<const uint4*>(h);
}

__global__ void __launch_bounds__(THREADS)
round_kernel(const Params p) {
    grid_launch_dependents();
    grid_dependency_wait();
    bool outside = false;
#pragma unroll
    for (int t = 0; t < 2; ++t) {
        const Operand& o = p.op[t];
        for (unsigned i = blockIdx.x * THREADS + threadIdx.x; i < o.pieces; i += gridDim.x * THREADS) {
            const float4* s = reinterpret_cast<const float4*>(piece_source(o, i));
            const float4 a = s[0], b = s[1];
            outside = to_fp16(o, i, a, b) || outside;
        }
    }
    clear_output(p, blockIdx.x * THREADS + threadIdx.x, gridDim.x * THREADS);
    const int any = __syncthreads_or(outside ? 1 : 0);
    if (threadIdx.x == 0) p.notes[blockIdx.x] = any;
}

__global__ void __launch_bounds__(THREADS)
settle_kernel(const Params p) {
    grid_launch_dependents();
    grid_dependency_wait();
    int outside = 0;
    for (int i = threadIdx.x; i < p.n_notes; i += THREADS) outside |= p.notes[i];
    outside = __syncthreads_or(outside);
    if (blockIdx.x == 0 && threadIdx.x == 0) *p.fmt = outside ? 1 : 0;
    if (!outside) return;
#pragma unroll
    for (int t = 0; t < 2; ++t) {
        const Operand& o = p.op[t];
        for (unsigned i = blockIdx.x * THREADS + threadIdx.x; i < o.pieces; i += gridDim.x * THREADS) to_bf16(o, i);
    }
}

// Both steps on one cluster of SMALL_CTAS CTAs.
__global__ void __launch_bounds__(SMALL_THREADS)
round_small_kernel(const Params p) {
    __shared__ uint32_t notes[SMALL_CTAS];
    grid_launch_dependents();
    smallq_cluster_arrive();
    grid_dependency_wait();
    const unsigned thread = blockIdx.x * SMALL_THREADS + threadIdx.x, threads = SMALL_CTAS * SMALL_THREADS;
    const unsigned first = p.op[0].pieces, all_pieces = first + p.op[1].pieces;
    bool outside = false;
    for (unsigned i0 = thread; i0 < all_pieces; i0 += 4 * threads) {     // four pieces of either operand in flight
        float4 a[4], b[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const unsigned i = i0 + j * threads;
            if (i >= all_pieces) break;
            const float4* s = reinterpret_cast<const float4*>(i < first ? piece_source(p.op[0], i) : piece_source(p.op[1], i - first));
            a[j] = s[0];
            b[j] = s[1];
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const unsigned i = i0 + j * threads;
            if (i >= all_pieces) break;
            outside = (i < first ? to_fp16(p.op[0], i, a[j], b[j]) : to_fp16(p.op[1], i - first, a[j], b[j])) || outside;
        }
    }
    clear_output(p, thread, threads);
    const int any = __syncthreads_or(outside ? 1 : 0);
    smallq_cluster_wait();       // (the other CTAs run)
    if (threadIdx.x < SMALL_CTAS) {
        uint32_t addr;
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(addr) : "r"(smem_u32(&notes[blockIdx.x])), "r"(threadIdx.x));
        asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(addr), "r"(any) : "memory");
    }
    __syncwarp();
    smallq_cluster_arrive();
    smallq_cluster_wait();
    uint32_t all = 0;
#pragma unroll
    for (int r = 0; r < SMALL_CTAS; ++r) all |= notes[r];
    if (thread == 0) *p.fmt = all ? 1 : 0;
    if (!all) return;
#pragma unroll
    for (int t = 0; t < 2; ++t) {
        const Operand& o = p.op[t];
        for (unsigned i = thread; i < o.pieces; i += threads) to_bf16(o, i);
    }
}

}  // namespace rnd
}  // namespace fcs
