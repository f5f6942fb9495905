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
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "sm100_ptx.cuh"

namespace fcs {
namespace rnd {

constexpr int THREADS = 256;
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
};

__device__ __forceinline__ const float* piece_source(const Operand& o, unsigned i) {
    if (o.dense) return o.src + (size_t)i * 8;
    const unsigned row = i / o.d8, e = i - row * o.d8;
    const unsigned unit = row / o.rows, r = row - unit * o.rows;
    const unsigned b = unit / o.H, h = unit - b * o.H;
    return o.src + (long long)b * o.sb + (long long)h * o.sh + (long long)r * o.ss + e * 8;
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
            const float m = fmaxf(fmaxf(fmaxf(fabsf(a.x), fabsf(a.y)), fmaxf(fabsf(a.z), fabsf(a.w))),
                                  fmaxf(fmaxf(fabsf(b.x), fabsf(b.y)), fmaxf(fabsf(b.z), fabsf(b.w))));
            outside = outside || m >= FP16_LIMIT;
            __half2 h[4] = {__floats2half2_rn(a.x, a.y), __floats2half2_rn(a.z, a.w), __floats2half2_rn(b.x, b.y),
                            __floats2half2_rn(b.z, b.w)};
            *reinterpret_cast<uint4*>(o.dst + (size_t)i * 8) = *reinterpret_cast<const uint4*>(h);
        }
    }
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
        for (unsigned i = blockIdx.x * THREADS + threadIdx.x; i < o.pieces; i += gridDim.x * THREADS) {
            const float4* s = reinterpret_cast<const float4*>(piece_source(o, i));
            const float4 a = s[0], b = s[1];
            __nv_bfloat162 h[4] = {__floats2bfloat162_rn(a.x, a.y), __floats2bfloat162_rn(a.z, a.w),
                                   __floats2bfloat162_rn(b.x, b.y), __floats2bfloat162_rn(b.z, b.w)};
            *reinterpret_cast<uint4*>(o.dst + (size_t)i * 8) = *reinterpret_cast<const uint4*>(h);
        }
    }
}

}  // namespace rnd
}  // namespace fcs
