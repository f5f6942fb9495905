// What the PyTorch binding (torch_binding.cpp) calls in the CUDA library: one call of the
// operator with the scratch taken from the caller's allocator as part of the call, so that the
// sizes are planned once.  Internal to this package; the C ABI for other hosts is
// include/flash_colsum_b200.h.
#pragma once

#include <stddef.h>
#include <stdint.h>

#include "../../include/flash_colsum_b200.h"

extern "C" {

// Operands that the library rounds itself (round_fp32.cuh); needs an allocator.
enum { FCS_DTYPE_FP32 = 2 };

typedef struct FcsCall {
    const void* q;
    const void* k;
    float* out;
    int64_t out_ld;
    int B, H, Sq, Sk, D;          // Sq: query rows of the tensor
    int dtype;                    // FCS_DTYPE_FP16 / _BF16 / _FP32
    int64_t q_stride[3], k_stride[3];   // batch, head, row; in elements
    float scale;
    int causal, k_past, cls_n, h_norm;  // as in fcs_colsum_causal_batched / fcs_colsum_batched
    int* status;
    void* stream;
    void* (*alloc)(void* ctx, size_t bytes);   // 256-byte aligned device memory, valid for the stream's work queued so far; NULL on failure
    void* alloc_ctx;
} FcsCall;

// A call whose query, key and result live in host memory (contiguous; pinned for copies that overlap).
// `call` describes the operands as they will lie on the device: q, k and out are device buffers of the whole
// operands' size, the strides dense.
typedef struct FcsHostCall {
    FcsCall call;
    const void* host_q;
    const void* host_k;
    float* host_out;
    int batch_chunk;              // batch entries per chunk, or 0: chunks that shrink towards the end
} FcsHostCall;

typedef int (*FcsRunCallFn)(const FcsCall*);
typedef int (*FcsRunHostCallFn)(const FcsHostCall*);
typedef int (*FcsSelectTopkFn)(const float*, int64_t, int, int, int, int*, float*, void*);
typedef int (*FcsSelectThresholdFn)(const float*, int64_t, int, int, float, int, int*, int*, void*);
typedef const char* (*FcsLastErrorFn)(void);

int fcs_run_call(const FcsCall* call);

// Copies in, computes, copies the result out; returns when the result is there.
int fcs_run_host_call(const FcsHostCall* call);
}
