// rotary.cuh -- launcher of the rotary-embedding kernels (see rotary.cu).
#pragma once
#include <cuda_runtime.h>

// What a rotary kernel leaves in page-locked memory when its last block is through: `call` last.
struct RotaryDone {
    unsigned long long start_ns, end_ns;  // of the kernel, by the device's clock
    const void *owner;                    // the host's record of this memory (the kernel leaves it alone)
    unsigned call;
};

// x: fp16, rotated in place; sin_t / cos_t: fp32 [seqlen][rotary_half]; strides in elements.
// All extents at least 1.  done: page-locked, `call` is written to done->call at the end.
cudaError_t of_launch_rotary(void *x, const void *sin_t, const void *cos_t, int batch, int seqlen,
                             int nheads, int rotary_half, long long stride_batch,
                             long long stride_seq, long long stride_head, int sm_count,
                             RotaryDone *done, unsigned call, cudaStream_t stream);
