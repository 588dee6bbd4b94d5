// rotary.cu -- in-place rotary position embedding on fp16 activations for sm_100a.
//
// Replaces rotary_emb_cuda / rotary_emb (src/nn_cuda.cu:10-40, src/rotary_emb_cuda.cuh:35-69):
// for every (batch, position, head) the pairs (i, i + rotary_half) of the head vector are
// rotated by the angle whose cosine/sine sit at [position][i] of two fp32 tables:
//   o0 = x0*cos - x1*sin,  o1 = x0*sin + x1*cos   (fp32 math, fp16 storage).
// The op is pure HBM streaming (read + write of the rotated part of x; the encoder's tensor at
// 0.88 of a copy's rate), so a thread moves V halves per access: it rotates V consecutive pairs of two
// heads with the same V angles, and a grid-stride loop over positions keeps every SM busy whatever
// the shape.  V is 8 (16-byte accesses) where the sizes and pointers allow it, else 4 (8-byte ones:
// a quarter of an 80-wide head); what allows neither takes a scalar kernel with the same arithmetic.
//
// A call is bound by what surrounds the kernel as well.  The last block to finish writes the kernel's
// start and end times and the call's number to page-locked memory, where the caller looks for them:
// 9 us for launch and wait together, against 18 with two timing events, a stream synchronisation
// and the events' difference (64 positions of two sequences: 21.5 -> 13.6 us for the whole call).  The report makes the
// kernel itself longer, since each block waits for its own stores first: 38 us instead of 32 for the encoder's
// tensor, whose call all the same takes 50 us instead of 55.
#include <cuda_fp16.h>
#include <stdint.h>

#include "rotary.cuh"

namespace {

struct RotArgs {
    __half *x;
    const float *cos_t;
    const float *sin_t;
    long long stride_batch, stride_seq, stride_head;
    int batch, seqlen, nheads, rotary_half;
    RotaryDone *done;
    unsigned call;
};

// Calls of one device follow one another on one stream: one set of counters is enough.
__device__ unsigned g_blocks_done;
__device__ unsigned long long g_started;

__device__ __forceinline__ unsigned long long now_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
__device__ __forceinline__ void block_starts() {
    if (blockIdx.x == 0 && threadIdx.x == 0 && threadIdx.y == 0) g_started = now_ns();
}
// At the end of the kernel, by every thread: the last block to come here reports.
__device__ __forceinline__ void block_ends(const RotArgs &a) {
    __syncthreads();
    if (threadIdx.x != 0 || threadIdx.y != 0) return;
    __threadfence();
    if (atomicAdd(&g_blocks_done, 1u) != gridDim.x - 1) return;
    g_blocks_done = 0;
    __threadfence();
    a.done->start_ns = *(volatile unsigned long long *)&g_started;
    a.done->end_ns = now_ns();
    __threadfence_system();
    *(volatile unsigned *)&a.done->call = a.call;
}

__device__ __forceinline__ void rotate(float x0, float x1, float c, float s, float &o0, float &o1) {
    // same operation order as the CPU routine (src/nn_cpu.c:36-37), no fused multiply-add
    o0 = __fsub_rn(__fmul_rn(x0, c), __fmul_rn(x1, s));
    o1 = __fadd_rn(__fmul_rn(x0, s), __fmul_rn(x1, c));
}

// V halves through one access.
template <int V> struct Vec;
template <> struct Vec<8> { typedef uint4 type; };
template <> struct Vec<4> { typedef uint2 type; };

// blockDim.x threads cover one position's (head group, pair group) items, blockDim.y positions
// per block; the grid strides over positions.  A thread keeps its pair group and its HPT heads for
// the whole launch, so the index arithmetic per position is one division, and the V cosines
// and sines it loads serve HPT heads.  All 2*HPT loads of a position are issued before the first is
// used.
template <int HPT, int V>
__global__ void __launch_bounds__(256) rotary_vec_kernel(const RotArgs a) {
    typedef typename Vec<V>::type vec;
    block_starts();
    const int groups = a.rotary_half / V;  // V pairs per item
    const int head_sets = a.nheads / HPT;
    const int per_pos = head_sets * groups;
    const long long positions = (long long)a.batch * a.seqlen;
    const long long hop = (long long)head_sets * a.stride_head;
    for (int r = threadIdx.x; r < per_pos; r += blockDim.x) {
        const int g = r % groups;
        const int h0 = r / groups;  // this thread's heads: h0, h0 + head_sets, ... (neighbours in a warp
                                    // take neighbouring heads, so each load instruction covers whole lines)
        for (long long pos = (long long)blockIdx.x * blockDim.y + threadIdx.y; pos < positions;
             pos += (long long)gridDim.x * blockDim.y) {
            const int t = (int)(pos % a.seqlen);
            const long long b = pos / a.seqlen;
            __half *base = a.x + b * a.stride_batch + (long long)t * a.stride_seq + h0 * a.stride_head + V * g;
            const float4 *cp = reinterpret_cast<const float4 *>(a.cos_t + (long long)t * a.rotary_half + V * g);
            const float4 *sp = reinterpret_cast<const float4 *>(a.sin_t + (long long)t * a.rotary_half + V * g);
            vec v0[HPT], v1[HPT];
#pragma unroll
            for (int k = 0; k < HPT; ++k) {
                v0[k] = *reinterpret_cast<const vec *>(base + k * hop);
                v1[k] = *reinterpret_cast<const vec *>(base + k * hop + a.rotary_half);
            }
            float c[V], s[V];
#pragma unroll
            for (int i = 0; i < V / 4; ++i) {
                const float4 cv = __ldg(cp + i), sv = __ldg(sp + i);
                c[4 * i] = cv.x; c[4 * i + 1] = cv.y; c[4 * i + 2] = cv.z; c[4 * i + 3] = cv.w;
                s[4 * i] = sv.x; s[4 * i + 1] = sv.y; s[4 * i + 2] = sv.z; s[4 * i + 3] = sv.w;
            }
#pragma unroll
            for (int k = 0; k < HPT; ++k) {
                __half2 *x0 = reinterpret_cast<__half2 *>(&v0[k]);
                __half2 *x1 = reinterpret_cast<__half2 *>(&v1[k]);
#pragma unroll
                for (int i = 0; i < V / 2; ++i) {
                    const float2 a0 = __half22float2(x0[i]);
                    const float2 a1 = __half22float2(x1[i]);
                    float o00, o10, o01, o11;
                    rotate(a0.x, a1.x, c[2 * i], s[2 * i], o00, o10);
                    rotate(a0.y, a1.y, c[2 * i + 1], s[2 * i + 1], o01, o11);
                    x0[i] = __floats2half2_rn(o00, o01);
                    x1[i] = __floats2half2_rn(o10, o11);
                }
                *reinterpret_cast<vec *>(base + k * hop) = v0[k];
                *reinterpret_cast<vec *>(base + k * hop + a.rotary_half) = v1[k];
            }
        }
    }
    block_ends(a);
}

__global__ void __launch_bounds__(256) rotary_scalar_kernel(const RotArgs a) {
    block_starts();
    const long long per_pos = (long long)a.nheads * a.rotary_half;
    const long long total = (long long)a.batch * a.seqlen * per_pos;
    for (long long w = (long long)blockIdx.x * blockDim.x + threadIdx.x; w < total;
         w += (long long)gridDim.x * blockDim.x) {
        const int i = (int)(w % a.rotary_half);
        const int h = (int)((w / a.rotary_half) % a.nheads);
        const long long bt = w / per_pos;
        const int t = (int)(bt % a.seqlen);
        const long long b = bt / a.seqlen;
        __half *p0 = a.x + b * a.stride_batch + (long long)t * a.stride_seq + h * a.stride_head + i;
        __half *p1 = p0 + a.rotary_half;
        float o0, o1;
        rotate(__half2float(*p0), __half2float(*p1), a.cos_t[(long long)t * a.rotary_half + i],
               a.sin_t[(long long)t * a.rotary_half + i], o0, o1);
        *p0 = __float2half_rn(o0);
        *p1 = __float2half_rn(o1);
    }
    block_ends(a);
}

template <int V>
void launch_vec(const RotArgs &a, int sm_count, cudaStream_t stream) {
    const int hpt = a.nheads % 2 == 0 ? 2 : 1;  // (four heads per thread measured slower than two)
    const int per_pos = (a.nheads / hpt) * (a.rotary_half / V);
    int bx = 1;
    while (bx < per_pos && bx < 256) bx <<= 1;  // 1..256 threads across one position
    const dim3 block(bx, 256 / bx);
    const long long positions = (long long)a.batch * a.seqlen;
    long long blocks = (positions + block.y - 1) / block.y;
    // Every block costs its start and its report, and many of them keep more loads under way.  The kernel with
    // four / eight blocks to the SM, by the bytes that are rotated, in us: 13.6 MB 6.7 / 6.6, 17.1 MB 7.4 / 8.3,
    // 20.5 MB 8.5 / 8.9, 27.3 MB 10.2 / 10.0, 34.1 MB 11.9 / 11.4, 54.6 MB 17.4 / 15.7, 109 MB 41.4 / 36.7 (42 with 32
    // blocks); the same order with inputs that come from HBM.
    const long long bytes = 4LL * positions * a.nheads * a.rotary_half;
    const long long cap = (long long)sm_count * (bytes < (32LL << 20) ? 4 : 8);
    if (blocks > cap) blocks = cap;
    if (hpt == 2) rotary_vec_kernel<2, V><<<(unsigned)blocks, block, 0, stream>>>(a);
    else rotary_vec_kernel<1, V><<<(unsigned)blocks, block, 0, stream>>>(a);
}

}  // namespace

cudaError_t of_launch_rotary(void *x, const void *sin_t, const void *cos_t, int batch, int seqlen,
                             int nheads, int rotary_half, long long stride_batch,
                             long long stride_seq, long long stride_head, int sm_count,
                             RotaryDone *done, unsigned call, cudaStream_t stream) {
    RotArgs a;
    a.x = static_cast<__half *>(x);
    a.cos_t = static_cast<const float *>(cos_t);
    a.sin_t = static_cast<const float *>(sin_t);
    a.stride_batch = stride_batch; a.stride_seq = stride_seq; a.stride_head = stride_head;
    a.done = done; a.call = call;
    a.batch = batch; a.seqlen = seqlen; a.nheads = nheads; a.rotary_half = rotary_half;
    // V halves at a time need V-multiples everywhere and pointers aligned to their accesses (the tables are
    // read four floats at a time)
    auto fits = [&](int v) {
        return rotary_half % v == 0 && stride_batch % v == 0 && stride_seq % v == 0 && stride_head % v == 0 &&
               (uintptr_t)x % (2 * v) == 0 && (uintptr_t)sin_t % 16 == 0 && (uintptr_t)cos_t % 16 == 0;
    };
    if (fits(8)) {
        launch_vec<8>(a, sm_count, stream);
    } else if (fits(4)) {
        launch_vec<4>(a, sm_count, stream);
    } else {
        const long long items = (long long)batch * seqlen * nheads * rotary_half;
        long long blocks = (items + 255) / 256;
        const long long cap = (long long)sm_count * 8;
        if (blocks > cap) blocks = cap;
        rotary_scalar_kernel<<<(unsigned)blocks, 256, 0, stream>>>(a);
    }
    return cudaGetLastError();
}
