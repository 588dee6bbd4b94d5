// scan_topo.cuh -- what the backward and the forward recursion of the CRF differ in (scan.cu, scan_ahead.cu).
#pragma once
#include <cuda_fp16.h>
#include <stdint.h>

namespace scan_topo {

// x plus one fp16 out of a 32-bit word: widened (exactly) and added with one rounding, in one instruction (a
// conversion and an addition before: a fifth of a state's instructions that are not exponentials.  256 states,
// T = 1666, a decode of 592 chunks 2.762 ms instead of 2.808, of 1024 4.78 instead of 4.87; 64 states, 1024 chunks
// 2.56 instead of 2.60).
__device__ __forceinline__ float add_half(float x, uint32_t word, int odd) {
    float r;
    if (odd) asm("{\n\t.reg .b16 a, b;\n\tmov.b32 {a, b}, %1;\n\tadd.f32.f16 %0, b, %2;\n\t}" : "=f"(r) : "r"(word), "f"(x));
    else asm("{\n\t.reg .b16 a, b;\n\tmov.b32 {a, b}, %1;\n\tadd.f32.f16 %0, a, %2;\n\t}" : "=f"(r) : "r"(word), "f"(x));
    return r;
}

// ------------------------------------------------------------------------------------------
// The two recursions differ only in which states a thread owns, which inputs they share, where
// their scores sit inside the 32-byte piece, and in the direction of time.

template <int NS>
struct BwdTopo {
    static constexpr int NJ = NS / 4;
    static constexpr bool kForward = false;
    // thread (j, slot k) owns state j + k*NJ; the four slots share the successors 4j..4j+3
    __device__ static int state(int j, int k) { return j + k * NJ; }
    __device__ static void shared_inputs(const float *in, int j, float (&x)[4]) {
        const float4 v = *reinterpret_cast<const float4 *>(in + 4 * j);
        x[0] = v.x; x[1] = v.y; x[2] = v.z; x[3] = v.w;
    }
    // score of (slot k, base b) is half number 4b + k of the piece
    __device__ static int half_index(int k, int b) { return 4 * b + k; }
    // the same out of the piece held as eight words, slot k0 + k with k0 (a multiple of SPT)
    // known only at run time: selects instead of strided shared-memory reads
    template <int SPT>
    __device__ static float plus_score(float x, const uint32_t (&w)[8], int k0, int k, int b) {
        static_assert(SPT == 2 || SPT == 4, "two or four states a thread");
        if (SPT == 4) return add_half(x, w[2 * b + (k >> 1)], k & 1);
        return add_half(x, k0 ? w[2 * b + 1] : w[2 * b], k);
    }
    __device__ static int j_of(int s) { return s % NJ; }
    __device__ static int k_of(int s) { return s / NJ; }
    // the states of the next row to be computed that read state s of this row, d = 0..3
    __device__ static int reader(int s, int d) { return (s >> 2) + d * NJ; }
    // time: step i reads score row T-1-i and produces output row T-1-i; row T is the zero row
    __device__ static int score_row(int i, int T) { return T - 1 - i; }
    __device__ static int out_row(int i, int T) { return T - 1 - i; }
    __device__ static int zero_row(int T) { return T; }
};

template <int NS>
struct FwdTopo {
    static constexpr int NJ = NS / 4;
    static constexpr bool kForward = true;
    // thread (j, slot k) owns state 4j + k; the four slots share the predecessors j + b*NJ
    __device__ static int state(int j, int k) { return 4 * j + k; }
    __device__ static void shared_inputs(const float *in, int j, float (&x)[4]) {
#pragma unroll
        for (int b = 0; b < 4; ++b) x[b] = in[j + b * NJ];
    }
    __device__ static int half_index(int k, int b) { return 4 * k + b; }
    template <int SPT>
    __device__ static float plus_score(float x, const uint32_t (&w)[8], int k0, int k, int b) {
        static_assert(SPT == 2 || SPT == 4, "two or four states a thread");
        const int c = b >> 1;
        if (SPT == 4) return add_half(x, w[2 * k + c], b & 1);
        return add_half(x, k0 ? w[4 + 2 * k + c] : w[2 * k + c], b & 1);
    }
    __device__ static int j_of(int s) { return s >> 2; }
    __device__ static int k_of(int s) { return s & 3; }
    __device__ static int reader(int s, int d) { return 4 * (s % NJ) + d; }
    __device__ static int score_row(int i, int) { return i; }
    __device__ static int out_row(int i, int) { return i + 1; }
    __device__ static int zero_row(int) { return 0; }
};

// The five terms of state s: inputs from row `in`, scores from the chunk's score row `row`.
template <class Topo>
__device__ __forceinline__ void terms_of(int s, const float *in, const unsigned char *row, float stay,
                                         float (&v)[5]) {
    const int j = Topo::j_of(s), k = Topo::k_of(s);
    const __half *piece = reinterpret_cast<const __half *>(row) + 16 * j;
    float x[4];
    Topo::shared_inputs(in, j, x);
    v[0] = in[s] + stay;
#pragma unroll
    for (int b = 0; b < 4; ++b) v[b + 1] = x[b] + __half2float(piece[Topo::half_index(k, b)]);
}

}  // namespace scan_topo
