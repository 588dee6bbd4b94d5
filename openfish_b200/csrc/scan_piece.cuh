// scan_piece.cuh -- what the scan kernels that run ahead of their checks share (scan_ahead.cu, scan_warp.cu).
#pragma once
#include <stdint.h>

#include "exact_math.cuh"
#include "scan_topo.cuh"

namespace scan_topo {

// The 16 scores of the four states that share j: 32 consecutive bytes of the score row.
struct Piece {
    uint32_t w[8];
    __device__ __forceinline__ Piece(const unsigned char *row, int j) { load(row, j); }
    __device__ __forceinline__ void load(const unsigned char *row, int j) {
        const uint4 lo = *reinterpret_cast<const uint4 *>(row + 32 * j);
        const uint4 hi = *reinterpret_cast<const uint4 *>(row + 32 * j + 16);
        w[0] = lo.x; w[1] = lo.y; w[2] = lo.z; w[3] = lo.w;
        w[4] = hi.x; w[5] = hi.y; w[6] = hi.z; w[7] = hi.w;
    }
};

// Terms of the SPT states (j, k0 .. k0+SPT-1) of one thread; `own` holds those states of row `in`
// (what the thread computed a timestep ago).
template <class Topo, int SPT>
__device__ __forceinline__ void thread_terms(const float *in, const Piece &piece, int j, int k0, float stay,
                                             float (*v)[5], const float *own) {
    float x[4];
    Topo::shared_inputs(in, j, x);
#pragma unroll
    for (int k = 0; k < SPT; ++k) {
        v[k][0] = own[k] + stay;
#pragma unroll
        for (int b = 0; b < 4; ++b) v[k][b + 1] = Topo::template plus_score<SPT>(x[b], piece.w, k0, k, b);
    }
}

template <class Topo, int SPT>
__device__ __forceinline__ void thread_store(float *dst, int j, int k0, const float *res) {
    if constexpr (Topo::kForward && SPT == 4) {
        *reinterpret_cast<float4 *>(dst + 4 * j) = make_float4(res[0], res[1], res[2], res[3]);
    } else if constexpr (Topo::kForward && SPT == 2) {
        *reinterpret_cast<float2 *>(dst + 4 * j + k0) = make_float2(res[0], res[1]);
    } else {
#pragma unroll
        for (int k = 0; k < SPT; ++k) dst[Topo::state(j, k0 + k)] = res[k];
    }
}

// Every state by the exact routine, judged by one of a row's scores: below FROM, or no finite number (then none of
// the row's states is certified and all would go through the checker; a batch of 300 chunks of T = 1000 with one infinite
// score took 3.70 ms instead of 2.43).
template <int FROM>
__device__ __forceinline__ bool exact_for_all(float score) {
    const uint32_t from = __float_as_uint((float)FROM), infinity = 0x7f800000u;
    return (__float_as_uint(score) & 0x7fffffffu) - from >= infinity - from;
}

// All states of a thread by the exact routine; out of line (the first hundred timesteps come here), so everything
// is passed in registers.
template <class Topo, int SPT>
__device__ __noinline__ float4 exact_step(const float *in, const unsigned char *row, int j, int k0, float stay,
                                          float4 own, const double *exp2_j, const double *rcp_c, const double *log_c) {
    float v[SPT][5], out[SPT];
    const float o[4] = {own.x, own.y, own.z, own.w};
    thread_terms<Topo, SPT>(in, Piece(row, j), j, k0, stay, v, o);
    const ofx::TabRef tr = {exp2_j, 1, rcp_c, log_c};
    ofx::lse5_batch_exact<SPT>(v, out, tr);
    return make_float4(out[0], SPT > 1 ? out[1 % SPT] : 0.f, SPT > 2 ? out[2 % SPT] : 0.f, SPT > 2 ? out[3 % SPT] : 0.f);
}

}  // namespace scan_topo
