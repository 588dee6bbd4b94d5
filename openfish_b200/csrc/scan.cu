// scan.cu -- backward and forward scans (and the posterior) of the CRF-CTC decode for sm_100a.
//
// Replaces the reference kernel bwd_scan (src/scan_cuda.cu:8-57) and the recursion half of
// fwd_post_scan (src/scan_cuda.cu:59-146), and reproduces the CPU routines backward_scan and
// forward_scan (src/decode_cpu.c:13-52, 54-119) bit for bit (see exact_math.cuh):
//   bwd[n][T][s] = 0,  bwd[n][t][s]   = LSE5( bwd[n][t+1][s] + stay, bwd[n][t+1][4j+b] + score[t][n][4(4j+b) + k] )
//                                       for s = j + k*ns/4
//   fwd[n][0][s] = 0,  fwd[n][t+1][s] = LSE5( fwd[n][t][s] + stay,   fwd[n][t][j + b*ns/4] + score[t][n][4s + b] )
//                                       for s = 4j + k                         (b = 0..3 in both)
// The two recursions do not depend on each other (only the posterior needs both).  This file's kernels
// are for batches that fill the GPU (scan_ahead.cu has one for smaller ones): the decode runs the
// backward scan first (the beam search waits for it) and the forward scan beside the beam search,
// which leaves most issue slots free.  For the 256- and 1024-state models the forward scan also
// forms the posterior (a warp of its own per block, see PosteriorRow) and its scores never leave the
// chip.  Of the 64-state model only the forward scan of a few batches is left to this file (scan_ahead.cu says which);
// its rows go to HBM for the kernel that forms the posterior.
//
// Shape of a block.  In either direction the four states that share j also share their four
// neighbour inputs, and their 16 transition scores are one contiguous 32-byte piece of the score
// row, so nothing is strided.  SPT of those four states go to one thread.  The previous row
// lives in shared memory (one block barrier per timestep); score rows arrive through a ring of
// 1-D bulk asynchronous copies tracked by mbarriers (no multicast), issued a ring length ahead
// by a copy warp of their own.  Output rows go straight to HBM.
//
// Neither scan is bound by HBM (each moves T*4ns*2 + (T+1)*ns*4 bytes per chunk); they are bound
// by the latency of one timestep's dependent arithmetic.
#include "scan.cuh"
#include "exact_math.cuh"
#include "fast_lse.cuh"
#include "of_device.cuh"
#include "prepare.cuh"
#include "scan_topo.cuh"

namespace {

using namespace scan_topo;

// Terms of the SPT states (j, k0 .. k0+SPT-1) of one thread.  The 32-byte piece is read as two
// 16-byte halves (a two-way bank conflict, which costs less than the selects that avoid it: the
// kernel is short of issue slots, not of shared-memory bandwidth).
// `own`, when given, holds the thread's own states of row `in` (what it computed a timestep ago),
// which saves reading them back.
template <class Topo, int SPT>
__device__ __forceinline__ void thread_terms(const float *in, const unsigned char *row, int j, int k0,
                                             float stay, float (&v)[SPT][5], const float *own = nullptr) {
    const unsigned char *piece = row + 32 * j;
    const uint4 lo = *reinterpret_cast<const uint4 *>(piece);
    const uint4 hi = *reinterpret_cast<const uint4 *>(piece + 16);
    float x[4];
    Topo::shared_inputs(in, j, x);
    const uint32_t w[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
#pragma unroll
    for (int k = 0; k < SPT; ++k) {
        v[k][0] = (own ? own[k] : in[Topo::state(j, k0 + k)]) + stay;
#pragma unroll
        for (int b = 0; b < 4; ++b) v[k][b + 1] = Topo::template plus_score<SPT>(x[b], w, k0, k, b);
    }
}

template <class Topo, int SPT>
__device__ __forceinline__ void thread_store(float *smem_row, float *gmem_row, int j, int k0,
                                             const float (&res)[SPT], bool to_gmem) {
    if constexpr (Topo::kForward && SPT == 4) {
        const float4 v = make_float4(res[0], res[1], res[2], res[3]);
        *reinterpret_cast<float4 *>(smem_row + 4 * j) = v;
        if (to_gmem) *reinterpret_cast<float4 *>(gmem_row + 4 * j) = v;
    } else if constexpr (Topo::kForward && SPT == 2) {
        const float2 v = make_float2(res[0], res[1]);
        *reinterpret_cast<float2 *>(smem_row + 4 * j + k0) = v;
        if (to_gmem) *reinterpret_cast<float2 *>(gmem_row + 4 * j + k0) = v;
    } else {
#pragma unroll
        for (int k = 0; k < SPT; ++k) {
            smem_row[Topo::state(j, k0 + k)] = res[k];
            if (to_gmem) gmem_row[Topo::state(j, k0 + k)] = res[k];
        }
    }
}

// ------------------------------------------------------------------------------------------
// One row of the posterior, softmax_s(fwd[s] + bwd[s]), by one warp: the forward row comes from
// shared memory and so does the backward row (it arrives beside the score row of the timestep
// during which it is needed; a load from HBM issued by this warp would put a microsecond of
// latency into every timestep, which is more than the scan warps take).  Lane l
// takes the states (q*32 + l)*VEC .. +VEC-1; the arithmetic and its order are those of the
// stand-alone posterior kernel in scan_ahead.cu (softmax offset m0 = the maximum of row 0, where
// fwd is zero: the log partition function is the same for every row, so exponents stay in range).
template <int NS>
struct PosteriorRow {
    static_assert(NS >= 128, "four states a lane and access");
    static constexpr int PERL = NS / 32;
    static constexpr int VEC = 4;
    static constexpr int NV = PERL / VEC;
    // two states in each arithmetic instruction: a 512-chunk decode of 256 states in 2.79 ms instead of 2.82, but
    // one of 256 chunks of 1024 states in 5.14 instead of 4.98
    static constexpr bool kPacked = PERL <= 8;

    __device__ static float row_max(const float *row, int lane) {
        float m = -3.0e38f;
        for (int st = lane; st < NS; st += 32) m = fmaxf(m, row[st]);
        return ofd::warp_max(m);
    }
    __device__ static void load(float *d, const float *p) {
        const float4 v = *reinterpret_cast<const float4 *>(p);
        d[0] = v.x; d[1] = v.y; d[2] = v.z; d[3] = v.w;
    }
    __device__ static void emit(const float *fwd_row, const float *bwd_row, float *post_row, float m0, int lane) {
        const float kLog2e = 1.4426950408889634f;
        float e[PERL];
        float part = 0.f;
#pragma unroll
        for (int q = 0; q < NV; ++q) {
            float f[VEC], b[VEC];
            load(f, fwd_row + (q * 32 + lane) * VEC);
            load(b, bwd_row + (q * 32 + lane) * VEC);
            if constexpr (kPacked) {
#pragma unroll
                for (int k = 0; k < VEC; k += 2) {
                    const ofd::f32x2 sum = ofd::add2(ofd::pack2(f[k], f[k + 1]), ofd::pack2(b[k], b[k + 1]));
                    float x0, x1;
                    ofd::unpack2(ofd::mul2(ofd::sub2(sum, ofd::pack2(m0, m0)), ofd::pack2(kLog2e, kLog2e)), x0, x1);
                    e[q * VEC + k] = ofd::ex2_approx(x0);
                    e[q * VEC + k + 1] = ofd::ex2_approx(x1);
                    part += e[q * VEC + k];
                    part += e[q * VEC + k + 1];
                }
            } else {
#pragma unroll
                for (int k = 0; k < VEC; ++k) {
                    e[q * VEC + k] = ofd::ex2_approx(((f[k] + b[k]) - m0) * kLog2e);
                    part += e[q * VEC + k];
                }
            }
        }
#pragma unroll
        for (int o = 16; o; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
        const float inv = 1.0f / part;
#pragma unroll
        for (int q = 0; q < NV; ++q) {
            float *x = e + q * VEC;
            if constexpr (kPacked) {
#pragma unroll
                for (int k = 0; k < VEC; k += 2)
                    ofd::unpack2(ofd::mul2(ofd::pack2(x[k], x[k + 1]), ofd::pack2(inv, inv)), x[k], x[k + 1]);
            } else {
#pragma unroll
                for (int k = 0; k < VEC; ++k) x[k] *= inv;
            }
            *reinterpret_cast<float4 *>(post_row + (q * 32 + lane) * VEC) = make_float4(x[0], x[1], x[2], x[3]);
        }
    }
};

// ------------------------------------------------------------------------------------------
// The scan of one chunk by one block.
//
// If a state whose rounding the fp32 evaluation cannot certify sent its warp through the
// value-exact routine before the timestep could end, that routine's latency would be paid on
// nearly every step: almost every timestep has a few such states.  Here the scan warps do not
// wait for it.  An uncertified state gets the likelier of its two candidate floats and is put on
// a list, together with its five terms; while the scan warps work on the next timestep, a
// checker warp recomputes the listed states exactly.  If every guess was right (most timesteps)
// nothing else happens.  If one was wrong the block pauses at the end of that next
// timestep: the checker corrects the value and recomputes exactly the five states of the next
// row that read it (the state itself and its four readers) before anybody reads those, and the
// scan carries on.  (Letting the scan run on and chasing the consequences a step behind does
// not work: a one-ulp change of an input moves an output by one ulp with a probability equal to
// that input's weight in the sum, and the weights of a state over its five readers add up to
// about one, so corrections would breed as fast as they die.)  What reaches HBM is, value for
// value, what the exact routine alone would have produced.  Three row buffers rotate so that the
// inputs of a timestep are still there while it is being checked, and score rows are released
// one timestep late.
template <int NS, int SPT, int RING, int COPIES, bool POST>
struct SpecSmem {
    static constexpr int kExpCopies = COPIES;  // of the 2^(j/64) table, by lane: their reads rarely meet in a bank
    static constexpr int kRowBytes = NS * 4 * 2;
    static constexpr int NW = NS / SPT / 32;  // scan warps
    static constexpr int kPerWarp = 16;       // listed states per warp and timestep, at most
    alignas(128) unsigned char ring[RING][kRowBytes];
    // with the posterior: the backward row that the posterior warp needs during a timestep
    // travels with that timestep's score row (same slot, same mbarrier)
    alignas(128) float bwd_ring[POST ? RING : 1][POST ? NS : 4];
    alignas(16) float alpha[3][NS];
    alignas(16) double exp2_rep[ofx::kExpTab * kExpCopies];
    double rcp_c[ofx::kLogTab];
    double log_c[ofx::kLogTab];
    alignas(8) uint64_t full[RING];
    // A listed state is handed to the checker with all it needs: its five terms, the guess and
    // the state's number (32 bytes), so that the checker's chain starts with one round trip to
    // shared memory instead of three dependent ones (list, then state, then the state's inputs).
    alignas(16) float4 listed[2][NW][kPerWarp][2];  // {v0 v1 v2 v3} {v4 guess state -}
    alignas(NW % 4 == 0 ? 16 : 4) int n_listed[2][NW];
    unsigned short wrong_state[NW * kPerWarp];
    float wrong_value[NW * kPerWarp];
    // settle-now path: a warp's uncertified states, dealt out to its lanes, and their exact values
    unsigned short redo_state[NW][32 * SPT];
    float redo_value[NW][32 * SPT];
    // The logarithm out of a table (fast_lse.cuh) where a row has so many states that one timestep in six had a wrong
    // guess: backward scan of 40 chunks of 1024 states, T = 300, both directions, 0.398 ms instead of 0.433, 256 chunks of
    // T = 1666 1.96 instead of 1.97 and with the posterior, beside the beam search, 2.80 instead of 2.84; for 256
    // states the look-up costs more than it saves (512 chunks 1.175 instead of 1.146).
    static constexpr bool kTable = NS == 1024;
    alignas(8) ofd::LogPair log_f[kTable ? ofd::kLogPairs : 1];
    int abort_flag;
};

// The exact routine for what happens seldom: inlined, it would be a good part of the block's code, and four
// blocks of this kernel and four beam searches that share an SM want their code to stay in its instruction
// cache.
__device__ __noinline__ float exact_out_of_line(float v0, float v1, float v2, float v3, float v4, const ofx::TabRef tr) {
    const float v[5] = {v0, v1, v2, v3, v4};
    return ofx::lse5_exact(v, tr);
}

// The scan warps' route for a timestep with more uncertified states than the usual one handles;
// out of line on purpose.  v: the thread's terms, res: its guesses (in) and, where states were
// settled, their exact values (out); bit k of okmask: state k was certified.  Returns the number of
// states the warp put on the list, or -1 if it settled its uncertified states here (res changed).
template <class Topo, int NS, int SPT, int RING, int COPIES, bool POST>
__device__ __noinline__ int crowded_step(SpecSmem<NS, SPT, RING, COPIES, POST> &sm, const float (*v)[5], float *res, uint32_t okmask,
                                         int par, int j, int k0, const float *in, const unsigned char *row,
                                         float stay, const ofx::TabRef tr) {
    constexpr int PER = SpecSmem<NS, SPT, RING, COPIES, POST>::kPerWarp;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t lt_mask = (1u << lane) - 1u;
    uint32_t bad[SPT];
    int total = 0;
#pragma unroll
    for (int k = 0; k < SPT; ++k) {
        bad[k] = __ballot_sync(0xffffffffu, !((okmask >> k) & 1u));
        total += __popc(bad[k]);
    }
    if (total > 16 * SPT) {
        // most states uncertified (the first few dozen timesteps, where scores are small and
        // the float grid fine): the exact routine for every state
        float out[SPT];
        ofx::lse5_batch_exact<SPT>(v, out, tr);
#pragma unroll
        for (int k = 0; k < SPT; ++k) res[k] = out[k];
        return -1;
    }
    if (total > PER) {
        // many uncertified states (the next hundred or two timesteps): settle them here and
        // now, nothing to check later.  They are dealt out evenly to the warp's lanes, so the
        // exact routine runs ceil(total / 32) times rather than once per state of the
        // unluckiest lane.
        int pos[SPT], base = 0;
#pragma unroll
        for (int k = 0; k < SPT; ++k) {
            pos[k] = base + __popc(bad[k] & lt_mask);
            if (!((okmask >> k) & 1u)) sm.redo_state[warp][pos[k]] = (unsigned short)Topo::state(j, k0 + k);
            base += __popc(bad[k]);
        }
        __syncwarp();
        for (int first = 0; first < total; first += 32) {
            const int e = first + lane;
            const int st = sm.redo_state[warp][e < total ? e : 0];
            float w[5];
            terms_of<Topo>(st, in, row, stay, w);
            const float x = ofx::lse5_exact(w, tr, e < total);
            if (e < total) sm.redo_value[warp][e] = x;
        }
        __syncwarp();
#pragma unroll
        for (int k = 0; k < SPT; ++k)
            if (!((okmask >> k) & 1u)) res[k] = sm.redo_value[warp][pos[k]];
        return -1;
    }
    int base = 0;
#pragma unroll
    for (int k = 0; k < SPT; ++k) {
        if (!((okmask >> k) & 1u)) {
            float4 *entry = sm.listed[par][warp][base + __popc(bad[k] & lt_mask)];
            entry[0] = make_float4(v[k][0], v[k][1], v[k][2], v[k][3]);
            entry[1] = make_float4(v[k][4], res[k], __int_as_float(Topo::state(j, k0 + k)), 0.f);
        }
        base += __popc(bad[k]);
    }
    return total;
}

//
// POST (forward direction only): the rows are not written out; a fourth kind of warp turns each
// row, once it is final, into the posterior row  softmax_s(fwd[t][s] + bwd[t][s])  and writes
// that (`out` is then the posterior tensor and `bwd_in` the finished backward scores).  Row r is
// final after the barrier that ends timestep r (its guesses have been checked by then) and its
// buffer is written again during timestep r+2, so the posterior warp takes it during timestep
// r+1; the last two rows are taken after the scan.
// Two states in each arithmetic instruction, roles by a warp number that the compiler knows to be the same for a warp:
// fewer instructions (256 states, 1024 chunks: 5.01 ms a decode instead of 5.11).
template <class Topo, int NS, int SPT, int RING, int COPIES, bool POST>
__device__ __forceinline__ void spec_body(unsigned char *smem_raw, int chunk, const __half *scores,
                                          float *out, const float *bwd_in, int T, int N, float stay,
                                          const ofx::Tables *tables, int *status, uint64_t wait_ns) {
    constexpr int NJ = NS / 4;
    constexpr int TPC = NS / SPT;
    using Smem = SpecSmem<NS, SPT, RING, COPIES, POST>;
    constexpr int NW = Smem::NW, PER = Smem::kPerWarp;
    constexpr int kExpCopies = Smem::kExpCopies;
    static_assert(!POST || Topo::kForward, "the posterior rides on the forward scan");
    static_assert(TPC % 32 == 0, "scan warps must be full");
    Smem &sm = *reinterpret_cast<Smem *>(smem_raw);

    const int tid = threadIdx.x, lane = tid & 31;
    const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    for (int i = tid; i < ofx::kExpTab * kExpCopies; i += blockDim.x)
        sm.exp2_rep[i] = tables->exp2_j[i / kExpCopies];
    for (int i = tid; i < ofx::kLogTab; i += blockDim.x) {
        sm.rcp_c[i] = tables->rcp_c[i];
        sm.log_c[i] = tables->log_c[i];
        if constexpr (Smem::kTable) sm.log_f[i] = {tables->rcp_f[i], tables->log_f[i]};
    }
    for (int i = tid; i < 2 * NW; i += blockDim.x) (&sm.n_listed[0][0])[i] = 0;
    for (int i = tid; i < NS; i += blockDim.x) sm.alpha[0][i] = 0.f;
    if (tid == 0) {
        sm.abort_flag = 0;
        for (int r = 0; r < RING; ++r) ofd::mbar_init(&sm.full[r], 1);
        ofd::mbar_fence_init();
    }
    __syncthreads();

    const size_t t_stride = (size_t)N * NS * 4;
    const __half *chunk_scores = scores + (size_t)chunk * NS * 4;
    float *out_chunk = out + (size_t)chunk * (size_t)(T + 1) * NS;
    const ofx::TabRef tr = {sm.exp2_rep + (tid & (kExpCopies - 1)), kExpCopies, sm.rcp_c, sm.log_c};

    if (warp == NW) {
        // ------------------------------------------------------------------ copy warp
        // A slot is refilled one timestep late: the checker still reads the scores of the
        // timestep it is checking.
        const bool issuer = lane == 0;
        int issued = 0;  // copies go out in row order; after an abort no more are issued
        auto fill = [&](int i) {
            if (sm.abort_flag) return;
            const int slot = i % RING;
            ofd::mbar_arrive_expect_tx(&sm.full[slot], Smem::kRowBytes + (POST ? NS * 4 : 0));
            ofd::bulk_g2s(sm.ring[slot], chunk_scores + t_stride * (size_t)Topo::score_row(i, T), Smem::kRowBytes,
                          &sm.full[slot]);
            // the posterior row formed during timestep i is row i-1 (row 0 during timestep 0)
            if (POST)
                ofd::bulk_g2s(sm.bwd_ring[slot], bwd_in + ((size_t)chunk * (size_t)(T + 1) + (size_t)(i ? i - 1 : 0)) * NS,
                              NS * 4, &sm.full[slot]);
            ++issued;
        };
        auto landed = [&](int i) {
            ofd::mbar_wait_bounded(&sm.full[i % RING], (uint32_t)(i / RING) & 1u, &sm.abort_flag, status, wait_ns);
        };
        if (issuer) {
            for (int i = 0; i < RING && i < T; ++i) fill(i);
            if (T > 0) landed(0);
        }
        __syncthreads();
        for (int i = 0; i < T; ++i) {
            if (issuer && i + 1 < T) landed(i + 1);
            if (__syncthreads_or(0)) __syncthreads();
            if (issuer && i >= 1 && i - 1 + RING < T) fill(i - 1 + RING);
        }
        if (POST) __syncthreads();  // the last row is final
        // after an abort the newest copies get a bounded chance to land before the block retires
        if (issuer && sm.abort_flag) ofd::mbar_drain_bounded(sm.full, RING, issued, wait_ns);
        return;
    }

    if constexpr (POST) if (warp == NW + 2) {
        // ------------------------------------------------------------------ posterior warp
        const float *bwd_chunk = bwd_in + (size_t)chunk * (size_t)(T + 1) * NS;
        const float m0 = PosteriorRow<NS>::row_max(bwd_chunk, lane);
        // inside the scan the backward row is in the slot of the timestep during which the
        // posterior row is formed; the last two rows take theirs from HBM
        auto emit = [&](int r, const float *bwd_row) {
            PosteriorRow<NS>::emit(sm.alpha[r % 3], bwd_row, out_chunk + (size_t)r * NS, m0, lane);
        };
        __syncthreads();  // start of the scan
        int next_row = 0;
        for (int i = 0; i < T; ++i) {
            // during timestep i the rows up to i-1 are final (and row 0 always is)
            if (next_row == 0 || next_row <= i - 1) {
                emit(next_row, sm.bwd_ring[i % RING]);  // next_row = i-1, or 0 when i = 0
                ++next_row;
            }
            if (__syncthreads_or(0)) __syncthreads();
        }
        while (next_row <= T - 1) {  // final since the last timestep's barrier
            emit(next_row, bwd_chunk + (size_t)next_row * NS);
            ++next_row;
        }
        __syncthreads();  // the last row is final
        emit(T, bwd_chunk + (size_t)T * NS);
        return;
    }

    if (warp == NW + 1) {
        // ------------------------------------------------------------------ checker warp
        __syncthreads();  // start of the scan
        for (int i = 0; i <= T; ++i) {
            // During timestep i (for i = T: after the last one) check the states listed during
            // timestep i-1; their terms and guesses come with the list, the guesses also stand in
            // alpha[i%3] and in the output row of timestep i-1.
            int nw = 0;
            if (i >= 1) {
                const int par = (i - 1) & 1;
                // An entry was written before the correction that ended its timestep, if there
                // was one: a state that read a corrected value stands on the list with the terms
                // from before.  The correction has recomputed every such state for good, so a
                // mismatch counts only if the entry's terms are still the state's terms.
                auto still_stands = [&](bool differs, const float (&v)[5], int s) {
                    if (__any_sync(0xffffffffu, differs)) {  // one timestep in seventeen
                        float now[5];
                        terms_of<Topo>(differs ? s : 0, sm.alpha[(i - 1) % 3], sm.ring[(i - 1) % RING], stay, now);
#pragma unroll
                        for (int q = 0; q < 5; ++q) differs = differs && __float_as_uint(now[q]) == __float_as_uint(v[q]);
                    }
                    return differs;
                };
                if constexpr (NW * PER <= 32) {
                    // a lane per slot: nothing to look up before the entry can be fetched
                    const int w = lane / PER, k = lane % PER;
                    const float4 a = sm.listed[par][w < NW ? w : 0][k][0], b = sm.listed[par][w < NW ? w : 0][k][1];
                    const bool mine = w < NW && k < sm.n_listed[par][w < NW ? w : 0];
                    if (__any_sync(0xffffffffu, mine)) {
                        const float v[5] = {a.x, a.y, a.z, a.w, b.x};
                        const float x = ofx::lse5_exact(v, tr, mine);
                        const bool wrong = still_stands(mine && __float_as_uint(x) != __float_as_uint(b.y), v, __float_as_int(b.z));
                        const uint32_t wm = __ballot_sync(0xffffffffu, wrong);
                        if (wrong) {
                            const int at = __popc(wm & ((1u << lane) - 1u));
                            sm.wrong_state[at] = (unsigned short)__float_as_int(b.z);
                            sm.wrong_value[at] = x;
                        }
                        nw = __popc(wm);
                    }
                } else {
                    // more slots than lanes: the filled ones are taken 32 at a time
                    int cnt[NW], total = 0;
#pragma unroll
                    for (int w = 0; w < NW; w += 4) {
                        const int4 c = *reinterpret_cast<const int4 *>(&sm.n_listed[par][w]);
                        cnt[w] = c.x; cnt[w + 1] = c.y; cnt[w + 2] = c.z; cnt[w + 3] = c.w;
                    }
#pragma unroll
                    for (int w = 0; w < NW; ++w) total += cnt[w];
                    for (int base = 0; base < total; base += 32) {
                        const int e = base + lane;
                        // the list that entry e is on: the last that starts at or before it
                        int at_w = 0, start = 0, acc = 0;
#pragma unroll
                        for (int w = 1; w < NW; ++w) {
                            acc += cnt[w - 1];
                            at_w += e >= acc;
                            start = e >= acc ? acc : start;
                        }
                        const int at_k = e < total ? e - start : 0;
                        const float4 a = sm.listed[par][at_w][at_k][0], b = sm.listed[par][at_w][at_k][1];
                        const float v[5] = {a.x, a.y, a.z, a.w, b.x};
                        const float x = ofx::lse5_exact(v, tr, e < total);
                        const bool wrong = still_stands(e < total && __float_as_uint(x) != __float_as_uint(b.y), v, __float_as_int(b.z));
                        const uint32_t wm = __ballot_sync(0xffffffffu, wrong);
                        if (wrong) {
                            const int at = nw + __popc(wm & ((1u << lane) - 1u));
                            sm.wrong_state[at] = (unsigned short)__float_as_int(b.z);
                            sm.wrong_value[at] = x;
                        }
                        nw += __popc(wm);
                    }
                }
                __syncwarp();
            }
            if (i == T) {
                // the last row: no timestep reads it any more, just correct it
                if (POST) {
                    for (int e = lane; e < nw; e += 32) sm.alpha[T % 3][sm.wrong_state[e]] = sm.wrong_value[e];
                    __syncthreads();  // the last row is final
                } else {
                    float *row = out_chunk + (size_t)Topo::out_row(T - 1, T) * NS;
                    for (int e = lane; e < nw; e += 32) row[sm.wrong_state[e]] = sm.wrong_value[e];
                }
                break;
            }
            // end of timestep i; the barrier itself tells every warp whether a guess was wrong
            __syncthreads_or(nw);
            if (nw) {
                float *prev_row = out_chunk + (size_t)Topo::out_row(i - 1, T) * NS;
                for (int e = lane; e < nw; e += 32) {
                    const int s = sm.wrong_state[e];
                    sm.alpha[i % 3][s] = sm.wrong_value[e];
                    if (!POST) prev_row[s] = sm.wrong_value[e];
                }
                __syncwarp();
                // the five states of timestep i's row that read a corrected value
                float *this_row = out_chunk + (size_t)Topo::out_row(i, T) * NS;
                for (int idx = lane; idx < 5 * nw; idx += 32) {
                    const int s = sm.wrong_state[idx / 5], d = idx % 5;
                    const int dep = d == 4 ? s : Topo::reader(s, d);
                    float v[5];
                    terms_of<Topo>(dep, sm.alpha[i % 3], sm.ring[i % RING], stay, v);
                    float x;  // certified fp32 evaluation first: it settles all but about 1 in 100
                    if (!ofd::lse5_try_fast(v, x)) x = exact_out_of_line(v[0], v[1], v[2], v[3], v[4], tr);
                    sm.alpha[(i + 1) % 3][dep] = x;
                    if (!POST) this_row[dep] = x;
                }
                __syncthreads();  // corrections in place
            }
        }
        return;
    }

    // ---------------------------------------------------------------------- scan warps
    const int j = tid % NJ;
    const int k0 = (tid / NJ) * SPT;
    if (!POST) {
#pragma unroll
        for (int k = 0; k < SPT; ++k) out_chunk[(size_t)Topo::zero_row(T) * NS + Topo::state(j, k0 + k)] = 0.f;
    }
    __syncthreads();
    const uint32_t lt_mask = (1u << lane) - 1u;
    float res[SPT];  // the thread's states of the current row: its stay terms for the next timestep
#pragma unroll
    for (int k = 0; k < SPT; ++k) res[k] = 0.f;
    // rotating pointers instead of i % 3 and i % RING: row i is read from `in`, row i+1 goes to `nxt`
    const float *in = sm.alpha[0];
    float *nxt = sm.alpha[1], *spare = sm.alpha[2];
    const unsigned char *row = sm.ring[0];
    float *gmem_out = out_chunk + (size_t)Topo::out_row(0, T) * NS;
    const ptrdiff_t gmem_step = Topo::kForward ? (ptrdiff_t)NS : -(ptrdiff_t)NS;
    for (int i = 0; i < T; ++i) {
        float v[SPT][5];
        bool ok[SPT];
        thread_terms<Topo, SPT>(in, row, j, k0, stay, v, res);
        const uint32_t bad = ofd::lse5_guess_pairs<SPT, Smem::kTable>(v, res, sm.log_f);  // bit k: state k is uncertified
#pragma unroll
        for (int k = 0; k < SPT; ++k) ok[k] = !((bad >> k) & 1u);
        // out they go at once (certified values and guesses alike), so that the stores issue in the
        // shadow of the vote below; the two routes that settle states here and now store again
        thread_store<Topo, SPT>(nxt, gmem_out, j, k0, res, !POST);
        int total = 0;
        // Both votes are taken here, where the warp is converged for certain, and nothing below
        // votes or diverges on the usual route: a vote or a lane-divergent branch inside
        // conditional code costs a hundred cycles and more of re-convergence.
        const uint32_t owners = __ballot_sync(0xffffffffu, bad != 0);  // non-zero about every other timestep per warp
        const uint32_t crowded = __ballot_sync(0xffffffffu, (bad & (bad - 1u)) != 0);
        // The usual case: a few lanes with one uncertified state each.  The first vote settles who
        // lists where, and the entry goes out through predicated stores.
        const bool few = owners != 0 && crowded == 0 && __popc(owners) <= PER;
        if (few) {
            const uint32_t entry = (uint32_t)__cvta_generic_to_shared(sm.listed[i & 1][warp][__popc(owners & lt_mask)]);
#pragma unroll
            for (int k = 0; k < SPT; ++k)
                ofd::sts_entry_if(!ok[k], entry, v[k], res[k], __int_as_float(Topo::state(j, k0 + k)));
            total = __popc(owners);
        } else if (owners) {
            // anything else (a lane with two uncertified states, more than a list takes, the first
            // few hundred timesteps where most states are uncertified) goes out of line: the
            // loop's instructions stay few and close together.  The copies live in local memory,
            // the arrays of the usual route in registers.
            float cv[SPT][5], cres[SPT];
            uint32_t okmask = 0;
#pragma unroll
            for (int k = 0; k < SPT; ++k) {
#pragma unroll
                for (int q = 0; q < 5; ++q) cv[k][q] = v[k][q];
                cres[k] = res[k];
                okmask |= (uint32_t)ok[k] << k;
            }
            total = crowded_step<Topo, NS, SPT, RING, COPIES, POST>(sm, cv, cres, okmask, i & 1, j, k0, in, row, stay, tr);
#pragma unroll
            for (int k = 0; k < SPT; ++k) res[k] = cres[k];
            if (total < 0) {  // states were settled here and now: their values replace the guesses
                thread_store<Topo, SPT>(nxt, gmem_out, j, k0, res, !POST);
                total = 0;
            }
        }
        if (lane == 0) sm.n_listed[i & 1][warp] = total;
        if (__syncthreads_or(0)) {
            __syncthreads();  // the checker is correcting this row's readers
#pragma unroll
            for (int k = 0; k < SPT; ++k) res[k] = nxt[Topo::state(j, k0 + k)];  // maybe corrected
        }
        float *const was_in = const_cast<float *>(in);
        in = nxt;
        nxt = spare;
        spare = was_in;
        row = (row == sm.ring[RING - 1]) ? sm.ring[0] : row + Smem::kRowBytes;
        gmem_out += gmem_step;
    }
    if (POST) __syncthreads();  // the last row is final
}

// ------------------------------------------------------------------------------------------
// One grid for the directions DIRS (kBackward, kForward or both): the first n_bwd_blocks blocks scan backwards, the
// rest forwards.
enum : int { kBackward = 1, kForward = 2 };

template <int NS, int SPT, int RING, int COPIES, int MINB, int DIRS>
__global__ void __launch_bounds__(NS / SPT + 64, MINB)
scan_spec_kernel(const __half *__restrict__ scores, float *__restrict__ bwd, float *__restrict__ fwd,
                 int T, int N, int n_bwd_blocks, float stay, const ofx::Tables *__restrict__ tables,
                 int *status, uint64_t wait_ns) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    const bool backward = DIRS == kBackward || (DIRS != kForward && (int)blockIdx.x < n_bwd_blocks);
    if constexpr (DIRS & kBackward)
        if (backward)
            spec_body<BwdTopo<NS>, NS, SPT, RING, COPIES, false>(smem_raw, blockIdx.x, scores, bwd, nullptr, T, N, stay, tables,
                                                                 status, wait_ns);
    if constexpr (DIRS & kForward)
        if (!backward)
            spec_body<FwdTopo<NS>, NS, SPT, RING, COPIES, false>(smem_raw, blockIdx.x - n_bwd_blocks, scores, fwd, nullptr, T, N,
                                                                 stay, tables, status, wait_ns);
}

// Forward scan with the posterior on top: one block per chunk, reads the finished backward scores.
template <int NS, int SPT, int RING, int COPIES, int MINB>
__global__ void __launch_bounds__(NS / SPT + 96, MINB)
scan_spec_posterior_kernel(const __half *__restrict__ scores, const float *__restrict__ bwd,
                           float *__restrict__ post, int T, int N, float stay,
                           const ofx::Tables *__restrict__ tables, int *status, uint64_t wait_ns) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    spec_body<FwdTopo<NS>, NS, SPT, RING, COPIES, true>(smem_raw, blockIdx.x, scores, post, bwd, T, N, stay, tables, status, wait_ns);
}

// The kernels are described once, for loading (of_load_scan) and for launching.
template <int NS, int SPT, int RING, int COPIES, int MINB, int DIRS>
struct Spec {
    static constexpr auto kern = scan_spec_kernel<NS, SPT, RING, COPIES, MINB, DIRS>;
    static constexpr size_t bytes = sizeof(SpecSmem<NS, SPT, RING, COPIES, false>);
    static cudaError_t launch(const __half *scores, float *bwd, float *fwd, int T, int N, float stay,
                              const ofx::Tables *tables, int *status, uint64_t wait_ns, cudaStream_t stream) {
        const int n_bwd = bwd ? N : 0, n_fwd = fwd ? N : 0;
        if ((bwd && !(DIRS & kBackward)) || (fwd && !(DIRS & kForward))) return cudaErrorInvalidValue;
        kern<<<n_bwd + n_fwd, NS / SPT + 64, bytes, stream>>>(scores, bwd, fwd, T, N, n_bwd, stay, tables, status, wait_ns);
        return cudaGetLastError();
    }
};

template <int NS, int SPT, int RING, int COPIES, int MINB>
struct SpecPosterior {
    static constexpr auto kern = scan_spec_posterior_kernel<NS, SPT, RING, COPIES, MINB>;
    static constexpr size_t bytes = sizeof(SpecSmem<NS, SPT, RING, COPIES, true>);
    static cudaError_t launch(const __half *scores, const float *bwd, float *post, int T, int N, float stay,
                              const ofx::Tables *tables, int *status, uint64_t wait_ns, cudaStream_t stream) {
        kern<<<N, NS / SPT + 96, bytes, stream>>>(scores, bwd, post, T, N, stay, tables, status, wait_ns);
        return cudaGetLastError();
    }
};

using Spec64 = Spec<64, 2, 8, 4, 12, kForward>;
// (Nothing launches the forward half of this one.  Without it the backward half takes 1.5 % longer, 1024 chunks of T =
// 1666 1.826 ms instead of 1.796, with the same registers: where the code comes to lie.)
using Spec256Many = Spec<256, 4, 6, 4, 7, kBackward | kForward>;
using Spec256Most = Spec<256, 4, 6, 4, 8, kBackward>;
using Spec1024 = Spec<1024, 4, 6, 16, 2, kBackward | kForward>;
using Spec1024Many = Spec<1024, 4, 4, 4, 3, kBackward | kForward>;
using SpecPosterior256 = SpecPosterior<256, 4, 6, 16, 5>;
using SpecPosterior256Many = SpecPosterior<256, 4, 6, 4, 5>;
using SpecPosterior256Most = SpecPosterior<256, 4, 6, 4, 6>;
using SpecPosterior1024 = SpecPosterior<1024, 4, 6, 8, 2>;  // (16 copies of the table: no difference)
using SpecPosterior1024Many = SpecPosterior<1024, 4, 3, 4, 3>;

}  // namespace

cudaError_t of_launch_forward_posterior(const void *scores_fp16, const float *bwd, float *post, int T, int N,
                                        int state_len, int sms, float stay, const ofx::Tables *tables, int *status,
                                        uint64_t wait_ns, cudaStream_t stream) {
    const __half *s = static_cast<const __half *>(scores_fp16);
    if (T < 1) return cudaErrorInvalidValue;
    switch (state_len) {
        // Of blocks with 36 KB an SM holds seven together with beam searches (20 KB): four of either would need
        // 512 bytes more than it has.  So a batch whose forward scans and beam searches are at most seven to the
        // SM has them all resident, and a larger one takes blocks of 30 KB (fewer copies of a table).  This
        // kernel beside the beam search, T = 800, large / small blocks: 500 chunks 0.796 / 0.815 ms, 518 0.797 /
        // 0.812, 540 1.120 / 0.817, 592 1.130 / 0.822.  Six of them to the SM instead of five (64 registers)
        // when there are several rounds of blocks, five / six: 1300 chunks 1.938 / 2.027 ms, 1480 2.130 / 2.088,
        // 1600 2.409 / 2.292, 3000 4.244 / 4.169.
        case 4:
            if (2 * N <= 7 * sms) return SpecPosterior256::launch(s, bwd, post, T, N, stay, tables, status, wait_ns, stream);
            if (N <= 10 * sms) return SpecPosterior256Many::launch(s, bwd, post, T, N, stay, tables, status, wait_ns, stream);
            return SpecPosterior256Most::launch(s, bwd, post, T, N, stay, tables, status, wait_ns, stream);
        // three blocks to the SM, with a ring of three rows, when two are not room enough: 444 chunks of T = 800
        // 2.23 ms instead of 2.63, 1000 chunks 5.30 instead of 5.67, but 256 chunks 1.92 instead of 1.58
        case 5:
            if (N > 2 * sms) return SpecPosterior1024Many::launch(s, bwd, post, T, N, stay, tables, status, wait_ns, stream);
            return SpecPosterior1024::launch(s, bwd, post, T, N, stay, tables, status, wait_ns, stream);
        default: return cudaErrorInvalidValue;
    }
}

cudaError_t of_launch_scans(const void *scores_fp16, float *bwd, float *fwd, int T, int N,
                            int state_len, int sms, float stay, const ofx::Tables *tables, int *status,
                            uint64_t wait_ns, cudaStream_t stream) {
    const __half *s = static_cast<const __half *>(scores_fp16);
    switch (state_len) {
        // (the forward scan of one to two chunks to the SM with many timesteps; all else of this model is scan_ahead.cu's and
        // scan_warp.cu's)
        case 3: return Spec64::launch(s, bwd, fwd, T, N, stay, tables, status, wait_ns, stream);
        // (more than five chunks to the SM, four if T is small; scan_ahead.cu has the kernel for fewer)  Seven blocks to the SM (72
        // registers) rather than four: what a block loses is less than what a half empty second round of blocks
        // costs: 740 chunks of T = 1666 1.43 ms instead of 1.86; 1024: 1.90 instead of 2.28.  Eight (64)
        // for many rounds.  Seven / eight, T = 800: 1490 chunks 1.453 / 1.495 ms, 1600 1.469 / 1.550, 1900 1.701 / 1.685, 2050 1.817 /
        // 1.807, 2200 1.996 / 1.913; T = 300: 1700 0.727 / 0.753.
        case 4:
            if (N > 12 * sms) return Spec256Most::launch(s, bwd, fwd, T, N, stay, tables, status, wait_ns, stream);
            return Spec256Many::launch(s, bwd, fwd, T, N, stay, tables, status, wait_ns, stream);
        // (three blocks to the SM, with a smaller ring, when two are not room enough: 444 chunks of T = 800 1.54 ms
        // instead of 1.91)
        case 5:
            if ((bwd && fwd ? 2 : 1) * N > 2 * sms) return Spec1024Many::launch(s, bwd, fwd, T, N, stay, tables, status, wait_ns, stream);
            return Spec1024::launch(s, bwd, fwd, T, N, stay, tables, status, wait_ns, stream);
        default: return cudaErrorInvalidValue;
    }
}

cudaError_t of_load_scan(int kernel) {
    switch (kernel) {
        case kFwd256: return of_load<SpecPosterior256>();
        case kBwd256Many: return of_load<Spec256Many>();
        case kFwd256Many: return of_load<SpecPosterior256Many>();
        case kFwd256Most: return of_load<SpecPosterior256Most>();
        case kBwd256Most: return of_load<Spec256Most>();
        case kScan1024: return of_load<Spec1024>();
        case kScan1024Many: return of_load<Spec1024Many>();
        case kFwd1024Many: return of_load<SpecPosterior1024Many>();
        case kFwd1024: return of_load<SpecPosterior1024>();
        case kFwd64: return of_load<Spec64>();
        default: return cudaSuccess;
    }
}
