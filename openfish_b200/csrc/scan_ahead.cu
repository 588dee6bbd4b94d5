// scan_ahead.cu -- scans that run ahead of their checks, for the 64- and the 256-state model, for sm_100a.
//
// Same recursions and, value for value, the same results as scan.cu (src/decode_cpu.c:13-52, 54-119), for batches
// that last as long as a chunk's chain of T dependent timesteps: up to five chunks of 256 states and eight of 64 to
// the SM.  While blocks have SMs to themselves one launch takes both directions (a block each for the backward and
// the forward scan of a chunk; they do not depend on each other); in larger batches it takes the backward scan,
// and in some of them the forward scan beside the beam search.  The forward rows go to HBM, and the posterior is formed by
// a kernel of its own.
//
// A state whose rounding the fp32 evaluation cannot certify (two or three of a row's 256, once the
// scores have grown) needs the value-exact routine, a chain of some 450 cycles on its own.  The scan
// warps never wait for it: such a state gets the likelier of its two candidate floats, a bit in its
// thread's mask says so, and the scan goes on.  Timesteps come in groups of E; while the scan warps work
// on a group, a checker warp recomputes the marked states of the group before, 32 at a time, puts those
// whose guess was wrong right in their row, and its verdict is looked at in the group after.  Was a guess
// wrong (one timestep in sixty), the scan goes back and carries on behind the first such timestep; the rows
// behind it, which followed from the wrong value, and whatever has been put right in them are written
// again.  What reaches HBM is what the exact routine alone would have produced.  While
// the scores are small and the float grid fine, guesses are too many and too often wrong: every state
// goes through the exact routine until the scores have passed FROM.
//
// What bounds it: the instructions of one timestep in one scan warp, issued two to three cycles apart.
// So a thread has two states (four warps for 256 states; with four states a thread a timestep takes a
// quarter longer), and everything that a timestep can do without sits elsewhere: waits for score rows,
// verdicts and ring bookkeeping once a group, copies in, rows out and checks in warps of their own,
// offsets inside a group as constants.
#include <type_traits>

#include "exact_math.cuh"
#include "fast_lse.cuh"
#include "group_order.h"
#include "of_device.cuh"
#include "prepare.cuh"
#include "scan.cuh"
#include "scan_piece.cuh"

namespace {

using namespace scan_topo;

template <int NS, int W, int E, int S>
struct AheadSmem {
    static constexpr int kRowBytes = NS * 4 * 2;
    static constexpr int H = E * (S + 1);  // rows kept: a row is overwritten only after it has gone out
    alignas(128) unsigned char ring[S][E][kRowBytes];
    alignas(16) float rows[H][NS];
    static constexpr bool kLogTable = NS > 64;  // the logarithm out of a table (fast_lse.cuh)
    alignas(8) ofd::LogPair log_f[kLogTable ? ofd::kLogPairs : 1];
    uint32_t mask[2][W][32];          // by group parity and scan thread: bit SPT*q + k, timestep q, state k
    uint32_t verdict[2];              // by group parity: bit q, a guess of timestep q was wrong
    unsigned short marked[64];        // marked states of a group, dealt out to the checker's lanes
    int ended[2];                     // by barrier parity: the group that ended there (group_order.h)
    double exp2_j[ofx::kExpTab];
    double rcp_c[ofx::kLogTab];
    double log_c[ofx::kLogTab];
    alignas(8) uint64_t full[S];      // score rows landed
    alignas(8) uint64_t done[S];      // group verified, its input rows final
    alignas(8) uint64_t empty[S];     // those rows gone out
    int abort_flag;
};

// Rounds of up to 64 marked states that a group's check goes through; with more the group is taken again exactly by
// the scan warps, which have a lane to two or four states.  Ordinary groups stay below four (FROM, below, says how many
// states are marked when guesses begin); it is for rows that turn infinite, whose first state, by which
// exact_for_all judges, is still finite: scans of 14 chunks of 256 states, T = 1000, infinite half way, 0.489 ms instead
// of 0.610.
constexpr int kRounds = 5;

template <int ID, int THREADS>
__device__ __forceinline__ void named_sync() {
    if constexpr (THREADS == 32) __syncwarp();
    else asm volatile("bar.sync %0, %1;" ::"n"(ID), "n"(THREADS) : "memory");
}

// One direction of one chunk by one block: W scan warps, a checker warp, a copy warp and an output warp.
// `out` gets the T+1 rows of the chunk.
template <class Topo, int NS, int W, int E, int S, int FROM>
__device__ __forceinline__ void scan_chunk(unsigned char *smem_raw, int chunk, const __half *scores, float *out,
                                           int T, int N, float stay, const ofx::Tables *tables, int *status,
                                           uint64_t wait_ns) {
    constexpr int SPT = NS / (32 * W);  // states per scan thread
    static_assert(SPT == 2 || SPT == 4, "a thread's states share one j");
    static_assert(W * E * SPT <= 32 && E >= 2 && S >= 4, "a mask word per group; three groups are under way");
    constexpr int NT = 32 * (W + 3);
    constexpr int kSync = 32 * (W + 1);  // threads at a group's end
    using Smem = AheadSmem<NS, W, E, S>;
    constexpr int H = Smem::H;
    Smem &sm = *reinterpret_cast<Smem *>(smem_raw);

    const int tid = threadIdx.x, lane = tid & 31;
    const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);  // (known to be the same for a whole warp)
    for (int i = tid; i < ofx::kExpTab; i += NT) sm.exp2_j[i] = tables->exp2_j[i];
    for (int i = tid; i < ofx::kLogTab; i += NT) {
        sm.rcp_c[i] = tables->rcp_c[i];
        sm.log_c[i] = tables->log_c[i];
        if constexpr (Smem::kLogTable) sm.log_f[i] = {tables->rcp_f[i], tables->log_f[i]};
    }
    for (int i = tid; i < NS; i += NT) sm.rows[0][i] = 0.f;
    for (int i = tid; i < 2 * W * 32; i += NT) (&sm.mask[0][0][0])[i] = 0;
    if (tid < 2) sm.verdict[tid] = 0;
    if (tid == 0) {
        sm.abort_flag = 0;
        for (int r = 0; r < S; ++r) {
            ofd::mbar_init(&sm.full[r], 1);
            ofd::mbar_init(&sm.done[r], 1);
            ofd::mbar_init(&sm.empty[r], 1);
        }
        ofd::mbar_fence_init();
    }
    __syncthreads();

    float *out_chunk = out + (size_t)chunk * (size_t)(T + 1) * NS;
    const int groups = (T + E - 1) / E;

    if (warp == W + 1) {
        // ------------------------------------------------------------------ copy warp
        if (lane == 0) {
            const size_t t_stride = (size_t)N * NS * 4;
            const __half *src = scores + (size_t)chunk * NS * 4 + t_stride * (size_t)Topo::score_row(0, T);
            const ptrdiff_t step = Topo::kForward ? (ptrdiff_t)t_stride : -(ptrdiff_t)t_stride;
            ofd::fill_ring_by_mbar<S>(groups, sm.full, sm.empty, &sm.abort_flag, status, wait_ns, [&](int g, int stage) {
                const int n = min(E, T - g * E);
                ofd::mbar_arrive_expect_tx(&sm.full[stage], n * Smem::kRowBytes);
                for (int q = 0; q < n; ++q) {
                    ofd::bulk_g2s(sm.ring[stage][q], src, Smem::kRowBytes, &sm.full[stage]);
                    src += step;
                }
            });
        }
        return;
    }

    if (warp == W + 2) {
        // ------------------------------------------------------------------ output warp
        // rows of a group leave once the group is verified; row T at the end
        constexpr int PERL = NS / 32, V = PERL >= 4 ? 4 : PERL;  // floats per lane, per access
        float *dst = out_chunk + (size_t)Topo::zero_row(T) * NS;
        const float *row = sm.rows[0];
        auto row_out = [&]() {
#pragma unroll
            for (int q = 0; q < PERL / V; ++q) {
                if constexpr (V == 4)
                    reinterpret_cast<float4 *>(dst)[q * 32 + lane] = reinterpret_cast<const float4 *>(row)[q * 32 + lane];
                else
                    reinterpret_cast<float2 *>(dst)[q * 32 + lane] = reinterpret_cast<const float2 *>(row)[q * 32 + lane];
            }
            dst += Topo::kForward ? NS : -NS;
            row = row == sm.rows[H - 1] ? sm.rows[0] : row + NS;
        };
        int stage = 0;
        uint32_t parity = 0;
        for (int g = 0; g < groups; ++g) {
            ofd::mbar_wait_bounded(&sm.done[stage], parity, &sm.abort_flag, status, wait_ns);
            const int n = min(E, T - g * E);
            for (int q = 0; q < n; ++q) row_out();
            __syncwarp();
            ofd::mbar_arrive_if(lane == 0, &sm.empty[stage]);
            if (++stage == S) {
                stage = 0;
                parity ^= 1u;
            }
        }
        row_out();
        return;
    }

    if (warp == W) {
        // ------------------------------------------------------------------ checker warp
        const ofx::TabRef tr = {sm.exp2_j, 1, sm.rcp_c, sm.log_c};
        const uint32_t lt_mask = (1u << lane) - 1u;
        for (int at = 0;; ++at) {
            named_sync<2, kSync>();
            const int g = group_told(sm.ended, at);  // has just ended
            if (g > groups) return;
            const int par = at & 1;
            uint32_t m = 0;  // marks of this lane's W scan threads, E*SPT bits each
#pragma unroll
            for (int w = 0; w < W; ++w) m |= sm.mask[par][w][lane] << (w * E * SPT);
            if (g >= groups) m = 0;
            const int h0 = (g * E) % H;
            const unsigned char *ring0 = sm.ring[g % S][0];
            uint32_t wrong = 0;
            int rounds = 0;
            // The marked states, 32 at a time.  A value put right here may be one that a later entry reads, or that was
            // itself worked out from a wrong one: both lie behind the first wrong timestep, from which on all is
            // taken again.  (Nobody else writes these rows before the next group's end.)
            for (uint32_t owners = __ballot_sync(0xffffffffu, m != 0); owners;) {
                if (NS > 64 && rounds++ == kRounds) {
                    wrong = kAllAnew;
                    break;
                }
                int n = 0;
                do {
                    if (m) sm.marked[n + __popc(owners & lt_mask)] = (unsigned short)(lane | (__ffs(m) - 1) << 5);
                    n += __popc(owners);
                    m &= m - 1u;
                    owners = __ballot_sync(0xffffffffu, m != 0);
                } while (owners && n + __popc(owners) <= 64);
                __syncwarp();
                for (int first = 0; first < n; first += 32) {
                    const bool mine = first + lane < n;
                    const int e = sm.marked[mine ? first + lane : 0];
                    const int bit = e >> 5, q = (bit / SPT) % E;
                    const int t = bit / (E * SPT) * 32 + (e & 31);  // the scan thread
                    const int s = Topo::state(t % Topo::NJ, (t / Topo::NJ) * SPT + bit % SPT);
                    const int h = h0 + q < H ? h0 + q : h0 + q - H;
                    float *const guess = &sm.rows[h + 1 == H ? 0 : h + 1][s];
                    float v[5];
                    terms_of<Topo>(s, sm.rows[h], ring0 + q * Smem::kRowBytes, stay, v);
                    const float was = *guess;
                    const float x = ofx::lse5_exact(v, tr);
                    __syncwarp();  // (every lane has its terms)
                    if (mine && __float_as_uint(x) != __float_as_uint(was)) {
                        wrong |= 1u << q;
                        *guess = x;
                    }
                    __syncwarp();
                }
            }
            wrong = __reduce_or_sync(0xffffffffu, wrong);
            if (lane == 0) sm.verdict[par] = wrong;
        }
    }

    // ---------------------------------------------------------------------- scan warps
    const int j = tid % Topo::NJ, k0 = (tid / Topo::NJ) * SPT;
    float res[SPT];  // the thread's states of the current row: its stay terms for the next timestep
#pragma unroll
    for (int k = 0; k < SPT; ++k) res[k] = 0.f;
    float *rows = sm.rows[0], *rows_next = sm.rows[E % H];  // row g*E, row (g+1)*E
    const unsigned char *ring = sm.ring[0][0];
    GroupOrder at;
    int stage = 0;
    uint32_t parity = 0;
    bool all = true;  // what exact_for_all said a group ago
    ofd::mbar_wait_bounded(&sm.full[0], 0u, &sm.abort_flag, status, wait_ns);
    Piece piece(ring, j);
    // (one group past the end for the last verdict, one more for the checker to leave)
    while (at.g <= groups + 1) {
        // The verdict on the group before the last was handed over at the barrier just passed (it stays
        // until the check of this group).  Nothing waits for it here: it is looked at when the first
        // timestep of this group has been computed.
        const uint32_t wrong = *(volatile uint32_t *)&sm.verdict[at.par];
        if (tid == 0) at.tell(sm.ended);
        const int next = stage + 1 == S ? 0 : stage + 1;
        const uint32_t next_parity = next ? parity : parity ^ 1u;
        const unsigned char *ring_next = next ? ring + E * Smem::kRowBytes : sm.ring[0][0];
        const float probe = rows[0];
        const int n = T - at.g * E;  // timesteps left
        const bool ready = at.g + 1 >= groups || ofd::mbar_try_wait(&sm.full[next], next_parity);
        const bool back = at.goes_back(wrong);
        uint32_t bad = 0;
        if (at.g < groups) {
#pragma unroll
            for (int q = 0; q < E; ++q) {
                if (q < at.from) continue;
                const float *in = rows + q * NS;
                float *nxt = q + 1 < E ? rows + (q + 1) * NS : rows_next;
                if (__builtin_expect(all, 0)) {
                    const float4 own = make_float4(res[0], res[1], SPT > 2 ? res[2 % SPT] : 0.f, SPT > 2 ? res[3 % SPT] : 0.f);
                    const float4 x = exact_step<Topo, SPT>(in, ring + q * Smem::kRowBytes, j, k0, stay, own, sm.exp2_j, sm.rcp_c, sm.log_c);
                    res[0] = x.x;
                    res[1] = x.y;
                    if constexpr (SPT > 2) {
                        res[2] = x.z;
                        res[3] = x.w;
                    }
                } else {
                    float v[SPT][5];
                    thread_terms<Topo, SPT>(in, piece, j, k0, stay, v, res);
                    bad |= ofd::lse5_guess_pairs<SPT, Smem::kLogTable>(v, res, sm.log_f) << (q * SPT);
                }
                if (q == 0 && back) break;
                // (timesteps past the end are taken like any other, on leftover scores: their rows lie
                // behind row T, and nothing reads them)
                thread_store<Topo, SPT>(nxt, j, k0, res);
                if (q + 1 < E) {
                    piece.load(ring + (q + 1) * Smem::kRowBytes, j);
                    named_sync<1, 32 * W>();
                }
            }
        }
        if (__builtin_expect(back, 0)) {
            // back to the group before the last, behind its first wrong timestep, which the checker has put right
            // (what follows it followed from it), or to its start, to take it exactly
            at.go_back(wrong);
            rows = sm.rows[(at.g * E) % H];
            rows_next = sm.rows[(at.g * E + E) % H];
            stage = at.g % S;
            parity = (uint32_t)(at.g / S) & 1u;
            ring = sm.ring[stage][0];
#pragma unroll
            for (int k = 0; k < SPT; ++k) res[k] = (at.from < E ? rows + at.from * NS : rows_next)[Topo::state(j, k0 + k)];
            piece.load(ring + (at.from < E ? at.from : 0) * Smem::kRowBytes, j);
            all = (wrong & kAllAnew) || exact_for_all<FROM>(rows[0]);
            continue;
        }
        // the group before the last is verified
        ofd::mbar_arrive_if(tid == 0 && at.verified(), &sm.done[stage >= 2 ? stage - 2 : stage - 2 + S]);
        if (n < E) bad &= n > 0 ? (1u << (n * SPT)) - 1u : 0u;
        sm.mask[at.par][warp][lane] = bad;
        if (!ready) ofd::mbar_wait_slow(&sm.full[next], next_parity, &sm.abort_flag, status, wait_ns);
        piece.load(ring_next, j);
        all = exact_for_all<FROM>(probe);
        named_sync<2, kSync>();
        at.next();
        stage = next;
        parity = next_parity;
        ring = ring_next;
        rows = rows_next;
        rows_next = rows_next == sm.rows[H - E] ? sm.rows[0] : rows_next + E * NS;
    }
}

// The first n_bwd blocks scan backwards, the others forwards.
template <int NS, int W, int E, int S, int MINB, int FROM>
__global__ void __launch_bounds__(32 * (W + 3), MINB)
scan_ahead_kernel(const __half *__restrict__ scores, float *__restrict__ bwd, float *__restrict__ fwd, int T, int N,
                  int n_bwd, float stay, const ofx::Tables *__restrict__ tables, int *status, uint64_t wait_ns) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    if ((int)blockIdx.x < n_bwd)
        scan_chunk<BwdTopo<NS>, NS, W, E, S, FROM>(smem_raw, blockIdx.x, scores, bwd, T, N, stay, tables, status, wait_ns);
    else
        scan_chunk<FwdTopo<NS>, NS, W, E, S, FROM>(smem_raw, blockIdx.x - n_bwd, scores, fwd, T, N, stay, tables, status, wait_ns);
}

template <int NS, int W, int E, int S, int MINB, int FROM>
struct Ahead {
    static constexpr auto kern = scan_ahead_kernel<NS, W, E, S, MINB, FROM>;
    static constexpr size_t bytes = sizeof(AheadSmem<NS, W, E, S>);
    static cudaError_t launch(const __half *scores, float *bwd, float *fwd, int T, int N, float stay,
                              const ofx::Tables *tables, int *status, uint64_t wait_ns, cudaStream_t stream) {
        const int n_bwd = bwd ? N : 0, n_fwd = fwd ? N : 0;
        kern<<<n_bwd + n_fwd, 32 * (W + 3), bytes, stream>>>(scores, bwd, fwd, T, N, n_bwd, stay, tables, status, wait_ns);
        return cudaGetLastError();
    }
};
// Longer groups: what a group costs besides its timesteps (250 cycles, and the checker's pass) is paid less often, and
// going back, rare and short, loses less than that.  One checker for a group instead of one for each of its
// timesteps, whose lists were nearly empty: both scans of one chunk of 64 states, T = 1000, 0.256 ms instead of 0.280
// (groups of four), 0.246 with groups of six (0.236 by now); of 14 chunks of 256 states, T = 1666, 0.560 instead of 0.572 (0.51 by now); the backward
// scan of 300 chunks 0.766 instead of 0.874.  (Groups of two with a checker for each timestep, and wrong guesses
// gone back to and taken again instead of put right: 0.345, 0.642, 0.979.)  Five stages of 256 states, so that three
// blocks fit an SM; four come too late (14 chunks 0.844).
// For more than three chunks of 256 states to the SM two scan warps of four states a thread, and blocks that fit four
// times: backward scan of 512 chunks 0.970 ms, 1.009 with four warps, 1.146 with scan.cu's kernel; of 601 chunks of T = 1201,
// which do not all fit, 1.132 with these, 1.030 with scan.cu's, and 0.989 with shorter groups, which fit five times.
// (Seven to the SM, with four stages of two timesteps: 1024 chunks 3.12 instead of scan.cu's 1.79.)  For more than five chunks of 64 states blocks that
// fit eight times (T = 800: 760 chunks 0.310 instead of 0.395 by a warp a chunk; 1300, which do not all fit, 0.511
// and 0.462).
// FROM, the score from which on guesses are made: at 512 one state in fourteen is marked, at 256 one in seven, and the fewer
// states there are, the fewer to go wrong.  Both scans of 40 chunks of T = 120, from 512 / 256 / 128: 64 states 0.069 / 0.065 /
// 0.067 ms, 256 states 0.076 / 0.085 / 0.094.  With two scan warps the exact routine is dearer, and so the more chunks there
// are to an SM: backward scan of T = 300, 512 chunks 0.256 / 0.259 / 0.279, 600 0.339 / 0.316 / 0.319; where scores grow slowly (by two a
// timestep, as stays do) 0.326 / 0.283 / 0.300 and 0.472 / 0.385 / 0.371, where all states are equal 0.317 / 0.229 / 0.184 and 0.468 /
// 0.326 / 0.255.
using Ahead64 = Ahead<64, 1, 6, 6, 5, 256>;
using Ahead64Mid = Ahead<64, 1, 4, 6, 8, 256>;
using Ahead256 = Ahead<256, 4, 4, 5, 3, 512>;
using Ahead256Mid = Ahead<256, 2, 3, 5, 4, 256>;
using Ahead256Five = Ahead<256, 2, 2, 5, 5, 128>;

// ------------------------------------------------------------------------------------------
// post (in: forward rows) = softmax over states of forward + backward, row by row: rows are independent,
// a warp takes a row straight from and to HBM.  No per-row maximum: the log partition function is the same
// for every row, so one offset, the maximum of row 0 (where the forward scores are zero), keeps every
// exponent in range.  Bound by HBM (12 bytes a state and row); it runs beside the beam search.
constexpr int kPostRows = 32;  // rows a block takes, eight warps

template <int NS>
__global__ void __launch_bounds__(256) posterior_kernel(const float *__restrict__ bwd, float *post, int T) {
    constexpr int PER = NS / 32, VEC = PER >= 4 ? 4 : PER, NV = PER / VEC;
    constexpr float kLog2e = 1.4426950408889634f;
    typedef typename std::conditional<VEC == 4, float4, float2>::type vec;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const size_t base = (size_t)blockIdx.y * (size_t)(T + 1) * NS;
    float m0 = -3.0e38f;
    for (int s = lane; s < NS; s += 32) m0 = fmaxf(m0, bwd[base + s]);
    m0 = ofd::warp_max(m0);
    const int last = min(T + 1, (int)(blockIdx.x + 1) * kPostRows);
    for (int t = blockIdx.x * kPostRows + warp; t < last; t += 8) {
        const vec *br = reinterpret_cast<const vec *>(bwd + base + (size_t)t * NS);
        vec *pr = reinterpret_cast<vec *>(post + base + (size_t)t * NS);
        vec f[NV], b[NV];
#pragma unroll
        for (int q = 0; q < NV; ++q) {
            f[q] = pr[q * 32 + lane];
            b[q] = br[q * 32 + lane];
        }
        float part = 0.f;
#pragma unroll
        for (int q = 0; q < NV; ++q) {
            float *e = reinterpret_cast<float *>(&f[q]);
            const float *d = reinterpret_cast<const float *>(&b[q]);
#pragma unroll
            for (int k = 0; k < VEC; ++k) {
                e[k] = ofd::ex2_approx(((e[k] + d[k]) - m0) * kLog2e);
                part += e[k];
            }
        }
#pragma unroll
        for (int o = 16; o; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
        const float inv = 1.0f / part;
#pragma unroll
        for (int q = 0; q < NV; ++q) {
            float *e = reinterpret_cast<float *>(&f[q]);
#pragma unroll
            for (int k = 0; k < VEC; ++k) e[k] *= inv;
            pr[q * 32 + lane] = f[q];
        }
    }
}

template <int NS>
struct Posterior {
    static constexpr auto kern = posterior_kernel<NS>;
    static constexpr size_t bytes = 0;
};

}  // namespace

cudaError_t of_launch_ahead(const void *scores_fp16, float *bwd, float *fwd, int T, int N, int state_len, int sms, float stay,
                            const ofx::Tables *tables, int *status, uint64_t wait_ns, cudaStream_t stream) {
    const __half *s = static_cast<const __half *>(scores_fp16);
    if (T < 1) return cudaErrorInvalidValue;
    switch (state_len) {
        case 3:
            if (N > 5 * sms) return Ahead64Mid::launch(s, bwd, fwd, T, N, stay, tables, status, wait_ns, stream);
            return Ahead64::launch(s, bwd, fwd, T, N, stay, tables, status, wait_ns, stream);
        case 4:
            if (N > 4 * sms) return Ahead256Five::launch(s, bwd, fwd, T, N, stay, tables, status, wait_ns, stream);
            if (N > 3 * sms) return Ahead256Mid::launch(s, bwd, fwd, T, N, stay, tables, status, wait_ns, stream);
            return Ahead256::launch(s, bwd, fwd, T, N, stay, tables, status, wait_ns, stream);
        default: return cudaErrorInvalidValue;
    }
}

cudaError_t of_launch_posterior(const float *bwd, float *post, int T, int N, int state_len, cudaStream_t stream) {
    // (65535 chunks are the most that a grid's second dimension holds)
    for (int first = 0; first < N; first += 65535) {
        const int n = N - first < 65535 ? N - first : 65535;
        const size_t skip = (size_t)first * (size_t)(T + 1) << (2 * state_len);
        const dim3 grid((T + 1 + kPostRows - 1) / kPostRows, n);
        switch (state_len) {
            case 3: posterior_kernel<64><<<grid, 256, 0, stream>>>(bwd + skip, post + skip, T); break;
            case 4: posterior_kernel<256><<<grid, 256, 0, stream>>>(bwd + skip, post + skip, T); break;
            case 5: posterior_kernel<1024><<<grid, 256, 0, stream>>>(bwd + skip, post + skip, T); break;
            default: return cudaErrorInvalidValue;
        }
    }
    return cudaGetLastError();
}

// Where the lines lie (decodes of T = 800, ms, by plan: together / ahead then forward / backward then forward):
//   256 states:  74 chunks 0.79 / 0.87 / 0.98;  111: 0.98 / 0.88 / 0.98;  296: 1.42 / 1.20 / 1.28;
//                at T = 1666 512: - / 2.56 / 2.73;  1024: - / 5.10 / 4.77;  at T = 1201 601: - / 2.69 / 2.73
//   64 states:   74 chunks 0.69 / 0.69 / 0.72;  296: 0.95 / 0.79 / 0.83;
//                ahead then forward / a warp to a chunk (their forward scan): 445 0.755 / 0.761, 500 0.781 / 0.774, 592 0.795 /
//                0.786, 700 1.086 / 0.919;  at T = 300 445 0.361 / 0.374, 592 0.379 / 0.380;  at T = 1666 445 1.406 / 1.404, 592
//                1.482 / 1.447, 1024 2.45 / 2.03
//   1024 states: 74 chunks 1.42 /  -   / 1.81;  222: 2.69 /  -   / 2.79;  240: 2.98 /  -   / 2.80
// Two directions on one SM are in each other's way beyond their number (their code is more than an
// instruction cache holds), which is why "together" ends where every block has an SM to itself, except for
// the 1024-state model, where one block is half an SM's work.
OfScanPlan of_scan_plan(int N, int state_len, int sms) {
    if (state_len == 5) return 2 * N <= 3 * sms ? OfScanPlan::kTogether : OfScanPlan::kBackwardThenForward;
    if (2 * N <= sms) return OfScanPlan::kTogether;
    if (N <= (state_len == 3 ? 3 : 5) * sms) return OfScanPlan::kAheadThenForward;
    return state_len == 3 ? OfScanPlan::kWarps : OfScanPlan::kBackwardThenForward;
}

cudaError_t of_launch_first_scans(OfScanPlan plan, const void *scores, float *bwd, float *post, int T, int N,
                                  int state_len, int sms, float stay, const ofx::Tables *tables, int *status,
                                  uint64_t wait_ns, cudaStream_t stream) {
    // (the backward scan of 1024 chunks of T = 1666 0.597 ms by the kernel that runs ahead and 0.742 by a warp each)
    if (plan == OfScanPlan::kWarps && N > 8 * sms)
        return of_launch_warp_backward(scores, bwd, T, N, stay, tables, status, wait_ns, stream);
    float *fwd = plan == OfScanPlan::kTogether ? post : nullptr;
    // (five chunks of 256 states to the SM, a few timesteps: all of them by the exact routine, at which scan.cu's kernel is no
    // slower.  Decodes with this file's kernel / scan.cu's, 593 and 740 chunks: T = 60 0.287 / 0.288 and 0.321 / 0.313 ms; 100
    // 0.406 / 0.412 and 0.446 / 0.446; 200 0.637 / 0.672 and 0.710 / 0.726)
    const bool early = state_len == 4 && N > 4 * sms && T < 100;
    if (plan == OfScanPlan::kBackwardThenForward || state_len == 5 || early)
        return of_launch_scans(scores, bwd, fwd, T, N, state_len, sms, stay, tables, status, wait_ns, stream);
    return of_launch_ahead(scores, bwd, fwd, T, N, state_len, sms, stay, tables, status, wait_ns, stream);
}

cudaError_t of_launch_rest_of_posterior(OfScanPlan plan, const void *scores, const float *bwd, float *post, int T,
                                        int N, int state_len, int sms, float stay, const ofx::Tables *tables, int *status,
                                        uint64_t wait_ns, cudaStream_t stream) {
    if (plan == OfScanPlan::kWarps)
        return of_launch_warp_forward_posterior(scores, bwd, post, T, N, stay, tables, status, wait_ns, stream);
    if (plan != OfScanPlan::kTogether) {
        // The forward scan beside the beam search: scan.cu's kernel is in its way least, the one that runs ahead
        // (followed by the posterior's kernel) has the shorter chain, above all of the first hundred timesteps.  So
        // the latter where the former would end after the beam search: in short and in small batches, up to two chunks to the
        // SM (three of 64 states).  Decodes with the former / the latter, ms, by chunks and T:
        //   256 states, a chunk to the SM:  75: 700 0.707 / 0.663, 1400 1.240 / 1.235;  100: 700 0.712 / 0.704, 1000 0.931 / 0.950;
        //   148: 500 0.572 / 0.552, 700 0.716 / 0.731.  Two:  149: 1666 1.729 / 1.678, 2000 2.084 / 2.064, 3000 3.17 / 3.27;  222: 1000
        //   1.176 / 1.152, 1400 1.541 / 1.541, 2000 2.162 / 2.248;  296: 700 0.921 / 0.898, 1000 1.202 / 1.207, 1666 1.810 / 1.891.
        //   Three:  297: 300 0.545 / 0.570, 1666 2.174 / 2.257.
        //   64 states:  75 to 148 within 1 % for every T (300 to 2000);  200: 300 0.330 / 0.321, 700 0.609 / 0.600, 1000 0.809 /
        //   0.820;  296: 300 0.339 / 0.337, 700 0.628 / 0.636, 1400 1.110 / 1.148.  Three:  310 of T = 800 0.765 / 0.733; 440 0.805 / 0.768.
        const long long steps = (long long)T * N;
        bool ahead = false;
        if (state_len == 3) ahead = N <= sms || N > 2 * sms || steps <= 1000ll * sms;
        if (state_len == 4) ahead = steps <= (N <= sms ? 600ll : 2000ll) * sms && N <= 2 * sms;
        // (a row of the 64-state model is too little work for a warp-wide reduction per chunk and timestep)
        if (!ahead && state_len != 3)
            return of_launch_forward_posterior(scores, bwd, post, T, N, state_len, sms, stay, tables, status, wait_ns, stream);
        const cudaError_t e =
            ahead ? of_launch_ahead(scores, nullptr, post, T, N, state_len, sms, stay, tables, status, wait_ns, stream)
                  : of_launch_scans(scores, nullptr, post, T, N, state_len, sms, stay, tables, status, wait_ns, stream);
        if (e != cudaSuccess) return e;
    }
    return of_launch_posterior(bwd, post, T, N, state_len, stream);
}

cudaError_t of_load_ahead(int kernel) {
    switch (kernel) {
        case kAhead256: return of_load<Ahead256>();
        case kAhead64Mid: return of_load<Ahead64Mid>();
        case kAhead256Mid: return of_load<Ahead256Mid>();
        case kAhead256Five: return of_load<Ahead256Five>();
        case kAhead64: return of_load<Ahead64>();
        case kPosterior64: return of_load<Posterior<64>>();
        case kPosterior256: return of_load<Posterior<256>>();
        case kPosterior1024: return of_load<Posterior<1024>>();
        default: return cudaSuccess;
    }
}
