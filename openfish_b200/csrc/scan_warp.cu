// scan_warp.cu -- a chunk's scan by one warp, for batches of the 64-state model that fill the GPU, for sm_100a.
//
// Same recursions and, value for value, the same results as scan.cu and scan_ahead.cu (src/decode_cpu.c:13-52,
// 54-119).  A block is a single warp: lane l has two of the 64 states, the previous row lies in shared memory, and
// nothing waits for anybody.  A state whose rounding the fp32 evaluation cannot certify gets the likelier of its two
// candidate floats and a bit in the lane's mask; after K timesteps the warp deals the marked states out to its
// lanes and works them out exactly, all at once.  Where a guess was wrong the value is put right in its row and
// the scan goes on from the timestep behind the first such (the rows in between are taken again: one group in
// ten, four timesteps on average).  Only then do the group's rows count, and with POST the posterior
// softmax_s(fwd + bwd) is formed from them, K rows at once.  While the scores are small every state goes through
// the exact routine.
//
// What bounds it: in a batch that fills the GPU, instructions.  Gone is what the kernels for fewer chunks spend so
// that a timestep is short: a checker's pass over a nearly empty list every timestep or two (one pass for eight
// here), barriers and votes, a copy warp's polling, and for the posterior a forward row that goes to HBM and back
// and a reduction over 32 lanes (four lanes to a row here).  A chunk alone takes longer than with those, and the
// backward scan does up to eight chunks to the SM (scan_ahead.cu: 1024 chunks of T = 1666 0.57 ms instead of 0.74).  Beside
// the beam search, with the posterior, T = 1666: 1024 chunks 1.31 ms instead of scan_ahead.cu's 1.72, 4096 4.71; backward scan of
// 4096 chunks 1.83 ms.  (The kernel before it, scan.cu's with a posterior kernel: 1.54 for 1024.)  K = 8: with 4 there are
// twice the passes (4096 chunks: backward scan 2.17 ms instead of 1.84); with 16 a block takes twice the shared memory (forward
// scan of 4096 chunks beside the beam search 5.4 ms instead of 4.7).
#include "exact_math.cuh"
#include "fast_lse.cuh"
#include "of_device.cuh"
#include "prepare.cuh"
#include "scan.cuh"
#include "scan_piece.cuh"

namespace {

using namespace scan_topo;

constexpr int NS = 64;
constexpr int K = 8;            // timesteps to a group
constexpr int STAGES = 2;       // groups of score rows kept
constexpr int H = K + 1;        // rows kept: a group's input row and the K behind it
constexpr int SPT = 2;          // states to a lane
constexpr int kGuessFrom = 256; // score from which on guesses are made
constexpr int kRowBytes = NS * 4 * 2;
static_assert(SPT * K <= 32, "a mask word holds a group's marks");

template <bool POST>
struct WarpSmem {
    alignas(128) unsigned char ring[STAGES][K][kRowBytes];
    // with the posterior: row t+1 of the backward scores beside score row t
    alignas(128) float bwd_ring[POST ? STAGES : 1][POST ? K : 1][POST ? NS : 4];
    alignas(16) float rows[H][NS];
    alignas(8) uint64_t full[STAGES];
    unsigned short marked[64];
    int abort_flag;
};

__device__ __forceinline__ int wrap(int row) { return row < H ? row : row - H; }

// Softmax of a sum of rows, in the order of scan_ahead.cu's posterior_kernel, so that both leave the same bits:
// states 2p and 2p+1 make pair p, and pairs are added up as its 32 lanes' partial sums are, distance 16 first.
// Four lanes have a row; lane m of them the pairs 2m, 2m+1 and so on at distances of 8 (float4 accesses).
template <bool ZERO>
__device__ __forceinline__ void posterior_row(const float *fwd, const float *bwd, float *post, float m0, int m, bool wanted) {
    const float kLog2e = 1.4426950408889634f;
    const ofd::f32x2 mm = ofd::pack2(m0, m0), l2 = ofd::pack2(kLog2e, kLog2e);
    float e[4][4];
    ofd::f32x2 sum[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float4 a = ZERO ? make_float4(0.f, 0.f, 0.f, 0.f) : *reinterpret_cast<const float4 *>(fwd + 16 * i + 4 * m);
        const float4 b = *reinterpret_cast<const float4 *>(bwd + 16 * i + 4 * m);
        ofd::unpack2(ofd::mul2(ofd::sub2(ofd::add2(ofd::pack2(a.x, a.y), ofd::pack2(b.x, b.y)), mm), l2), e[i][0], e[i][1]);
        ofd::unpack2(ofd::mul2(ofd::sub2(ofd::add2(ofd::pack2(a.z, a.w), ofd::pack2(b.z, b.w)), mm), l2), e[i][2], e[i][3]);
#pragma unroll
        for (int k = 0; k < 4; ++k) e[i][k] = ofd::ex2_approx(e[i][k]);
        sum[i] = ofd::pack2(e[i][0] + e[i][1], e[i][2] + e[i][3]);
    }
    float p0, p1;
    ofd::unpack2(ofd::add2(ofd::add2(sum[0], sum[2]), ofd::add2(sum[1], sum[3])), p0, p1);
#pragma unroll
    for (int o = 2; o; o >>= 1) {
        p0 += __shfl_xor_sync(0xffffffffu, p0, o);
        p1 += __shfl_xor_sync(0xffffffffu, p1, o);
    }
    const float inv = 1.0f / (p0 + p1);
    if (wanted) {
#pragma unroll
        for (int i = 0; i < 4; ++i)
            *reinterpret_cast<float4 *>(post + 16 * i + 4 * m) = make_float4(e[i][0] * inv, e[i][1] * inv, e[i][2] * inv, e[i][3] * inv);
    }
}

// out: the rows [T+1][64] of every chunk, or with POST the posterior's (bwd_in: the finished backward scores).
template <class Topo, bool POST>
__global__ void __launch_bounds__(32, 16)
scan_warp_kernel(const __half *__restrict__ scores, float *__restrict__ out, const float *__restrict__ bwd_in, int T, int N,
                 float stay, const ofx::Tables *__restrict__ tables, int *status, uint64_t wait_ns) {
    static_assert(!POST || Topo::kForward, "the posterior rides on the forward scan");
    using Smem = WarpSmem<POST>;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    Smem &sm = *reinterpret_cast<Smem *>(smem_raw);
    const int lane = threadIdx.x;
    const int chunk = blockIdx.x;
    const uint32_t lt_mask = (1u << lane) - 1u;
    const int groups = (T + K - 1) / K;
    const size_t t_stride = (size_t)N * NS * 4;
    const __half *const chunk_scores = scores + (size_t)chunk * NS * 4;
    float *const out_chunk = out + (size_t)chunk * (size_t)(T + 1) * NS;
    const float *const bwd_chunk = POST ? bwd_in + (size_t)chunk * (size_t)(T + 1) * NS : nullptr;
    // (the tables stay where they are: a block per chunk, and the exact routine once a group)
    const ofx::TabRef tr = {tables->exp2_j, 1, tables->rcp_c, tables->log_c};

    reinterpret_cast<float2 *>(sm.rows[0])[lane] = make_float2(0.f, 0.f);
    if (lane == 0) {
        sm.abort_flag = 0;
        for (int r = 0; r < STAGES; ++r) ofd::mbar_init(&sm.full[r], 1);
        ofd::mbar_fence_init();
    }
    __syncwarp();
    // The copies of group g, by lane 0 alone; after an abort no more are issued.
    int issued = 0;
    auto fill = [&](int g) {
        if (sm.abort_flag) return;
        const int stage = g % STAGES, n = min(K, T - g * K);
        ofd::mbar_arrive_expect_tx(&sm.full[stage], n * (kRowBytes + (POST ? NS * 4 : 0)));
        for (int q = 0; q < n; ++q) {
            ofd::bulk_g2s(sm.ring[stage][q], chunk_scores + t_stride * (size_t)Topo::score_row(g * K + q, T), kRowBytes, &sm.full[stage]);
            if (POST) ofd::bulk_g2s(sm.bwd_ring[stage][q], bwd_chunk + (size_t)(g * K + q + 1) * NS, NS * 4, &sm.full[stage]);
        }
        ++issued;
    };
    if (lane == 0)
        for (int g = 0; g < STAGES && g < groups; ++g) fill(g);

    float m0 = 0.f;  // softmax offset: the maximum of row 0, where the forward scores are zero
    if constexpr (POST) {
        m0 = ofd::warp_max(fmaxf(fmaxf(-3.0e38f, bwd_chunk[lane]), bwd_chunk[lane + 32]));
        posterior_row<true>(nullptr, bwd_chunk, out_chunk, m0, lane & 3, lane < 4);
    } else {
        reinterpret_cast<float2 *>(out_chunk + (size_t)Topo::zero_row(T) * NS)[lane] = make_float2(0.f, 0.f);
    }

    const int j = lane % Topo::NJ, k0 = (lane / Topo::NJ) * SPT;
    float res[SPT] = {0.f, 0.f};  // the lane's states of the current row: its stay terms for the next timestep
    const ptrdiff_t out_step = Topo::kForward ? (ptrdiff_t)NS : -(ptrdiff_t)NS;
    int stage = 0, at = 0;  // at: the group's input row
    uint32_t parity = 0;
    for (int g = 0; g < groups; ++g) {
        if (!ofd::mbar_try_wait(&sm.full[stage], parity))
            ofd::mbar_wait_slow(&sm.full[stage], parity, &sm.abort_flag, status, wait_ns);
        __syncwarp();
        const int n = min(K, T - g * K);
        for (int q = 0;;) {
            // timesteps q .. n-1 of the group
            const float *in = sm.rows[wrap(at + q)];
            const unsigned char *row = sm.ring[stage][q];
            float *gmem_out = out_chunk + (ptrdiff_t)Topo::out_row(g * K + q, T) * NS;
            const bool all = exact_for_all<kGuessFrom>(in[0]);
            uint32_t mask = 0;  // bit SPT*q + k: state k of timestep q is a guess
            Piece piece(row, j);
#pragma unroll 1
            for (; q < n; ++q) {
                float *const nxt = in == sm.rows[H - 1] ? sm.rows[0] : const_cast<float *>(in) + NS;
                if (__builtin_expect(all, 0)) {
                    const float4 x = exact_step<Topo, SPT>(in, row, j, k0, stay, make_float4(res[0], res[1], 0.f, 0.f),
                                                           tr.exp2_j, tr.rcp_c, tr.log_c);
                    res[0] = x.x;
                    res[1] = x.y;
                } else {
                    float v[SPT][5];
                    thread_terms<Topo, SPT>(in, piece, j, k0, stay, v, res);
                    mask |= ofd::lse5_guess_pairs<SPT, false>(v, res, nullptr) << (SPT * q);
                }
                row += kRowBytes;
                if (q + 1 < n) piece.load(row, j);
                thread_store<Topo, SPT>(nxt, j, k0, res);
                if (!POST) thread_store<Topo, SPT>(gmem_out, j, k0, res);
                gmem_out += out_step;
                in = nxt;
                __syncwarp();
            }
            // The marked states, 32 at a time.  A value put right here may be one that a later entry reads, or that
            // was itself worked out from a wrong one: both lie behind the first wrong timestep, from which on all
            // is taken again.  (scan_ahead.cu's checker deals its marks out the same way.  As a function that both call the
            // compiler lays 64-state scan_ahead's code out so that 300 to 444 chunks take 5 % longer.)
            int first_wrong = K;
            for (uint32_t owners = __ballot_sync(0xffffffffu, mask != 0); owners;) {
                int count = 0;
                do {
                    if (mask) sm.marked[count + __popc(owners & lt_mask)] = (unsigned short)(lane | (__ffs(mask) - 1) << 5);
                    count += __popc(owners);
                    mask &= mask - 1u;
                    owners = __ballot_sync(0xffffffffu, mask != 0);
                } while (owners && count + __popc(owners) <= 64);
                __syncwarp();
                for (int first = 0; first < count; first += 32) {
                    const bool mine = first + lane < count;
                    const int e = sm.marked[mine ? first + lane : 0];
                    const int l = e & 31, bit = e >> 5, t = bit / SPT;
                    const int s = Topo::state(l % Topo::NJ, (l / Topo::NJ) * SPT + bit % SPT);
                    const int r = wrap(at + t);
                    float *const guess = &sm.rows[wrap(r + 1)][s];
                    float v[5];
                    terms_of<Topo>(s, sm.rows[r], sm.ring[stage][t], stay, v);
                    const float x = ofx::lse5_exact(v, tr);
                    const bool wrong = mine && __float_as_uint(x) != __float_as_uint(*guess);
                    if (__any_sync(0xffffffffu, wrong)) {
                        first_wrong = min(first_wrong, (int)__reduce_min_sync(0xffffffffu, wrong ? (uint32_t)t : (uint32_t)K));
                        __syncwarp();  // (every lane has its terms)
                        if (wrong) {
                            *guess = x;
                            if (!POST) out_chunk[(ptrdiff_t)Topo::out_row(g * K + t, T) * NS + s] = x;
                        }
                    }
                    __syncwarp();
                }
            }
            if (first_wrong == K) break;
            q = first_wrong + 1;
#pragma unroll
            for (int k = 0; k < SPT; ++k) res[k] = sm.rows[wrap(at + q)][Topo::state(j, k0 + k)];
            if (q == n) break;
        }
        if constexpr (POST) {
            const int r = lane >> 2;  // (a row behind the last is formed from leftovers and not written)
            posterior_row<false>(sm.rows[wrap(at + 1 + r)], sm.bwd_ring[stage][r], out_chunk + (size_t)(g * K + r + 1) * NS, m0,
                                 lane & 3, r < n);
        }
        __syncwarp();  // the group's rows have been read by every lane
        if (lane == 0 && g + STAGES < groups) fill(g + STAGES);
        at = wrap(at + n);
        if (++stage == STAGES) {
            stage = 0;
            parity ^= 1u;
        }
    }
    // after an abort the newest copies get a bounded chance to land before the block retires
    if (lane == 0 && sm.abort_flag) ofd::mbar_drain_bounded(sm.full, STAGES, issued, wait_ns);
}

template <class Topo, bool POST>
struct WarpScan {
    static constexpr auto kern = scan_warp_kernel<Topo, POST>;
    static constexpr size_t bytes = sizeof(WarpSmem<POST>);
};
using WarpBwd = WarpScan<BwdTopo<NS>, false>;
using WarpFwd = WarpScan<FwdTopo<NS>, true>;

}  // namespace

cudaError_t of_launch_warp_backward(const void *scores_fp16, float *bwd, int T, int N, float stay, const ofx::Tables *tables,
                                    int *status, uint64_t wait_ns, cudaStream_t stream) {
    if (T < 1) return cudaErrorInvalidValue;
    WarpBwd::kern<<<N, 32, WarpBwd::bytes, stream>>>(static_cast<const __half *>(scores_fp16), bwd, nullptr, T, N, stay, tables,
                                                     status, wait_ns);
    return cudaGetLastError();
}

cudaError_t of_launch_warp_forward_posterior(const void *scores_fp16, const float *bwd, float *post, int T, int N, float stay,
                                             const ofx::Tables *tables, int *status, uint64_t wait_ns, cudaStream_t stream) {
    if (T < 1) return cudaErrorInvalidValue;
    WarpFwd::kern<<<N, 32, WarpFwd::bytes, stream>>>(static_cast<const __half *>(scores_fp16), post, bwd, T, N, stay, tables,
                                                     status, wait_ns);
    return cudaGetLastError();
}

cudaError_t of_load_warp(int kernel) {
    switch (kernel) {
        case kWarpBwd64: return of_load<WarpBwd>();
        case kWarpFwd64: return of_load<WarpFwd>();
        default: return cudaSuccess;
    }
}
