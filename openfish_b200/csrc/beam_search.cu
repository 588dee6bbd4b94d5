// beam_search.cu -- the beam search of the CRF-CTC decode, one warp per chunk, for sm_100a.
//
// Replaces the reference kernel beam_search (src/beam_search_cuda.cu:139-528) up to, but not
// including, its traceback.  It follows the reference's CPU routine beam_search_cpu
// (src/beam_search.c:117-428) -- including its bisection of the pruning threshold, which the
// reference's CUDA kernel lacks -- because output parity is defined against the CPU decoder.
//
// A block is one chunk: a beam warp and a copy warp.
//   beam warp    lane = beam slot (width <= 32).  Everything is warp-synchronous and, where
//                lanes differ, branch free: candidate scores, duplicate-prefix merges (CRC32C
//                hashes; a stay merges with the step whose parent hash equals the stay's hash
//                run backwards through the CRC), maximum, threshold bisection by warp
//                reductions, order-preserving compaction by ballots.  One packed back-pointer
//                byte per slot and timestep goes to HBM (prev slot 5 bits | stay 1 bit | base
//                2 bits), plus the 32 initial k-mers; the traceback happens in the kernel that
//                also needs the posterior (posterior_seq.cu).
//   copy warp    one lane issues 1-D bulk asynchronous copies (no multicast) of score row t
//                (timesteps strided by N*C as in src/decode_cpu.c:204,216) and backward row t
//                into a ring; the beam warp releases a slot through an mbarrier.
// The kernel is a chain of T dependent, latency-bound steps per chunk and leaves most issue
// slots free, which is why the forward scan runs beside it on another stream.
#include <float.h>

#include "beam_post.cuh"
#include "exact_math.cuh"
#include "fast_lse.cuh"
#include "of_device.cuh"
#include "prepare.cuh"

namespace {

constexpr int kBeam = 32;
// Threads per block: the beam warp, the copy warp and a padding warp that exits at once.  With
// two-warp blocks the warp slots of an SM fill in pairs and every beam warp lands on the same two
// of the four schedulers, where they queue behind each other; a block of three warps rotates them
// over all four (measured on the hac decode: 3.87 -> 3.58 ms; fast, with seven blocks per SM:
// 4.84 -> 4.39 ms).
constexpr int kBeamBlock = 96;


// Warp maximum of a float through the sm_100a float reduction instruction.
__device__ __forceinline__ float warp_max_f32(float v) {
    float r;
    asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
    return r;
}

// The reference's two-term fold (src/beam_search.c:43-47): certified fp32 evaluation first (same
// interval argument as fast_lse.cuh: log1p(exp(-d)) in fp32 is within 2^-20.5 of the reference's
// double value; if both ends of that interval round to the same float next to m, that float is
// the reference's).  Branch free; `sure` says whether the result is certain, and the caller goes to
// the value-exact routine when it is not.
__device__ __forceinline__ float fold2_fast(float x, float y, bool &sure) {
    const float d = fabsf(x - y);
    const float m = x > y ? x : y;
    const float e = ofd::ex2_approx(-d * 1.4426950408889634f);
    const float l = ofd::lg2_approx(1.0f + e) * 0.6931471805599453f;
    const float eps = 6.75e-7f;  // 2^-20.5
    const float lo = m + (l - eps), hi = m + (l + eps);
    const bool adds = d < 17.0f;
    sure = !adds || (lo == hi && fabsf(lo) < 3.0e38f);
    return adds ? lo : m;
}

// x plus an fp16, widened (exactly) and added with one rounding, in one instruction  (Alone no faster; beside the
// forward scan of 1024 chunks of 64 states 1.13 ms instead of 1.15.)
__device__ __forceinline__ float add_half(float x, __half h) {
    float r;
    asm("add.f32.f16 %0, %1, %2;" : "=f"(r) : "h"(__half_as_ushort(h)), "f"(x));
    return r;
}

// CRC32C over two input bits, table form of src/beam_search.c:103-115:
// crc' = (crc >> 2) ^ tab[(crc ^ bits) & 3], tab = {0, 0x417B1DBC, 0x82F63B78, 0xC38D26C4}.
__device__ __forceinline__ uint32_t crc_tab2(uint32_t x) {
    return ((x & 1u) ? 0x417B1DBCu : 0u) ^ ((x & 2u) ? 0x82F63B78u : 0u);
}
__device__ __forceinline__ uint32_t crc_step2(uint32_t crc, uint32_t bits) {
    return (crc >> 2) ^ crc_tab2((crc ^ bits) & 3u);
}
// The update is a bijection for fixed input bits (the table's top two bits equal its index),
// so the parent hash that would step to `crc` by appending `bits` is unique.
__device__ __forceinline__ uint32_t crc_unstep2(uint32_t crc, uint32_t bits) {
    const uint32_t idx = crc >> 30;
    return ((crc ^ crc_tab2(idx)) << 2) | (idx ^ bits);
}
__device__ __forceinline__ uint32_t crc32c_bits(uint32_t crc, uint32_t v, int n) {
    for (int i = 0; i < n; ++i) {
        const uint32_t b = (v ^ crc) & 1u;
        crc >>= 1;
        if (b) crc ^= 0x82f63b78u;
        v >>= 1;
    }
    return crc;
}

// Number of entries of the owner table; 32 elements land on distinct ones in all but 11 % of the timesteps.
constexpr int kOwner = 4096;

// GROUP timesteps share an mbarrier pair (fewer waits and releases on the beam warp's chain), STAGES
// such groups make the ring.
template <int NS, int STAGES, int GROUP>
struct BeamSmem {
    static constexpr int kScoreRow = NS * 8;  // bytes of one fp16 score row
    static constexpr int kBwdRow = NS * 4;    // bytes of one fp32 backward row
    static constexpr int kSlot = kScoreRow + kBwdRow;
    // The beam: {score, hash, k-mer | back-pointer << 16, score before the subtraction}.  Only 32
    // elements live on; the room behind them is for the survivors beyond the 32nd in a timestep that
    // runs out of bisection guesses.
    alignas(16) uint4 rec[5 * kBeam];
    alignas(16) float4 step[kBeam];           // step scores of the timestep's candidates, by parent slot
    unsigned char owner[kOwner + 32];         // (+ one spare per lane) hash -> slot + 1 of the beam element owning it
    int init_state[kBeam];
    alignas(8) uint64_t full[STAGES];
    alignas(8) uint64_t empty[STAGES];
    int abort_flag;
    // slot of timestep t: score row t, then backward row t+1
    alignas(128) unsigned char ring[STAGES * GROUP][kSlot];
};

template <int NS, int STAGES, int GROUP, bool SCALED>
__global__ void __launch_bounds__(kBeamBlock)
beam_search_kernel(const OfDecodeArgs a) {
    constexpr int BITS = (NS == 64) ? 6 : (NS == 256 ? 8 : 10);
    constexpr int MSB = NS / 4;
    constexpr int NT = kBeamBlock;
    using Smem = BeamSmem<NS, STAGES, GROUP>;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    Smem &sm = *reinterpret_cast<Smem *>(smem_raw);

    const int tid = threadIdx.x;
    const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);  // (known to be the same for a whole warp)
    const int lane = tid & 31;
    const int chunk = blockIdx.x;
    const int T = a.T, N = a.N;
    for (int i = tid; i < (kOwner + 32) / 4; i += NT) reinterpret_cast<uint32_t *>(sm.owner)[i] = 0;
    if (tid == 0) {
        sm.abort_flag = 0;
        for (int r = 0; r < STAGES; ++r) {
            ofd::mbar_init(&sm.full[r], 1);
            ofd::mbar_init(&sm.empty[r], 1);
        }
        ofd::mbar_fence_init();
    }
    __syncthreads();

    const float *bwd_chunk = a.bwd + (size_t)chunk * (size_t)(T + 1) * NS;
    unsigned char *bp_chunk = a.bp + (size_t)chunk * (size_t)(T + 1) * kBeam;

    if (warp >= 2) return;  // the padding warp: it has helped to set shared memory up, that is all
    if (warp == 1) {
        // ------------------------------------------------------------------ copy warp
        if (lane == 0) {
            // the beam search strides timesteps by N*C (src/decode_cpu.c:204,216)
            const __half *src = a.scores + (size_t)chunk * NS * 4;
            const float *bwd_src = bwd_chunk + NS;
            const size_t beam_stride = (size_t)N * a.C;
            ofd::fill_ring_by_mbar<STAGES>((T + GROUP - 1) / GROUP, sm.full, sm.empty, &sm.abort_flag, a.status, a.wait_ns,
                                           [&](int g, int stage) {
                const int rows = min(GROUP, T - g * GROUP);
                ofd::mbar_arrive_expect_tx(&sm.full[stage], rows * Smem::kSlot);
                for (int r = 0; r < rows; ++r) {
                    unsigned char *dst = sm.ring[stage * GROUP + r];
                    ofd::bulk_g2s(dst + Smem::kScoreRow, bwd_src, Smem::kBwdRow, &sm.full[stage]);
                    ofd::bulk_g2s(dst, src, Smem::kScoreRow, &sm.full[stage]);
                    bwd_src += NS;
                    src += beam_stride;
                }
            });
        }
        return;
    }
    // ------------------------------------------------------------------ beam warp
    // (so seldom needed that the tables stay where they are: a smaller block leaves the forward scan more room)
    const ofx::TabRef tr = {a.tables->exp2_j, 1, a.tables->rcp_c, a.tables->log_c};
    const uint32_t lt_mask = (1u << lane) - 1u;
    // initial beam: first <= 32 states, in state order, reaching the 32nd largest bwd[0]
    // (src/beam_search.c:151-175).  Radix-select the 32nd largest key bit by bit.
    {
        constexpr int PER = NS / 32;
        uint32_t key[PER];
#pragma unroll
        for (int i = 0; i < PER; ++i)
            key[i] = (uint32_t)ofd::float_order_key(bwd_chunk[lane + 32 * i]) ^ 0x80000000u;
        uint32_t thr = 0;
        for (int bit = 31; bit >= 0; --bit) {
            const uint32_t cand = thr | (1u << bit);
            int c = 0;
#pragma unroll
            for (int i = 0; i < PER; ++i) c += key[i] >= cand;
            c = __reduce_add_sync(0xffffffffu, c);
            if (c >= kBeam) thr = cand;
        }
        int filled = 0;
#pragma unroll
        for (int i = 0; i < PER; ++i) {
            const bool f = key[i] >= thr;
            const uint32_t bal = __ballot_sync(0xffffffffu, f);
            const int pos = filled + __popc(bal & lt_mask);
            if (f && pos < kBeam) sm.init_state[pos] = lane + 32 * i;
            filled += __popc(bal);
        }
        __syncwarp();
    }
    int W = kBeam;
    {
        const int state = sm.init_state[lane];
        sm.rec[lane] = make_uint4(__float_as_uint(0.f), crc32c_bits(0x12345678u, (uint32_t)state, 32),
                                  (uint32_t)state | (uint32_t)(state & 3) << 22, __float_as_uint(0.f));
        a.init_kmers[(size_t)chunk * kBeam + lane] = state;  // for the traceback's benefit
    }
    __syncwarp();

    // Bound: the chain of one timestep's dependent instructions in this one warp (two to three cycles
    // an instruction), so the usual route is one long basic block up to the first count, and what
    // happens in one timestep of six (a merge, two elements on one table entry) redoes the end of it.
    unsigned char *bp = bp_chunk + lane;
    const unsigned char *slot = sm.ring[0];
    int stage = 0, in_group = 0;
    uint32_t parity = 0;
    ofd::mbar_wait_bounded(&sm.full[0], 0u, &sm.abort_flag, a.status, a.wait_ns);
    for (int t = 0; t < T; ++t) {
        const uint4 mine = sm.rec[lane];
        const bool act = lane < W;
        // (idle slots hold a valid, stale k-mer: they read like everybody else, and a score of -inf
        // voids their candidates)
        const float score = act ? __uint_as_float(mine.x) : -INFINITY;
        const uint32_t hash = mine.y;
        const int state = (int)(mine.z & (uint32_t)(NS - 1));
        const int q = state & (MSB - 1);
        const int top = state >> (BITS - 2);
        const uint32_t b_own = (uint32_t)state & 3u;

        // duplicate-prefix detection (src/beam_search.c:281-316): a stay can only merge with a
        // step whose parent's hash is `need`.  Every element writes its slot number into an
        // owner table indexed by its hash; a stay then finds the one candidate parent by a single
        // look-up and confirms it by comparing the full hash.
        // (idle slots use a private spare entry so that nothing here branches)
        const uint32_t own_at = act ? (hash & (kOwner - 1)) : kOwner + lane;
        sm.owner[own_at] = (unsigned char)(lane + 1);

        // candidates: 4 steps (state' = 4q + b, column 16q + 4b + top) and the stay
        const __half *sp = reinterpret_cast<const __half *>(slot) + 16 * q + top;
        const float *brow = reinterpret_cast<const float *>(slot + Smem::kScoreRow);
        const float4 bw = *reinterpret_cast<const float4 *>(brow + 4 * q);
        const float bs = brow[state];
        const __half s0 = sp[0], s1 = sp[4], s2 = sp[8], s3 = sp[12];
        const uint32_t need = crc_unstep2(hash, b_own);
        __syncwarp();
        const int mine_back = sm.owner[own_at];
        const int cand = sm.owner[need & (kOwner - 1)];
        bp[0] = (unsigned char)(act ? mine.z >> 16 : 0u);  // back-pointer row t
        bp += kBeam;
        // the children's hashes (the CRC is linear: appending base b adds tab[b])
        const uint32_t h0 = crc_step2(hash, 0u);
        float c0, c1, c2, c3, c4;
        {
            // (float)score * score_scale, rounded before it is added (src/beam_search.c:233-234)
            auto plus = [&](float x, __half h) {
                return SCALED ? __fadd_rn(x, __fmul_rn(__half2float(h), a.score_scale)) : add_half(x, h);
            };
            c0 = __fadd_rn(plus(score, s0), bw.x);
            c1 = __fadd_rn(plus(score, s1), bw.y);
            c2 = __fadd_rn(plus(score, s2), bw.z);
            c3 = __fadd_rn(plus(score, s3), bw.w);
            c4 = __fadd_rn(__fadd_rn(score, a.stay), bs);
        }
        // pruning threshold (src/beam_search.c:320-381): best - ln(beam_cut); if more than 32
        // candidates pass, bisect towards 25..32 survivors for at most 9 further guesses.  The first
        // of those guesses is known from the start and counted together with the threshold itself.
        float best, cut, mid;
        uint32_t both;
        auto passing = [&](float th) {
            return (uint32_t)((c0 >= th) + (c1 >= th) + (c2 >= th) + (c3 >= th) + (c4 >= th));
        };
        auto threshold = [&]() {
            best = warp_max_f32(ofd::max3(ofd::max3(c0, c1, c2), c3, c4));
            cut = __fsub_rn(best, a.log_beam_cut);
            mid = __fmul_rn(__fadd_rn(cut, best), 0.5f);
            both = __reduce_add_sync(0xffffffffu, passing(cut) + (passing(mid) << 16));
        };
        const uint32_t cand_hash = __shfl_sync(0xffffffffu, hash, (cand - 1) & 31);
        int mate = (act && cand > 0 && cand_hash == need) ? cand - 1 : -1;
        const bool odd = __any_sync(0xffffffffu, mate >= 0 || mine_back != lane + 1);
        __syncwarp();  // (a vote orders no memory: the entries are cleared only after every lane's look-ups)
        sm.owner[own_at] = 0;
        threshold();
        if (__builtin_expect(odd, 0)) {
            bool conflict = false;
            // elements that found another on their table entry: the table does not know them, so
            // every lane compares with each of them (one, nearly always)
            for (uint32_t left = __ballot_sync(0xffffffffu, mine_back != lane + 1); left; left &= left - 1u) {
                const int l = __ffs(left) - 1;
                const uint32_t h = __shfl_sync(0xffffffffu, hash, l);
                const uint32_t same = __ballot_sync(0xffffffffu, act && hash == h);
                if (same & (same - 1u)) conflict = true;  // a hash that occurs twice in the beam
                if (act && need == h) mate = l;
            }
            const bool merges = __any_sync(0xffffffffu, mate >= 0);
            if (merges) {
                sm.step[lane] = make_float4(c0, c1, c2, c3);
                __syncwarp();
            }
            if (merges && !conflict) {
                // every stay has at most one partner and no step has two: the folds are independent.
                // The stay reads its partner's step score, folds, and puts the partner's new score back.
                float *theirs = reinterpret_cast<float *>(&sm.step[mate >= 0 ? mate : lane]) + b_own;
                const float x = c4, y = *theirs;
                bool sure;
                float f = fold2_fast(x, y, sure);
                if (mate >= 0) {
                    if (!sure) f = ofx::fold2_exact(x, y, tr);
                    const bool stay_wins = x > y;
                    c4 = stay_wins ? f : -FLT_MAX;
                    *theirs = stay_wins ? -FLT_MAX : f;
                }
            } else if (merges) {
                // repeated hashes inside the beam (CRC collisions): replay the reference's
                // nested loop, stay-major then slot-minor, on one lane
                sm.rec[lane] = make_uint4(hash, b_own, __float_as_uint(c4), 0u);
                __syncwarp();
                if (lane == 0) {
                    float *cstep = reinterpret_cast<float *>(sm.step);
                    for (int i = 0; i < W; ++i) {
                        const uint32_t h_i = sm.rec[i].x, b_i = sm.rec[i].y;
                        for (int jj = 0; jj < W; ++jj) {
                            if (h_i != crc_step2(sm.rec[jj].x, b_i)) continue;
                            const float x = __uint_as_float(sm.rec[i].z);
                            const float y = cstep[4 * jj + b_i];
                            const float f = ofx::fold2_exact(x, y, tr);
                            if (x > y) {
                                sm.rec[i].z = __float_as_uint(f);
                                cstep[4 * jj + b_i] = -FLT_MAX;
                            } else {
                                cstep[4 * jj + b_i] = f;
                                sm.rec[i].z = __float_as_uint(-FLT_MAX);
                            }
                        }
                    }
                }
                __syncwarp();
                if (act) c4 = __uint_as_float(sm.rec[lane].z);
            }
            if (merges) {
                __syncwarp();
                const float4 r = sm.step[lane];
                c0 = r.x; c1 = r.y; c2 = r.z; c3 = r.w;
                threshold();
            }
        }
        int kept = (int)(both & 0xffffu);
        if (kept > kBeam) {
            float lo = cut, hi = best;
            cut = mid;
            kept = (int)(both >> 16);
            int guesses = 2;
#pragma unroll 2
            for (int g = 0; g < 8; ++g) {
                if (kept <= kBeam && kept >= 25) break;
                const bool many = kept > kBeam;
                lo = many ? cut : lo;
                hi = many ? hi : cut;
                cut = __fmul_rn(__fadd_rn(cut, many ? hi : lo), 0.5f);
                kept = (int)__reduce_add_sync(0xffffffffu, passing(cut));
                ++guesses;
            }
            if (guesses == 10) {
                cut = hi;
                kept = (int)__reduce_add_sync(0xffffffffu, passing(cut));
            }
        }

        // survivors keep candidate order: steps (slot-major, base-minor), then stays.  Every
        // survivor goes to its new slot complete: score less the backward score, hash, k-mer and
        // back-pointer, so that the next timestep starts with one read.
        {
            const bool k0 = c0 >= cut, k1 = c1 >= cut, k2 = c2 >= cut, k3 = c3 >= cut, k4 = c4 >= cut;
            const uint32_t B0 = __ballot_sync(0xffffffffu, k0), B1 = __ballot_sync(0xffffffffu, k1);
            const uint32_t B2 = __ballot_sync(0xffffffffu, k2), B3 = __ballot_sync(0xffffffffu, k3);
            const uint32_t B4 = __ballot_sync(0xffffffffu, k4);
            uint4 *to = sm.rec + ((__popc(B0 & lt_mask) + __popc(B1 & lt_mask)) + (__popc(B2 & lt_mask) + __popc(B3 & lt_mask)));
            uint4 *to4 = sm.rec + (kept - __popc(B4 & ~lt_mask));
            const uint32_t word = (uint32_t)(4 * q) | (uint32_t)lane << 16;
            if (k0) *to = make_uint4(__float_as_uint(__fsub_rn(c0, bw.x)), h0, word, __float_as_uint(c0));
            to += k0;
            if (k1) *to = make_uint4(__float_as_uint(__fsub_rn(c1, bw.y)), h0 ^ crc_tab2(1u), word | (1u | 1u << 22), __float_as_uint(c1));
            to += k1;
            if (k2) *to = make_uint4(__float_as_uint(__fsub_rn(c2, bw.z)), h0 ^ crc_tab2(2u), word | (2u | 2u << 22), __float_as_uint(c2));
            to += k2;
            if (k3) *to = make_uint4(__float_as_uint(__fsub_rn(c3, bw.w)), h0 ^ crc_tab2(3u), word | (3u | 3u << 22), __float_as_uint(c3));
            if (k4) *to4 = make_uint4(__float_as_uint(__fsub_rn(c4, bs)), hash, (uint32_t)state | (uint32_t)(lane | 32) << 16 | b_own << 22, __float_as_uint(c4));
        }
        W = min(kept, kBeam);
        __syncwarp();
        slot += Smem::kSlot;
        if (++in_group == GROUP) {
            // the group's rows have been read by every lane
            in_group = 0;
            ofd::mbar_arrive_if(lane == 0, &sm.empty[stage]);
            if (++stage == STAGES) {
                stage = 0;
                slot = sm.ring[0];
                parity ^= 1u;
            }
            if (t + 1 < T && !ofd::mbar_try_wait(&sm.full[stage], parity))
                ofd::mbar_wait_slow(&sm.full[stage], parity, &sm.abort_flag, a.status, a.wait_ns);
        }
    }
    if (T > 0) {
        // best survivor swaps into slot 0 (src/beam_search.c:398-414); of the last row only the
        // back-pointers matter any more
        const uint4 mine = sm.rec[lane];
        const float sc = lane < W ? __uint_as_float(mine.w) : -INFINITY;
        const float top_s = warp_max_f32(sc);
        const uint32_t eq = __ballot_sync(0xffffffffu, lane < W && sc == top_s && sc > -FLT_MAX);
        const int at = eq ? __ffs(eq) - 1 : 0;
        uint32_t meta = lane < W ? mine.z >> 16 : 0u;
        const uint32_t m0 = __shfl_sync(0xffffffffu, meta, 0), ma = __shfl_sync(0xffffffffu, meta, at);
        if (lane == at) meta = m0;
        if (lane == 0) meta = ma;
        bp[0] = (unsigned char)meta;
    }
}

template <int NS, int STAGES, int GROUP, bool SCALED>
struct Beam {
    static constexpr auto kern = beam_search_kernel<NS, STAGES, GROUP, SCALED>;
    static constexpr size_t bytes = sizeof(BeamSmem<NS, STAGES, GROUP>);
    static cudaError_t launch(const OfDecodeArgs &a, cudaStream_t stream) {
        kern<<<a.N, kBeamBlock, bytes, stream>>>(a);
        return cudaGetLastError();
    }
};
template <bool SCALED> using Beam64 = Beam<64, 2, 4, SCALED>;
template <bool SCALED> using Beam256 = Beam<256, 2, 2, SCALED>;
template <bool SCALED> using Beam1024 = Beam<1024, 4, 1, SCALED>;
// For a batch that has an SM to a beam search (no forward scan beside it): longer groups, since a group's end (arrival, wait,
// the next slot's address) is on the chain and costs as much as a tenth of a timestep.  The kernel with groups of
// 4 / 6 / 8 / 12 / 16 timesteps: 64 states, T = 1000, 0.432 / 0.426 / 0.426 / 0.422 / 0.422 ms; 256 states, T = 1666, 0.702 /
// 0.694 / 0.688 / 0.678 / 0.684 (0.735 with two); 1024 states, 74 chunks of T = 800, with 1 / 2 / 5 / 6 / 8: 0.469 / 0.487 / 0.422
// / 0.426 / 0.446.  Beside forward scans the larger blocks push those together on fewer SMs: 148 chunks of 256 states, T =
// 1666, 2.70 ms a decode instead of 1.52.
template <bool SCALED> using BeamFew64 = Beam<64, 2, 12, SCALED>;
template <bool SCALED> using BeamFew256 = Beam<256, 2, 12, SCALED>;
template <bool SCALED> using BeamFew1024 = Beam<1024, 2, 5, SCALED>;

// (a scale of one leaves every score as it is: no multiplication then)
template <template <bool> class B>
cudaError_t launch_beam_of(const OfDecodeArgs &a, cudaStream_t stream) {
    return a.score_scale == 1.0f ? B<false>::launch(a, stream) : B<true>::launch(a, stream);
}
template <template <bool> class B, template <bool> class FEW>
cudaError_t launch_beam(const OfDecodeArgs &a, int sms, cudaStream_t stream) {
    // (the batches whose scans are both done when the beam search starts, see of_scan_plan)
    const bool few = a.state_len == 5 ? a.N <= sms : 2 * a.N <= sms;
    return few ? launch_beam_of<FEW>(a, stream) : launch_beam_of<B>(a, stream);
}

}  // namespace

cudaError_t of_launch_beam_search(const OfDecodeArgs &a, int sms, cudaStream_t stream) {
    switch (a.state_len) {
        case 3: return launch_beam<Beam64, BeamFew64>(a, sms, stream);
        case 4: return launch_beam<Beam256, BeamFew256>(a, sms, stream);
        case 5: return launch_beam<Beam1024, BeamFew1024>(a, sms, stream);
        default: return cudaErrorInvalidValue;
    }
}

cudaError_t of_load_beam_search(int kernel) {
    switch (kernel) {
        case kBeam64: return of_load<Beam64<false>>();
        case kBeam256: return of_load<Beam256<false>>();
        case kBeam1024: return of_load<Beam1024<false>>();
        case kBeam64Scaled: return of_load<Beam64<true>>();
        case kBeam256Scaled: return of_load<Beam256<true>>();
        case kBeam1024Scaled: return of_load<Beam1024<true>>();
        case kBeamFew64: return of_load<BeamFew64<false>>();
        case kBeamFew256: return of_load<BeamFew256<false>>();
        case kBeamFew1024: return of_load<BeamFew1024<false>>();
        case kBeamFew64Scaled: return of_load<BeamFew64<true>>();
        case kBeamFew256Scaled: return of_load<BeamFew256<true>>();
        case kBeamFew1024Scaled: return of_load<BeamFew1024<true>>();
        default: return cudaSuccess;
    }
}
