// posterior_seq.cu -- traceback, per-base quality and sequence/qstring generation for
// one chunk per block, for sm_100a.
//
// Replaces the traceback at the end of beam_search (src/beam_search_cuda.cu:517-527) and the kernels
// compute_qual_data (:530-605) and generate_sequence (:52-121); semantics are those of the CPU
// routines (src/beam_search.c:430-496 and 49-99).
//
// The whole block walks the back-pointers the beam search left in HBM (staged through shared memory
// in windows), rebuilds the k-mer of every path element from the emitted bases, gathers the
// posterior of each path k-mer and its shifted neighbours, and emits moves, sequence and qstring,
// zero-filling the unused tail of each row.
#include <float.h>

#include "beam_post.cuh"
#include "of_device.cuh"
#include "prepare.cuh"

namespace {

constexpr int kBeam = 32;

// A chunk's row of n bytes to host memory, in stores of 16 bytes (what crosses the bus should be as few
// requests as possible).  The caller's buffer may start anywhere: where its rows don't lie as the device's do,
// the 16 bytes of a store are gathered one by one (601 chunks of T = 1201: 0.125 ms for the kernel either way; by
// way of the staging area the call took 2.97 ms instead of 2.83, of 4095 chunks 19.5 instead of 17.9).
__device__ __forceinline__ void row_to_host(unsigned char *to, const unsigned char *from, int n, int tid, int threads) {
    const int head = min(n, (int)((16u - ((uintptr_t)to & 15u)) & 15u));
    if (tid < head) to[tid] = from[tid];
    const int pieces = (n - head) >> 4;
    const bool alike = (((uintptr_t)(from + head)) & 15u) == 0;
    for (int i = tid; i < pieces; i += threads) {
        const unsigned char *src = from + head + 16 * i;
        uint4 v;
        if (alike) {
            v = *reinterpret_cast<const uint4 *>(src);
        } else {
            uint32_t w[4];
#pragma unroll
            for (int k = 0; k < 4; ++k)
                w[k] = src[4 * k] | (uint32_t)src[4 * k + 1] << 8 | (uint32_t)src[4 * k + 2] << 16 | (uint32_t)src[4 * k + 3] << 24;
            v = make_uint4(w[0], w[1], w[2], w[3]);
        }
        reinterpret_cast<uint4 *>(to + head)[i] = v;
    }
    const int done = head + 16 * pieces;
    if (tid < n - done) to[done + tid] = from[done + tid];
}

template <int NS, int NT>
struct PostSmem {
    int part[NT / 32];  // steps in each warp's timesteps
    int init_kmers[kBeam];
    // the tail phase's arrays start here and run into the dynamic shared memory behind
    alignas(128) unsigned char tail[128];
};

// What bounds it: in a large batch the posterior's gather, whose 32-byte pieces use half of what a read of
// the memory brings; in a small one the chain of phases.  1024 threads to a chunk, with the next window's
// rows on their way: 0.133 ms for 512 chunks of T = 1666 instead of 0.162 with 256 threads that fetch as they
// go, 0.032 instead of 0.048 for 16, 0.153 instead of 0.217 for 1024 of the 64-state model.
template <int NS, int NT>
__global__ void __launch_bounds__(NT)
posterior_seq_kernel(const OfDecodeArgs a) {
    constexpr int BITS = (NS == 64) ? 6 : (NS == 256 ? 8 : 10);
    constexpr int SL = BITS / 2;
    constexpr int MSB = NS / 4;
    constexpr int kWin = NT / 2;  // traceback window, timesteps: a thread stages one 16-byte piece of it
    using Smem = PostSmem<NS, NT>;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    Smem &sm = *reinterpret_cast<Smem *>(smem_raw);

    const int tid = threadIdx.x;
    const int chunk = blockIdx.x;
    const int T = a.T;
    const float *post_chunk = a.post + (size_t)chunk * (size_t)(T + 1) * NS;
    const unsigned char *bp_chunk = a.bp + (size_t)chunk * (size_t)(T + 1) * kBeam;

    unsigned char *tail = sm.tail;
    const int Tp = (T + 16) & ~15;
    unsigned char *win = tail;                          // kWin * 32 bytes
    unsigned char *bexit = win + kWin * kBeam;          // [kWin/8][32] slot reached below an 8-row block
    int *bentry = reinterpret_cast<int *>(bexit + (kWin / 8) * kBeam);  // [kWin/8] slot entering each block
    unsigned char *path = reinterpret_cast<unsigned char *>(bentry + kWin / 8);  // [T+1] packed back-pointer of the path
    unsigned char *ext = path + Tp;                     // [SL + T] initial k-mer bases then steps
    unsigned short *cnt = reinterpret_cast<unsigned short *>(ext + Tp + 16);  // [T+1] steps so far
    float *qp = reinterpret_cast<float *>(reinterpret_cast<unsigned char *>(cnt) + 2 * Tp);  // [T]

    // traceback from slot 0 of the last row (src/beam_search.c:430-438), window by window.
    // Following one pointer per row is a chain of dependent shared-memory reads, so the chain is
    // shortened eightfold: for every block of 8 rows and each of the 32 slots one could enter it
    // with, all threads first work out where one leaves it (independent short walks); one thread
    // then hops block to block; finally all threads replay their block with the known entry.
    // The next window's rows are on their way while this one is walked.
    if (tid < kBeam) sm.init_kmers[tid] = a.init_kmers[(size_t)chunk * kBeam + tid];
    uint4 piece = make_uint4(0, 0, 0, 0);
    auto fetch = [&](int hi_r) {
        const int lo_r = max(1, hi_r - kWin + 1);
        if (tid < 2 * (hi_r - lo_r + 1)) piece = __ldcg(reinterpret_cast<const uint4 *>(bp_chunk + (size_t)lo_r * kBeam) + tid);
    };
    fetch(T);
    int at = 0;
    for (int hi_r = T; hi_r >= 1; hi_r -= kWin) {
        const int lo_r = max(1, hi_r - kWin + 1);
        const int rows = hi_r - lo_r + 1;
        const int nblk = (rows + 7) >> 3;
        if (tid < 2 * rows) reinterpret_cast<uint4 *>(win)[tid] = piece;
        __syncthreads();
        fetch(hi_r - kWin);
        for (int w = tid; w < nblk * kBeam; w += NT) {
            const int g = w >> 5;
            int e = w & 31;
            const int top_r = hi_r - 8 * g, bot_r = max(lo_r, top_r - 7);
            for (int r = top_r; r >= bot_r; --r) e = win[(r - lo_r) * kBeam + e] & 31;
            bexit[w] = (unsigned char)e;
        }
        __syncthreads();
        if (tid == 0) {
            for (int g = 0; g < nblk; ++g) {
                bentry[g] = at;
                at = bexit[g * kBeam + at];
            }
        }
        __syncthreads();
        for (int g = tid; g < nblk; g += NT) {
            int e = bentry[g];
            const int top_r = hi_r - 8 * g, bot_r = max(lo_r, top_r - 7);
            for (int r = top_r; r >= bot_r; --r) {
                const unsigned char b = win[(r - lo_r) * kBeam + e];
                path[r] = b;
                e = b & 31;
            }
        }
        __syncthreads();
    }
    if (tid == 0) {
        const int st0 = sm.init_kmers[at];
#pragma unroll
        for (int i = 0; i < SL; ++i) ext[i] = (unsigned char)((st0 >> (2 * (SL - 1 - i))) & 3);
    }
    __syncthreads();

    // running count of true steps along the path, and the stepped bases in order
    const int seg = (T + NT - 1) / NT;
    const int r_lo = 1 + tid * seg, r_hi = min(T, r_lo + seg - 1);
    int local = 0;
    for (int r = r_lo; r <= r_hi; ++r) local += !((path[r] >> 5) & 1);
    int run = local;
#pragma unroll
    for (int d = 1; d < 32; d *= 2) {
        const int below = __shfl_up_sync(0xffffffffu, run, d);
        run += (tid & 31) >= d ? below : 0;
    }
    if ((tid & 31) == 31) sm.part[tid >> 5] = run;
    __syncthreads();
    run -= local;
    for (int w = 0; w < tid >> 5; ++w) run += sm.part[w];
    for (int r = r_lo; r <= r_hi; ++r) {
        const unsigned char b = path[r];
        if (!((b >> 5) & 1)) {
            ext[SL + run] = b >> 6;
            ++run;
        }
        cnt[r] = (unsigned short)run;
    }
    if (tid == 0) cnt[0] = 0;
    __syncthreads();

    // per-timestep quality (src/beam_search.c:441-496)
    const size_t ct = (size_t)chunk * T;
    for (int t = tid; t < T; t += NT) {
        const int r = t + 1;
        const int c = cnt[r];
        int st = 0;
#pragma unroll
        for (int i = 0; i < SL; ++i) st = (st << 2) | ext[c + i];
        const int base = st & 3;
        const float *pr = post_chunk + (size_t)r * NS;
        int nb[8];
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            nb[2 * b] = (st >> 2) + MSB * b;
            nb[2 * b + 1] = ((st << 2) & (NS - 1)) + b;
        }
        // all nine posteriors are fetched before any is used, the four that lie together at once: one memory
        // round trip of six requests
        float prob = __ldcg(pr + st);
        const float4 next = __ldcg(reinterpret_cast<const float4 *>(pr + nb[1]));
        const float pv[8] = {__ldcg(pr + nb[0]), next.x, __ldcg(pr + nb[2]), next.y,
                             __ldcg(pr + nb[4]), next.z, __ldcg(pr + nb[6]), next.w};
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            bool fresh = nb[k] != st;
#pragma unroll
            for (int m = 0; m < k; ++m) fresh = fresh && (nb[m] != nb[k]);
            prob = fresh ? __fadd_rn(prob, pv[k]) : prob;
        }
        prob = prob > 1.0f ? 1.0f : (prob < 0.0f ? 0.0f : prob);
        prob = powf(prob, 0.4f);
        const float other = __fdiv_rn(__fsub_rn(1.0f, prob), 3.0f);
        qp[t] = prob;
        *reinterpret_cast<float4 *>(a.qual + (ct + t) * 4) =
            make_float4(base == 0 ? prob : other, base == 1 ? prob : other,
                        base == 2 ? prob : other, base == 3 ? prob : other);
        a.states[ct + t] = base;
        a.moves[ct + t] = (uint8_t)((t == 0) ? 1 : !((path[r] >> 5) & 1));
    }
    __syncthreads();

    // bases and quality string (src/beam_search.c:49-99).  Position of timestep t =
    // (number of moves up to and including t) - 1; move 0 is forced.
    const int forced = (T > 0 && ((path[1] >> 5) & 1)) ? 1 : 0;
    const int seq_len = T > 0 ? cnt[T] + forced : 0;
    for (int t = tid; t < T; t += NT) {
        const bool starts = (t == 0) || !((path[t + 1] >> 5) & 1);
        if (!starts) continue;
        const int pos = cnt[t + 1] + forced - 1;
        const int b_emit = path[t + 1] >> 6;
        float bsum = 0.f, tsum = 0.f;
        for (int u = t; u < T; ++u) {
            if (u > t && !((path[u + 1] >> 5) & 1)) break;
            const int b = path[u + 1] >> 6;
            const float pq = qp[u];
            const float other = __fdiv_rn(__fsub_rn(1.0f, pq), 3.0f);
            bsum = __fadd_rn(bsum, pq);
#pragma unroll
            for (int k = 0; k < 4; ++k) tsum = __fadd_rn(tsum, k == b ? pq : other);
        }
        float v = __fsub_rn(1.0f, __fdiv_rn(bsum, tsum));
        v = __fmul_rn(-10.0f, log10f(v));
        float qs = __fadd_rn(__fmul_rn(v, a.q_scale), a.q_shift);
        if (qs > 50.0f) qs = 50.0f;
        if (qs < 1.0f) qs = 1.0f;
        a.base_probs[ct + pos] = v;
        a.total_probs[ct + pos] = tsum;
        a.sequence[ct + pos] = "ACGT"[b_emit];
        a.qstring[ct + pos] = (char)(33.5f + qs);
    }
    for (int i = seq_len + tid; i < T; i += NT) {
        a.sequence[ct + i] = 0;
        a.qstring[ct + i] = 0;
        a.base_probs[ct + i] = 0.f;
        a.total_probs[ct + i] = 0.f;
    }

    // The results' way to the host, while other blocks are still at work (a copy after the kernel took
    // 65 us for 512 chunks, 400 for 4096, 18 for one).
    if (a.host_status != nullptr) {
        __syncthreads();
        constexpr int part = NT / 4;
        const unsigned char *rows[3] = {a.moves, reinterpret_cast<const unsigned char *>(a.sequence),
                                        reinterpret_cast<const unsigned char *>(a.qstring)};
#pragma unroll
        for (int k = 0; k < 3; ++k)
            if (tid / part == k) row_to_host(a.host_results[k] + ct, rows[k] + ct, T, tid % part, part);
        // (every kernel that waits for anything has ended)
        if (chunk == 0 && tid == 0) *a.host_status = *a.status;
    }
}

constexpr size_t kMostBytes = 227 * 1024;  // of dynamic shared memory: what a block can have

template <int NS, int NT>
struct Seq {
    static constexpr auto kern = posterior_seq_kernel<NS, NT>;
    static constexpr size_t bytes = kMostBytes;
    static size_t bytes_for(int T) {
        constexpr size_t win = NT / 2;
        const size_t Tp = (T + 16) & ~15;
        return sizeof(PostSmem<NS, NT>) + win * kBeam + (win / 8) * (kBeam + 4) + 8 * Tp + 64;
    }
    static cudaError_t launch(const OfDecodeArgs &a, cudaStream_t stream) {
        const size_t need = bytes_for(a.T);
        if (need > kMostBytes) return cudaErrorInvalidValue;
        kern<<<a.N, NT, need, stream>>>(a);
        return cudaGetLastError();
    }
};

// 1024 threads shorten a chunk's chain of phases, 512 keep more chunks' gathers under way: many rounds of blocks
// want the latter.  ms with 1024 / 512 threads: 256 states, T = 1666, 16 chunks 0.032 / 0.038, 296 0.098 / 0.102, 512
// 0.131 / 0.139; T = 800, 600 chunks 0.091 / 0.085, 2072 0.236 / 0.211, 4096 0.427 / 0.382; 64 states, T = 800, 1036
// chunks 0.090 / 0.088, 2072 0.152 / 0.145, 8000 0.500 / 0.467; 1024 states, T = 400, 600 chunks 0.062 / 0.057, 2072
// 0.149 / 0.141, 4096 0.267 / 0.253.  From 4 chunks to the SM on 512 are the better, by at most 0.5 % of a
// decode (25 us of 5.06 ms at 14), and the line lies at 14.
template <int NS>
cudaError_t launch_seq(const OfDecodeArgs &a, int sms, cudaStream_t stream) {
    return a.N > 14 * sms ? Seq<NS, 512>::launch(a, stream) : Seq<NS, 1024>::launch(a, stream);
}

}  // namespace

cudaError_t of_launch_posterior_seq(const OfDecodeArgs &a, int sms, cudaStream_t stream) {
    switch (a.state_len) {
        case 3: return launch_seq<64>(a, sms, stream);
        case 4: return launch_seq<256>(a, sms, stream);
        case 5: return launch_seq<1024>(a, sms, stream);
        default: return cudaErrorInvalidValue;
    }
}

cudaError_t of_load_posterior_seq(int kernel) {
    switch (kernel) {
        case kSeq64: return of_load<Seq<64, 1024>>();
        case kSeq64Many: return of_load<Seq<64, 512>>();
        case kSeq256: return of_load<Seq<256, 1024>>();
        case kSeq256Many: return of_load<Seq<256, 512>>();
        case kSeq1024: return of_load<Seq<1024, 1024>>();
        case kSeq1024Many: return of_load<Seq<1024, 512>>();
        default: return cudaSuccess;
    }
}
