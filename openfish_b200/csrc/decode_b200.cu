// decode_b200.cu -- device buffers, stream and launch orchestration of the decode path.
//
// Replaces gpubuf_init_cuda / gpubuf_free_cuda / decode_cuda (src/decode_cuda.cu:11-212).
// Differences in design: the caller-visible openfish_gpubuf_t sits at the start of a private
// record that also owns two streams, events, the arithmetic tables and a page-locked staging
// area; one decode is four or five kernel launches -- the scans that the beam search waits for; beam
// search with the rest of the way to the posterior beside it on the second stream; traceback +
// sequence, which also writes the results to the host -- all stream ordered, with a single host
// wait at the end (the reference launches five kernels and three memsets with a device-wide
// synchronisation after each and copies with three blocking pageable transfers).
#include <cuda.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdarg.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include <atomic>
#include <mutex>

#include "backend.h"
#include "scan.cuh"
#include "exact_math.cuh"
#include "beam_post.cuh"
#include "cpu_relax.h"
#include "host_view.h"
#include "of_device.cuh"
#include "prepare.cuh"
#include "openfish_b200.h"
#include "rotary.cuh"

namespace {

constexpr uint32_t kMagic = 0x0F15B200u;

struct GpuBuf {
    openfish_gpubuf_t pub;  // must stay first: the public pointer is the record's address
    uint32_t magic;
    int T, N, state_len, device;
    cudaStream_t stream;   // the main one; blocking, see ofb_gpubuf_create
    cudaStream_t stream2;  // what runs beside the beam search, ordered against `stream` by events only
    // 0 start, 1 first scans done, 2 beam search done, 3 all done, 4 and 5 start and end of what runs beside the
    // beam search, 6 blank-column strip start; two sets, so that the times of the last decode can be
    // worked out when somebody asks for them, whether or not another is in flight
    cudaEvent_t ev[2][7];
    cudaEvent_t caller_ev;  // the caller's stream at submit time
    int set;                // of the decode in flight, or else of the last one
    int done_set;           // of the last completed decode, -1 before the first
    uint64_t wait_ns;      // how long a kernel waits for an asynchronous copy before it raises d_status
    int *d_init_kmers;     // inside the beam_vector allocation, behind the back-pointers
    ofx::Tables *d_tables;
    int *d_status;
    void *d_scores4;           // 4-wide copy of 5-wide scores, made on the first 5-wide decode (null before)
    int sms;
    unsigned char *d_small;    // the allocation of all device buffers but the two large tensors
    unsigned char *h_stage;    // page-locked, three results of N*T bytes, each on a 16-byte boundary, and a status word
    unsigned char *d_stage;    // the same for the device
    int *h_status;
    // decode in flight
    bool pending;
    uint8_t *dst_moves;
    char *dst_sequence, *dst_qstring;
    bool via_stage;
    bool stripped[2];  // the decode of this set of events began with the blank-column strip
};

thread_local char g_err[512] = "";

int fail(int code, const char *fmt, ...) {
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(g_err, sizeof(g_err), fmt, ap);
    va_end(ap);
    return code;
}

#define CU(call)                                                                              \
    do {                                                                                      \
        cudaError_t e_ = (call);                                                              \
        if (e_ != cudaSuccess)                                                                \
            return fail(e_ == cudaErrorMemoryAllocation ? OPENFISH_B200_ERR_ALLOC             \
                                                        : OPENFISH_B200_ERR_CUDA,             \
                        "%s failed: %s", #call, cudaGetErrorString(e_));                      \
    } while (0)

// Bytes from one result to the next, in the staging area and on the device.
size_t stage_pitch(const GpuBuf *g) { return ((size_t)g->N * g->T + 15) & ~(size_t)15; }

GpuBuf *priv(const openfish_gpubuf_t *g) {
    return reinterpret_cast<GpuBuf *>(const_cast<openfish_gpubuf_t *>(g));
}

// Where the device can write all `bytes` bytes of a host buffer; null if it cannot.  (The runtime knows
// nothing of a registration's extent, so the driver is asked: 0.06 us, as much as the runtime's answer takes.)
unsigned char *device_view(void *p, size_t bytes) {
    typedef CUresult (*Attribute)(void *, CUpointer_attribute, CUdeviceptr);
    static const Attribute attribute = [] {
        void *f = nullptr;
        cudaDriverEntryPointQueryResult found;
        if (cudaGetDriverEntryPoint("cuPointerGetAttribute", &f, cudaEnableDefault, &found) != cudaSuccess) {
            cudaGetLastError();
            f = nullptr;
        }
        return reinterpret_cast<Attribute>(f);
    }();
    if (!attribute) return nullptr;
    cudaPointerAttributes at;
    if (cudaPointerGetAttributes(&at, p) != cudaSuccess) {
        cudaGetLastError();
        return nullptr;
    }
    HostRange r = {at.type == cudaMemoryTypeHost, reinterpret_cast<uintptr_t>(at.devicePointer), 0, 0};
    if (!r.page_locked) return nullptr;
    CUdeviceptr start = 0;
    if (attribute(&start, CU_POINTER_ATTRIBUTE_RANGE_START_ADDR, (CUdeviceptr)r.device) != CUDA_SUCCESS ||
        attribute(&r.size, CU_POINTER_ATTRIBUTE_RANGE_SIZE, (CUdeviceptr)r.device) != CUDA_SUCCESS)
        return nullptr;
    r.start = start;
    return writable_by_device(r, bytes);
}

int destroy(GpuBuf *g) {
    if (!g) return OPENFISH_B200_OK;
    if (g->pending && g->stream) cudaStreamSynchronize(g->stream);
    if (g->pending && g->stream2) cudaStreamSynchronize(g->stream2);
    cudaFree(g->pub.bwd_NTC);
    cudaFree(g->pub.post_NTC);
    cudaFree(g->d_small);
    cudaFree(g->d_scores4);
    if (g->h_stage) cudaFreeHost(g->h_stage);
    for (int i = 0; i < 14; ++i)
        if (g->ev[i / 7][i % 7]) cudaEventDestroy(g->ev[i / 7][i % 7]);
    if (g->caller_ev) cudaEventDestroy(g->caller_ev);
    if (g->stream2) cudaStreamDestroy(g->stream2);
    if (g->stream) cudaStreamDestroy(g->stream);
    g->magic = 0;
    free(g);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return fail(OPENFISH_B200_ERR_CUDA, "releasing device buffers failed: %s", cudaGetErrorString(e));
    return OPENFISH_B200_OK;
}

}  // namespace

// The kernels are loaded here, all at once and always in the same order, instead of each at its first
// launch: kernels that run beside one another get in each other's way in the instruction caches according
// to where their code has come to lie.  A 512-chunk decode of the 256-state model took 2.96 ms in a process
// that began with one and 3.10 in one that had decoded 74 chunks before.
// What is loaded and how much shared memory a kernel may have belongs to the current context and ends with it
// (cudaDeviceReset), so nothing is remembered here: every set of device buffers asks again (2 us).
cudaError_t of_prepare_device() {
    static std::mutex lock;
    std::lock_guard<std::mutex> hold(lock);
    cudaError_t e = cudaSuccess;
    for (int k = 0; k < kKernels && e == cudaSuccess; ++k) {
        e = of_load_scan(k);
        if (e == cudaSuccess) e = of_load_ahead(k);
        if (e == cudaSuccess) e = of_load_warp(k);
        if (e == cudaSuccess) e = of_load_beam_search(k);
        if (e == cudaSuccess) e = of_load_posterior_seq(k);
    }
    return e;
}

extern "C" const char *ofb_error_text(void) { return g_err; }

extern "C" int ofb_gpubuf_create(int T, int N, int state_len, openfish_gpubuf_t **out) {
    *out = nullptr;
    GpuBuf *g = static_cast<GpuBuf *>(calloc(1, sizeof(GpuBuf)));
    if (!g) return fail(OPENFISH_B200_ERR_ALLOC, "out of host memory");
    g->T = T; g->N = N; g->state_len = state_len;
    const size_t ns = (size_t)1 << (2 * state_len);
    const size_t nt = (size_t)N * T;
    const size_t tens = (size_t)N * (T + 1) * ns * sizeof(float);
    int rc = [&]() -> int {
        CU(cudaGetDevice(&g->device));
        CU(of_prepare_device());
        CU(cudaDeviceGetAttribute(&g->sms, cudaDevAttrMultiProcessorCount, g->device));
        // a blocking stream: ordered after work the caller queued on the legacy default
        // stream (where the reference runs), so freshly written scores are seen
        CU(cudaStreamCreateWithFlags(&g->stream, cudaStreamDefault));
        CU(cudaStreamCreateWithFlags(&g->stream2, cudaStreamNonBlocking));
        for (int i = 0; i < 14; ++i) CU(cudaEventCreate(&g->ev[i / 7][i % 7]));
        CU(cudaEventCreateWithFlags(&g->caller_ev, cudaEventDisableTiming));
        g->done_set = -1;
        g->wait_ns = ofd::kDefaultWaitLimitNs;
        // same ten buffers and sizes as the reference (src/decode_cuda.cu:22-45)
        CU(cudaMalloc(&g->pub.bwd_NTC, tens));
        CU(cudaMalloc(&g->pub.post_NTC, tens));
        // (everything but the two large tensors in one allocation)
        size_t bytes = 0;
        auto piece = [&](size_t n) {
            const size_t at = bytes;
            bytes += (n + 255) & ~(size_t)255;
            return at;
        };
        const size_t o_results = piece(3 * stage_pitch(g));
        // reference-sized (8 bytes per beam slot and timestep); this library uses 1 byte of the 8
        // for its packed back-pointers and 128 bytes per chunk behind them for the initial k-mers
        const size_t o_beam = piece((size_t)8 * N * 32 * (T + 1));
        const size_t o_states = piece(sizeof(int32_t) * nt), o_qual = piece(sizeof(float) * nt * 4);
        const size_t o_base = piece(sizeof(float) * nt), o_total = piece(sizeof(float) * nt);
        const size_t o_tables = piece(sizeof(ofx::Tables)), o_status = piece(sizeof(int));
        CU(cudaMalloc(&g->d_small, bytes));
        unsigned char *const d = g->d_small;
        g->pub.moves = d + o_results;
        g->pub.sequence = reinterpret_cast<char *>(d + o_results + stage_pitch(g));
        g->pub.qstring = reinterpret_cast<char *>(d + o_results + 2 * stage_pitch(g));
        g->pub.beam_vector = d + o_beam;
        g->d_init_kmers = reinterpret_cast<int *>(d + o_beam + (((size_t)N * 32 * (T + 1) + 255) & ~(size_t)255));
        g->pub.states = d + o_states;
        g->pub.qual_data = reinterpret_cast<float *>(d + o_qual);
        g->pub.base_probs = reinterpret_cast<float *>(d + o_base);
        g->pub.total_probs = reinterpret_cast<float *>(d + o_total);
        g->d_tables = reinterpret_cast<ofx::Tables *>(d + o_tables);
        g->d_status = reinterpret_cast<int *>(d + o_status);
        CU(cudaHostAlloc(&g->h_stage, 3 * stage_pitch(g) + 16, cudaHostAllocMapped));
        CU(cudaHostGetDevicePointer(&g->d_stage, g->h_stage, 0));
        g->h_status = reinterpret_cast<int *>(g->h_stage + 3 * stage_pitch(g));
        *g->h_status = ofd::kStatusOk;
        static const ofx::Tables host_tables = [] {
            ofx::Tables t;
            ofx::fill_tables(&t);
            return t;
        }();
        CU(cudaMemcpy(g->d_tables, &host_tables, sizeof(host_tables), cudaMemcpyHostToDevice));
        CU(cudaMemset(g->d_status, 0, sizeof(int)));
        return OPENFISH_B200_OK;
    }();
    if (rc != OPENFISH_B200_OK) {
        char keep[sizeof(g_err)];
        memcpy(keep, g_err, sizeof(keep));
        destroy(g);
        memcpy(g_err, keep, sizeof(keep));
        return rc;
    }
    g->magic = kMagic;
    *out = &g->pub;
    return OPENFISH_B200_OK;
}

extern "C" int ofb_gpubuf_destroy(openfish_gpubuf_t *gpubuf) {
    if (!gpubuf) return OPENFISH_B200_OK;
    GpuBuf *g = priv(gpubuf);
    if (g->magic != kMagic) return fail(OPENFISH_B200_ERR_ARGUMENT, "gpubuf was not created by openfish_gpubuf_init");
    return destroy(g);
}

extern "C" int ofb_gpubuf_check_owner(const openfish_gpubuf_t *gpubuf) {
    if (!gpubuf) return fail(OPENFISH_B200_ERR_ARGUMENT, "gpubuf is NULL");
    if (priv(gpubuf)->magic != kMagic) return fail(OPENFISH_B200_ERR_ARGUMENT, "gpubuf was not created by openfish_gpubuf_init");
    return OPENFISH_B200_OK;
}

extern "C" int ofb_gpubuf_check(const openfish_gpubuf_t *gpubuf, int T, int N, int state_len) {
    if (!gpubuf) return fail(OPENFISH_B200_ERR_ARGUMENT, "gpubuf is NULL");
    const GpuBuf *g = priv(gpubuf);
    if (g->magic != kMagic) return fail(OPENFISH_B200_ERR_ARGUMENT, "gpubuf was not created by openfish_gpubuf_init");
    if (g->T != T || g->N != N || g->state_len != state_len)
        return fail(OPENFISH_B200_ERR_SHAPE, "gpubuf was sized for T=%d N=%d state_len=%d, decode asked for T=%d N=%d state_len=%d",
                    g->T, g->N, g->state_len, T, N, state_len);
    return OPENFISH_B200_OK;
}

extern "C" int ofb_decode_submit(int T, int N, int C, const void *scores, int state_len,
                                 const ofb_decode_params_t *params, const openfish_gpubuf_t *gpubuf,
                                 uint8_t *moves, char *sequence, char *qstring) {
    GpuBuf *g = priv(gpubuf);
    const float beam_cut = params->beam_cut, blank_score = params->blank_score;
    const float q_shift = params->q_shift, q_scale = params->q_scale;
    if (g->pending) return fail(OPENFISH_B200_ERR_ARGUMENT, "a decode is already in flight on this gpubuf");
    int dev = -1;
    CU(cudaGetDevice(&dev));
    if (dev != g->device) return fail(OPENFISH_B200_ERR_ARGUMENT, "gpubuf belongs to device %d, current device is %d", g->device, dev);

    OfDecodeArgs a;
    // the last kernel writes the results to the host itself: into the caller's buffers if all of them are
    // page-locked from end to end, else into the staging area
    void *const dst[3] = {moves, sequence, qstring};
    g->via_stage = false;
    for (int i = 0; i < 3; ++i) {
        a.host_results[i] = device_view(dst[i], (size_t)N * T);
        if (!a.host_results[i]) g->via_stage = true;
    }
    if (g->via_stage)
        for (int i = 0; i < 3; ++i) a.host_results[i] = g->d_stage + i * stage_pitch(g);
    a.host_status = reinterpret_cast<int *>(g->d_stage + 3 * stage_pitch(g));
    a.scores = static_cast<const __half *>(scores);
    a.bwd = g->pub.bwd_NTC;
    a.post = g->pub.post_NTC;
    a.bp = static_cast<unsigned char *>(g->pub.beam_vector);
    a.init_kmers = g->d_init_kmers;
    a.moves = g->pub.moves;
    a.sequence = g->pub.sequence;
    a.qstring = g->pub.qstring;
    a.states = static_cast<int *>(g->pub.states);
    a.qual = g->pub.qual_data;
    a.base_probs = g->pub.base_probs;
    a.total_probs = g->pub.total_probs;
    a.tables = g->d_tables;
    a.status = g->d_status;
    a.wait_ns = g->wait_ns;
    a.T = T; a.N = N; a.C = C; a.state_len = state_len;
    a.stay = blank_score;
    a.log_beam_cut = beam_cut > 0.0f ? logf(beam_cut) : 3.402823466e+38f;  // src/beam_search.c:135
    a.q_shift = q_shift;
    a.q_scale = q_scale;
    a.score_scale = params->score_scale;

    // stream:  scans as far as the beam search needs them -> beam search -----> sequence
    // stream2:                    the rest of the way to the posterior (beside it) --^
    // Ordering against the producer of the scores: the gpubuf's main stream is a blocking one, so it
    // runs after whatever the caller queued on the legacy default stream (the reference's stream);
    // a caller that works on a stream of its own names it, and the decode waits for that stream's
    // work as of now.
    if (params->on_caller_stream) {
        cudaStream_t caller = static_cast<cudaStream_t>(params->caller_stream);
        CU(cudaEventRecord(g->caller_ev, caller));
        CU(cudaStreamWaitEvent(g->stream, g->caller_ev, 0));
    }
    // (one decode is in flight at a time: the other set is free)
    cudaEvent_t *const ev = g->ev[g->set = g->done_set == 0 ? 1 : 0];
    CU(cudaEventRecord(ev[0], g->stream));
    const OfScanPlan plan = of_scan_plan(N, state_len, g->sms);
    CU(of_launch_first_scans(plan, scores, g->pub.bwd_NTC, g->pub.post_NTC, T, N, state_len, g->sms, blank_score,
                             g->d_tables, g->d_status, g->wait_ns, g->stream));
    CU(cudaEventRecord(ev[1], g->stream));
    CU(cudaStreamWaitEvent(g->stream2, ev[1], 0));
    CU(cudaEventRecord(ev[4], g->stream2));
    CU(of_launch_rest_of_posterior(plan, scores, g->pub.bwd_NTC, g->pub.post_NTC, T, N, state_len, g->sms, blank_score,
                                   g->d_tables, g->d_status, g->wait_ns, g->stream2));
    CU(cudaEventRecord(ev[5], g->stream2));
    CU(of_launch_beam_search(a, g->sms, g->stream));
    CU(cudaEventRecord(ev[2], g->stream));
    CU(cudaStreamWaitEvent(g->stream, ev[5], 0));
    CU(of_launch_posterior_seq(a, g->sms, g->stream));
    CU(cudaEventRecord(ev[3], g->stream));
    g->dst_moves = moves;
    g->dst_sequence = sequence;
    g->dst_qstring = qstring;
    g->stripped[g->set] = false;
    g->pending = true;
    return OPENFISH_B200_OK;
}

namespace {
// Waits for the gpubuf's main stream, then looks at the status word its kernels share (brought to
// the host by the last operation queued): a raised status is reported and cleared on the device.
int stream_done_and_status(GpuBuf *g) {
    CU(cudaStreamSynchronize(g->stream));
    if (*g->h_status != ofd::kStatusOk) {
        const int st = *g->h_status;
        *g->h_status = ofd::kStatusOk;
        CU(cudaMemsetAsync(g->d_status, 0, sizeof(int), g->stream));
        return fail(OPENFISH_B200_ERR_DEVICE_WAIT, "a kernel raised device status %d (an asynchronous copy did not complete in time)", st);
    }
    return OPENFISH_B200_OK;
}
}  // namespace

extern "C" int ofb_decode_submit_5wide(int T, int N, const void *scores5, int state_len, float clamp,
                                       const ofb_decode_params_t *params, const openfish_gpubuf_t *gpubuf,
                                       uint8_t *moves, char *sequence, char *qstring) {
    GpuBuf *g = priv(gpubuf);
    if (g->pending) return fail(OPENFISH_B200_ERR_ARGUMENT, "a decode is already in flight on this gpubuf");
    int dev = -1;
    CU(cudaGetDevice(&dev));
    if (dev != g->device) return fail(OPENFISH_B200_ERR_ARGUMENT, "gpubuf belongs to device %d, current device is %d", g->device, dev);
    const size_t ns = (size_t)1 << (2 * state_len);
    if (!g->d_scores4) CU(cudaMalloc(&g->d_scores4, (size_t)T * N * 4 * ns * sizeof(__half)));
    if (params->on_caller_stream) {
        cudaStream_t caller = static_cast<cudaStream_t>(params->caller_stream);
        CU(cudaEventRecord(g->caller_ev, caller));
        CU(cudaStreamWaitEvent(g->stream, g->caller_ev, 0));
    }
    const int set = g->done_set == 0 ? 1 : 0;  // (what the submit below takes)
    CU(cudaEventRecord(g->ev[set][6], g->stream));
    CU(of_launch_strip_blank(scores5, g->d_scores4, (long long)T * N, state_len, clamp, g->sms, g->stream));
    ofb_decode_params_t p = *params;
    p.on_caller_stream = 0;  // (already ordered: the copy above runs on the gpubuf's stream)
    const int rc = ofb_decode_submit(T, N, (int)(4 * ns), g->d_scores4, state_len, &p, gpubuf, moves, sequence, qstring);
    g->stripped[set] = true;
    return rc;
}

extern "C" int ofb_decode_wait(const openfish_gpubuf_t *gpubuf) {
    GpuBuf *g = priv(gpubuf);
    if (!g->pending) return OPENFISH_B200_OK;
    g->pending = false;
    const int rc = stream_done_and_status(g);
    if (rc != OPENFISH_B200_OK) return rc;
    if (g->via_stage) {
        const size_t nt = (size_t)g->N * g->T;
        memcpy(g->dst_moves, g->h_stage, nt);
        memcpy(g->dst_sequence, g->h_stage + stage_pitch(g), nt);
        memcpy(g->dst_qstring, g->h_stage + 2 * stage_pitch(g), nt);
    }
    g->done_set = g->set;
    return OPENFISH_B200_OK;
}

extern "C" int ofb_stream_wait_decode(void *stream, const openfish_gpubuf_t *gpubuf) {
    GpuBuf *g = priv(gpubuf);
    if (!g->pending) return OPENFISH_B200_OK;  // nothing in flight: nothing to wait for
    CU(cudaStreamWaitEvent(static_cast<cudaStream_t>(stream), g->ev[g->set][3], 0));
    return OPENFISH_B200_OK;
}

extern "C" int ofb_selfcheck_wait(const openfish_gpubuf_t *gpubuf, unsigned limit_us) {
    GpuBuf *g = priv(gpubuf);
    if (g->pending) return fail(OPENFISH_B200_ERR_ARGUMENT, "a decode is in flight on this gpubuf");
    int dev = -1;
    CU(cudaGetDevice(&dev));
    if (dev != g->device) return fail(OPENFISH_B200_ERR_ARGUMENT, "gpubuf belongs to device %d, current device is %d", g->device, dev);
    CU(of_launch_wait_that_runs_out(g->d_status, (uint64_t)limit_us * 1000ull, g->stream));
    CU(cudaMemcpyAsync(g->h_status, g->d_status, sizeof(int), cudaMemcpyDeviceToHost, g->stream));
    return stream_done_and_status(g);
}

// 0 the scans before the beam search, 1 everything after them (beam search with the rest of the posterior
// beside it, then sequence), 2 zero (the last kernel writes the results to the host), 3 all of it; detail:
// 4 beam search, 5 the rest of the posterior, 6 sequence (from the later of its two inputs), 7 the
// blank-column strip in front of a 5-wide decode (0 otherwise)
extern "C" int ofb_last_decode_ms(const openfish_gpubuf_t *gpubuf, float ms[8]) {
    const GpuBuf *g = priv(gpubuf);
    for (int i = 0; i < 8; ++i) ms[i] = 0.f;
    if (g->done_set < 0) return OPENFISH_B200_OK;
    const cudaEvent_t *ev = g->ev[g->done_set];
    float from_beam = 0.f, from_rest = 0.f;
    CU(cudaEventElapsedTime(&ms[0], ev[0], ev[1]));
    CU(cudaEventElapsedTime(&ms[1], ev[1], ev[3]));
    CU(cudaEventElapsedTime(&ms[3], ev[0], ev[3]));
    CU(cudaEventElapsedTime(&ms[4], ev[1], ev[2]));
    CU(cudaEventElapsedTime(&ms[5], ev[4], ev[5]));
    CU(cudaEventElapsedTime(&from_beam, ev[2], ev[3]));
    CU(cudaEventElapsedTime(&from_rest, ev[5], ev[3]));
    ms[6] = from_beam < from_rest ? from_beam : from_rest;
    if (g->stripped[g->done_set]) CU(cudaEventElapsedTime(&ms[7], ev[6], ev[0]));
    return OPENFISH_B200_OK;
}

// Rotary: where a call's kernel reports its end.  A record belongs to one thread at a time; a thread
// that ends leaves its record for the next one that needs one, so there are never more of them than
// there have been threads at work at once.
namespace {
constexpr int kMaxDevices = 64;
struct RotaryRecord {
    RotaryDone *done;  // page-locked, portable: any device may write it
    unsigned calls;
    RotaryRecord *next;
};
std::mutex g_rotary_lock;
RotaryRecord *g_rotary_free = nullptr;
std::atomic<int> g_sms[kMaxDevices];

struct RotaryThread {
    RotaryRecord *mine = nullptr;
    float last_ms = 0.f;
    ~RotaryThread() {
        if (!mine) return;
        std::lock_guard<std::mutex> hold(g_rotary_lock);
        mine->next = g_rotary_free;
        g_rotary_free = mine;
    }
};
thread_local RotaryThread t_rotary;

// Is the record's memory still there?  It goes when the program resets the device on which it was made, and
// other memory may since have come to lie at its address; writing to that, or to none, must not happen.
// (0.05 us)
bool still_there(const RotaryRecord *r) {
    cudaPointerAttributes at;
    if (cudaPointerGetAttributes(&at, r->done) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return at.type == cudaMemoryTypeHost && at.devicePointer == r->done && r->done->owner == r;
}

int rotary_record(RotaryRecord **out) {
    if (!t_rotary.mine) {
        std::lock_guard<std::mutex> hold(g_rotary_lock);
        if (g_rotary_free) {
            t_rotary.mine = g_rotary_free;
            g_rotary_free = g_rotary_free->next;
        } else {
            t_rotary.mine = static_cast<RotaryRecord *>(calloc(1, sizeof(RotaryRecord)));
            if (!t_rotary.mine) return fail(OPENFISH_B200_ERR_ALLOC, "out of host memory");
        }
    }
    RotaryRecord *r = t_rotary.mine;
    if (!r->done || !still_there(r)) {
        r->done = nullptr;  // (what a reset has taken needs no freeing)
        RotaryDone *d = nullptr;
        CU(cudaHostAlloc(&d, sizeof(RotaryDone), cudaHostAllocPortable | cudaHostAllocMapped));
        memset(d, 0, sizeof(*d));
        d->owner = r;
        r->calls = 0;
        r->done = d;
    }
    *out = r;
    return OPENFISH_B200_OK;
}
}  // namespace

extern "C" int ofb_rotary(void *x, const void *sin_t, const void *cos_t, int batch, int seqlen,
                          int nheads, int rotary_half, long long stride_batch,
                          long long stride_seq, long long stride_head) {
    t_rotary.last_ms = 0.f;
    if ((long long)batch * seqlen * nheads * rotary_half <= 0) return OPENFISH_B200_OK;
    int dev = 0;
    CU(cudaGetDevice(&dev));
    if (dev < 0 || dev >= kMaxDevices) return fail(OPENFISH_B200_ERR_ARGUMENT, "device %d out of range", dev);
    int sms = g_sms[dev].load(std::memory_order_relaxed);
    if (!sms) {
        CU(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
        g_sms[dev].store(sms, std::memory_order_relaxed);
    }
    RotaryRecord *r = nullptr;
    const int rc = rotary_record(&r);
    if (rc != OPENFISH_B200_OK) return rc;
    const unsigned call = ++r->calls;
    // the reference launches on the legacy default stream and waits for the device
    // (src/nn_cuda.cu:27-39); same stream here, and a wait for this kernel only
    CU(of_launch_rotary(x, sin_t, cos_t, batch, seqlen, nheads, rotary_half, stride_batch,
                        stride_seq, stride_head, sms, r->done, call, 0));
    // The kernel's own report first (nothing is nearer); work queued before it may keep it for longer, and
    // an error would keep it for good: then the stream is asked.
    volatile unsigned *seen = &r->done->call;
    for (int spin = 0; *seen != call && spin < 20000; ++spin) cpu_relax();
    if (*seen != call) CU(cudaStreamSynchronize(0));
    if (*seen != call) return fail(OPENFISH_B200_ERR_CUDA, "the rotary kernel did not report its end");
    std::atomic_thread_fence(std::memory_order_acquire);
    t_rotary.last_ms = (float)((r->done->end_ns - r->done->start_ns) * 1e-6);
    return OPENFISH_B200_OK;
}

extern "C" float ofb_last_rotary_ms(void) { return t_rotary.last_ms; }

// ---- helpers for a driver program in the style of the reference's (src/decode_cuda.cu:214-240)
extern "C" int ofb_set_device(int device) {
    CU(cudaSetDevice(device));
    return OPENFISH_B200_OK;
}
extern "C" int ofb_device_upload(const void *host, size_t bytes, void **out) {
    void *d = nullptr;
    CU(cudaMalloc(&d, bytes ? bytes : 1));
    cudaError_t e = cudaMemcpy(d, host, bytes, cudaMemcpyHostToDevice);
    if (e != cudaSuccess) {
        cudaFree(d);
        return fail(OPENFISH_B200_ERR_CUDA, "host-to-device copy failed: %s", cudaGetErrorString(e));
    }
    *out = d;
    return OPENFISH_B200_OK;
}
extern "C" int ofb_device_free(void *device) {
    CU(cudaFree(device));
    return OPENFISH_B200_OK;
}
extern "C" int ofb_device_download(void *host, const void *device, size_t bytes) {
    CU(cudaMemcpy(host, device, bytes, cudaMemcpyDeviceToHost));
    return OPENFISH_B200_OK;
}

