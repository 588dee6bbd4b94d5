// scan.cuh -- launchers of the scan kernels and of two small ones beside them.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
namespace ofx { struct Tables; }

// scores_fp16: [T][N][4*ns] fp16, 16-byte aligned; bwd, fwd: [N][T+1][ns] fp32 out; tables: device copy
// of ofx::Tables; status: device int raised when a wait for an asynchronous copy runs out, which it
// does after wait_ns nanoseconds.

// sms: the GPU's multiprocessors.

// How the scans of a batch are best run.
enum class OfScanPlan {
    kTogether,           // both in one launch, the posterior by a kernel of its own
    kAheadThenForward,   // the backward one by of_launch_ahead (with few timesteps, of five chunks to the multiprocessor, by
                         // scan.cu's kernel), the forward one afterwards, beside the beam search, by either file's
    kBackwardThenForward,// both by scan.cu's kernels
    kWarps               // the 64-state model: the forward one by scan_warp.cu's kernel, a warp to a chunk; the backward one by
                         // of_launch_ahead, and in batches of more than eight chunks to the multiprocessor by a warp to a chunk
};
OfScanPlan of_scan_plan(int N, int state_len, int sms);

// One or both scans (bwd or fwd null: not that direction) by the kernel for batches that fill the GPU: 64 states
// forwards only, 256 states backwards only.  (scan.cu)
cudaError_t of_launch_scans(const void *scores_fp16, float *bwd, float *fwd, int T, int N, int state_len, int sms,
                            float stay, const ofx::Tables *tables, int *status, uint64_t wait_ns, cudaStream_t stream);

// Forward scan and posterior in one kernel, for the 256- and the 1024-state model: reads the finished
// backward scores, writes post = softmax_s(fwd + bwd) [N][T+1][ns]; the forward scores never leave the chip.
cudaError_t of_launch_forward_posterior(const void *scores_fp16, const float *bwd, float *post, int T, int N,
                                        int state_len, int sms, float stay, const ofx::Tables *tables, int *status,
                                        uint64_t wait_ns, cudaStream_t stream);

// One or both scans by the kernel that runs ahead of its checks, for the 64- and the 256-state model.  (scan_ahead.cu)
cudaError_t of_launch_ahead(const void *scores_fp16, float *bwd, float *fwd, int T, int N, int state_len, int sms, float stay,
                            const ofx::Tables *tables, int *status, uint64_t wait_ns, cudaStream_t stream);

// Backward scan, and forward scan with the posterior, of the 64-state model by one warp a chunk.  (scan_warp.cu)
cudaError_t of_launch_warp_backward(const void *scores_fp16, float *bwd, int T, int N, float stay, const ofx::Tables *tables,
                                    int *status, uint64_t wait_ns, cudaStream_t stream);
cudaError_t of_launch_warp_forward_posterior(const void *scores_fp16, const float *bwd, float *post, int T, int N, float stay,
                                             const ofx::Tables *tables, int *status, uint64_t wait_ns, cudaStream_t stream);

// post holds the forward rows and gets softmax_s(fwd + bwd) in their place.  (scan_ahead.cu)
cudaError_t of_launch_posterior(const float *bwd, float *post, int T, int N, int state_len, cudaStream_t stream);

// The scans of a batch up to the backward scores (and, as the plan has it, forward scores in `post`), and what
// is left to make of `post` the posterior, which may run beside the beam search.
cudaError_t of_launch_first_scans(OfScanPlan plan, const void *scores_fp16, float *bwd, float *post, int T, int N,
                                  int state_len, int sms, float stay, const ofx::Tables *tables, int *status,
                                  uint64_t wait_ns, cudaStream_t stream);
cudaError_t of_launch_rest_of_posterior(OfScanPlan plan, const void *scores_fp16, const float *bwd, float *post, int T,
                                        int N, int state_len, int sms, float stay, const ofx::Tables *tables, int *status,
                                        uint64_t wait_ns, cudaStream_t stream);

// Scores with every state's stay score in front of its four transition scores, [rows][5*ns] fp16,
// to the [rows][4*ns] layout the decode reads (adaptor.cu); clamp > 0 also bounds the values.
cudaError_t of_launch_strip_blank(const void *in, void *out, long long rows, int state_len, float clamp, int sms,
                                  cudaStream_t stream);

// One block, one bounded wait of wait_ns nanoseconds on a barrier that nothing completes (no copy is
// issued at all); the wait runs out, *status becomes ofd::kStatusWaitTimeout and the kernel returns.
// Exists so that the path from a kernel's timeout to the host's error can be exercised without anything
// being wrong.  (selfcheck.cu)
cudaError_t of_launch_wait_that_runs_out(int *status, uint64_t wait_ns, cudaStream_t stream);
