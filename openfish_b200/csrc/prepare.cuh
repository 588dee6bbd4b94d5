// prepare.cuh -- loading kernels.
#pragma once
#include <cuda_runtime.h>

// The decode's kernels, in the order in which they are loaded.
enum OfKernel : int {
    kFwd256, kBeam256, kFwd256Many, kFwd256Most, kSeq256, kBwd256Many, kBwd256Most, kAhead256,
    kPosterior256, kBeam256Scaled,
    kScan1024, kFwd1024, kFwd1024Many, kBeam1024, kSeq1024, kPosterior1024, kBeam1024Scaled, kScan1024Many,
    kAhead64, kFwd64, kWarpBwd64, kWarpFwd64, kBeam64, kPosterior64, kSeq64, kBeam64Scaled,
    kSeq256Many, kSeq1024Many, kSeq64Many,
    kBeamFew256, kBeamFew64, kBeamFew1024, kBeamFew256Scaled, kBeamFew64Scaled, kBeamFew1024Scaled, kAhead256Mid, kAhead256Five, kAhead64Mid,
    kKernels
};

// Loads a kernel (a type with `kern` and the dynamic shared memory `bytes` it may be launched with) on the
// current device.
template <class K>
cudaError_t of_load() {
    return cudaFuncSetAttribute(K::kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)K::bytes);
}

// Each loads the kernel if it is one of its file's, and else does nothing.
cudaError_t of_load_scan(int kernel);           // scan.cu
cudaError_t of_load_ahead(int kernel);          // scan_ahead.cu
cudaError_t of_load_warp(int kernel);           // scan_warp.cu
cudaError_t of_load_beam_search(int kernel);    // beam_search.cu
cudaError_t of_load_posterior_seq(int kernel);  // posterior_seq.cu

// All of them on the current device (decode_b200.cu); before the first launch in its present context.
cudaError_t of_prepare_device();
