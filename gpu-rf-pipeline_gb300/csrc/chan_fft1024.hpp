// The 1024-point inverse transform of the plain channelizer (chan_fft1024.cu): internal interface.
#pragma once

#include <cuda_runtime.h>

namespace rfx {

// z (cf32), or |z| (float) with `magnitude`, of `frames` frames of 1024 branch sums u; out may be u.
cudaError_t chan_fft1024_launch(const void* u, void* out, long long frames, bool magnitude,
                                cudaStream_t stream);

// Longest plan this kernel transforms; longer ones use cuFFT's plan. Measured, sums and transform, 32
// taps per branch (us, this kernel / cuFFT): 44 frames 8.4 / 9.8, 4096 frames 32.5 / 37.1, 16384 frames
// 99.0 / 102.6, 65536 frames 361 / 355. Magnitudes go the way of the complex outputs, whose bits they
// have (65536 frames 469 with cuFFT and a magnitude pass; this kernel, which writes them directly, 329).
constexpr long long kFft1024Frames = 8192;

}  // namespace rfx
