// The fused channelizer (chan_fused.cuh): internal launch interface.
#pragma once

#include <cuda_runtime.h>

namespace rfx {

// Whether the fused kernel takes this shape: 8, 16, ..., 512 channels, at most 32 taps in any
// branch.
inline bool chan_fused_supported(int channels, int num_taps)
{
    return channels >= 8 && channels <= 512 && (channels & (channels - 1)) == 0 &&
           num_taps >= 1 && num_taps <= 32 * channels;
}

#define RFX_CHAN_FUSED(M)                                                                          \
    cudaError_t chan_fused_launch_##M(const void* x, const float* taps, void* out,                 \
                                      long long frames, int num_taps, bool magnitude, int format,  \
                                      cudaStream_t stream);
RFX_CHAN_FUSED(8)
RFX_CHAN_FUSED(16)
RFX_CHAN_FUSED(32)
RFX_CHAN_FUSED(64)
RFX_CHAN_FUSED(128)
RFX_CHAN_FUSED(256)
RFX_CHAN_FUSED(512)
#undef RFX_CHAN_FUSED

// z (or |z| with `magnitude`) of `frames` frames of x, stored in `format` (rfx_sample_format), for
// a supported shape; the newest sample read is x[(frames - 1) channels].
inline cudaError_t chan_fused_launch(const void* x, const float* taps, void* out, long long frames,
                                     int channels, int num_taps, bool magnitude, int format,
                                     cudaStream_t stream)
{
    if (frames <= 0) {
        return cudaSuccess;
    }
    switch (channels) {
    case 8: return chan_fused_launch_8(x, taps, out, frames, num_taps, magnitude, format, stream);
    case 16: return chan_fused_launch_16(x, taps, out, frames, num_taps, magnitude, format, stream);
    case 32: return chan_fused_launch_32(x, taps, out, frames, num_taps, magnitude, format, stream);
    case 64: return chan_fused_launch_64(x, taps, out, frames, num_taps, magnitude, format, stream);
    case 128: return chan_fused_launch_128(x, taps, out, frames, num_taps, magnitude, format, stream);
    case 256: return chan_fused_launch_256(x, taps, out, frames, num_taps, magnitude, format, stream);
    case 512: return chan_fused_launch_512(x, taps, out, frames, num_taps, magnitude, format, stream);
    default: return cudaErrorInvalidValue;
    }
}

}  // namespace rfx
