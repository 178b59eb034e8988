// The fused channelizer's kernels at 8 channels (chan_fused.cuh; one translation unit per
// channel count, compiled in parallel).
#include "chan_fused.cuh"

namespace rfx {

cudaError_t chan_fused_launch_8(const void* x, const float* taps, void* out, long long frames,
                                 int num_taps, bool magnitude, int format, cudaStream_t stream)
{
    return fused::launch_channels<8>(x, taps, out, frames, num_taps, magnitude, format, stream);
}

}  // namespace rfx
