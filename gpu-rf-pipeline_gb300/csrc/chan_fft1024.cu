// The inverse transform of the 1024-channel plain channelizer in FP32: frames of 1024 branch sums
// (chan_plain.cu) to channels, or to their magnitudes.
//
//   z[t][k] = sum_m u[t][m] e^{+2 pi i k m / 1024}                           src/channelize.cu:70-71
//
// One warp per frame, 32 x 32 (m = m1 + 32 m2, k = k2 + 32 k1): lane m1 holds the 32 sums
// u[m1 + 32 m2], transforms them over m2 in registers, multiplies by w_1024^(k2 m1), hands them to
// lane k2 through shared memory, which transforms over m1 and writes z[k2 + 32 k1]. Every load and
// store instruction of a warp is one row of 256 contiguous bytes. In place where out is u: a warp
// reads its whole frame before it writes it.
#include "chan_fft1024.hpp"
#include "fft_small.cuh"
#include "launch.hpp"
#include "magnitude.cuh"

#include <cuda_runtime.h>

namespace rfx {

namespace {

constexpr int kM = 1024;
constexpr int kWarps = 4;
constexpr int kThreads = kWarps * 32;
constexpr int kBlocks = 4;                     // per SM: 16 warps of 128 registers
constexpr int kRow = 33;                       // exchange rows padded by one element (banks)
constexpr uint32_t kTwBytes = 8u * kM;
constexpr uint32_t kBytes = kTwBytes + kWarps * 8u * 32u * kRow;

static __device__ const fft::Roots<kM> kRoots1024 = fft::make_roots<kM>();

}  // namespace

template <bool kMag>
__global__ void __launch_bounds__(kThreads, kBlocks)
chan_fft1024_kernel(const f32x2* u, void* out, int frames)
{
    extern __shared__ __align__(16) unsigned char smem[];
    // w_1024^(k2 m1), two k2 per 16-byte entry: tw[k2 / 2][m1].
    float4* const tw = reinterpret_cast<float4*>(smem);
    const float2* const roots = reinterpret_cast<const float2*>(kRoots1024.v);
    for (int i = threadIdx.x; i < kM / 2; i += kThreads) {
        const int k2 = 2 * (i >> 5);
        const int m1 = i & 31;
        const float2 a = roots[k2 * m1];
        const float2 b = roots[(k2 + 1) * m1];
        tw[i] = make_float4(a.x, a.y, b.x, b.y);
    }
    __syncthreads();
    wait_for_stream();
    allow_next();
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    f32x2* const ex = reinterpret_cast<f32x2*>(smem + kTwBytes) + warp * (32 * kRow);
    for (int t = static_cast<int>(blockIdx.x) * kWarps + warp; t < frames;
         t += static_cast<int>(gridDim.x) * kWarps) {
        const f32x2* src = u + static_cast<long long>(t) * kM + lane;
        f32x2 v[32];
#pragma unroll
        for (int i = 0; i < 32; ++i) {
            v[i] = src[32 * i];
        }
        fft::dft32(v);
#pragma unroll
        for (int k2 = 0; k2 < 32; k2 += 2) {
            const float4 w = tw[16 * k2 + lane];
            ex[lane * kRow + k2] = fft::cmul(v[k2], make_float2(w.x, w.y));
            ex[lane * kRow + k2 + 1] = fft::cmul(v[k2 + 1], make_float2(w.z, w.w));
        }
        __syncwarp();
#pragma unroll
        for (int m1 = 0; m1 < 32; ++m1) {
            v[m1] = ex[m1 * kRow + lane];
        }
        __syncwarp();
        fft::dft32(v);
        const long long o = static_cast<long long>(t) * kM + lane;
#pragma unroll
        for (int k1 = 0; k1 < 32; ++k1) {
            const float2 z = unpack2(v[k1]);
            if constexpr (kMag) {
                static_cast<float*>(out)[o + 32 * k1] = cmag(z.x, z.y);
            } else {
                static_cast<float2*>(out)[o + 32 * k1] = z;
            }
        }
    }
}

cudaError_t chan_fft1024_launch(const void* u, void* out, long long frames, bool magnitude,
                                cudaStream_t stream)
{
    int device = 0;
    int sms = 0;
    cudaError_t err = cudaGetDevice(&device);
    if (err != cudaSuccess ||
        (err = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device)) !=
            cudaSuccess) {
        return err;
    }
    auto kernel = magnitude ? chan_fft1024_kernel<true> : chan_fft1024_kernel<false>;
    const long long want = (frames + kWarps - 1) / kWarps;
    const long long cap = static_cast<long long>(sms) * kBlocks;
    const unsigned grid = static_cast<unsigned>(want < cap ? want : cap);
    return launch_overlapped(kernel, grid, kThreads, kBytes, stream, static_cast<const f32x2*>(u),
                             out, static_cast<int>(frames));
}

}  // namespace rfx
