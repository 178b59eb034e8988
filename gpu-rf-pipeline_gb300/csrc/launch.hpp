// Kernel launches that overlap the end of the kernel before them (programmatic dependent launch).
//
// A kernel launched here may be scheduled while the previous kernel of its stream drains: its
// blocks take the multiprocessors that fall idle, set up their barriers and tensor memory, and
// wait in wait_for_stream() (ptx.cuh) until every earlier kernel has completed and its writes are
// visible. Every thread of such a kernel calls wait_for_stream() before it touches global memory
// and allow_next() after it (a kernel that allocates tensor memory has a block barrier behind the
// allocation and before both), or never where the kernel after it is better held back (chan_wide.cu). A kernel launched in the ordinary way, a copy or an event after it
// still waits for its completion. Back to back on one stream this took 2 to 3 us off every call
// (64 channels, 2^24 samples: 53.8 -> 51.5 us; 2^21 ci16 samples to magnitudes: 14.0 -> 10.9).
#pragma once

#include <cuda_runtime.h>

#include <utility>

namespace rfx {

template <class... Params, class... Args>
cudaError_t launch_overlapped(void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem,
                              cudaStream_t stream, Args&&... args)
{
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t config{};
    config.gridDim = grid;
    config.blockDim = block;
    config.dynamicSmemBytes = smem;
    config.stream = stream;
    config.attrs = &attr;
    config.numAttrs = 1;
    return cudaLaunchKernelEx(&config, kernel, std::forward<Args>(args)...);
}

// Lets launches of `kernel` (which has no static shared memory) ask for `bytes` of dynamic shared
// memory. The limit belongs to the function, not to the launch: set to what one call needs, it fails
// a call of another thread, or a plan made before, that needs more and launches after it. So always
// the device's limit.
inline cudaError_t opt_in_smem(const void* kernel, size_t bytes)
{
    if (bytes <= 48u * 1024u) {
        return cudaSuccess;
    }
    int device = 0;
    int limit = 0;
    cudaError_t err = cudaGetDevice(&device);
    if (err == cudaSuccess) {
        err = cudaDeviceGetAttribute(&limit, cudaDevAttrMaxSharedMemoryPerBlockOptin, device);
    }
    if (err != cudaSuccess) {
        return err;
    }
    return bytes > static_cast<size_t>(limit)
               ? cudaErrorInvalidValue
               : cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, limit);
}

template <class... Params>
cudaError_t opt_in_smem(void (*kernel)(Params...), size_t bytes)
{
    return opt_in_smem(reinterpret_cast<const void*>(kernel), bytes);
}

constexpr size_t kSmemPerSm = 228u * 1024u;    // shared memory of an SM
constexpr size_t kSmemPerBlock = 1024u;        // of which the system takes this much per block

// Dynamic shared memory to ask for so that no multiprocessor takes more than its share,
// ceil(blocks / sms), of a launch smaller than one full wave (`bytes` needed, `fit` blocks fit an
// SM). Launched in the ordinary way blocks spread evenly; while the kernel before still holds its
// multiprocessors they gather on the ones that fall idle first (350 blocks of the plain FIR at 511
// taps: 48.1 us with up to four on one SM against 36.8 with three).
inline size_t even_spread_smem(size_t bytes, long long blocks, int sms, int fit)
{
    const long long share = (blocks + sms - 1) / sms;
    if (share >= fit || 2 * blocks <= sms) {
        return bytes;   // a full wave, or few enough that idle multiprocessors remain
    }
    const size_t more_than = kSmemPerSm / static_cast<size_t>(share + 1) - kSmemPerBlock;
    const size_t padded = (more_than / 128u + 1u) * 128u;   // share + 1 blocks do not fit
    return bytes > padded ? bytes : padded;
}

}  // namespace rfx
