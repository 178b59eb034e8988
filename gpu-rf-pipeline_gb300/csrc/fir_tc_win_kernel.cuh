// The resident-window FIR's single-capture kernel and its launch, one instance per reach-back C,
// sample format and tile (fir_tc_win.cu: 1 to 3 blocks back; fir_tc_win_long.cu: 4 to 8).
#pragma once

#include "fir_tc.cuh"
#include "fir_tc_win.cuh"
#include "launch.hpp"
#include "tmap.hpp"

#include <cuda.h>
#include <cuda_runtime.h>

namespace rfx {

// One fault word per translation unit.
static __device__ unsigned int g_fault_fir_tcw;

// wmap: x as rows of 256 components (one 128-sample block per row, full blocks only), boxes
// of 256 components x (NB + C) rows (one tile window). kFmt: 0 cf32, 1 ci16, 2 ci8 (the copy
// moves the components as stored; the producers decode them).
template <int C, int kFmt, int NB>
__global__ void __launch_bounds__(tcw::kThreads, 1)
fir_tcw_kernel(const __grid_constant__ CUtensorMap wmap, const void* __restrict__ x,
               const float* __restrict__ taps, float2* __restrict__ y, long long n, int num_taps,
               int num_tiles)
{
    extern __shared__ __align__(1024) unsigned char smem[];
    tcw::Ctrl& ctl = *reinterpret_cast<tcw::Ctrl*>(smem);
    // The tensor-memory base travels through the last word of the control block's kilobyte.
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + 1020);
    const int warp = threadIdx.x >> 5;
    if (warp == tcw::kMmaWarp) {
        tc::tmem_alloc(smem_u32(tmem_slot), tcw::kTmemCols);
    }
    if (threadIdx.x == 0) {
        tcw::tcw_init<8>(ctl);
    }
    tc::fence_before();
    __syncthreads();
    tc::fence_after();
    const uint32_t tmem = *tmem_slot;
    wait_for_stream();
    allow_next();
    const tcw::TcwSingleSrc src{&wmap, tcw::WinCapture{x, y, taps, n, num_taps, 0}, num_tiles};
    tcw::tcw_pipeline<C, kFmt, 8, tcw::TcwSingleSrc, 2, NB>(src, smem, ctl, tmem, &g_fault_fir_tcw);
    if (warp == tcw::kMmaWarp) {
        tc::tmem_dealloc(tmem, tcw::kTmemCols);
    }
}

template <int C, int kFmt, int NB>
static cudaError_t launch_tcw(const void* x, const float* taps, void* y, long long n, int num_taps,
                              cudaStream_t stream)
{
    constexpr int es = tc::component_bytes(kFmt);
    const tcw::Layout lay = tcw::win_layout(C, 8, 1, es, NB);
    if (lay.bytes > tcw::kSmemMax) {
        return cudaErrorInvalidValue;
    }
    int device = 0;
    cudaError_t err = cudaGetDevice(&device);
    if (err != cudaSuccess) {
        return err;
    }
    int optin = 0;
    int sms = 0;
    if ((err = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin,
                                      device)) != cudaSuccess ||
        (err = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device)) !=
            cudaSuccess) {
        return err;
    }
    // At least 120 KB per block keeps one block per SM: each block owns all 512 TMEM columns.
    const uint32_t bytes = lay.bytes > 120u * 1024u ? lay.bytes : 120u * 1024u;
    if (bytes > static_cast<uint32_t>(optin)) {
        return cudaErrorInvalidValue;
    }
    err = cudaFuncSetAttribute(fir_tcw_kernel<C, kFmt, NB>,
                               cudaFuncAttributeMaxDynamicSharedMemorySize,
                               static_cast<int>(bytes));
    if (err != cudaSuccess) {
        return err;
    }
    // x as rows of 256 components (one 128-sample block per row), full blocks only; one box
    // is a tile window.
    CUtensorMap map;
    err = encode_rows(&map, x, es, n / tcw::kB, 2 * tcw::kB, 2 * tcw::kB,
                      static_cast<uint32_t>(NB + C));
    if (err != cudaSuccess) {
        return err;
    }
    const long long blocks = (n + tcw::kB - 1) / tcw::kB;
    const int tiles = static_cast<int>((blocks + NB - 1) / NB);
    const int grid = tiles < sms ? tiles : sms;
    return launch_overlapped(fir_tcw_kernel<C, kFmt, NB>, grid, tcw::kThreads, bytes, stream, map, x,
                             taps, static_cast<float2*>(y), n, num_taps, tiles);
}

template <int C, int NB>
static cudaError_t launch_formats(int format, const void* x, const float* taps, void* y,
                                  long long n, int num_taps, cudaStream_t stream)
{
    switch (format) {
    case 0: return launch_tcw<C, 0, NB>(x, taps, y, n, num_taps, stream);
    case 1: return launch_tcw<C, 1, NB>(x, taps, y, n, num_taps, stream);
    case 2: return launch_tcw<C, 2, NB>(x, taps, y, n, num_taps, stream);
    default: return cudaErrorInvalidValue;
    }
}

}  // namespace rfx
