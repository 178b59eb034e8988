// Plain FP32 FIR kernels for sm_103a: one tile per block (fir_plain_tile.cuh holds the tile
// function, its arithmetic and its staging), for one capture (cf32 or integer input) and for
// captures sharing one tap set in tiles of 384 to 2304 outputs by the amount of work and the filter's
// shared memory (tile_shape), and for captures with their own taps in tiles of 2304.
#include "fir_plain.cuh"
#include "fir_plain_tile.cuh"
#include "launch.hpp"
#include "ptx.cuh"

#include <cuda_runtime.h>

#include <type_traits>

namespace rfx {

static __device__ unsigned int g_fault_fir_plain;

namespace {

constexpr int kThreads = kPlainThreads;

// One tile per block, the whole block as the tile's thread group.
template <int kFmt = 0, int R = kPlainOutputsPerThread, int T = kPlainThreads>
__device__ __forceinline__ void plain_block_tile(const void* x, const float* taps, float2* y,
                                                 long long n, int num_taps, long long tile,
                                                 unsigned char* smem)
{
    uint32_t phase = 0;
    fir_plain_tile<kFmt, R, T>(x, taps, y, n, num_taps, tile, smem, &g_fault_fir_plain,
                               static_cast<int>(threadIdx.x), PlainBlockSync{}, phase, true);
}

}  // namespace

// kFmt: cf32 input, or integer I/Q (1 ci16, 2 ci8) decoded in the load stage.
template <int kFmt, int R, int T>
__global__ void __launch_bounds__(T, 1024 / T)
fir_plain_kernel(const void* __restrict__ x, const float* __restrict__ taps,
                 float2* __restrict__ y, long long n, int num_taps)
{
    extern __shared__ __align__(128) unsigned char smem[];
    wait_for_stream();
    allow_next();
    plain_block_tile<kFmt, R, T>(x, taps, y, n, num_taps, blockIdx.x, smem);
}

// The capture c that block `block` works on: the last with tile0[c] <= block. Through a warp
// reduction, so that the compiler knows it to be the same on every lane and keeps the capture's
// fields and what follows from them in uniform registers: 2^22 samples, 700 taps 188.3 us, as for one
// capture in the kernel's parameters, against 198 with the search's own result (more register bank
// conflicts on the packed multiply-adds).
template <class Captures>
__device__ __forceinline__ int capture_of(const Captures& captures, int block)
{
    int lo = 0;
    int hi = captures.count;
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (captures.tile0[mid] <= block) {
            lo = mid;
        } else {
            hi = mid;
        }
    }
    return static_cast<int>(__reduce_max_sync(0xFFFFFFFFu, static_cast<unsigned>(lo)));
}

// Several captures sharing one tap set. kRows, captures of about the same length: a row of blocks each
// (blockIdx.y). Otherwise block b takes tile b - tile0[c] of the capture c whose tiles hold b, so that no
// block is launched without work: of 64 captures, one of 2^22 samples and 63 of 4096, 63 taps 23.6 us,
// against 247 in rows of the longest capture's tiles; but the search costs 32 captures of 2^18 samples,
// 31 taps 2 us (27.0 against 25.0). (Both in one kernel: 390 us against 373 for 2^23 samples, 700 taps,
// the index no longer uniform.)
template <int R, int T, bool kRows>
__global__ void __launch_bounds__(T, 1024 / T)
fir_plain_batched_kernel(const __grid_constant__ PlainBatch batch, const float* __restrict__ taps,
                         int num_taps)
{
    extern __shared__ __align__(128) unsigned char smem[];
    wait_for_stream();
    allow_next();
    if constexpr (kRows) {
        const int c = blockIdx.y;
        const long long n = batch.num_samples[c];
        if (static_cast<long long>(blockIdx.x) * (T * R) >= n) {
            return;
        }
        plain_block_tile<0, R, T>(batch.x[c], taps, static_cast<float2*>(batch.y[c]), n, num_taps,
                                  blockIdx.x, smem);
    } else {
        const int block = static_cast<int>(blockIdx.x);
        const int c = capture_of(batch, block);
        plain_block_tile<0, R, T>(batch.x[c], taps, static_cast<float2*>(batch.y[c]),
                                  batch.num_samples[c], num_taps, block - batch.tile0[c], smem);
    }
}

// Captures with their own taps: block b takes tile b - tile0[c] of the capture c whose tiles
// contain it (same arithmetic per capture as fir_plain_kernel, so the same bits).
__global__ void __launch_bounds__(kThreads, 4)
fir_plain_caps_kernel(const __grid_constant__ PlainCaps caps)
{
    extern __shared__ __align__(128) unsigned char smem[];
    wait_for_stream();
    allow_next();
    const int block = static_cast<int>(blockIdx.x);
    const int c = capture_of(caps, block);
    plain_block_tile(caps.x[c], caps.taps[c], static_cast<float2*>(caps.y[c]), caps.num_samples[c],
                     caps.num_taps[c], block - caps.tile0[c], smem);
}

// Blocks of `threads` threads (1024 to an SM: the kernels' launch bounds) and `bytes` of shared memory
// that fit an SM.
static int tiles_that_fit(int threads, size_t bytes)
{
    const int by_smem = static_cast<int>(kSmemPerSm / (bytes + kSmemPerBlock));
    return by_smem < 1024 / threads ? by_smem : 1024 / threads;
}

// Shared memory for a launch of `blocks` tiles and the function's opt-in to it.
static cudaError_t spread_tiles(const void* fn, long long blocks, int sms, int threads,
                                size_t* bytes)
{
    *bytes = even_spread_smem(*bytes, blocks, sms, tiles_that_fit(threads, *bytes));
    return opt_in_smem(fn, *bytes);
}

static cudaError_t sm_count(int* sms)
{
    int device = 0;
    const cudaError_t err = cudaGetDevice(&device);
    return err == cudaSuccess
               ? cudaDeviceGetAttribute(sms, cudaDevAttrMultiProcessorCount, device)
               : err;
}

// The tile of a launch over `outputs` outputs: threads and outputs per thread.
struct TileShape {
    int threads;
    int outputs;
};

// By the time of the busiest SM, in cycles: w warps per scheduler (at least one), each R cycles of
// a tap. Fitted to times on 152 SMs at 16 to 1025 taps: a warp alone on its scheduler takes 12.5,
// 18.6 and 26 cycles per tap for 3, 5 and 9 outputs per thread, several share it at 12.5, 15.2,
// 18.9 and 23.3 each (the fewer outputs, the more sample loads per tap), and no fewer than `least`
// with staging. Measured, 1025 taps (us): 4096 samples 8.6 (3 outputs) against 25.5 for the tile of
// 256 threads and 9 outputs that every call took, 65536 samples 11.5 (5) against 25.4, 2^18 samples
// 20.9 (7) against 25.6; 63 taps: 10007 samples 2.4 against 4.0, 2^24 75.6 (9 outputs, 128 threads)
// against 78.1. Long filters take so much shared memory that one or two blocks fill an SM: a warp is
// alone on its scheduler then, however many tiles wait, and the larger block is the better one (2^22
// samples of cf32, 8192 taps 2185 us with 256 threads of 9 outputs against 2371 with 128).
// tiles_of(outputs): the launch's tiles of that many outputs each.
template <class Tiles>
static TileShape tile_shape(Tiles tiles_of, int num_taps, int fmt, int sms)
{
    struct Candidate {
        TileShape shape;
        double per_tap;      // cycles per tap and warp of a scheduler
        double alone;        // cycles per tap of one warp
        double least;        // cycles per warp
        double floor_cycles; // of the launch
    };
    static constexpr Candidate kCandidates[] = {
        {{128, 9}, 23.3, 26.0, 780.0, 2500.0},
        {{256, 9}, 23.3, 26.0, 780.0, 3100.0},
        {{256, 7}, 18.9, 18.9, 620.0, 3100.0},
        {{128, 5}, 15.2, 18.6, 480.0, 1400.0},
        {{128, 3}, 12.5, 12.5, 460.0, 1500.0},
    };
    TileShape best = kCandidates[0].shape;
    double best_cycles = 1e300;
    for (const Candidate& c : kCandidates) {
        const long long tile = static_cast<long long>(c.shape.threads) * c.shape.outputs;
        const long long per_sm = (tiles_of(tile) + sms - 1) / sms;
        const double w = static_cast<double>(per_sm) * c.shape.threads / 128.0;
        const long long fit = tiles_that_fit(
            c.shape.threads, plain_layout(num_taps, fmt, static_cast<int>(tile)).bytes);
        const double live = static_cast<double>(per_sm < fit ? per_sm : fit) * c.shape.threads / 128.0;
        // Fewer than four warps on a scheduler, though more wait: 2 % of staging in the open.
        const double open = per_sm > fit && live < 4.0 ? 1.02 : 1.0;
        const double tap = w * (live > 1.0 ? open * c.per_tap : c.alone);
        double cycles = num_taps * tap;
        cycles = cycles > w * c.least ? cycles : w * c.least;
        cycles = cycles > c.floor_cycles ? cycles : c.floor_cycles;
        if (cycles < best_cycles) {
            best_cycles = cycles;
            best = c.shape;
        }
    }
    return best;
}

// Calls run(R, T) as integral constants for a shape.
template <class Run>
static cudaError_t with_shape(TileShape shape, Run run)
{
    using std::integral_constant;
    if (shape.threads == 256 && shape.outputs == 9) {
        return run(integral_constant<int, 9>{}, integral_constant<int, 256>{});
    }
    switch (shape.outputs) {
    case 3: return run(integral_constant<int, 3>{}, integral_constant<int, 128>{});
    case 5: return run(integral_constant<int, 5>{}, integral_constant<int, 128>{});
    case 7: return run(integral_constant<int, 7>{}, integral_constant<int, 256>{});
    default: return run(integral_constant<int, 9>{}, integral_constant<int, 128>{});
    }
}

template <int kFmt>
static cudaError_t launch_plain(const void* x, const float* taps, void* y, long long n,
                                int num_taps, cudaStream_t stream)
{
    if (n <= 0) {
        return cudaSuccess;
    }
    int sms = 0;
    const cudaError_t err = sm_count(&sms);
    if (err != cudaSuccess) {
        return err;
    }
    auto tiles_of = [n](long long tile) { return (n + tile - 1) / tile; };
    return with_shape(tile_shape(tiles_of, num_taps, kFmt, sms), [&](auto r, auto t) {
        constexpr int R = decltype(r)::value;
        constexpr int T = decltype(t)::value;
        auto kernel = fir_plain_kernel<kFmt, R, T>;
        const long long tiles = tiles_of(T * R);
        size_t bytes = plain_layout(num_taps, kFmt, T * R).bytes;
        const cudaError_t e =
            spread_tiles(reinterpret_cast<const void*>(kernel), tiles, sms, T, &bytes);
        if (e != cudaSuccess) {
            return e;
        }
        return launch_overlapped(kernel, static_cast<unsigned>(tiles), T, bytes, stream, x, taps,
                                 static_cast<float2*>(y), n, num_taps);
    });
}

cudaError_t fir_plain_launch(const void* x, const float* taps, void* y, long long n,
                             int num_taps, cudaStream_t stream)
{
    return launch_plain<0>(x, taps, y, n, num_taps, stream);
}

cudaError_t fir_plain_batched_launch(PlainBatch& batch, const float* taps, int num_taps,
                                     cudaStream_t stream)
{
    // Every capture ends in a tile of its own: 16 captures of 2^14 samples are 160 tiles of 1792
    // outputs, two rounds of 152 SMs, though their samples would fit 147.
    auto tiles_of = [&batch](long long tile) {
        long long tiles = 0;
        for (int c = 0; c < batch.count; ++c) {
            tiles += (batch.num_samples[c] + tile - 1) / tile;
        }
        return tiles;
    };
    if (tiles_of(1) == 0) {
        return cudaSuccess;
    }
    int sms = 0;
    const cudaError_t err = sm_count(&sms);
    if (err != cudaSuccess) {
        return err;
    }
    return with_shape(tile_shape(tiles_of, num_taps, 0, sms), [&](auto r, auto t) {
        constexpr int R = decltype(r)::value;
        constexpr int T = decltype(t)::value;
        const long long tiles = tiles_of(T * R);
        long long longest = 0;
        batch.tile0[0] = 0;
        for (int c = 0; c < batch.count; ++c) {
            const long long own = (batch.num_samples[c] + T * R - 1) / (T * R);
            longest = own > longest ? own : longest;
            batch.tile0[c + 1] = batch.tile0[c] + static_cast<int>(own);
        }
        // Rows where no more than one block in nine has no work.
        const bool rows = longest * batch.count <= tiles + tiles / 8;
        const dim3 grid(static_cast<unsigned>(rows ? longest : tiles), rows ? batch.count : 1);
        auto kernel = rows ? fir_plain_batched_kernel<R, T, true>
                           : fir_plain_batched_kernel<R, T, false>;
        size_t bytes = plain_layout(num_taps, 0, T * R).bytes;
        const cudaError_t e =
            spread_tiles(reinterpret_cast<const void*>(kernel), tiles, sms, T, &bytes);
        if (e != cudaSuccess) {
            return e;
        }
        return launch_overlapped(kernel, grid, T, bytes, stream, batch, taps, num_taps);
    });
}

cudaError_t fir_plain_launch_format(int format, const void* x, const float* taps, void* y,
                                    long long n, int num_taps, cudaStream_t stream)
{
    switch (format) {
    case 1: return launch_plain<1>(x, taps, y, n, num_taps, stream);
    case 2: return launch_plain<2>(x, taps, y, n, num_taps, stream);
    default: return launch_plain<0>(x, taps, y, n, num_taps, stream);
    }
}

cudaError_t fir_plain_caps_launch(const PlainCaps& caps, cudaStream_t stream)
{
    const int tiles = caps.tile0[caps.count];
    if (caps.count == 0 || tiles == 0) {
        return cudaSuccess;
    }
    int kmax = 1;
    for (int c = 0; c < caps.count; ++c) {
        kmax = caps.num_taps[c] > kmax ? caps.num_taps[c] : kmax;
    }
    int sms = 0;
    cudaError_t err = sm_count(&sms);
    if (err != cudaSuccess) {
        return err;
    }
    size_t bytes = plain_layout(kmax).bytes;
    err = spread_tiles(reinterpret_cast<const void*>(fir_plain_caps_kernel), tiles, sms, kThreads,
                       &bytes);
    if (err != cudaSuccess) {
        return err;
    }
    return launch_overlapped(fir_plain_caps_kernel, static_cast<unsigned>(tiles), kThreads, bytes,
                             stream, caps);
}

cudaError_t fir_plain_take_fault(unsigned int* code)
{
    unsigned int zero = 0;
    cudaError_t err = cudaMemcpyFromSymbol(code, g_fault_fir_plain, sizeof(unsigned int));
    if (err != cudaSuccess) {
        return err;
    }
    return cudaMemcpyToSymbol(g_fault_fir_plain, &zero, sizeof(unsigned int));
}

}  // namespace rfx
