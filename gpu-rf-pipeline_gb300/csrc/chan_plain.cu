// Plain channelizer: FP32 polyphase branch sums, then cuFFT's batched inverse transform in
// place — the structure of the project's channelize_device (src/channelize.cu:56-72).
//
//   u[t][m] = sum_p h[pM + m] x[tM - pM - m]          (x[i < 0] = 0)
//   z[t][k] = sum_m u[t][m] e^{+2 pi i k m / M}        (cuFFT inverse, unnormalized)
//
// The branch sums use the project's arithmetic (src/channelize.cu:35-46): one fused
// multiply-add per tap, l = m, m + M, ... ascending from +0, skipping the terms before the start
// of the input, so u is bit-identical to its kernel's. The project runs one thread per (frame,
// branch), which reads every sample once per tap of its branch (32 times at 32 taps per branch)
// through the caches. Here the frames of one branch are a FIR over the decimated sequence
// s_d = x[dM - m] with taps g_p = h[pM + m], and consecutive threads take consecutive branches,
// so every sample and tap load of a warp is one coalesced 256-byte row; the I/Q pair is one
// packed f32x2 fused multiply-add. Two forms:
//  - chan_branch_ring_kernel (up to 32 taps per branch): a thread walks one branch through a
//    segment of frames keeping the window of its current 8 frames in registers, so each sample is
//    loaded once (2^26 samples, 1024 channels, 32 taps per branch: 187 us under
//    the profiler, 84 % of the HBM copy rate, against 350 us for the form below);
//  - chan_branch_kernel (more taps): a thread computes R = 8 consecutive frames of one
//    branch with two alternating 8-sample register blocks, so each sample is loaded
//    (R + P - 1) / R times instead of P times.
// Frame groups whose terms fall before the input, and the last group (past its end), take a
// path that tests every term.
#include "chan_plain.cuh"
#include "launch.hpp"
#include "ptx.cuh"

#include <cuda_runtime.h>
#include <cufft.h>

#include <type_traits>

namespace rfx {

namespace {
constexpr int kBranchThreads = 256;
constexpr int kR = 8;   // frames per thread

// Taps p0 + q (q < nq) of one branch: acc[i] += g_p s_{t0 + i - p}, with cur[i] = s_{t0 - 8g + i}
// and nxt[i] = s_{t0 - 8(g+1) + i} for p0 = 8 g. Guarded: only terms whose sample index is >= 0.
template <bool kGuard>
__device__ __forceinline__ void taps_block(f32x2 (&acc)[kR], const f32x2 (&cur)[kR],
                                           const f32x2 (&nxt)[kR], const float* tcol,
                                           int tstride, int p0, int nq, long long t0,
                                           int first_valid_d)
{
#pragma unroll
    for (int q = 0; q < kR; ++q) {
        if (q < nq) {
            const float hv = tcol[(p0 + q) * tstride];
            const f32x2 h2 = pack2(hv, hv);
#pragma unroll
            for (int i = 0; i < kR; ++i) {
                const f32x2 v = i >= q ? cur[i - q] : nxt[kR + i - q];
                if (!kGuard || t0 + i - (p0 + q) >= first_valid_d) {
                    acc[i] = fma2(h2, v, acc[i]);
                }
            }
        }
    }
}

// Sample s of x in format kFmt (0 cf32; 1 ci16, 2 ci8: components converted as the project's
// SigMF reader converts them, src/io.cpp:110-148, so the sums are those of the converted input).
template <int kFmt>
__device__ __forceinline__ f32x2 load_sample(const void* __restrict__ x, long long s)
{
    if constexpr (kFmt == 0) {
        const float2 w = __ldg(static_cast<const float2*>(x) + s);
        return pack2(w.x, w.y);
    } else if constexpr (kFmt == 1) {
        const short2 w = __ldg(static_cast<const short2*>(x) + s);
        return pack2(static_cast<float>(w.x) * (1.0f / 32768.0f),
                     static_cast<float>(w.y) * (1.0f / 32768.0f));
    } else {
        const char2 w = __ldg(static_cast<const char2*>(x) + s);
        return pack2(static_cast<float>(w.x) * (1.0f / 128.0f),
                     static_cast<float>(w.y) * (1.0f / 128.0f));
    }
}

template <bool kGuard, int kFmt>
__device__ __forceinline__ void load_block(f32x2 (&blk)[kR], const void* __restrict__ x,
                                           long long n, int channels, int m, long long d0)
{
#pragma unroll
    for (int i = 0; i < kR; ++i) {
        const long long s = (d0 + i) * channels - m;
        f32x2 v = 0ull;
        if (!kGuard || (s >= 0 && s < n)) {
            v = load_sample<kFmt>(x, s);
        }
        blk[i] = v;
    }
}

template <bool kGuard, int kFmt>
__device__ __forceinline__ void branch_frames(f32x2 (&acc)[kR], const void* __restrict__ x,
                                              const float* tcol, int tstride, long long n,
                                              int channels, int m, int P, long long t0)
{
    const int first_valid_d = m > 0 ? 1 : 0;   // x[dM - m] >= 0 from this d on
    const int groups = P / kR;
    const int rem = P - groups * kR;
    f32x2 a[kR];
    f32x2 b[kR];
    load_block<kGuard, kFmt>(a, x, n, channels, m, t0);
    int g = 0;
    for (; g + 2 <= groups; g += 2) {
        load_block<kGuard, kFmt>(b, x, n, channels, m, t0 - kR * (g + 1));
        taps_block<kGuard>(acc, a, b, tcol, tstride, kR * g, kR, t0, first_valid_d);
        load_block<kGuard, kFmt>(a, x, n, channels, m, t0 - kR * (g + 2));
        taps_block<kGuard>(acc, b, a, tcol, tstride, kR * (g + 1), kR, t0, first_valid_d);
    }
    if (g < groups) {
        load_block<kGuard, kFmt>(b, x, n, channels, m, t0 - kR * (g + 1));
        taps_block<kGuard>(acc, a, b, tcol, tstride, kR * g, kR, t0, first_valid_d);
        if (rem > 0) {
            load_block<kGuard, kFmt>(a, x, n, channels, m, t0 - kR * (g + 2));
            taps_block<kGuard>(acc, b, a, tcol, tstride, kR * (g + 1), rem, t0,
                               first_valid_d);
        }
    } else if (rem > 0) {
        load_block<kGuard, kFmt>(b, x, n, channels, m, t0 - kR * (g + 1));
        taps_block<kGuard>(acc, a, b, tcol, tstride, kR * g, rem, t0, first_valid_d);
    }
}
}  // namespace

// Block: `width` consecutive branches x (256 / width) frame groups of kR frames per step, over
// kGroupSteps consecutive steps. With kSmemTaps the block's taps (max_p x width) are staged in
// shared memory once, and its consecutive frame groups reuse each other's samples through L1
// (measured at 2^26 samples, 1024 channels, 32 taps per branch: 490 us against 533 us reading
// taps through the caches one frame group per block). Groups with t0 < guard_frames or
// reaching past the last frame test every load and term.
constexpr int kGroupSteps = 16;

template <int kFmt, bool kSmemTaps>
__global__ void __launch_bounds__(kBranchThreads)
chan_branch_kernel(const void* __restrict__ x, const float* __restrict__ taps,
                   float2* __restrict__ u, long long n, long long frames, int channels,
                   int num_taps, int width, int guard_frames)
{
    extern __shared__ float taps_s[];   // [p][j]: tap p of branch blockIdx.y * width + j
    wait_for_stream();
    allow_next();
    const int j = static_cast<int>(threadIdx.x) % width;
    const int m = static_cast<int>(blockIdx.y) * width + j;
    if (kSmemTaps) {
        const int max_p = (num_taps + channels - 1) / channels;
        for (int i = threadIdx.x; i < max_p * width; i += kBranchThreads) {
            const int p = i / width;
            const int jj = i - p * width;
            const int mm = static_cast<int>(blockIdx.y) * width + jj;
            const long long l = static_cast<long long>(p) * channels + mm;
            taps_s[i] = (mm < channels && l < num_taps) ? __ldg(taps + l) : 0.0f;
        }
        __syncthreads();
    }
    if (m >= channels) {
        return;
    }
    // Taps of branch m: l = pM + m < num_taps; read from column j of the staged table, or from
    // global memory at stride `channels`.
    const int P = m < num_taps ? (num_taps - m + channels - 1) / channels : 0;
    const float* tcol = kSmemTaps ? taps_s + j : taps + m;
    const int tstride = kSmemTaps ? width : channels;
    const int steps = kSmemTaps ? kGroupSteps : 1;
    for (int it = 0; it < steps; ++it) {
        const long long group = (static_cast<long long>(blockIdx.x) * steps + it) *
                                    (kBranchThreads / width) + threadIdx.x / width;
        const long long t0 = group * kR;
        if (t0 >= frames) {
            return;
        }
        f32x2 acc[kR];
#pragma unroll
        for (int i = 0; i < kR; ++i) {
            acc[i] = 0ull;
        }
        if (t0 < guard_frames || t0 + kR > frames) {
            branch_frames<true, kFmt>(acc, x, tcol, tstride, n, channels, m, P, t0);
        } else {
            branch_frames<false, kFmt>(acc, x, tcol, tstride, n, channels, m, P, t0);
        }
#pragma unroll
        for (int i = 0; i < kR; ++i) {
            if (t0 + i < frames) {
                u[(t0 + i) * channels + m] = unpack2(acc[i]);
            }
        }
    }
}

// Register-ring form, for filters of up to 32 taps per branch. A thread owns one branch m and one
// segment of consecutive frames, which it walks in steps of kR = 8 frames. The samples of its
// branch for the current step and the kPG steps before it (kPG tap groups of eight) stay in
// registers as kPG + 1 blocks of eight, so every sample is loaded once per segment instead of once
// per tap group, and the branch's taps stay in registers too. The next blocks stream in by
// per-thread asynchronous copies, kRingStages steps ahead, into the thread's own slots of a
// shared-memory stage ring (a warp's copies and reads of one block row are 256 contiguous bytes);
// ci8 samples, narrower than such a copy, are loaded one step ahead into registers. Terms are
// summed in branch_frames' order: taps ascending from +0, one fused multiply-add each, absent
// taps and samples before the input left out.
// Three forms of the step (Ring), which differ in the tests around the tap loop:
//  * kLong: 8 kPG taps in every branch, long segments. No test in the loop (a per-tap test of the
//    branch's tap count doubled the instructions issued); the segment that starts the input sums
//    its first frames with branch_frames' tested path, from global memory.
//  * kUniform: the same taps, short segments. The first frames too come from the window, each term
//    tested, in a second copy of the loop: 1024 channels, 32 taps, sums and transform (us): 2^20
//    samples 15.3 against 18.5 for kLong, 2^22 39.5 against 41.1, but 2^26 389 against 348 (the
//    longer step code falls out of the instruction cache).
//  * kAny: any tap count, any format; the last tap group tests the branch's tap count as well, and
//    beyond 16 taps the window moves on one block per step instead of the code being repeated per
//    position (32763 taps, 2^22 samples: 41.7 us against 80). Against chan_branch_kernel, which
//    took these filters: 2^20 samples, 12287 taps 12.9 against 28.7, 32763 taps 22.4 against 52.2.
constexpr int kRingThreads = 128;
constexpr int kRingStages = 4;

template <int kFmt>
__device__ __forceinline__ f32x2 ring_lds(uint32_t addr)
{
    if constexpr (kFmt == 0) {
        return lds64(addr);
    } else {
        uint32_t w;
        asm volatile("ld.shared.u32 %0, [%1];" : "=r"(w) : "r"(addr));
        return pack2(static_cast<float>(static_cast<int>(w << 16) >> 16) * (1.0f / 32768.0f),
                     static_cast<float>(static_cast<int>(w) >> 16) * (1.0f / 32768.0f));
    }
}

// Blocks per SM: what the registers of the window and the taps leave.
__host__ __device__ constexpr int ring_blocks(int groups)
{
    return groups == 1 ? 5 : groups == 2 ? 4 : 3;
}

enum class Ring { kLong, kUniform, kAny };

template <int kPG, int kFmt, Ring kRing>
__global__ void __launch_bounds__(kRingThreads, ring_blocks(kPG))
chan_branch_ring_kernel(const void* __restrict__ x, const float* __restrict__ taps,
                        float2* __restrict__ u, long long n, long long frames, int channels,
                        int num_taps, int width, long long seg_frames, int guard_frames)
{
    constexpr int kN = kPG + 1;                  // register blocks
    constexpr int kP = kR * kPG;                 // taps per branch
    constexpr int kSb = kFmt == 0 ? 8 : kFmt == 1 ? 4 : 2;       // bytes per stored sample
    constexpr bool kCopies = kFmt != 2;
    constexpr bool kGeneral = kRing == Ring::kAny;
    constexpr bool kGuard = kRing != Ring::kLong;    // the first frames from the window too
    constexpr bool kRotate = !kGeneral || kPG <= 2;   // else the window moves on one block per step
    constexpr uint32_t kStageBytes = kR * kRingThreads * kSb;
    __shared__ __align__(16) unsigned char stage[kCopies ? kRingStages * kStageBytes : 16];
    wait_for_stream();
    allow_next();
    const int tid = static_cast<int>(threadIdx.x);
    const int j = tid % width;
    const int m = static_cast<int>(blockIdx.y) * width + j;
    const long long seg = static_cast<long long>(blockIdx.x) * (kRingThreads / width) + tid / width;
    const long long f0 = seg * seg_frames;
    if (m >= channels || f0 >= frames) {
        return;
    }
    const long long f1 = f0 + seg_frames < frames ? f0 + seg_frames : frames;
    float g[kP];
#pragma unroll
    for (int p = 0; p < kP; ++p) {
        const long long l = static_cast<long long>(p) * channels + m;
        g[p] = !kGeneral || l < num_taps ? __ldg(taps + l) : 0.0f;
    }
    const int my_taps = m < num_taps ? (num_taps - m + channels - 1) / channels : 0;
    const bool full = num_taps == kP * channels;
    const long long first_valid = m > 0 ? 1 : 0;   // x[dM - m] lies in the input from this d on
    long long t0 = f0;
    if constexpr (!kGuard) {
        for (; t0 < f1 && t0 < guard_frames; t0 += kR) {
            f32x2 acc[kR];
#pragma unroll
            for (int i = 0; i < kR; ++i) {
                acc[i] = 0ull;
            }
            branch_frames<true, kFmt>(acc, x, taps + m, channels, n, channels, m, kP, t0);
#pragma unroll
            for (int i = 0; i < kR; ++i) {
                if (t0 + i < f1) {
                    u[(t0 + i) * channels + m] = unpack2(acc[i]);
                }
            }
        }
        if (t0 >= f1) {
            return;
        }
    }
    // Ring slot k % kN holds block B(t0 + 8k) (decimated samples t0 + 8k .. + 7) during step k;
    // the blocks before step 0 go to slots kN - q, q = 1 .. kPG (zeros before the input).
    f32x2 R[kN][kR];
#pragma unroll
    for (int q = 1; q <= kPG; ++q) {
#pragma unroll
        for (int i = 0; i < kR; ++i) {
            const long long s = (t0 - kR * q + i) * channels - m;
            R[kN - q][i] = s >= 0 ? load_sample<kFmt>(x, s) : 0ull;
        }
    }
    // Sample d of the branch is at byte (d M - m) kSb of x: consecutive d are `row` bytes apart.
    const long long row = static_cast<long long>(channels) * kSb;
    // Slot (stage s, sample i) of this thread: stage + s * kStageBytes + (i * 128 + tid) * kSb.
    const uint32_t sbase = smem_u32(stage) + static_cast<uint32_t>(tid * kSb);
    const long long nb = (f1 - t0 + kR - 1) / kR;
    // The next block to copy: its first sample's address and how many of its samples lie in
    // the segment.
    const char* src = static_cast<const char*>(x) + (t0 * channels - m) * kSb;
    long long src_left = f1 - t0;
    bool src_first = t0 == 0;   // its frame 0 reads x[-m] in all branches but the first
    uint32_t src_stage = 0;
    unsigned short pre[kCopies ? 1 : kR];   // ci8: the next step's samples
    auto issue = [&]() {
        if constexpr (!kCopies) {
#pragma unroll
            for (int i = 0; i < kR; ++i) {
                const bool ok = i < src_left && (i > 0 || !src_first || m == 0);
                pre[i] = ok ? __ldg(reinterpret_cast<const unsigned short*>(src + i * row))
                            : static_cast<unsigned short>(0);
            }
            src += kR * row;
            src_left -= kR;
            src_first = false;
            return;
        }
        const uint32_t dst = sbase + src_stage * kStageBytes;
        if (src_left >= kR && !src_first) {
            const char* s = src;
#pragma unroll
            for (int i = 0; i < kR; ++i) {
                cp_async<kSb>(dst + static_cast<uint32_t>(i * kRingThreads * kSb), s, kSb);
                s += row;
            }
        } else {
            const char* s = src;
#pragma unroll
            for (int i = 0; i < kR; ++i) {
                const bool ok = i < src_left && (i > 0 || !src_first || m == 0);
                cp_async<kSb>(dst + static_cast<uint32_t>(i * kRingThreads * kSb),
                              ok ? s : static_cast<const char*>(x), ok ? kSb : 0);
                s += row;
            }
        }
        cp_async_commit();
        src += kR * row;
        src_left -= kR;
        src_first = false;
        src_stage = src_stage + 1 == kRingStages ? 0 : src_stage + 1;
    };
#pragma unroll
    for (int s = 0; s < (kCopies ? kRingStages - 1 : 1); ++s) {
        issue();
    }
    float2* dst = u + t0 * channels + m;
    long long dst_left = f1 - t0;
    uint32_t read_stage = 0;
    constexpr int kRots = kRotate ? kN : 1;
    for (long long k0 = 0; k0 < nb; k0 += kRots) {
#pragma unroll
        for (int rot = 0; rot < kRots; ++rot) {
            if (k0 + rot < nb) {
                if constexpr (kCopies) {
                    // Refills the stage read in the step before with the block kRingStages - 1
                    // steps ahead, then waits for this step's block.
                    issue();
                    cp_async_wait<kRingStages - 1>();
                    const uint32_t rs = sbase + read_stage * kStageBytes;
                    read_stage = read_stage + 1 == kRingStages ? 0 : read_stage + 1;
#pragma unroll
                    for (int i = 0; i < kR; ++i) {
                        R[rot][i] =
                            ring_lds<kFmt>(rs + static_cast<uint32_t>(i * kRingThreads * kSb));
                    }
                } else {
#pragma unroll
                    for (int i = 0; i < kR; ++i) {
                        const int v = pre[i];
                        R[rot][i] = pack2(
                            static_cast<float>(static_cast<int>(static_cast<uint32_t>(v) << 24) >> 24) *
                                (1.0f / 128.0f),
                            static_cast<float>(static_cast<int>(static_cast<uint32_t>(v) << 16) >> 24) *
                                (1.0f / 128.0f));
                    }
                    issue();
                }
                f32x2 acc[kR];
#pragma unroll
                for (int i = 0; i < kR; ++i) {
                    acc[i] = 0ull;
                }
                // Tap group gq: cur = B(T - 8 gq), nxt = B(T - 8 gq - 8), T = t0 + 8 k.
                const long long T = t0 + kR * (k0 + rot);
#pragma unroll
                for (int gq = 0; gq < kPG; ++gq) {
                    const int cs = (rot - gq + 2 * kN) % kN;
                    const int ns = (rot - gq - 1 + 2 * kN) % kN;
                    auto tap = [&](int q, auto guarded) {
                        const f32x2 h2 = pack2(g[kR * gq + q], g[kR * gq + q]);
#pragma unroll
                        for (int i = 0; i < kR; ++i) {
                            if (!decltype(guarded)::value ||
                                T + i - (kR * gq + q) >= first_valid) {
                                acc[i] = fma2(h2, i >= q ? R[cs][i - q] : R[ns][kR + i - q],
                                              acc[i]);
                            }
                        }
                    };
                    if (kGuard && T < guard_frames) {
#pragma unroll
                        for (int q = 0; q < kR; ++q) {
                            if (!kGeneral || kR * gq + q < my_taps) {
                                tap(q, std::true_type{});
                            }
                        }
                    } else if (!kGeneral || gq < kPG - 1 || full) {
#pragma unroll
                        for (int q = 0; q < kR; ++q) {
                            tap(q, std::false_type{});
                        }
                    } else {
#pragma unroll
                        for (int q = 0; q < kR; ++q) {
                            if (kR * gq + q < my_taps) {
                                tap(q, std::false_type{});
                            }
                        }
                    }
                }
                if (dst_left >= kR) {
                    float2* o = dst;
#pragma unroll
                    for (int i = 0; i < kR; ++i) {
                        *o = unpack2(acc[i]);
                        o += channels;
                    }
                } else {
                    float2* o = dst;
#pragma unroll
                    for (int i = 0; i < kR; ++i) {
                        if (i < dst_left) {
                            *o = unpack2(acc[i]);
                        }
                        o += channels;
                    }
                }
                dst += static_cast<long long>(kR) * channels;
                dst_left -= kR;
                if constexpr (!kRotate) {
                    // Every block one place older.
#pragma unroll
                    for (int q = 1; q < kN; ++q) {
#pragma unroll
                        for (int i = 0; i < kR; ++i) {
                            R[q][i] = R[(q + 1) % kN][i];
                        }
                    }
                }
            }
        }
    }
    if constexpr (kCopies) {
        cp_async_wait<0>();
    }
}

using RingKernel = void (*)(const void*, const float*, float2*, long long, long long, int, int, int,
                            long long, int);

template <int kFmt, Ring kRing>
static RingKernel ring_kernel(int groups)
{
    switch (groups) {
    case 1: return chan_branch_ring_kernel<1, kFmt, kRing>;
    case 2: return chan_branch_ring_kernel<2, kFmt, kRing>;
    case 3: return chan_branch_ring_kernel<3, kFmt, kRing>;
    default: return chan_branch_ring_kernel<4, kFmt, kRing>;
    }
}

template <int kFmt>
static RingKernel ring_kernel(int groups, Ring ring)
{
    return ring == Ring::kLong      ? ring_kernel<kFmt, Ring::kLong>(groups)
           : ring == Ring::kUniform ? ring_kernel<kFmt, Ring::kUniform>(groups)
                                    : ring_kernel<kFmt, Ring::kAny>(groups);
}

static cudaError_t ring_launch(const void* x, const float* taps, float2* u, long long n,
                               long long frames, int channels, int num_taps, cudaStream_t stream,
                               int format, bool before_dft)
{
    const int groups = static_cast<int>((num_taps + static_cast<long long>(kR) * channels - 1) /
                                        (static_cast<long long>(kR) * channels));
    int device = 0;
    int sms = 0;
    cudaError_t err = cudaGetDevice(&device);
    if (err != cudaSuccess ||
        (err = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device)) !=
            cudaSuccess) {
        return err;
    }
    // Branches per block: all (up to 128), or the power of two >= channels with several
    // segments per block. One wave of blocks: segments of equal length cover the frames.
    int w = 32;
    while (w < channels && w < kRingThreads) {
        w *= 2;
    }
    const int per_block = kRingThreads / w;
    const long long gy = (channels + w - 1) / w;
    const long long capacity = static_cast<long long>(sms) * ring_blocks(groups);
    const long long bx_target = capacity / gy > 0 ? capacity / gy : 1;
    const long long segs_target = bx_target * per_block;
    long long seg_frames = (frames + segs_target - 1) / segs_target;
    seg_frames = (seg_frames + kR - 1) / kR * kR;
    const long long segs = (frames + seg_frames - 1) / seg_frames;
    const long long bx = (segs + per_block - 1) / per_block;
    if (bx > 0x7FFFFFFFLL) {
        return cudaErrorInvalidConfiguration;
    }
    const int guard_frames = kR * (groups + 1);
    // Few channels reach long segments' form sooner: its tested first frames are in the caches there
    // (3 channels, 24 taps per branch, segments of 192 frames 26.1 us against 29.0 for kUniform, 64
    // frames 12.1 against 11.6; 1024 channels, 192 frames 41 against 34). So does the largest form before
    // the tensor-core transform (1024 channels, 32 taps per branch, whole call: segments of 40 frames 31.5
    // against 33.5, 72 47.7 against 54.5, 32 27.9 against 26.2; at 24 taps kUniform is faster at 72, 36.4
    // against 41.1).
    const long long long_segment = channels < 128                ? (groups == 4 ? 128 : 96)
                                   : groups == 4 && before_dft ? 40
                                   : groups == 4               ? 160
                                                               : 256;
    const Ring ring = num_taps != kR * groups * channels ? Ring::kAny
                      : seg_frames < long_segment        ? Ring::kUniform
                                                         : Ring::kLong;
    const RingKernel fn = format == 2   ? ring_kernel<2, Ring::kAny>(groups)
                          : format == 1 ? ring_kernel<1>(groups, ring)
                                        : ring_kernel<0>(groups, ring);
    const dim3 grid(static_cast<unsigned>(bx), static_cast<unsigned>(gy));
    return launch_overlapped(fn, grid, kRingThreads, 0, stream, x, taps, u, n, frames, channels,
                             num_taps, w, seg_frames, guard_frames);
}

cudaError_t chan_branch_launch(const void* x, const float* taps, void* u, long long frames,
                               int channels, int num_taps, cudaStream_t stream, int format,
                               bool before_dft)
{
    if (frames == 0 || channels < 1) {
        return cudaSuccess;
    }
    {
        const long long n = (frames - 1) * static_cast<long long>(channels) + 1;
        // (The grid has room for 65535 rows of blocks: of 128 branches each in the ring form, of 256
        // in the one below.)
        if (num_taps <= 4LL * kR * channels && channels <= 65535LL * kRingThreads) {
            return ring_launch(x, taps, static_cast<float2*>(u), n, frames, channels, num_taps,
                               stream, format, before_dft);
        }
    }
    // The newest sample any frame reads is the last frame's x[(frames - 1) M], which lies in the
    // input: loads are bounded by that index.
    const long long n = (frames - 1) * static_cast<long long>(channels) + 1;
    // Branches per block: the power of two >= channels, between one warp and the whole block.
    int w = 32;
    while (w < channels && w < kBranchThreads) {
        w *= 2;
    }
    const long long groups = (frames + kR - 1) / kR;
    const int per_block = kBranchThreads / w;
    const long long gy = (channels + w - 1) / w;
    // Frame groups before this one load samples before the input (the lowest sample block a
    // group loads starts kR * ceil(P / kR) frames back): they take the tested path.
    const int max_p = (num_taps + channels - 1) / channels;
    const int guard_frames = kR * ((max_p + kR - 1) / kR + 1);
    const size_t smem_bytes = static_cast<size_t>(max_p) * w * sizeof(float);
    int device = 0;
    int optin = 0;
    cudaError_t err = cudaGetDevice(&device);
    if (err != cudaSuccess ||
        (err = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, device)) !=
            cudaSuccess) {
        return err;
    }
    const bool staged = smem_bytes <= static_cast<size_t>(optin);
    const long long steps = staged ? kGroupSteps : 1;
    const long long gx = (groups + per_block * steps - 1) / (per_block * steps);
    if (gx > 0x7FFFFFFFLL || gy > 65535) {
        return cudaErrorInvalidConfiguration;
    }
    const dim3 grid(static_cast<unsigned>(gx), static_cast<unsigned>(gy));
    float2* uo = static_cast<float2*>(u);
    auto run = [&](auto kernel, size_t bytes) -> cudaError_t {
        const cudaError_t e = opt_in_smem(kernel, bytes);
        if (e != cudaSuccess) {
            return e;
        }
        return launch_overlapped(kernel, grid, kBranchThreads, bytes, stream, x, taps, uo, n, frames,
                                 channels, num_taps, w, guard_frames);
    };
    switch (format * 2 + (staged ? 1 : 0)) {
    case 0: err = run(chan_branch_kernel<0, false>, 0); break;
    case 1: err = run(chan_branch_kernel<0, true>, smem_bytes); break;
    case 2: err = run(chan_branch_kernel<1, false>, 0); break;
    case 3: err = run(chan_branch_kernel<1, true>, smem_bytes); break;
    case 4: err = run(chan_branch_kernel<2, false>, 0); break;
    case 5: err = run(chan_branch_kernel<2, true>, smem_bytes); break;
    default: return cudaErrorInvalidValue;
    }
    if (err != cudaSuccess) {
        return err;
    }
    return cudaGetLastError();
}

}  // namespace rfx
