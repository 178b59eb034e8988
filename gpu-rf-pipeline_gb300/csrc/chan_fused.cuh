// Fused channelizer for M = 8, 16, ..., 512 channels and up to 32 taps per branch: polyphase
// branch sums and the M-point inverse transform in one pass over memory, in FP32.
//
//   u[t][m] = sum_p h[pM + m] x[tM - pM - m]           (x[i < 0] = 0)      src/channelize.cu:25-49
//   z[t][k] = sum_m u[t][m] e^{+2 pi i k m / M}                              src/channelize.cu:70-71
//
// A group of M threads walks one segment of consecutive frames, eight per step.
//  1. Branch sums: thread m owns branch m. The window of the current eight frames (the block of
//     eight decimated samples x[(t + i) M - m] and the PG blocks before it, PG = ceil(P / 8)) stays
//     in registers, so every sample is loaded once per segment, straight into the register block
//     that has just become the oldest; the load of the next step's block is issued before the
//     transform of this one, which covers its latency. One fused multiply-add per tap in ascending
//     order, absent terms skipped: u is bit-identical to the project's kernel.
//  2. The transform of the eight frames, in shared memory: Stockham stages of radix 8, 4 or 2,
//     eight points per thread and stage in registers, the first stage reading u, the last one
//     writing z (or |z|) to global memory.
// The sums u never leave the SM: 16 bytes of HBM per sample where branch sums + cuFFT move 32.
//
// What bounds it (64 channels, 16 taps per branch, 2^24 cf32 samples): HBM takes 39.5 us at the
// copy rate, the FP32 pipe 27 us (per sample 32 lane operations of sums, about 24 of transform).
// Measured 50.5 us (5.3 TB/s) against 67.9 us for the dense GEMM form (chan_tc.cu), whose workers
// spend more than the FP32 transform on staging split operands, and 88.9 us for branch sums +
// cuFFT. The rest is latency at 16 warps per SM (fixed-latency waits, group barriers, loads); the
// launch is one wave of equal segments, and two waves took 52.1 us (shorter segments reread more
// history). Copying the samples through shared memory asynchronously took 59.5 us: the exchanges
// of the transform already keep the load/store pipe half busy.
#pragma once

#include "fft_small.cuh"
#include "launch.hpp"
#include "magnitude.cuh"
#include "ptx.cuh"
#include "sample_fmt.cuh"

#include <cuda_runtime.h>

#include <type_traits>

namespace rfx {
namespace fused {

using fft::cmul;
using fft::small_dft;

constexpr int kR = 8;                  // frames per step
constexpr int kMaxGroups = 4;          // tap groups of eight per branch
constexpr int kTablePoints = 512;      // e^{2 pi i k / 512}: every M divides it

// ---- geometry ---------------------------------------------------------------------------------

// Radices of the M-point transform, first to last (0: no such stage). The last radix leaves at
// least eight consecutive channels per frame to eight consecutive lanes (64-byte stores; four at
// eight channels).
template <int M>
struct Radices;
template <> struct Radices<8> { static constexpr int r[3] = {4, 2, 0}; };
template <> struct Radices<16> { static constexpr int r[3] = {8, 2, 0}; };
template <> struct Radices<32> { static constexpr int r[3] = {8, 4, 0}; };
template <> struct Radices<64> { static constexpr int r[3] = {8, 8, 0}; };
template <> struct Radices<128> { static constexpr int r[3] = {8, 4, 4}; };
template <> struct Radices<256> { static constexpr int r[3] = {8, 8, 4}; };
template <> struct Radices<512> { static constexpr int r[3] = {8, 8, 8}; };

__host__ __device__ constexpr int sample_bytes(int fmt) { return fmt == 0 ? 8 : fmt == 1 ? 4 : 2; }

// The shape of a block. The rules follow times at 2^24 cf32 samples (us, 64 channels unless said):
//  * blocks per SM: 5 of 128 threads (96 registers) up to 8 taps per branch (45.1 against 47.5 for
//    4) and up to 16 taps at 16 and 32 channels (47.5 against 49.7 at 32); 4 (128 registers)
//    beyond (16 taps 50.5, 24 taps 55.9 against 72.9 for 5); 3 (168 registers) where the window
//    spills at 4 (32 taps: 71.0 against 81.0);
//  * the window as a ring of blocks with the step code repeated per position, or moved one block
//    per step: repeated, 32 taps are 28 KB of step code and miss the instruction cache (97.7
//    against 71.0 moved); up to 16 taps the moves cost up to 1 us;
//  * the taps in shared memory only where registers run out (32 taps at 128 channels: 82.2 against
//    96.2; at 64 channels 77.8 against 71.0 in registers).
template <int M, int PG, int kFmt>
struct Cfg {
    static constexpr int kThreads = M < 128 ? 128 : M;
    static constexpr int kGroups = kThreads / M;
    static constexpr int kBlocks = (PG == 1 && M <= 64) || (PG == 2 && M <= 32)   ? 5
                                   : (PG == 3 && M <= 32) || (PG == 4 && M <= 64) ? 3
                                                                                  : 512 / kThreads;
    static constexpr bool kRotate = PG <= 2 || (PG == 3 && M >= 64);
    static constexpr bool kSmemTaps = (PG == 4 && M >= 128) || (PG == 3 && M == 512);
    static constexpr int kFrameU = M + M / 8;    // pitch of a frame in the u buffer (banks)
    static constexpr int kFrameA = M + M / 8;    // and in the padded stage buffers
    static constexpr uint32_t kTw1 = 0;                        // second stage's factors
    static constexpr uint32_t kTw2 = kTw1 + 8u * Radices<M>::r[0] * Radices<M>::r[1];   // third's
    static constexpr uint32_t kTaps = kTw2 + (Radices<M>::r[2] != 0 ? 8u * M : 0u);
    static constexpr uint32_t kBuf = kTaps + (kSmemTaps ? 4u * kR * PG * M : 0u);
    static constexpr uint32_t kBufBytes = 8u * kR * kFrameU;   // one of a group's two buffers
    static constexpr uint32_t kBytes = kBuf + 2u * kGroups * kBufBytes;
};

// Barrier of a group of M threads.
template <int M, int kThreads>
__device__ __forceinline__ void group_sync(int group)
{
    if constexpr (M <= 32) {
        __syncwarp();
    } else if constexpr (M == kThreads) {
        __syncthreads();
    } else {
        // Named by constants: an identifier in a register reserves all sixteen of a block.
        static_assert(kThreads == 2 * M, "two groups per block");
        if (group == 0) {
            asm volatile("bar.sync 1, %0;" ::"n"(M) : "memory");
        } else {
            asm volatile("bar.sync 2, %0;" ::"n"(M) : "memory");
        }
    }
}

// Element e of a padded stage buffer: one extra element per eight (strides of 8 between lanes
// fall on distinct banks).
__device__ __forceinline__ constexpr int padded(int e) { return e + e / 8; }

// The factors w_{Ns r}^{q i}, q < r, i < Ns, of a stage of radix r after Ns points, two q per
// 16-byte entry: tw[q / 2][i], so that a stage reads them with r / 2 conflict-free loads.
template <int M, int r, int Ns>
__device__ __forceinline__ void fill_factors(float4* tw, int tid, int threads, const float2* roots)
{
    constexpr int kStep = kTablePoints / (Ns * r);
    for (int e = tid; e < Ns * r / 2; e += threads) {
        const int q = 2 * (e / Ns);
        const int i = e % Ns;
        const float2 a = roots[q * i * kStep];
        const float2 b = roots[(q + 1) * i * kStep];
        tw[e] = make_float4(a.x, a.y, b.x, b.y);
    }
}

// One Stockham stage of radix r after Ns points: butterfly j takes elements j + q J (J = M / r),
// multiplied by w_{Ns r}^{q (j mod Ns)}, to elements (j / Ns) Ns r + j mod Ns + q Ns. Thread tau of
// the group takes butterfly j = tau % J of the frames tau / J + r i. `out(f, e, v)` stores.
template <int M, int r, int Ns, bool kFirst, class Out>
__device__ __forceinline__ void stage(const f32x2* in, int pitch, const float4* tw, int tau,
                                      Out out)
{
    constexpr int J = M / r;
    const int j = tau % J;
    const int f0 = tau / J;
    float2 w[r];
    if constexpr (!kFirst) {
#pragma unroll
        for (int q = 0; q < r; q += 2) {
            const float4 t = tw[(q / 2) * Ns + j % Ns];
            w[q] = make_float2(t.x, t.y);
            w[q + 1] = make_float2(t.z, t.w);
        }
    }
    const int e0 = (j / Ns) * Ns * r + j % Ns;
#pragma unroll
    for (int i = 0; i < 8 / r; ++i) {
        const int f = f0 + r * i;
        f32x2 v[r];
#pragma unroll
        for (int q = 0; q < r; ++q) {
            const int e = j + q * J;
            v[q] = in[f * pitch + (kFirst ? e : padded(e))];
        }
        if constexpr (!kFirst) {
#pragma unroll
            for (int q = 1; q < r; ++q) {
                v[q] = cmul(v[q], w[q]);
            }
        }
        small_dft<r>(v);
#pragma unroll
        for (int q = 0; q < r; ++q) {
            out(f, e0 + q * Ns, v[q]);
        }
    }
}

// A stored sample, read once (no L1 allocation), as raw bits in the low bytes of a register
// pair; and its components.
template <int kFmt>
__device__ __forceinline__ f32x2 load_raw(const char* p)
{
    f32x2 v;
    if constexpr (kFmt == 0) {
        asm volatile("ld.global.nc.L1::no_allocate.b64 %0, [%1];" : "=l"(v) : "l"(p));
    } else if constexpr (kFmt == 1) {
        uint32_t w;
        asm volatile("ld.global.nc.L1::no_allocate.b32 %0, [%1];" : "=r"(w) : "l"(p));
        v = w;
    } else {
        unsigned short w;
        asm volatile("ld.global.nc.L1::no_allocate.u16 %0, [%1];" : "=h"(w) : "l"(p));
        v = w;
    }
    return v;
}

template <int kFmt>
__device__ __forceinline__ f32x2 decode(f32x2 raw)
{
    if constexpr (kFmt == 0) {
        return raw;
    } else {
        // Each component, offset to unsigned, as the low mantissa bits of 2^23 + value; one fused
        // multiply-add takes the offset off and scales, exactly (an integer conversion runs at
        // a quarter of the rate).
        constexpr uint32_t kFlip = kFmt == 1 ? 0x80008000u : 0x8080u;
        constexpr float kScale = kFmt == 1 ? 1.0f / 32768.0f : 1.0f / 128.0f;
        constexpr float kOffset = -(8388608.0f + (kFmt == 1 ? 32768.0f : 128.0f)) * kScale;
        const uint32_t w = static_cast<uint32_t>(raw) ^ kFlip;
        const uint32_t re = __byte_perm(w, 0x4B000000u, kFmt == 1 ? 0x7610 : 0x7650);
        const uint32_t im = __byte_perm(w, 0x4B000000u, kFmt == 1 ? 0x7632 : 0x7651);
        return fma2(pack2(__uint_as_float(re), __uint_as_float(im)), pack2(kScale, kScale),
                    pack2(kOffset, kOffset));
    }
}

static __device__ const fft::Roots<kTablePoints> kRootTable = fft::make_roots<kTablePoints>();

// kFmt: sample format of x (0 cf32, 1 ci16, 2 ci8). n: one past the newest sample any frame
// reads. seg_frames: frames per segment, a multiple of eight. guard_frames: frames before it have
// terms before the input. full: every branch has 8 PG taps.
template <int M, int PG, int kFmt, bool kMag>
__global__ void __launch_bounds__(Cfg<M, PG, kFmt>::kThreads, Cfg<M, PG, kFmt>::kBlocks)
chan_fused_kernel(const void* __restrict__ x, const float* __restrict__ taps,
                  void* __restrict__ out, long long n, int frames, int num_taps, int seg_frames,
                  int guard_frames, int full)
{
    using C = Cfg<M, PG, kFmt>;
    constexpr int T = C::kThreads;
    constexpr int kN = PG + 1;                 // register blocks of the ring
    constexpr int kP = kR * PG;
    constexpr int kSb = sample_bytes(kFmt);
    extern __shared__ __align__(128) unsigned char smem[];
    const int tid = static_cast<int>(threadIdx.x);
    const int m = tid % M;
    const int group = tid / M;
    const int f0 = (static_cast<int>(blockIdx.x) * C::kGroups + group) * seg_frames;
    const int f1 = min(f0 + seg_frames, frames);   // f0 >= frames: loads and stores all tested

    constexpr int r0 = Radices<M>::r[0];
    constexpr int r1 = Radices<M>::r[1];
    constexpr int r2 = Radices<M>::r[2];
    wait_for_stream();
    allow_next();
    // This branch's taps: in registers, or column m of taps_s[p][m].
    const int my_taps = m < num_taps ? (num_taps - m + M - 1) / M : 0;
    const int first_valid = m > 0 ? 1 : 0;   // x[dM - m] lies in the input from this d on
    float g[C::kSmemTaps ? 1 : kP];
    float* const taps_s = reinterpret_cast<float*>(smem + C::kTaps);
    if constexpr (!C::kSmemTaps) {
#pragma unroll
        for (int p = 0; p < kP; ++p) {
            const int l = p * M + m;
            g[p] = l < num_taps ? __ldg(taps + l) : 0.0f;
        }
    }
    const float4* const tw1 = reinterpret_cast<const float4*>(smem + C::kTw1);
    const float4* const tw2 = reinterpret_cast<const float4*>(smem + C::kTw2);
    f32x2* ubuf = reinterpret_cast<f32x2*>(smem + C::kBuf + 2u * group * C::kBufBytes);
    f32x2* abuf = reinterpret_cast<f32x2*>(smem + C::kBuf + (2u * group + 1u) * C::kBufBytes);
    // The window in register blocks: with kRotate slot k % kN holds the samples
    // x[(f0 + 8 k + i) M - m], i < 8, of step k, else slot 0 does and the older ones move on; the
    // blocks before step 0 start in slots kN - q, q = 1 .. PG. A step's block is loaded, as stored,
    // once the step before it has summed (its slot then holds the oldest block) and arrives
    // during that step's transform. Zeros outside the input and past the segment.
    const char* const xb = static_cast<const char*>(x) - static_cast<long long>(m) * kSb;
    f32x2 R[kN][kR];
    auto load_block = [&](f32x2 (&blk)[kR], int b, int last) {
        const char* src = xb + static_cast<long long>(b) * (M * kSb);
        if (b > 0 && b + kR <= last) {
#pragma unroll
            for (int i = 0; i < kR; ++i) {
                blk[i] = load_raw<kFmt>(src + i * (M * kSb));
            }
        } else {
#pragma unroll
            for (int i = 0; i < kR; ++i) {
                const long long s = static_cast<long long>(b + i) * M - m;
                blk[i] = 0ull;
                if (b + i < last && s >= 0 && s < n) {
                    blk[i] = load_raw<kFmt>(src + i * (M * kSb));
                }
            }
        }
    };
    load_block(R[0], f0, f1);
#pragma unroll
    for (int q = 1; q <= PG; ++q) {
        load_block(R[kN - q], f0 - kR * q, f1);
    }
    // The stage factors and the longer filters' taps while those loads are in flight.
    const float2* const roots = reinterpret_cast<const float2*>(kRootTable.v);
    fill_factors<M, r1, r0>(reinterpret_cast<float4*>(smem + C::kTw1), tid, T, roots);
    if constexpr (r2 != 0) {
        fill_factors<M, r2, r0 * r1>(reinterpret_cast<float4*>(smem + C::kTw2), tid, T, roots);
    }
    if constexpr (C::kSmemTaps) {
        for (int i = tid; i < kP * M; i += T) {
            taps_s[i] = i < num_taps ? __ldg(taps + i) : 0.0f;
        }
    }
#pragma unroll
    for (int q = 1; q <= PG; ++q) {
#pragma unroll
        for (int i = 0; i < kR; ++i) {
            R[kN - q][i] = decode<kFmt>(R[kN - q][i]);
        }
    }
    __syncthreads();   // factors (and taps) in shared memory

    const int steps = seg_frames / kR;
    int rot = 0;
    for (int k = 0; k < steps; ++k) {
        const int t0 = f0 + kR * k;
        f32x2 acc[kR];
        // One step with the newest block in ring slot c.
        auto step = [&](auto slot) {
            constexpr int c = decltype(slot)::value;
#pragma unroll
            for (int i = 0; i < kR; ++i) {
                R[c][i] = decode<kFmt>(R[c][i]);
            }
            // Tap group gq: cur = block of frame t0 - 8 gq, nxt = the block before it. A tap is
            // applied to frame t0 + i where the branch has it and its sample lies in the input;
            // away from the first frames, and in all but the last tap group, it always does.
#pragma unroll
            for (int gq = 0; gq < PG; ++gq) {
                constexpr int kTwice = 2 * kN;
                const int cs = (c - gq + kTwice) % kN;
                const int ns = (c - gq - 1 + kTwice) % kN;
                auto tap = [&](int q, auto guarded) {
                    const int p = kR * gq + q;
                    const float h = C::kSmemTaps ? taps_s[p * M + m] : g[C::kSmemTaps ? 0 : p];
                    const f32x2 h2 = pack2(h, h);
#pragma unroll
                    for (int i = 0; i < kR; ++i) {
                        if (!decltype(guarded)::value || t0 + i - p >= first_valid) {
                            acc[i] = fma2(h2, i >= q ? R[cs][i - q] : R[ns][kR + i - q], acc[i]);
                        }
                    }
                };
                if (t0 < guard_frames) {
#pragma unroll
                    for (int q = 0; q < kR; ++q) {
                        if (kR * gq + q < my_taps) {
                            tap(q, std::true_type{});
                        }
                    }
                } else if (gq < PG - 1 || full) {
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
            if constexpr (!C::kRotate) {
                // Every block one place older.
#pragma unroll
                for (int q = 1; q < kN; ++q) {
#pragma unroll
                    for (int i = 0; i < kR; ++i) {
                        R[q][i] = R[(q + 1) % kN][i];
                    }
                }
            }
            load_block(R[C::kRotate ? (c + 1) % kN : 0], t0 + kR, f1);
        };
#pragma unroll
        for (int i = 0; i < kR; ++i) {
            acc[i] = 0ull;
        }
        if constexpr (C::kRotate) {
            switch (rot) {
            case 0: step(std::integral_constant<int, 0>{}); break;
            case 1: step(std::integral_constant<int, 1>{}); break;
            case 2:
                if constexpr (kN > 2) {
                    step(std::integral_constant<int, 2>{});
                }
                break;
            default:
                if constexpr (kN > 3) {
                    step(std::integral_constant<int, 3>{});
                }
                break;
            }
            rot = rot + 1 == kN ? 0 : rot + 1;
        } else {
            step(std::integral_constant<int, 0>{});
        }

        // ---- the transform of frames t0 .. t0 + 7 -------------------------------------------
#pragma unroll
        for (int i = 0; i < kR; ++i) {
            ubuf[i * C::kFrameU + m] = acc[i];
        }
        group_sync<M, T>(group);
        auto to_buf = [&](f32x2* buf) {
            return [buf](int f, int e, f32x2 v) { buf[f * C::kFrameA + padded(e)] = v; };
        };
        auto to_out = [&](int f, int e, f32x2 v) {
            if (t0 + f < f1) {
                const long long o = static_cast<long long>(t0 + f) * M + e;
                const float2 z = unpack2(v);
                if constexpr (kMag) {
                    static_cast<float*>(out)[o] = cmag(z.x, z.y);
                } else {
                    static_cast<float2*>(out)[o] = z;
                }
            }
        };
        stage<M, r0, 1, true>(ubuf, C::kFrameU, nullptr, m, to_buf(abuf));
        group_sync<M, T>(group);
        if constexpr (r2 == 0) {
            stage<M, r1, r0, false>(abuf, C::kFrameA, tw1, m, to_out);
        } else {
            stage<M, r1, r0, false>(abuf, C::kFrameA, tw1, m, to_buf(ubuf));
            group_sync<M, T>(group);
            stage<M, r2, r0 * r1, false>(ubuf, C::kFrameA, tw2, m, to_out);
            group_sync<M, T>(group);   // ubuf read before the next step's sums
        }
    }
}

// One launch: a wave of equal segments over the frames.
template <int M, int PG, int kFmt, bool kMag>
cudaError_t launch(const void* x, const float* taps, void* out, long long frames, int num_taps,
                   cudaStream_t stream)
{
    using C = Cfg<M, PG, kFmt>;
    int device = 0;
    int sms = 0;
    cudaError_t err = cudaGetDevice(&device);
    if (err != cudaSuccess ||
        (err = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device)) !=
            cudaSuccess) {
        return err;
    }
    const long long groups = static_cast<long long>(sms) * C::kBlocks * C::kGroups;
    long long seg = (frames + groups - 1) / groups;
    seg = (seg + kR - 1) / kR * kR;
    const long long segs = (frames + seg - 1) / seg;
    const unsigned blocks = static_cast<unsigned>((segs + C::kGroups - 1) / C::kGroups);
    const long long n = (frames - 1) * M + 1;
    const int guard = kR * (PG + 1);
    const size_t bytes = even_spread_smem(C::kBytes, blocks, sms, C::kBlocks);
    auto kernel = chan_fused_kernel<M, PG, kFmt, kMag>;
    if ((err = opt_in_smem(kernel, bytes)) != cudaSuccess) {
        return err;
    }
    return launch_overlapped(kernel, blocks, C::kThreads, bytes, stream, x, taps, out, n,
                             static_cast<int>(frames), num_taps, static_cast<int>(seg), guard,
                             num_taps == kR * PG * M ? 1 : 0);
}

template <int M, int PG>
cudaError_t launch_forms(const void* x, const float* taps, void* out, long long frames,
                         int num_taps, bool magnitude, int format, cudaStream_t stream)
{
    switch (2 * format + (magnitude ? 1 : 0)) {
    case 0: return launch<M, PG, 0, false>(x, taps, out, frames, num_taps, stream);
    case 1: return launch<M, PG, 0, true>(x, taps, out, frames, num_taps, stream);
    case 2: return launch<M, PG, 1, false>(x, taps, out, frames, num_taps, stream);
    case 3: return launch<M, PG, 1, true>(x, taps, out, frames, num_taps, stream);
    case 4: return launch<M, PG, 2, false>(x, taps, out, frames, num_taps, stream);
    case 5: return launch<M, PG, 2, true>(x, taps, out, frames, num_taps, stream);
    default: return cudaErrorInvalidValue;
    }
}

// The launch of one channel count (one translation unit each, chan_fused_*.cu).
template <int M>
cudaError_t launch_channels(const void* x, const float* taps, void* out, long long frames,
                            int num_taps, bool magnitude, int format, cudaStream_t stream)
{
    const int groups = (num_taps + kR * M - 1) / (kR * M);
    switch (groups) {
    case 1: return launch_forms<M, 1>(x, taps, out, frames, num_taps, magnitude, format, stream);
    case 2: return launch_forms<M, 2>(x, taps, out, frames, num_taps, magnitude, format, stream);
    case 3: return launch_forms<M, 3>(x, taps, out, frames, num_taps, magnitude, format, stream);
    case 4: return launch_forms<M, 4>(x, taps, out, frames, num_taps, magnitude, format, stream);
    default: return cudaErrorInvalidValue;
    }
}

}  // namespace fused
}  // namespace rfx
