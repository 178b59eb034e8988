// Tensor-core FIR on sm_103a, resident-window form (2 to 385 taps): the block-Toeplitz GEMM
// of fir_tc.cu, tiled so that each sample crosses HBM and the copy engine once.
//
//   y[n] = sum_{k<K} h[k] x[n-k],  x[m < 0] = 0                              (src/fir.cu:1-5)
//
// Blocks of B = 128 outputs; a block reaches back C = floor((K + 126) / 128) blocks (1 to 3):
//   Y[:, j] = sum_{c=0}^{C} T_c X[:, j - c],   T_c(r, s) = h[cB + r - s]  (0 outside [0, K)).
// A tile is NB blocks, 48 (6144 outputs) in long captures and 8 to 32 where smaller tiles spread
// a short one over more SMs (fir_tcw_tile_blocks); its input window is blocks j0 - C .. j0 + NB - 1.
// The GEMM per tile is D (128 x 2 NB) += A (128 x 16) B (16 x 2 NB) over K-steps (c, st): A is a
// descriptor into the tap strip (fir_tc.cu's layout: output rows stored reversed, so every 8 x 8
// core matrix of every T_c is one strip element), B the FP16 planes of K-step st (16 samples of
// each window row, N index 2 j + {0: I, 1: Q}). Chunk C of a K-step whose taps are all zero
// (16 st <= C B - K - 15) is skipped: 63 taps need 12 of the 16 chunk-steps.
//
// What differs from fir_tc.cu (which keeps the longest filters: its N = 192 tiles spread a tap
// matrix's read over twice the columns):
//  * tap matrices (128 x 16 FP16) sit in tensor memory beside the accumulators as far as its columns
//    go: both splits' up to C = 1 and the high split's up to C = 3 at 32 blocks, two chunks of the
//    high split at 48. Read from the strip in shared memory, 4 KB per MMA, they set the MMAs' pace
//    (99 cycles an MMA at N = 96 against 51 of the tensor cores) and took the bandwidth that the
//    copies, the scan and the converters need. 2^24 samples (us): 63 taps 51.1 -> 46.1, 255 taps 70.4
//    -> 60.5, 385 taps 82.6 -> 73; 2^20 samples, 255 taps 10.8 -> 10.1, 1025 taps 19.2 -> 18.2. Tiles of
//    8 and 16 blocks at C <= 2 keep the strip: one such tile is over before the copies to tensor
//    memory are paid back (63 taps, 2^16 samples 4.6 against 5.0);
//  * the whole window arrives by ONE 2-D TMA copy (rows of 1 KB for cf32) into a ring of three
//    window buffers, issued by a copy warp as soon as a buffer is converted: each sample
//    crosses HBM once and the TMA engine once (fir_tc.cu copies it twice: a scan slice and a
//    K-step box);
//  * the tile's power-of-two scale (largest |component| of the window brought into
//    [2^14, 2^15)) is a scan of that resident window by two scan warps as soon as it lands;
//    the eight producer warps only convert, from the same buffer, four K-steps at a time (a
//    thread's items of four K-steps are independent, so their loads, splits and stores overlap;
//    one K-step at a time took 62.7 us at 63 taps against 53.7 us);
//  * the large product h_hi x_hi goes to accumulator H in groups of whole K-steps of at most 18
//    MMAs (round-toward-zero accumulation: fir_tc.cu measured 5e-7 at 9 MMAs, 8e-7 at 18), H
//    double-buffered; the cross products go to X once per tile, X double-buffered: the MMAs of
//    one group or tile run while eight drain warps add the previous one into FP32 running sums.
// Split precision as in fir_tc.cu: x' = 2^ex x = x_hi + x_lo, h' = 2^eh h = h_hi + h_lo in FP16;
// the MMAs sum h_hi x_hi + h_hi x_lo + h_lo x_hi with FP32 accumulation; the drain scales by
// 2^-(ex + eh).
//
// The pipeline itself is in fir_tc_win.cuh (the batch kernel runs it over lists of captures).
//
// Roles (640 threads): warp 0 copies windows; warp 1 owns tensor memory and issues the MMAs (the
// warp runs the loop, one elected lane issues); warps 2-9 produce (FP16 hi/lo planes); warps
// 10-17 drain (warp w reads TMEM lane quarter w % 4, the columns of half h of the tile's blocks
// with h = (w - 10) / 4); warps 18-19 scan windows. Every wait is an mbarrier wait bounded in
// time, polled by every lane of a waiting warp (measured: lane 0 polling alone and handing the
// result to the warp by a shuffle took 18 us longer at 63 taps, the hand-off latency landing on
// every K-step); a give-up sets the fault word and every role stops.
#include "fir_tc_win_kernel.cuh"

namespace rfx {

// Several cf32 captures with one tap set, each tile as in fir_tcw_kernel: the same bits as the capture
// alone where that takes the same tile (a tile's scale is taken over its own window).
template <int C, int NB>
__global__ void __launch_bounds__(tcw::kThreads, 1)
fir_tcw_shared_kernel(const __grid_constant__ tcw::SharedCaptures list)
{
    extern __shared__ __align__(1024) unsigned char smem[];
    tcw::Ctrl& ctl = *reinterpret_cast<tcw::Ctrl*>(smem);
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
    const tcw::TcwSharedSrc src{list};
    tcw::tcw_pipeline<C, 0, 8, tcw::TcwSharedSrc, 1, NB>(src, smem, ctl, tmem, &g_fault_fir_tcw);
    if (warp == tcw::kMmaWarp) {
        tc::tmem_dealloc(tmem, tcw::kTmemCols);
    }
}

bool fir_tcw_supported(int num_taps)
{
    return num_taps >= 2 && (num_taps + tcw::kB - 2) / tcw::kB <= tcw::kCMax &&
           tcw::win_layout((num_taps + tcw::kB - 2) / tcw::kB, 8, 1, 4).bytes <= tcw::kSmemMax;
}

// Form and tile by the time of the busiest SM (us, a step per tile fitted to measurements on 152 SMs;
// C = blocks reached back to). Resident window: a first tile through the whole pipeline, then one
// step per further tile; long-filter form (96 blocks a tile): one step per tile. So short captures
// take small tiles on more SMs, middling ones the tile that fills the last round, long ones the
// largest tile of the window form or, beyond 385 taps, the long-filter form where it is faster.
// Measured, 63 / 255 / 385 taps: one tile of 8, 16, 24, 32, 48 blocks 4.6 / 5.9 / 6.8, 5.0 / 6.2 / 7.1,
// 5.6 / 6.6 / 7.4, 5.8 / 7.0 / 7.3, 6.0 / 7.3 / 8.3, each further one 1.5 / 2.4 / 1.9 (8 blocks) to
// 2.3 / 3.0 / 3.8 (48); 511 / 1025 taps: 2^16 samples 7.6 / 10.5 (16 blocks) against 18.9 / 24.3 in the
// long-filter form, 2^20 12.5 / 18.3 (32) against 20.5 / 25.3, 2^22 31.9 / 51.2 against 50.6 / 58.6,
// 2^23 56.0 / 94.8 against 72.6 / 83.9, 2^24 101 / 175 against 118 / 138 (768 taps 143 against 125).
// The rule's choice was within 0.2 % of the best on average over 144 cases, 7 % at worst.
int fir_tcw_tile_blocks(int num_taps, long long n)
{
    int device = 0;
    int sms = 0;
    if (cudaGetDevice(&device) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess ||
        sms < 1) {
        cudaGetLastError();
        sms = 152;
    }
    const int C = (num_taps + tcw::kB - 2) / tcw::kB;
    const long long blocks = (n + tcw::kB - 1) / tcw::kB;
    auto rounds = [&](int nb) {
        const long long tiles = (blocks + nb - 1) / nb;
        return static_cast<double>((tiles + sms - 1) / sms);
    };
    int best = 0;
    double best_us = 1e30;
    if (!fir_tcw_supported(num_taps)) {
        const double r = rounds(96);
        best_us = 9.0 + r * (10.3 + 0.5 * C) + (r < 3.0 ? r - 1.0 : 2.0) * 3.0;
    }
    for (int nb : {48, 32, 24, 16, 8}) {
        if (!fir_tcw_takes(num_taps, nb)) {
            continue;
        }
        const double step = C <= tcw::kCMax ? 0.75 + 0.53 * C + (0.02 + 0.007 * C) * nb
                                            : 0.2 + 0.5 * C + (0.02 + 0.006 * C) * nb;
        const double us =
            4.0 + 0.75 * C + (0.045 + 0.004 * C) * nb + (rounds(nb) - 1.0) * step;
        if (us < best_us) {
            best_us = us;
            best = nb;
        }
    }
    return best;
}

template <int NB>
static cudaError_t launch_reach(int format, const void* x, const float* taps, void* y, long long n,
                                int num_taps, cudaStream_t stream)
{
    switch ((num_taps + tcw::kB - 2) / tcw::kB) {
    case 1: return launch_formats<1, NB>(format, x, taps, y, n, num_taps, stream);
    case 2: return launch_formats<2, NB>(format, x, taps, y, n, num_taps, stream);
    case 3: return launch_formats<3, NB>(format, x, taps, y, n, num_taps, stream);
    default: return cudaErrorInvalidValue;
    }
}

bool fir_tcw_takes(int num_taps, int tile_blocks)
{
    if (fir_tcw_supported(num_taps)) {
        return is_window_tile(tile_blocks);
    }
    const int C = (num_taps + tcw::kB - 2) / tcw::kB;
    return C > tcw::kCMax && C <= kTcWindowReach &&
           (tile_blocks == 16 || tile_blocks == 24 || tile_blocks == 32);
}

cudaError_t fir_tcw_launch(int tile_blocks, int format, const void* x, const float* taps, void* y,
                           long long n, int num_taps, cudaStream_t stream)
{
    if (n < tcw::kB || !fir_tcw_takes(num_taps, tile_blocks)) {
        return cudaErrorInvalidValue;
    }
    if (!fir_tcw_supported(num_taps)) {
        return fir_tcw_long_launch(tile_blocks, format, x, taps, y, n, num_taps, stream);
    }
    switch (tile_blocks) {
    case 8: return launch_reach<8>(format, x, taps, y, n, num_taps, stream);
    case 16: return launch_reach<16>(format, x, taps, y, n, num_taps, stream);
    case 24: return launch_reach<24>(format, x, taps, y, n, num_taps, stream);
    case 32: return launch_reach<32>(format, x, taps, y, n, num_taps, stream);
    case 48: return launch_reach<48>(format, x, taps, y, n, num_taps, stream);
    default: return cudaErrorInvalidValue;
    }
}

template <int C, int NB>
static cudaError_t launch_shared(tcw::SharedCaptures& list, int sms, cudaStream_t stream)
{
    const tcw::Layout lay = tcw::win_layout(C, 8, 1, 4, NB);
    const uint32_t bytes = lay.bytes > 120u * 1024u ? lay.bytes : 120u * 1024u;
    cudaError_t err = cudaFuncSetAttribute(fir_tcw_shared_kernel<C, NB>,
                                           cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           static_cast<int>(bytes));
    if (err != cudaSuccess) {
        return err;
    }
    list.tiles = 0;
    for (int c = 0; c < list.count; ++c) {
        tcw::WinCapture& cap = list.cap[c];
        err = encode_rows(&list.map[c], cap.x, 4, cap.n / tcw::kB, 2 * tcw::kB, 2 * tcw::kB,
                          static_cast<uint32_t>(NB + C));
        if (err != cudaSuccess) {
            return err;
        }
        cap.item0 = list.tiles;
        list.tiles += static_cast<int>(((cap.n + tcw::kB - 1) / tcw::kB + NB - 1) / NB);
    }
    const int grid = list.tiles < sms ? list.tiles : sms;
    return launch_overlapped(fir_tcw_shared_kernel<C, NB>, grid, tcw::kThreads, bytes, stream, list);
}

template <int NB>
static cudaError_t launch_shared_reach(tcw::SharedCaptures& list, int num_taps, int sms,
                                       cudaStream_t stream)
{
    switch ((num_taps + tcw::kB - 2) / tcw::kB) {
    case 1: return launch_shared<1, NB>(list, sms, stream);
    case 2: return launch_shared<2, NB>(list, sms, stream);
    case 3: return launch_shared<3, NB>(list, sms, stream);
    default: return cudaErrorInvalidValue;
    }
}

cudaError_t fir_tcw_shared_launch(int tile_blocks, const void* const* x, void* const* y,
                                  const int64_t* n, int count, const float* taps, int num_taps,
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
    if (!fir_tcw_supported(num_taps)) {
        return cudaErrorInvalidValue;
    }
    if (count < 1 || count > kTcSharedMax) {
        return cudaErrorInvalidValue;
    }
    tcw::SharedCaptures list;   // 11 KB
    list.count = count;
    long long total = 0;
    for (int c = 0; c < count; ++c) {
        if (n[c] < tcw::kB) {
            return cudaErrorInvalidValue;
        }
        list.cap[c] =
            tcw::WinCapture{x[c], static_cast<float2*>(y[c]), taps, n[c], num_taps, 0};
        total += n[c];
    }
    switch (tile_blocks != 0 ? tile_blocks : fir_tcw_tile_blocks(num_taps, total)) {
    case 8: return launch_shared_reach<8>(list, num_taps, sms, stream);
    case 16: return launch_shared_reach<16>(list, num_taps, sms, stream);
    case 24: return launch_shared_reach<24>(list, num_taps, sms, stream);
    case 32: return launch_shared_reach<32>(list, num_taps, sms, stream);
    case 48: return launch_shared_reach<48>(list, num_taps, sms, stream);
    default: return cudaErrorInvalidValue;
    }
}

cudaError_t fir_tcw_take_fault(unsigned int* code)
{
    unsigned int zero = 0;
    unsigned int more = 0;
    cudaError_t err = cudaMemcpyFromSymbol(code, g_fault_fir_tcw, sizeof(unsigned int));
    if (err != cudaSuccess ||
        (err = cudaMemcpyToSymbol(g_fault_fir_tcw, &zero, sizeof(unsigned int))) != cudaSuccess ||
        (err = fir_tcw_long_take_fault(&more)) != cudaSuccess) {
        return err;
    }
    *code |= more;
    return cudaSuccess;
}

}  // namespace rfx
