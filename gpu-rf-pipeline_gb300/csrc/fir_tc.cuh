// Tensor-core FIR (fir_tc.cu) and the per-capture batch (fir_batch.cu): internal interface.
#pragma once

#include "rfx.h"

#include <cuda_runtime.h>

namespace rfx {

// Form and tile shape of the tensor-core FIR, chosen by the tuner.
struct TcConfig {
    int tile_blocks;  // 128-output blocks per tile: 96 = one CTA per tile (fir_tc.cu),
                      // 192 = a CTA pair per tile of 96 256-output blocks (fir_tc2.cu),
                      // 8, 16, 24, 32 or 48 = the resident-window form, 2 to 385 taps, and 16,
                      // 24 or 32 up to 1025 (fir_tc_win.cu)
    int stages;       // operand ring depth cap (the largest that fits is used)
};
constexpr int kTcPairTile = 192;

// Whether a tile shape is the resident-window form's.
constexpr bool is_window_tile(int tile_blocks)
{
    return tile_blocks == 8 || tile_blocks == 16 || tile_blocks == 24 || tile_blocks == 32 ||
           tile_blocks == 48;
}

constexpr int kTcBatchMax = 4096;

// Whether the tensor-core kernel takes this tap count. One tap is an exact elementwise scale,
// which the plain kernel computes exactly; the split form would round it.
bool fir_tc_supported(int num_taps);

cudaError_t fir_tc_launch(const void* x, const float* taps, void* y, long long n, int num_taps,
                          TcConfig config, cudaStream_t stream);
cudaError_t fir_tc_take_fault(unsigned int* code);

// The resident-window form (fir_tc_win.cu): 2 to 385 taps (fir_tcw_supported), for short captures
// up to 1025 (fir_tcw_takes says which tiles), tiles of `tile_blocks` blocks whose
// whole input window arrives by one TMA copy; format 0 cf32, 1 ci16, 2 ci8 (decoded in the load stage, the
// same bits as over the converted samples). n >= 128.
bool fir_tcw_supported(int num_taps);
bool fir_tcw_takes(int num_taps, int tile_blocks);
cudaError_t fir_tcw_launch(int tile_blocks, int format, const void* x, const float* taps, void* y,
                           long long n, int num_taps, cudaStream_t stream);
// Its instances for 386 to 1025 taps (fir_tc_win_long.cu).
constexpr int kTcWindowReach = 8;   // blocks of 128 outputs a block may reach back
cudaError_t fir_tcw_long_launch(int tile_blocks, int format, const void* x, const float* taps,
                                void* y, long long n, int num_taps, cudaStream_t stream);
cudaError_t fir_tcw_long_take_fault(unsigned int* code);
// Up to kTcSharedMax captures sharing one tap set (cf32, each of at least 128 samples, none
// touching what another writes) in one launch, in tiles of `tile_blocks` blocks (0: by the built-in
// rule over all their samples).
constexpr int kTcSharedMax = 64;
cudaError_t fir_tcw_shared_launch(int tile_blocks, const void* const* x, void* const* y,
                                  const int64_t* n, int count, const float* taps, int num_taps,
                                  cudaStream_t stream);
// The tile the form takes for a capture of n samples by the built-in rule; 0 where the form for long
// filters (fir_tc.cu) is the faster one.
int fir_tcw_tile_blocks(int num_taps, long long n);
cudaError_t fir_tcw_take_fault(unsigned int* code);

// The same FIR over integer I/Q input decoded in the load stage (format 1 = ci16, 2 = ci8; 0 =
// cf32, fir_tc_launch): the copies move the stored components, the producers convert them as
// the project's SigMF reader does. Results have the bits of fir_tc_launch over the converted
// samples in the single-CTA form (the form integer input always takes).
cudaError_t fir_tc_launch_format(int format, const void* x, const float* taps, void* y,
                                 long long n, int num_taps, TcConfig config, cudaStream_t stream);
long long fir_tc_tile_outputs_format(int format, int num_taps, long long n, TcConfig config);

// Outputs per tile of the form fir_tc_launch picks for (num_taps, n, config): tiles start at
// multiples of this, and each tile's results depend only on the samples from one tile before
// its start to its end (its window reaches back C blocks, C * 128 <= 3456 < one tile), so a
// run over any tile-aligned stretch with one tile of history reproduces the whole run's bits
// there. 1 when the plain kernel runs instead.
long long fir_tc_tile_outputs(int num_taps, long long n, TcConfig config);

// Per-capture-taps batch: tensor core (or auto) = one persistent launch of fir_batch.cu per
// 96 captures; plain = one launch per capture.
cudaError_t fir_batch_launch(int impl, const rfx_fir_capture* captures, int count,
                             cudaStream_t stream);
cudaError_t fir_batch_tc_launch(const rfx_fir_capture* captures, int count, cudaStream_t stream);
bool fir_batch_supported(int num_taps);

// A batch plan: the work list of one batch (capture tables, tensor maps, per-block ranges) in
// device memory, built once; every run is ONE persistent launch of fir_batch.cu that takes the
// tensor-core captures and, with groups of its threads, the plain captures' tiles.
struct BatchPlan;
cudaError_t fir_batch_plan_make(int impl, const rfx_fir_capture* captures, int count,
                                BatchPlan** out);
cudaError_t fir_batch_plan_run(const BatchPlan* plan, cudaStream_t stream);
void fir_batch_plan_free(BatchPlan* plan);
void fir_batch_plan_counts(const BatchPlan* plan, int* tc_captures, int* plain_captures,
                           int* launches);
cudaError_t fir_batch_take_fault(unsigned int* code);

}  // namespace rfx
