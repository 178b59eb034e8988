// The tuned-configuration tables consulted by RFX_FIR_AUTO, the tensor-core FIR launches and
// RFX_CHAN_AUTO plans (tuning.cu), filled by rfx_autotune_fir / rfx_autotune_channelize and
// persisted with rfx_autotune_save/load.
#pragma once

#include "fir_tc.cuh"

namespace rfx {

int tuned_fir_impl(int num_taps, long long n);
int tuned_fir_batch_impl(int num_taps, long long n);
int tuned_fir_batch_launch_impl(int num_taps, long long n);
TcConfig tuned_fir_tc_config(int num_taps, long long n);
// Whether a tuned entry names the tensor-core form for this case, and its configuration.
bool tuned_fir_tc_entry(int num_taps, long long n, TcConfig* config);
// *fused: the plan's calls of any length that the fused FP32 kernel takes run it (64 channels, no tuned
// entry for the tensor-core form). The result then says what becomes of the others: RFX_CHAN_TC, no
// tuned entry, refused as the tensor-core form's plans refuse them; RFX_CHAN_PLAIN, tuned, the plain form.
int tuned_chan_impl(int channels, long long n, bool* fused);

}  // namespace rfx
