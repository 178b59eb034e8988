// The resident-window FIR for filters that reach back 4 to 8 blocks (386 to 1025 taps): the form short
// captures of long filters take (fir_tc_win.cu has the algorithm and the rule).
#include "fir_tc_win_kernel.cuh"

namespace rfx {

template <int NB>
static cudaError_t launch_long(int format, const void* x, const float* taps, void* y, long long n,
                               int num_taps, cudaStream_t stream)
{
    static_assert(kTcWindowReach == 8, "reach-backs instantiated below");
    switch ((num_taps + tcw::kB - 2) / tcw::kB) {
    case 4: return launch_formats<4, NB>(format, x, taps, y, n, num_taps, stream);
    case 5: return launch_formats<5, NB>(format, x, taps, y, n, num_taps, stream);
    case 6: return launch_formats<6, NB>(format, x, taps, y, n, num_taps, stream);
    case 7: return launch_formats<7, NB>(format, x, taps, y, n, num_taps, stream);
    case 8: return launch_formats<8, NB>(format, x, taps, y, n, num_taps, stream);
    default: return cudaErrorInvalidValue;
    }
}

cudaError_t fir_tcw_long_launch(int tile_blocks, int format, const void* x, const float* taps,
                                void* y, long long n, int num_taps, cudaStream_t stream)
{
    switch (tile_blocks) {
    case 16: return launch_long<16>(format, x, taps, y, n, num_taps, stream);
    case 24: return launch_long<24>(format, x, taps, y, n, num_taps, stream);
    case 32: return launch_long<32>(format, x, taps, y, n, num_taps, stream);
    default: return cudaErrorInvalidValue;
    }
}

cudaError_t fir_tcw_long_take_fault(unsigned int* code)
{
    unsigned int zero = 0;
    cudaError_t err = cudaMemcpyFromSymbol(code, g_fault_fir_tcw, sizeof(unsigned int));
    if (err != cudaSuccess) {
        return err;
    }
    return cudaMemcpyToSymbol(g_fault_fir_tcw, &zero, sizeof(unsigned int));
}

}  // namespace rfx
