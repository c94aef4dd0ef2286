// transform kernels of the line lengths in PL_FFT_LEN2
#include "fft_kernels.cuh"

namespace pl {
PL_FFT_LEN2(PL_FFT_INSTANTIATE)
} // namespace pl
