// transform kernels of the line lengths in PL_FFT_LEN1
#include "fft_kernels.cuh"

namespace pl {
PL_FFT_LEN1(PL_FFT_INSTANTIATE)
} // namespace pl
