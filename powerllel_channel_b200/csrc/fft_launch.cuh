// fft_launch.cuh -- launchers of the transform kernels compiled per line length (fft_kernels.cuh),
// instantiated in fft_len*.cu so that the lengths compile side by side.
#pragma once

#include <algorithm>

#include "ppe.cuh"

namespace pl {

// Line lengths with compile-time kernels: every even 2^a 3^b from 16 to 1024.
// Shorter and longer lines use the runtime-length kernels (ppe.cu).
#define PL_FFT_LEN1(X) X(64) X(128) X(192) X(256) X(16) X(18) X(24) X(32) X(36) X(48)
#define PL_FFT_LEN2(X) X(384) X(512) X(54) X(72) X(96) X(108) X(144)
#define PL_FFT_LEN3(X) X(768) X(162) X(216) X(288) X(324) X(432)
#define PL_FFT_LEN4(X) X(1024) X(486) X(576) X(648) X(864) X(972)
#define PL_FFT_CT_SIZES(X) PL_FFT_LEN1(X) PL_FFT_LEN2(X) PL_FFT_LEN3(X) PL_FFT_LEN4(X)

inline int sm_count()
{
    static int n = 0;
    if (n == 0) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
        if (n <= 0) n = 1;
    }
    return n;
}

// per plan: shared-memory limits and persistent grids of the kernels below
template <typename T, int N> int prepare_x_ct(Ppe *s);
template <typename T, int N> int prepare_y_ct(Ppe *s);
// x transform (fused: whether the pressure update ran with it)
template <typename T, int N, bool FWD>
int launch_x_ct(const Ppe *s, const T *in, size_t in_off, size_t in_sj, size_t in_sk, T *out, size_t out_off,
                size_t out_sj, size_t out_sk, T scale, cudaStream_t st, const PressureUpdate *pu, bool *fused);
// y transform, in place (ps: the plane sums that a forward one forms as well)
template <typename T, int N, bool FWD> int launch_y_ct(const Ppe *s, T *data, cudaStream_t st, const PlaneSums &ps);
// calcRHS and the forward x transform
template <typename T, int N> int launch_xdiv(Ppe *s, const DivIn &d, T *out, double *part, cudaStream_t st);

// line pairs per group of launch_xdiv: short lines are taken several at a
// time, one radix-8 butterfly per thread
__host__ __device__ constexpr int xdiv_lines(int n) { return n < 192 ? 512 / n : 1; }

} // namespace pl
