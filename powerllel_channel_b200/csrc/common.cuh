// common.cuh -- shared definitions of the B200 channel-flow step library.
//
// Device layout (all fields, both precisions): x fastest, then y, then z.
//   velocity-like fields  [k = 0 .. nz+1][j = 0 .. ny-1][i = 0 .. nx-1]
//       (wall ghost planes k = 0 and k = nz+1 are stored; x and y are periodic
//        and are indexed modulo nx / ny, so no x/y ghost cells exist)
//   pressure / PPE work    [k = 0 .. nz-1][j][i]   (interior only)
// The reference's ghosted Fortran array u(0:nx+1,0:ny+1,0:nz+1)
// (mod_variables.f90:21-41) maps to this layout by dropping the x/y ghosts,
// which on one rank always equal the periodic images of the interior
// (imposePeriodicBC, mod_updateBound.f90:241-272, and the self-exchange of
// updateHalo, :364-396).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <cstdio>
#include <string>

namespace pl {

// last error message of the calling host thread (C ABI: pl_last_error)
void set_error(const std::string &msg);
const char *get_error();

#define PL_CUDA_TRY(expr)                                                                  \
    do {                                                                                   \
        cudaError_t _e = (expr);                                                           \
        if (_e != cudaSuccess) {                                                           \
            ::pl::set_error(std::string(#expr) + ": " + cudaGetErrorString(_e) + " at " +  \
                            __FILE__ + ":" + std::to_string(__LINE__));                    \
            return -1;                                                                     \
        }                                                                                  \
    } while (0)

#define PL_CHECK_LAUNCH()                                                                  \
    do {                                                                                   \
        cudaError_t _e = cudaGetLastError();                                               \
        if (_e != cudaSuccess) {                                                           \
            ::pl::set_error(std::string("kernel launch: ") + cudaGetErrorString(_e) +      \
                            " at " + __FILE__ + ":" + std::to_string(__LINE__));           \
            return -1;                                                                     \
        }                                                                                  \
    } while (0)

// Launch of a kernel that begins with pdl_enter(): its launch is prepared while
// the stream's previous kernel runs, and its CTAs start as that one's end.  The
// step is a chain of seven short kernels, whose launch latencies add up on
// small grids.
template <typename... K, typename... A>
inline cudaError_t launch_chained(void (*kern)(K...), dim3 grid, dim3 block, size_t shm, cudaStream_t st, A &&...args)
{
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = shm;
    cfg.stream = st;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kern, static_cast<K>(args)...);
}

// First statement of such a kernel: waits until the previous kernel of the
// stream has completed and its writes are visible (it waited for its own
// predecessor in turn).  Without the launch attribute it is a no-op.  The next
// kernel is released by this one's end: releasing it here as well
// (griddepcontrol.launch_dependents) let its waiting CTAs take the room and
// the shared-memory split that the running kernel's own tail needs, and cost
// more than the launches it hid (step back to back, us: plain launches 50.4,
// wait alone 36.8, early release 42.8 at 64x64x64; 334, 316 and 350 at
// 256x192x128 PDD-4; 2435, 2428 and 2592 at 512x384x256, all FP64).
__device__ __forceinline__ void pdl_enter()
{
    asm volatile("griddepcontrol.wait;\n" ::: "memory");
}

template <typename T> struct cplx_of;
template <> struct cplx_of<double> { using type = double2; };
template <> struct cplx_of<float> { using type = float2; };

template <typename V>
__host__ __device__ __forceinline__ V cmul(V a, V b)
{
    V r;
    r.x = a.x * b.x - a.y * b.y;
    r.y = a.x * b.y + a.y * b.x;
    return r;
}

// a * conj(b)
template <typename V>
__host__ __device__ __forceinline__ V cmulc(V a, V b)
{
    V r;
    r.x = a.x * b.x + a.y * b.y;
    r.y = a.y * b.x - a.x * b.y;
    return r;
}

template <typename V> __host__ __device__ __forceinline__ V cadd(V a, V b)
{
    V r;
    r.x = a.x + b.x;
    r.y = a.y + b.y;
    return r;
}

template <typename V> __host__ __device__ __forceinline__ V csub(V a, V b)
{
    V r;
    r.x = a.x - b.x;
    r.y = a.y - b.y;
    return r;
}

__host__ __device__ __forceinline__ size_t idx3(int i, int j, int k, int nx, int ny)
{
    return (size_t)i + (size_t)nx * ((size_t)j + (size_t)ny * (size_t)k);
}

} // namespace pl
