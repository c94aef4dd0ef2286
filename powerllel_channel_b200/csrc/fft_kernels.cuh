// fft_kernels.cuh -- the transform kernels compiled per line length, and their launchers
// (declared in fft_launch.cuh, instantiated in fft_len*.cu).
//
// Reference: src/src_c/mod_fft_fftw.inc (init_fft :35-90, execute_fft :92-95).
#pragma once

#include <algorithm>
#include <cstdint>

#include "fft_launch.cuh"

namespace pl {

// Compile-time-length version of k_xfft (same layout, same arithmetic): N is
// the line length, the batch per CTA is a constant, and the twiddle table is
// staged in shared memory.  Used for the strided (ghosted) layout of the
// host-pointer drop-in.
template <int N> __host__ __device__ constexpr int ct_x_lines() { return N >= 1024 ? 1 : 1024 / N; }

template <typename T, int N, bool FWD>
__global__ void __launch_bounds__(256) k_xfft_ct(const T *__restrict__ in, size_t in_off, size_t in_sj, size_t in_sk,
                                                 T *__restrict__ out, size_t out_off, size_t out_sj, size_t out_sk,
                                                 const typename cplx_of<T>::type *__restrict__ twg, int ny, T scale)
{
    pdl_enter();
    using V = typename cplx_of<T>::type;
    constexpr int NB = ct_x_lines<N>(), BUF = fpad_elems<V>(NB * N);
    extern __shared__ __align__(16) unsigned char smem_raw[];
    V *buf0 = reinterpret_cast<V *>(smem_raw);
    V *buf1 = buf0 + BUF;
    V *tw = buf1 + BUF;
    const int k = blockIdx.y;
    const int p0 = blockIdx.x * NB;
    const int nb = (NB == 1 ? 1 : min(NB, ny / 2 - p0));
    const int tid = threadIdx.x;
    ct_build_twiddles<V, N, 256>(twg, tw, tid);
    for (int e = tid; e < nb * 2 * N; e += 256) {
        const int m = e % N, r = (e / N) & 1, b = e / (2 * N);
        const int j = 2 * (p0 + b) + r;
        T val = in[in_off + (size_t)m + (size_t)j * in_sj + (size_t)k * in_sk];
        reinterpret_cast<T *>(&buf0[fpad<V>(b * N + m)])[r] = val;
    }
    __syncthreads();
    if (FWD) {
        V *res = ct_batch<V, true, false, N, NB, 1, N, 256>(buf0, buf1, nb, tw, tid);
        for (int e = tid; e < nb * N; e += 256) {
            const int m = e % N, b = e / N;
            V A = res[fpad<V>(b * N + m)], Bc = res[fpad<V>(b * N + (m == 0 ? 0 : N - m))];
            V h = split_hc(A, Bc, m, N);
            const int j = 2 * (p0 + b);
            out[out_off + (size_t)m + (size_t)j * out_sj + (size_t)k * out_sk] = h.x;
            out[out_off + (size_t)m + (size_t)(j + 1) * out_sj + (size_t)k * out_sk] = h.y;
        }
    } else {
        for (int e = tid; e < nb * N; e += 256) {
            const int m = e % N, b = e / N;
            V P = buf0[fpad<V>(b * N + m)], Q = buf0[fpad<V>(b * N + (m == 0 ? 0 : N - m))];
            buf1[fpad<V>(b * N + m)] = merge_hc(P, Q, m, N);
        }
        __syncthreads();
        V *res = ct_batch<V, false, false, N, NB, 1, N, 256>(buf1, buf0, nb, tw, tid);
        for (int e = tid; e < nb * N; e += 256) {
            const int m = e % N, b = e / N;
            V z = res[fpad<V>(b * N + m)];
            const int j = 2 * (p0 + b);
            out[out_off + (size_t)m + (size_t)j * out_sj + (size_t)k * out_sk] = z.x * scale;
            out[out_off + (size_t)m + (size_t)(j + 1) * out_sj + (size_t)k * out_sk] = z.y * scale;
        }
    }
}

// threadIdx.x through a volatile move: index arithmetic derived from it inside
// a persistent loop is recomputed per iteration instead of being hoisted and
// held in registers across the whole loop (which cost occupancy)
__device__ __forceinline__ int opaque_tid()
{
    int t;
    asm volatile("mov.u32 %0, %%tid.x;" : "=r"(t));
    return t;
}

// pressure update of one point o (PressureUpdate in ppe.cuh) from the increment dp, the staged
// prediction q and old pressure pold; the prediction is stored first (see pressure_update)
__device__ __forceinline__ void pressure_update_staged(const PressureUpdate &pu, size_t o, float dp, float q,
                                                       float pold)
{
    const float pn = (pu.incremental ? q : 0.f) + dp;
    pu.qnext[o] = pu.qmode ? 2.f * pn - pold : pn;
    pu.p[o] = pn;
}

// Persistent versions on the compact layout [k][j][i] (the device solves).
// Each CTA walks line groups g = blockIdx.x, + gridDim.x, ...  The raw data
// of the next group is copied global -> shared with cp.async into a staging
// buffer while the current group is transformed in place in the work
// buffer, so load latency overlaps the butterflies without holding the data
// in registers.  The staging copy into the work buffer pairs the two real
// lines into complex values (and, for the inverse, merges the half-complex
// spectra).  The y kernel moves whole 32-byte sectors: W column pairs of V
// per row (W * sizeof(V) = 64 bytes when N allows).
// (FP64 at N = 384: the forward transform measured faster with 8 columns,
// 0.173 -> 0.160 ms at 512x384x256, the inverse with 4, 0.177 against 0.182.)
// Short lines take more columns, so that a stage has work for the 256 threads.
// Long lines take whole 64-byte row segments at one CTA per SM rather than
// parts of them at two: FP32 at 1024x768x512, ny = 768, 4 -> 8 columns 1.015
// -> 0.868 ms forward, 1.026 -> 0.892 ms inverse.  FP64 lines of 432 to 512
// take two columns, 32-byte segments; no wider choice was measured there.
template <typename V, int N, bool FWD> __host__ __device__ constexpr int pf_y_cols()
{
    constexpr bool fp32 = sizeof(V) == 8;
    if (N <= 48) return 32;
    if (N <= 96) return 16;
    if (N >= 576) return fp32 ? 8 : 4;
    if (fp32) return 3072 / N >= 8 ? 8 : 4;
    return (FWD ? 3072 / N : 1536 / N) >= 8 ? 8 : (1536 / N >= 4 ? 4 : 2);
}

// threads per CTA of the persistent x kernel, and line pairs per group: one
// radix-8 stage of a group is one butterfly per thread
template <typename T> __host__ __device__ constexpr int pf_y_threads() { return 256; }
template <typename T> __host__ __device__ constexpr int pf_x_threads() { return sizeof(T) == 8 ? 64 : 256; }
template <typename T, int N> __host__ __device__ constexpr int pf_x_lines()
{
    return (pf_x_threads<T>() * 8 / N) < 1 ? 1 : pf_x_threads<T>() * 8 / N;
}
// shared memory of the persistent kernels, in V elements: work buffer,
// staging buffer (rounded to an even count), per-stage twiddle table
template <typename T, int N> __host__ __device__ constexpr int pf_x_smem_elems()
{
    using V = typename cplx_of<T>::type;
    return (fpad_elems<V>(pf_x_lines<T, N>() * N) + 1) / 2 * 2 + pf_x_lines<T, N>() * N + N;
}
// ... and with the mixed pressure update fused (FP32 inverse): the group's
// rows of the prediction q and of the old pressure, staged (bytes)
template <typename T, int N> __host__ __device__ constexpr int pf_x_pu_bytes()
{
    return 2 * 2 * pf_x_lines<T, N>() * N * 4;
}
template <typename T, int N, bool FWD> __host__ __device__ constexpr int pf_y_smem_elems()
{
    using V = typename cplx_of<T>::type;
    return (fpad_elems<V>(pf_y_cols<V, N, FWD>() * N) + 1) / 2 * 2 + pf_y_cols<V, N, FWD>() * N + N;
}

// PU (FP32 inverse only): the pressure update of the mixed path is fused
// into the last stage; the group's rows of q and of the old pressure are
// copied into shared memory when the group starts, so their latency hides
// behind its butterflies instead of sitting in the epilogue.
template <typename T, int N, bool FWD, bool PU = false>
__global__ void __launch_bounds__(pf_x_threads<T>()) k_xfft_pf(const T *__restrict__ in, T *__restrict__ out,
                                                               const typename cplx_of<T>::type *__restrict__ twg,
                                                               int ny, int total, T scale, PressureUpdate pu)
{
    pdl_enter();
    static_assert(!PU || (sizeof(T) == 4 && !FWD), "the fused pressure update is the FP32 inverse's");
    using V = typename cplx_of<T>::type;
    constexpr int NT = pf_x_threads<T>();
    constexpr int NB = pf_x_lines<T, N>(), BUF = (fpad_elems<V>(NB * N) + 1) / 2 * 2;
    constexpr int CH = 16 / sizeof(T); // T values per 16-byte copy
    extern __shared__ __align__(16) unsigned char smem_raw[];
    V *buf = reinterpret_cast<V *>(smem_raw);
    T *stage = reinterpret_cast<T *>(buf + BUF); // 2 NB rows of N values, 16-byte aligned
    V *tw = reinterpret_cast<V *>(stage + 2 * NB * N);
    float *pst = reinterpret_cast<float *>(tw + N); // PU: [2][2 NB N], q then the old pressure
    const int tid = threadIdx.x;
    const int gpk = (ny / 2 + NB - 1) / NB; // groups per k-plane
    ct_build_twiddles<V, N, NT>(twg, tw, tid);
    // PU: the group's rows of q and p (the run the group writes), one commit group
    auto fetch_pu = [&](int g) {
        const int k = g / gpk, p0 = (g % gpk) * NB, cnt = (NB == 1 ? 1 : min(NB, ny / 2 - p0)) * 2 * N;
        const size_t o = (size_t)k * N * ny + (size_t)2 * p0 * N;
        for (int e = tid * 4; e < cnt; e += NT * 4) {
            if (pu.incremental) cp_async_16(pst + e, pu.q + o + e);
            cp_async_16(pst + 2 * NB * N + e, pu.p + o + e);
        }
        cp_async_commit();
    };
    // rows 2 p0 .. 2 p0 + 2 nb - 1 of plane k are one contiguous run
    auto fetch = [&](int g) {
        const int k = g / gpk, p0 = (g % gpk) * NB, cnt = (NB == 1 ? 1 : min(NB, ny / 2 - p0)) * 2 * N;
        const T *src = in + (size_t)k * N * ny + (size_t)2 * p0 * N;
        for (int e = tid * CH; e < cnt; e += NT * CH) cp_async_16(stage + e, src + e);
        cp_async_commit();
    };
    if (blockIdx.x < total) fetch(blockIdx.x);
    for (int g = blockIdx.x; g < total; g += gridDim.x) {
        const int tid = opaque_tid();
        const int k = g / gpk, p0 = (g % gpk) * NB, nb = (NB == 1 ? 1 : min(NB, ny / 2 - p0));
        cp_async_wait<0>(); // this thread's copies of group g have landed
        __syncthreads();    // ... and everyone's; the previous group is done with buf (and pst)
        if (PU) fetch_pu(g);
        // first stage straight from the staged rows: line b pairs rows 2b, 2b+1
        auto in = [&](int b, int m) {
            const T *r0 = stage + 2 * b * N, *r1 = r0 + N;
            V z;
            if (FWD) {
                z.x = r0[m];
                z.y = r1[m];
            } else {
                const int mc = (m == 0) ? 0 : N - m;
                V P, Q;
                P.x = r0[m];
                P.y = r1[m];
                Q.x = r0[mc];
                Q.y = r1[mc];
                z = merge_hc(P, Q, m, N);
            }
            return z;
        };
        ct_first_stage<V, FWD, false, N, NB, 1, N, NT>(buf, nb, in, tid);
        __syncthreads();
        if (g + (int)gridDim.x < total)
            fetch(g + gridDim.x);
        else if (PU)
            cp_async_commit(); // one group after fetch_pu(g), as in the other rounds
        T *dst = out + (size_t)k * N * ny + (size_t)2 * p0 * N;
        if constexpr (FWD) {
            ct_batch_ip<V, FWD, false, N, NB, 1, N, NT, 1, ct_nstages(N) - 1>(buf, nb, tw, tid);
            // the last stage splits line b into its two half-complex rows from registers
            auto put = [&](int b, int m, V A, V Bc) {
                const V h = split_hc(A, Bc, m, N);
                dst[(size_t)2 * b * N + m] = h.x;
                dst[(size_t)(2 * b + 1) * N + m] = h.y;
            };
            ct_last_stage_pairs<V, FWD, false, N, NB, 1, N, NT>(buf, nb, tw, tid, put);
        } else {
            ct_batch_ip<V, FWD, false, N, NB, 1, N, NT, 1, ct_nstages(N) - 1>(buf, nb, tw, tid);
            if (PU) {
                cp_async_wait<1>(); // fetch_pu(g) landed (the next group's fetch may be in flight)
                __syncthreads();
            }
            // the last stage writes the two real rows of line b from registers
            auto put = [&](int b, int m, V z) {
                const T d0 = z.x * scale, d1 = z.y * scale;
                dst[(size_t)2 * b * N + m] = d0; // mixed: the increment itself, for the correction
                dst[(size_t)(2 * b + 1) * N + m] = d1;
                if (PU) {
                    const int r = 2 * b * N + m;
                    const size_t o = (size_t)k * N * ny + (size_t)2 * p0 * N + r;
                    pressure_update_staged(pu, o, (float)d0, pst[r], pst[2 * NB * N + r]);
                    pressure_update_staged(pu, o + N, (float)d1, pst[r + N], pst[2 * NB * N + r + N]);
                }
            };
            ct_last_stage<V, FWD, false, N, NB, 1, N, NT>(buf, nb, tw, tid, put);
        }
    }
    cp_async_wait<0>();
}

template <typename T, int N, bool FWD>
// CTAs per SM the register budget is cut for, as measured fastest at
// N = 384: up to 80 registers (three CTAs) for FP32 lines up to 512 and for
// the FP64 inverse (a spill of 4-16 bytes, served from L1, costs less than
// the third CTA gains), 128 (two) for the FP64 forward, which would spill
// 80 bytes at 80; longer lines keep more registers rather than spill
__global__ void __launch_bounds__(pf_y_threads<T>(),
                                  sizeof(T) == 4 ? (N <= 512 ? 3 : 2) : (N <= 512 ? (FWD ? 2 : 3) : 1))
    k_yfft_pf(T *__restrict__ data, const typename cplx_of<T>::type *__restrict__ twg, int nx, int total, PlaneSums ps)
{
    pdl_enter();
    using V = typename cplx_of<T>::type;
    constexpr int NT = pf_y_threads<T>();
    constexpr int W = pf_y_cols<V, N, FWD>(), BUF = (fpad_elems<V>(W * N) + 1) / 2 * 2, RAW = W * N;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int ncol = nx / 2;
    V *buf = reinterpret_cast<V *>(smem_raw);
    V *stage = buf + BUF; // [m][c], dense
    V *tw = stage + RAW;
    const int tid = threadIdx.x;
    const int gpk = (ncol + W - 1) / W;
    ct_build_twiddles<V, N, NT>(twg, tw, tid);
    auto fetch = [&](int g) {
        const int k = g / gpk, c0 = (g % gpk) * W, nb = min(W, ncol - c0);
        const V *plane = reinterpret_cast<const V *>(data) + (size_t)k * N * ncol;
        if (sizeof(V) == 8 && W % 2 == 0 && ncol % 2 == 0) {
            // FP32: two columns per 16-byte copy (c0 and c even, rows of even
            // length: 16-byte aligned); a lone last column takes an 8-byte one
            for (int e = 2 * tid; e < RAW; e += 2 * NT) {
                const int c = e % W, m = e / W;
                if (c + 1 < nb)
                    cp_async_16(stage + e, plane + (size_t)m * ncol + c0 + c);
                else if (c < nb)
                    cp_async_8(stage + e, plane + (size_t)m * ncol + c0 + c);
            }
        } else {
            for (int e = tid; e < RAW; e += NT) {
                const int c = e % W, m = e / W;
                if (c < nb) {
                    if (sizeof(V) == 16)
                        cp_async_16(stage + e, plane + (size_t)m * ncol + c0 + c);
                    else
                        cp_async_8(stage + e, plane + (size_t)m * ncol + c0 + c);
                }
            }
        }
        cp_async_commit();
    };
    if (blockIdx.x < total) fetch(blockIdx.x);
    if constexpr (FWD && sizeof(T) == 4) {
        // plane sums, while the first group's copies are in flight: launch_plane_sums' tree
        if (ps.part != nullptr) {
            __shared__ double sh[NT];
            for (int k = blockIdx.x; k < ps.nz; k += gridDim.x) {
                double sum = 0.0;
                for (int b = tid; b < ps.nper; b += NT) sum += __ldg(ps.part + (size_t)k * ps.nper + b);
                sh[tid] = sum;
                __syncthreads();
                for (int o = NT / 2; o > 0; o >>= 1) {
                    if (tid < o) sh[tid] += sh[tid + o];
                    __syncthreads();
                }
                if (tid == 0) ps.out[k] = sh[0];
                __syncthreads();
            }
        }
    }
    for (int g = blockIdx.x; g < total; g += gridDim.x) {
        const int k = g / gpk, c0 = (g % gpk) * W, nb = min(W, ncol - c0);
        V *plane = reinterpret_cast<V *>(data) + (size_t)k * N * ncol;
        cp_async_wait<0>();
        __syncthreads();
        // first stage straight from the staged columns ([m][c])
        auto in = [&](int c, int m) {
            if (FWD) return stage[m * W + c];
            return merge_hc(stage[m * W + c], stage[(m == 0 ? 0 : N - m) * W + c], m, N);
        };
        ct_first_stage<V, FWD, true, N, W, W, 1, NT>(buf, nb, in, tid);
        __syncthreads();
        if (g + (int)gridDim.x < total) fetch(g + gridDim.x);
        if constexpr (FWD) {
            ct_batch_ip<V, FWD, true, N, W, W, 1, NT, 1, ct_nstages(N) - 1>(buf, nb, tw, tid);
            auto put = [&](int c, int m, V A, V Bc) { plane[(size_t)m * ncol + c0 + c] = split_hc(A, Bc, m, N); };
            ct_last_stage_pairs<V, FWD, true, N, W, W, 1, NT>(buf, nb, tw, tid, put);
        } else {
            ct_batch_ip<V, FWD, true, N, W, W, 1, NT, 1, ct_nstages(N) - 1>(buf, nb, tw, tid);
            auto put = [&](int c, int m, V z) { plane[(size_t)m * ncol + c0 + c] = z; };
            ct_last_stage<V, FWD, true, N, W, W, 1, NT>(buf, nb, tw, tid, put);
        }
    }
    cp_async_wait<0>();
}
// calcRHS (mod_calcRHS.f90:19-33) fused into the forward x transform.  One
// group is xdiv_lines(N) line pairs (pair p: rows 2p, 2p+1 of interior plane
// k); its staging holds, as FP64 rows of the ghosted fields (plane kg = k + 1),
// the pairs' u, v and w rows, the v row below the first (periodic), and the w
// rows of plane kg - 1.  The first Stockham stage forms rhs = div(u)/dt
// with k_calc_rhs_fp64's expression (u_{i-1} is in the same periodic row)
// and pairs them into one complex line, so neither the right-hand side nor
// its re-read crosses HBM.  When `part` is given, each group also writes the
// FP64 sum of its rhs values (in a fixed order) for the plane sums of the
// mixed path's (0,0) mode.
// one radix-8 butterfly of a stage per thread, up to 128 threads
template <int N> __host__ __device__ constexpr int xdiv_threads() { return N > 512 ? 128 : 64; }

template <typename T, int N> __host__ __device__ constexpr int xdiv_smem_bytes()
{
    using V = typename cplx_of<T>::type;
    constexpr int NB = xdiv_lines(N);
    // work buffer, 8 NB + 1 staged FP64 rows, per-stage twiddles, warp sums
    return (int)(sizeof(V) * ((fpad_elems<V>(NB * N) + 1) / 2 * 2) + 8 * (8 * NB + 1) * N + sizeof(V) * N + 32);
}

template <typename T, int N>
__global__ void __launch_bounds__(xdiv_threads<N>()) k_xfft_div_pf(DivIn d, T *__restrict__ out,
                                                              const typename cplx_of<T>::type *__restrict__ twg,
                                                              int ny, int total, double *__restrict__ part)
{
    pdl_enter();
    using V = typename cplx_of<T>::type;
    constexpr int NT = xdiv_threads<N>(), NB = xdiv_lines(N), BUF = (fpad_elems<V>(NB * N) + 1) / 2 * 2;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    V *buf = reinterpret_cast<V *>(smem_raw);
    // rows of a group of nb <= NB line pairs: u (2 NB) | v (the row below, 2 NB) | w (2 NB) | w below (2 NB)
    double *su = reinterpret_cast<double *>(buf + BUF), *sv = su + 2 * NB * N, *sw = sv + (2 * NB + 1) * N,
           *sm = sw + 2 * NB * N;
    V *tw = reinterpret_cast<V *>(sm + 2 * NB * N);
    double *wsum = reinterpret_cast<double *>(tw + N);
    const int tid = threadIdx.x;
    const int gpk = (ny / 2 + NB - 1) / NB; // groups per plane
    const size_t sk = (size_t)N * ny;
    ct_build_twiddles<V, N, NT>(twg, tw, tid);
    auto copy_rows = [&](double *dst, const double *src, int n) {
        for (int e = tid * 2; e < n; e += NT * 2) cp_async_16(dst + e, src + e);
    };
    auto fetch = [&](int g) {
        const int k = g / gpk, p = (g % gpk) * NB, kg = k + 1, nb = NB == 1 ? 1 : min(NB, ny / 2 - p);
        const size_t r0 = sk * kg + (size_t)2 * p * N;
        copy_rows(su, d.u + r0, 2 * nb * N);
        copy_rows(sv, d.v + sk * kg + (size_t)(p == 0 ? ny - 1 : 2 * p - 1) * N, N);
        copy_rows(sv + N, d.v + r0, 2 * nb * N);
        copy_rows(sw, d.w + r0, 2 * nb * N);
        copy_rows(sm, d.w + r0 - sk, 2 * nb * N);
        cp_async_commit();
    };
    if (blockIdx.x < total) fetch(blockIdx.x);
    for (int g = blockIdx.x; g < total; g += gridDim.x) {
        const int k = g / gpk, p = (g % gpk) * NB, nb = NB == 1 ? 1 : min(NB, ny / 2 - p);
        const double dtidzi_k = __ldg(d.dzf_inv + k + 1);
        cp_async_wait<0>();
        __syncthreads();
        double acc = 0.0;
        auto in = [&](int b, int m) {
            const int mm = (m == 0) ? N - 1 : m - 1;
            if (NB == 1) b = 0; // known at compile time
            const double *u0 = su + 2 * b * N, *u1 = u0 + N, *vm = sv + 2 * b * N, *v0 = vm + N, *v1 = v0 + N;
            const double *w0 = sw + 2 * b * N, *w1 = w0 + N, *w0m = sm + 2 * b * N, *w1m = w0m + N;
            const double r0 = (u0[m] - u0[mm]) * d.dtidxi + (v0[m] - vm[m]) * d.dtidyi + (w0[m] - w0m[m]) * d.dti * dtidzi_k;
            const double r1 = (u1[m] - u1[mm]) * d.dtidxi + (v1[m] - v0[m]) * d.dtidyi + (w1[m] - w1m[m]) * d.dti * dtidzi_k;
            acc += r0 + r1;
            V z;
            z.x = (T)r0;
            z.y = (T)r1;
            return z;
        };
        ct_first_stage<V, true, false, N, NB, 1, N, NT>(buf, nb, in, tid);
        if (part != nullptr) { // the group's sum, in a fixed order
            for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
            if ((tid & 31) == 0) wsum[tid >> 5] = acc;
        }
        __syncthreads();
        if (part != nullptr && tid == 0)
            part[g] = NT == 64 ? wsum[0] + wsum[1] : (wsum[0] + wsum[1]) + (wsum[2] + wsum[3]);
        if (g + (int)gridDim.x < total) fetch(g + gridDim.x);
        T *dst = out + (size_t)k * N * ny + (size_t)2 * p * N;
        ct_batch_ip<V, true, false, N, NB, 1, N, NT, 1, ct_nstages(N) - 1>(buf, nb, tw, tid);
        auto put = [&](int b, int m, V A, V Bc) {
            if (NB == 1) b = 0;
            const V h = split_hc(A, Bc, m, N);
            dst[(size_t)2 * b * N + m] = h.x;
            dst[(size_t)(2 * b + 1) * N + m] = h.y;
        };
        ct_last_stage_pairs<V, true, false, N, NB, 1, N, NT>(buf, nb, tw, tid, put);
    }
    cp_async_wait<0>();
}

// shared memory (bytes) of the kernels of a length
template <typename T, int N> constexpr size_t x_pf_bytes() { return sizeof(typename cplx_of<T>::type) * (size_t)pf_x_smem_elems<T, N>(); }
template <typename T, int N> constexpr size_t x_ct_bytes()
{
    using V = typename cplx_of<T>::type;
    return sizeof(V) * (2 * (size_t)fpad_elems<V>(ct_x_lines<N>() * N) + N);
}
template <typename T, int N, bool FWD> constexpr size_t y_pf_bytes()
{
    return sizeof(typename cplx_of<T>::type) * (size_t)pf_y_smem_elems<T, N, FWD>();
}
template <typename T, int N> int x_pf_groups(const Ppe *s) { return ((s->ny / 2 + pf_x_lines<T, N>() - 1) / pf_x_lines<T, N>()) * s->nz; }
template <typename T, int N, bool FWD> int y_pf_groups(const Ppe *s)
{
    constexpr int W = pf_y_cols<typename cplx_of<T>::type, N, FWD>();
    return ((s->nx / 2 + W - 1) / W) * s->nz;
}
template <int N> int xdiv_groups(const Ppe *s) { return ((s->ny / 2 + xdiv_lines(N) - 1) / xdiv_lines(N)) * s->nz; }

// the kernel's shared-memory limit and its grid: all groups, or what the chip holds at once
template <typename K> int persistent_grid(K kernel, size_t shm, int total, int threads, int *grid)
{
    if (shm > 48 * 1024)
        PL_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)shm));
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, shm) != cudaSuccess || per_sm < 1)
        per_sm = 1;
    *grid = std::max(1, std::min(total, per_sm * sm_count()));
    return 0;
}

template <typename T, int N> int prepare_x_ct(Ppe *s)
{
    constexpr int NT = pf_x_threads<T>();
    const int groups = x_pf_groups<T, N>(s);
    if (x_ct_bytes<T, N>() > 48 * 1024) {
        PL_CUDA_TRY(cudaFuncSetAttribute(k_xfft_ct<T, N, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)x_ct_bytes<T, N>()));
        PL_CUDA_TRY(cudaFuncSetAttribute(k_xfft_ct<T, N, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)x_ct_bytes<T, N>()));
    }
    if (persistent_grid(k_xfft_pf<T, N, true>, x_pf_bytes<T, N>(), groups, NT, &s->grid_x[0]) ||
        persistent_grid(k_xfft_pf<T, N, false>, x_pf_bytes<T, N>(), groups, NT, &s->grid_x[1]) ||
        persistent_grid(k_xfft_div_pf<T, N>, xdiv_smem_bytes<T, N>(), xdiv_groups<N>(s), xdiv_threads<N>(), &s->grid_x[3]))
        return -1;
    if constexpr (sizeof(T) == 4)
        return persistent_grid(k_xfft_pf<T, N, false, true>, x_pf_bytes<T, N>() + pf_x_pu_bytes<T, N>(), groups, NT,
                               &s->grid_x[2]);
    return 0;
}

template <typename T, int N> int prepare_y_ct(Ppe *s)
{
    constexpr int NT = pf_y_threads<T>();
    return persistent_grid(k_yfft_pf<T, N, true>, y_pf_bytes<T, N, true>(), y_pf_groups<T, N, true>(s), NT, &s->grid_y[0]) ||
                   persistent_grid(k_yfft_pf<T, N, false>, y_pf_bytes<T, N, false>(), y_pf_groups<T, N, false>(s), NT,
                                   &s->grid_y[1])
               ? -1
               : 0;
}

template <typename T, int N, bool FWD>
int launch_x_ct(const Ppe *s, const T *in, size_t in_off, size_t in_sj, size_t in_sk, T *out, size_t out_off,
                size_t out_sj, size_t out_sk, T scale, cudaStream_t st, const PressureUpdate *pu, bool *fused)
{
    using V = typename cplx_of<T>::type;
    const V *tw = reinterpret_cast<const V *>(sizeof(T) == 8 ? (const void *)s->d_twx64 : (const void *)s->d_twx32);
    const size_t sk = (size_t)N * s->ny;
    const bool aligned = ((uintptr_t)in % 16 == 0) && ((uintptr_t)out % 16 == 0);
    *fused = false;
    if (aligned && in_off == 0 && out_off == 0 && in_sj == (size_t)N && out_sj == (size_t)N && in_sk == sk &&
        out_sk == sk) {
        constexpr int NT = pf_x_threads<T>();
        const int groups = x_pf_groups<T, N>(s);
        if constexpr (sizeof(T) == 4 && !FWD) {
            if (pu != nullptr) {
                *fused = true;
                PL_CUDA_TRY(launch_chained(k_xfft_pf<T, N, false, true>, s->grid_x[2], NT,
                                           x_pf_bytes<T, N>() + pf_x_pu_bytes<T, N>(), st, in, out, tw, s->ny, groups,
                                           scale, *pu));
                return 0;
            }
        }
        PL_CUDA_TRY(launch_chained(k_xfft_pf<T, N, FWD>, s->grid_x[FWD ? 0 : 1], NT, x_pf_bytes<T, N>(), st, in, out,
                                   tw, s->ny, groups, scale, PressureUpdate{}));
        return 0;
    }
    constexpr int NB = ct_x_lines<N>();
    PL_CUDA_TRY(launch_chained(k_xfft_ct<T, N, FWD>, dim3((s->ny / 2 + NB - 1) / NB, s->nz), 256, x_ct_bytes<T, N>(), st,
                               in, in_off, in_sj, in_sk, out, out_off, out_sj, out_sk, tw, s->ny, scale));
    return 0;
}

template <typename T, int N, bool FWD> int launch_y_ct(const Ppe *s, T *data, cudaStream_t st, const PlaneSums &ps)
{
    using V = typename cplx_of<T>::type;
    const V *tw = reinterpret_cast<const V *>(sizeof(T) == 8 ? (const void *)s->d_twy64 : (const void *)s->d_twy32);
    PL_CUDA_TRY(launch_chained(k_yfft_pf<T, N, FWD>, s->grid_y[FWD ? 0 : 1], pf_y_threads<T>(), y_pf_bytes<T, N, FWD>(),
                               st, data, tw, s->nx, y_pf_groups<T, N, FWD>(s), ps));
    return 0;
}

template <typename T, int N> int launch_xdiv(Ppe *s, const DivIn &d, T *out, double *part, cudaStream_t st)
{
    using V = typename cplx_of<T>::type;
    const V *tw = reinterpret_cast<const V *>(sizeof(T) == 8 ? (const void *)s->d_twx64 : (const void *)s->d_twx32);
    PL_CUDA_TRY(launch_chained(k_xfft_div_pf<T, N>, s->grid_x[3], xdiv_threads<N>(), xdiv_smem_bytes<T, N>(), st, d, out, tw,
                               s->ny, xdiv_groups<N>(s), part));
    return 0;
}

#define PL_FFT_INSTANTIATE_T(T, n)                                                                                     \
    template int prepare_x_ct<T, n>(Ppe *);                                                                            \
    template int prepare_y_ct<T, n>(Ppe *);                                                                            \
    template int launch_x_ct<T, n, true>(const Ppe *, const T *, size_t, size_t, size_t, T *, size_t, size_t, size_t,  \
                                         T, cudaStream_t, const PressureUpdate *, bool *);                             \
    template int launch_x_ct<T, n, false>(const Ppe *, const T *, size_t, size_t, size_t, T *, size_t, size_t, size_t, \
                                          T, cudaStream_t, const PressureUpdate *, bool *);                            \
    template int launch_y_ct<T, n, true>(const Ppe *, T *, cudaStream_t, const PlaneSums &);                           \
    template int launch_y_ct<T, n, false>(const Ppe *, T *, cudaStream_t, const PlaneSums &);                          \
    template int launch_xdiv<T, n>(Ppe *, const DivIn &, T *, double *, cudaStream_t);
#define PL_FFT_INSTANTIATE(n) PL_FFT_INSTANTIATE_T(double, n) PL_FFT_INSTANTIATE_T(float, n)

} // namespace pl
