// rk_mixed.cu -- the mixed-precision path's fused RK2 kernel: both stages of
// timeIntVelRK1 / timeIntVelRK2 (mod_calcVel.f90:52-146, 240-334) with their
// wall fills, in FP32 flux form.
//
// The tile and the flux form are the FP64 kernel's (rk_fused.cu): a 32 x 16
// tile whose 256 threads own two x-adjacent points each, rings of u, v, w
// (FP32, halo 2) and of the stage-1 field u1 = u + d1 (FP32, halo 1), one z flux
// per face carried up the march.  HBM sees u, v, w read once, the new fields
// written once and the FP32 pressure prediction read once.  What differs:
//   * the kernel waits more than it computes (half its issue slots are used, at
//     the 16 warps that its registers allow), so what shortens a plane's chain
//     of loads counts: the points of a pair are evaluated in packed FP32 (one
//     two-lane instruction for both, each lane rounded as the scalar
//     operation), pairs move as 8-byte shared and 16-byte global accesses, and
//     stage 2's operands and the prediction (read by this kernel alone, so cold)
//     are fetched ahead of stage 1's barrier and planes ahead into L2;
//   * two planes per ring and two barriers per plane: stage 1 on plane k, then
//     stage 2 on plane k-1 and the conversion of plane k+2.  Three planes, one
//     barrier and stage 2 a plane later keep d1 and the centres in registers
//     for longer and were slower (0.767 against 0.821 ms at 512x384x256); a third
//     CTA per SM at 80 registers (0.806), four points per thread (1.22) and a
//     warp-specialised split of the stages (1.09) were slower as well;
//   * the FP64 planes arrive in a staging area by 16-byte cp.async copies a
//     plane ahead; each thread converts the pairs that it copied itself, so the
//     conversion waits on the thread's own copies only;
//   * the stage-1 increment d1 = dt RHS(u) of the tile's own points stays in
//     the thread's registers from stage 1 of plane k to stage 2 of plane k
//     (the thread that forms it consumes it), so only u1 goes through
//     shared memory.
// 512x384x256: 0.902 -> 0.743 ms (54 % of the measured copy bandwidth at
// 52 B/point); 256x192x128 0.135 -> 0.095; 1024x768x512 6.21 -> 5.24-5.56; 64x64x64
// 0.041 -> 0.017; 324x162x150, which ran two stage kernels, 0.622 -> 0.223 ms
// (WIDE below).
//
// Stage 2 forms u_hat = u + [ (d1 + d2)/2 - dt G p_pred ] with the bracket in
// FP32 (WIDE: in FP64) and the sum in FP64: u, v, w stay FP64, and the projection residual of
// the increment solve is the FP64 divergence of the stored u_hat, whatever
// rounding the bracket carries.
#include <type_traits>

#include "fft.cuh" // cp.async helpers
#include "stencil.cuh"
#include "stencil_rhs.cuh"

namespace pl {

namespace {

constexpr int MX = 32, MY = 16;         // tile; each thread owns two x-adjacent points
constexpr int MT = 256;                 // threads
constexpr int MW = 36, MH = MY + 4;     // ring plane with a halo of 2
constexpr int MPS = MW * MH;            // values per field and plane
constexpr int MSS = 3 * MPS;            // ring layout [slot][field][xy]
constexpr int MPAIRS = MH * (MW / 2);   // aligned pairs of a field and plane
constexpr int MX_KCHUNK = 80;           // longest z-chunk (planes)

// Packed FP32 pairs: .x belongs to a thread's point at even i, .y to the one at i + 1.
typedef float2 f2;

// coefficients of a plane, as the FP64 kernel's FPlane, and the run's, stored
// twice (a packed operand); with the sign of their use
struct MPlane {
    float a, b, nrz, nhz, nrw, nhw;
};
struct MConst {
    f2 nhx, nhy, ngx, ngy, cxx, cyy, ncc, nucx;
};

__device__ __forceinline__ f2 pk2(float a, float b) { return make_float2(a, b); }
__device__ __forceinline__ f2 bc2(float s) { return make_float2(s, s); }
__device__ __forceinline__ f2 add2(f2 a, f2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ f2 sub2(f2 a, f2 b) { return __ffma2_rn(b, bc2(-1.f), a); }
__device__ __forceinline__ f2 mul2(f2 a, f2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ f2 ld2(const float *q) { return *reinterpret_cast<const float2 *>(q); }

__device__ __forceinline__ MPlane m_plane(const float4 *tab, int k)
{
    const float4 x = tab[2 * k], y = tab[2 * k + 1];
    return MPlane{x.x, x.y, x.z, x.w, y.x, y.y};
}

// one point's convective edge product of the u (v) top face (a quarter of the
// reference's), its z flux, and w's between the levels k and k+1
__device__ __forceinline__ float top_edge(const MPlane &P, float q, float qz, float w2)
{
    return __fmul_rn(fmaf(P.b, qz, __fmul_rn(P.a, q)), w2);
}
__device__ __forceinline__ float top_flux(const MPlane &P, float e, float q, float qz)
{
    return fmaf(P.nrz, qz - q, e);
}
__device__ __forceinline__ float w_flux(const MPlane &P, float q, float qz)
{
    const float s = q + qz;
    return fmaf(P.nrw, qz - q, __fmul_rn(__fmul_rn(0.25f, s), s));
}
// the same for a pair
__device__ __forceinline__ f2 top_edge2(const MPlane &P, f2 q, f2 qz, f2 w2)
{
    return mul2(fma2(bc2(P.b), qz, mul2(bc2(P.a), q)), w2);
}
__device__ __forceinline__ f2 top_flux2(const MPlane &P, f2 e, f2 q, f2 qz) { return fma2(bc2(P.nrz), sub2(qz, q), e); }
__device__ __forceinline__ f2 w_flux2(const MPlane &P, f2 q, f2 qz)
{
    const f2 s = add2(q, qz);
    return fma2(bc2(P.nrw), sub2(qz, q), mul2(mul2(bc2(0.25f), s), s));
}

struct MPair { // a thread's pair: centre values, fluxes through the bottom faces
    f2 u, v, w, fu, fv, fw;
};

// the top fluxes of the pair at c (plane k; p: plane k+1)
__device__ __forceinline__ void top_fluxes2(const float *c, const float *p, const MPlane &P, MPair &S)
{
    const float *cw = c + 2 * MPS;
    const f2 u = ld2(c), v = ld2(c + MPS), w = ld2(cw);
    const f2 uz = ld2(p), vz = ld2(p + MPS), wz = ld2(p + 2 * MPS);
    S.fu = top_flux2(P, top_edge2(P, u, uz, add2(w, pk2(w.y, cw[2]))), u, uz);
    S.fv = top_flux2(P, top_edge2(P, v, vz, add2(w, ld2(cw + MW))), v, vz);
    S.fw = w_flux2(P, w, wz);
    S.u = uz;
    S.v = vz;
    S.w = wz;
}

// x and y parts and the assembly of one component's increment (rk_fused.cu's
// assemble): sx, sy the neighbour sums, cx, cy, dz the flux differences
template <bool CRF>
__device__ __forceinline__ f2 assemble2(const MConst &K, f2 sx, f2 sy, f2 q, f2 nhx, f2 cx, f2 nhy, f2 cy, float nhz, f2 dz,
                                        f2 dq)
{
    f2 r = mul2(K.cxx, sx);
    r = fma2(K.cyy, sy, r);
    r = fma2(K.ncc, q, r);
    r = fma2(nhx, cx, r);
    r = fma2(nhy, cy, r);
    r = fma2(bc2(nhz), dz, r);
    if (CRF) r = fma2(K.nucx, dq, r);
    return r;
}

// dt * (momentum right-hand side) of the pair at c (plane k; p: plane k+1).
// S: on entry the centres of plane k and the fluxes through the bottom faces,
// on return those of plane k+1.
template <bool CRF>
__device__ __forceinline__ void rhs_pair2(const float *c, const float *p, const MPlane &P, const MConst &K, MPair &S,
                                          f2 &du, f2 &dv, f2 &dw)
{
    const float *cv = c + MPS, *cw = c + 2 * MPS, *pv = p + MPS, *pw = p + 2 * MPS;
    const f2 u = S.u, v = S.v, w = S.w;
    const f2 uz = ld2(p), vz = ld2(pv), wz = ld2(pw);
    const f2 uS = ld2(c - MW), uN = ld2(c + MW), vS = ld2(cv - MW), vN = ld2(cv + MW), wS = ld2(cw - MW),
             wN = ld2(cw + MW);
    const float uw = c[-1], vw = cv[-1], ww = cw[-1];
    const f2 uE = pk2(u.y, c[2]), uW = pk2(uw, u.x), vE = pk2(v.y, cv[2]), vW = pk2(vw, v.x), wE = pk2(w.y, cw[2]),
             wW = pk2(ww, w.x);
    // edges: (i+1/2, j+-1/2), and west of the pair
    const f2 n = mul2(add2(u, uN), add2(v, vE)), nS = mul2(add2(uS, u), add2(vS, pk2(vS.y, cv[2 - MW])));
    const float nw = __fmul_rn(uw + c[MW - 1], vw + v.x);
    // (i+1/2, k+1/2) and west of the pair, (j+-1/2, k+1/2)
    const f2 t = top_edge2(P, u, uz, add2(w, wE));
    const float tw = top_edge(P, uw, p[-1], ww + w.x);
    const f2 s = top_edge2(P, v, vz, add2(w, wN)), sS = top_edge2(P, vS, ld2(pv - MW), add2(wS, w));
    {
        const f2 sx = add2(uE, uW), dx = sub2(uE, uW), f = top_flux2(P, t, u, uz);
        du = assemble2<CRF>(K, sx, add2(uN, uS), u, K.nhx, mul2(dx, fma2(bc2(2.f), u, sx)), K.nhy, sub2(n, nS), P.nhz,
                            sub2(f, S.fu), dx);
        S.fu = f;
    }
    {
        const f2 sy = add2(vN, vS), dy = sub2(vN, vS), f = top_flux2(P, s, v, vz);
        dv = assemble2<CRF>(K, add2(vE, vW), sy, v, K.nhx, sub2(n, pk2(nw, n.x)), K.nhy,
                            mul2(dy, fma2(bc2(2.f), v, sy)), P.nhz, sub2(f, S.fv), sub2(vE, vW));
        S.fv = f;
    }
    {
        const f2 f = w_flux2(P, w, wz);
        dw = assemble2<CRF>(K, add2(wE, wW), add2(wN, wS), w, K.ngx, sub2(t, pk2(tw, t.x)), K.ngy, sub2(s, sS), P.nhw,
                            sub2(f, S.fw), sub2(wE, wW));
        S.fw = f;
    }
    S.u = uz;
    S.v = vz;
    S.w = wz;
}

// the same for one point (the stage-1 halo); f: its carried fluxes
__device__ __forceinline__ void top_fluxes1(const float *c, const float *p, const MPlane &P, float *f)
{
    const float *cw = c + 2 * MPS;
    f[0] = top_flux(P, top_edge(P, c[0], p[0], cw[0] + cw[1]), c[0], p[0]);
    f[1] = top_flux(P, top_edge(P, c[MPS], p[MPS], cw[0] + cw[MW]), c[MPS], p[MPS]);
    f[2] = w_flux(P, cw[0], p[2 * MPS]);
}
template <bool CRF>
__device__ __forceinline__ float assemble1(const MConst &K, float sx, float sy, float q, f2 nhx, float cx, f2 nhy,
                                           float cy, float nhz, float dz, float dq)
{
    float r = __fmul_rn(K.cxx.x, sx);
    r = fmaf(K.cyy.x, sy, r);
    r = fmaf(K.ncc.x, q, r);
    r = fmaf(nhx.x, cx, r);
    r = fmaf(nhy.x, cy, r);
    r = fmaf(nhz, dz, r);
    if (CRF) r = fmaf(K.nucx.x, dq, r);
    return r;
}
template <bool CRF>
__device__ __forceinline__ void rhs_one(const float *c, const float *p, const MPlane &P, const MConst &K, float *f,
                                        float &du, float &dv, float &dw)
{
    const float *cv = c + MPS, *cw = c + 2 * MPS, *pv = p + MPS, *pw = p + 2 * MPS;
    const float uc = c[0], vc = cv[0], wc = cw[0], uz = p[0], vz = pv[0], wz = pw[0];
    const float uS = c[-MW], uN = c[MW], uW = c[-1], uE = c[1];
    const float vS = cv[-MW], vN = cv[MW], vW = cv[-1], vE = cv[1];
    const float wS = cw[-MW], wN = cw[MW], wW = cw[-1], wE = cw[1];
    const float nS = __fmul_rn(uS + uc, vS + cv[1 - MW]), nC = __fmul_rn(uc + uN, vc + vE),
                nW = __fmul_rn(uW + c[MW - 1], vW + vc);
    const float t = top_edge(P, uc, uz, wc + wE), tW = top_edge(P, uW, p[-1], wW + wc);
    const float s = top_edge(P, vc, vz, wc + wN), sS = top_edge(P, vS, pv[-MW], wS + wc);
    const float fu = top_flux(P, t, uc, uz), fv = top_flux(P, s, vc, vz), fw = w_flux(P, wc, wz);
    const float sx = uE + uW, dx = uE - uW, sy = vN + vS, dy = vN - vS;
    du = assemble1<CRF>(K, sx, uN + uS, uc, K.nhx, __fmul_rn(dx, fmaf(2.f, uc, sx)), K.nhy, nC - nS, P.nhz, fu - f[0], dx);
    dv = assemble1<CRF>(K, vE + vW, sy, vc, K.nhx, nC - nW, K.nhy, __fmul_rn(dy, fmaf(2.f, vc, sy)), P.nhz, fv - f[1],
                        vE - vW);
    dw = assemble1<CRF>(K, wE + wW, wN + wS, wc, K.ngx, t - tW, K.ngy, s - sS, P.nhw, fw - f[2], wE - wW);
    f[0] = fu;
    f[1] = fv;
    f[2] = fw;
}

} // namespace

// WIDE: the stage-1 field and stage 2's update are formed in FP64, from the
// FP64 fields and the FP32 increments, as the stage kernels (stencil.cu) form
// them: u1 = (float)(u + d1), u_hat = ((u + d1) + d2 + u) / 2 - dt G p_pred.
// Otherwise u1 = (float)u + d1 and the bracket are FP32, where stage 2 sees the
// rounding of u that stage 1 saw and another one.
template <bool CRF, bool WIDE>
__global__ void __launch_bounds__(MT, 2) k_rk_mixed(const double *__restrict__ u, const double *__restrict__ v,
                                                   const double *__restrict__ w, double *__restrict__ uo,
                                                   double *__restrict__ vo, double *__restrict__ wo, StepParams p,
                                                   MeshDev m, MConst K, MeanRed red, int kchunk,
                                                   const float *__restrict__ pq, int pinc)
{
    pdl_enter();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double2 *stg = reinterpret_cast<double2 *>(smem_raw);    // FP64 staging, [field][pair]
    float *ur = reinterpret_cast<float *>(stg + 3 * MPAIRS); // u, v, w rings, two planes
    float *sr = ur + 2 * MSS;                                // u1 rings, two planes
    float4 *tab = reinterpret_cast<float4 *>(sr + 2 * MSS);  // plane coefficients, 2 per plane
    double *pzl = reinterpret_cast<double *>(tab + 2 * (MX_KCHUNK + 4)); // dzf / lz
    const int lane = threadIdx.x, wid = threadIdx.y, tid = lane + MX * wid;
    const int i0 = blockIdx.x * MX, j0 = blockIdx.y * MY;
    const int kbeg = blockIdx.z * kchunk + 1, kend = min(kbeg + kchunk - 1, p.nz);
    const size_t sk = (size_t)p.nx * p.ny;

    // Copies: 20 rows of 18 aligned pairs per field and plane; thread t takes
    // pair t and, for t >= 152, pair t + 104 (warps 0-3 have the stage-1 halo
    // instead).  x and y wrap; nx is even, so a pair never straddles the wrap
    // and, i0 being even, starts on a 16-byte boundary.
    constexpr int PAIR2 = MT - (MPAIRS - MT);
    int soff[2], pk[2];
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const int q = h == 0 ? tid : (tid >= PAIR2 ? tid + (MPAIRS - MT) : 0);
        const int r = q / 18, c = q % 18;
        const int gx = (i0 - 2 + 2 * c + p.nx) % p.nx, gy = (j0 - 2 + r + p.ny) % p.ny;
        soff[h] = gy * p.nx + gx;
        pk[h] = r * MW + 2 * c;
    }
    const bool pv2 = tid >= PAIR2;
    // stage 1 runs one plane beyond the chunk, but not on a wall plane; at a
    // slab interface it runs on the halo
    const int mstart = max(kbeg - 1, p.wlo ? 1 : 0), mend = min(kend + 1, p.whi ? p.nz : p.nz + 1);
    // u, v, w plane kq (none past the last that stage 1 reads) into staging
    auto issue = [&](int kq) {
        if (kq <= mend + 1) {
            const long long off = (long long)sk * kq; // kq >= -1 (a slab's lower halo)
            double2 *d = stg + tid;
#pragma unroll
            for (int h = 0; h < 2; h++) {
                if (h == 0 || pv2) {
                    const long long o = off + soff[h];
                    cp_async_16(d + h * (MPAIRS - MT), u + o);
                    cp_async_16(d + h * (MPAIRS - MT) + MPAIRS, v + o);
                    cp_async_16(d + h * (MPAIRS - MT) + 2 * MPAIRS, w + o);
                }
            }
        }
        cp_async_commit();
    };
    // the thread's own staged pairs, once landed, into ring slot s
    auto convert = [&](int s) {
        cp_async_wait<0>();
        const double2 *d = stg + tid;
        float *o = ur + s * MSS;
#pragma unroll
        for (int h = 0; h < 2; h++) {
            if (h == 0 || pv2) {
#pragma unroll
                for (int f = 0; f < 3; f++) {
                    const double2 x = d[h * (MPAIRS - MT) + f * MPAIRS];
                    *reinterpret_cast<float2 *>(o + f * MPS + pk[h]) = make_float2((float)x.x, (float)x.y);
                }
            }
        }
    };

    // stage 1 covers x 1..34, y 1..18 of the ring plane: the thread's pair,
    // and on warps 0-3 one point of the rim: rows 1 and 18 (warps 0, 1), the
    // columns 1 and 34 (warp 2 and 4 lanes of warp 3)
    const int hxy0 = (2 + 2 * wid + (lane >> 4)) * MW + 2 + 2 * (lane & 15);
    const int he = (wid - 2) * 32 + lane;
    const int hxy1 = wid < 2 ? (wid == 0 ? 1 : 18) * MW + 2 + lane : (1 + he % 18) * MW + (he < 18 ? 1 : 34);
    const bool hval = wid < 3 || (wid == 3 && lane < 4);

    // the thread's points in the domain (the last tiles of a row or column of
    // tiles reach past it; nx is even, so a pair lies inside or outside), and
    // the pair's neighbours in the pressure prediction, +x and +y
    const int gi = i0 + 2 * (lane & 15), gj = j0 + 2 * wid + (lane >> 4);
    const bool inside = gi < p.nx && gj < p.ny;
    const size_t gA = (size_t)gi + (size_t)p.nx * gj;
    const size_t gE = gi == p.nx - 2 ? gA - gi : gA + 2, gN = gj == p.ny - 1 ? gi : gA + p.nx;
    // WIDE: where the FP64 values of the thread's pair and rim point are (wrapped)
    const int swA = WIDE ? gj % p.ny * p.nx + gi % p.nx : 0;
    const int swH = WIDE ? (j0 - 2 + hxy1 / MW + p.ny) % p.ny * p.nx + (i0 - 2 + hxy1 % MW + p.nx) % p.nx : 0;

    issue(mstart - 1);
    for (int k = mstart - 1 + tid; k <= mend; k += MT) {
        const double ci = __ldg(m.dzc_inv + k);
        const int r = k - mstart + 1;
        const float fa = (float)(0.25 * (__ldg(m.dzf + k + 1) * ci)), fb = (float)(0.25 * (__ldg(m.dzf + k) * ci));
        const float rz = (float)(-p.re_inv * ci), hz = (float)(-p.dt * __ldg(m.dzf_inv + k));
        const float rw = (float)(-p.re_inv * __ldg(m.dzf_inv + k + 1)), hw = (float)(-p.dt * ci);
        tab[2 * r] = make_float4(fa, fb, rz, hz);
        tab[2 * r + 1] = make_float4(rw, hw, 0.f, 0.f);
        pzl[r] = __ldg(m.dzflzi + k);
    }
    tab -= 2 * (mstart - 1); // indexed by the plane
    pzl -= mstart - 1;
    // slots: u plane k in ring slot (k - mstart + 1) % 2, u1 plane k in slot (k - mstart) % 2
    convert(0);
    issue(mstart);
    convert(1);
    issue(mstart + 1);
    __syncthreads();
    MPair s1, s2 = {};
    float fh[3] = {0.f, 0.f, 0.f};
    {
        const MPlane P = m_plane(tab, mstart - 1);
        top_fluxes2(ur + hxy0, ur + MSS + hxy0, P, s1);
        if (hval) top_fluxes1(ur + hxy1, ur + MSS + hxy1, P, fh);
    }
    __syncthreads(); // ring slot 0 is free
    convert(0);
    issue(mstart + 2);
    __syncthreads();
    // d1 of the own pair at the planes mq and mq - 1; the prediction at stage
    // 2's next plane
    f2 d1[3] = {}, e1[3] = {};
    // WIDE: the pair's FP64 values at those planes, loaded once for both stages
    // (loading them for each: 0.237 against 0.223 ms at 324x162x150)
    double2 q1[3] = {}, e64[3] = {};
    f2 qc = bc2(0.f);
    double su = 0.0;
    const double b2 = 2.0 * (0.0 - p.u_crf); // imposeNoSlipBC's image
    const float bcu2 = (float)b2;
    float eh = 0.f; // WIDE: the rim point's stage-1 increment of u
    // FP64 value and increment, rounded once
    auto sum32 = [](double2 q, f2 d) { return make_float2((float)(q.x + (double)d.x), (float)(q.y + (double)d.y)); };
    auto image32 = [&](double2 q, f2 d) {
        return make_float2((float)((b2 - q.x) - (double)d.x), (float)((b2 - q.y) - (double)d.y));
    };
    auto pair64 = [&](const double *f, size_t at) { return __ldg(reinterpret_cast<const double2 *>(f + at)); };

    // one plane of the march: PH = (mq - mstart) % 2
    auto march = [&](auto PH, int mq) {
        constexpr int a = decltype(PH)::value, b = a ^ 1;
        const int kq = mq - 1; // stage 2: u1 plane kq in slot b, kq + 1 in slot a
        const bool do2 = kq >= kbeg && kq <= kend;
        const size_t pl = sk * kq;
        // the prediction is read here alone: its plane kq + 4 on its way to L2
        if (do2 && pinc && inside && kq + 4 <= min(kend + 1, p.nz))
            asm volatile("prefetch.global.L2 [%0];" ::"l"(pq + (pl + 3 * sk) + gA));
        if (mq <= mend) {
            const MPlane P = m_plane(tab, mq);
            const bool top = p.whi && mq == p.nz; // w1(nz) = 0, the wall
            float *o = sr + a * MSS;
            const float *h0 = ur + b * MSS + hxy0;
            [[maybe_unused]] const f2 cu = s1.u, cv = s1.v;
            const f2 cw = s1.w;
            [[maybe_unused]] double h64[3] = {0.0, 0.0, 0.0};
            if constexpr (WIDE) {
                const size_t at = sk * mq + swA, ah = sk * mq + swH;
                q1[0] = pair64(u, at);
                q1[1] = pair64(v, at);
                q1[2] = pair64(w, at);
                if (hval) {
                    h64[0] = __ldg(u + ah);
                    h64[1] = __ldg(v + ah);
                    h64[2] = __ldg(w + ah);
                }
            }
            rhs_pair2<CRF>(h0, ur + a * MSS + hxy0, P, K, s1, d1[0], d1[1], d1[2]);
            if (top) d1[2] = make_float2(-cw.x, -cw.y);
            f2 nu, nv, nw;
            if constexpr (WIDE) {
                nu = sum32(q1[0], d1[0]);
                nv = sum32(q1[1], d1[1]);
                nw = top ? bc2(0.f) : sum32(q1[2], d1[2]);
            } else {
                nu = add2(cu, d1[0]);
                nv = add2(cv, d1[1]);
                nw = add2(cw, d1[2]);
            }
            *reinterpret_cast<float2 *>(o + hxy0) = nu;
            *reinterpret_cast<float2 *>(o + hxy0 + MPS) = nv;
            *reinterpret_cast<float2 *>(o + hxy0 + 2 * MPS) = nw;
            if (hval) {
                const float *h = ur + b * MSS + hxy1;
                float eu, ev, ew;
                rhs_one<CRF>(h, ur + a * MSS + hxy1, P, K, fh, eu, ev, ew);
                if constexpr (WIDE) {
                    o[hxy1] = (float)(h64[0] + (double)eu);
                    o[hxy1 + MPS] = (float)(h64[1] + (double)ev);
                    o[hxy1 + 2 * MPS] = top ? 0.f : (float)(h64[2] + (double)ew);
                    eh = eu;
                } else {
                    o[hxy1] = h[0] + eu;
                    o[hxy1 + MPS] = h[MPS] + ev;
                    o[hxy1 + 2 * MPS] = top ? 0.f : h[2 * MPS] + ew;
                }
            }
        } else if (p.whi && mq == p.nz + 1) {
            // imposeNoSlipBC on the stage-1 field: plane nz+1 from plane nz
            float *o = sr + a * MSS;
            const float *n = sr + b * MSS;
            auto image = [&](int xy) {
                o[xy] = bcu2 - n[xy]; // exact where u_crf is zero
                o[xy + MPS] = -n[xy + MPS];
                o[xy + 2 * MPS] = 0.f;
            };
            image(hxy0);
            image(hxy0 + 1);
            if (hval) image(hxy1);
            if constexpr (WIDE && CRF) { // the image in FP64
                *reinterpret_cast<float2 *>(o + hxy0) = image32(q1[0], d1[0]);
                if (hval) o[hxy1] = (float)((b2 - __ldg(u + sk * p.nz + swH)) - (double)eh);
            }
        }
        // stage 2's operands from global memory, ahead of the barrier
        double2 u0 = {}, v0 = {}, w0 = {};
        f2 qy = bc2(0.f), qz = bc2(0.f);
        float qE = 0.f;
        if (do2 && inside) {
            if (pinc) {
                const float *q = pq + (pl - sk);
                qE = __ldg(q + gE);
                qy = __ldg(reinterpret_cast<const float2 *>(q + gN));
                qz = (kq < p.nz) ? __ldg(reinterpret_cast<const float2 *>(q + sk + gA)) : qc;
            }
            u0 = WIDE ? e64[0] : pair64(u, pl + gA);
            v0 = WIDE ? e64[1] : pair64(v, pl + gA);
            w0 = WIDE ? e64[2] : pair64(w, pl + gA);
        }
        __syncthreads();
        // ring slot of plane mq, which stage 1 above has finished with
        if (mq + 2 <= mend + 1) convert(b);
        issue(mq + 3);
        if (do2) {
            const MPlane P = m_plane(tab, kq);
            f2 du, dv, dw;
            rhs_pair2<CRF>(sr + b * MSS + hxy0, sr + a * MSS + hxy0, P, K, s2, du, dv, dw);
            double2 nu, nv, nw;
            if constexpr (WIDE) {
                // ((q + d1) + d2 + q) / 2 - dt G p_pred
                auto mean = [](double q, float a, float b) { return ((q + (double)a) + (double)b + q) * 0.5; };
                nu = make_double2(mean(u0.x, e1[0].x, du.x), mean(u0.y, e1[0].y, du.y));
                nv = make_double2(mean(v0.x, e1[1].x, dv.x), mean(v0.y, e1[1].y, dv.y));
                nw = make_double2(mean(w0.x, e1[2].x, dw.x), mean(w0.y, e1[2].y, dw.y));
                if (pinc) {
                    const double gx = p.dt * p.dx_inv, gy = p.dt * p.dy_inv, gz = p.dt * __ldg(m.dzc_inv + kq);
                    const double q0 = qc.x, q1 = qc.y;
                    nu.x -= (q1 - q0) * gx;
                    nu.y -= ((double)qE - q1) * gx;
                    nv.x -= ((double)qy.x - q0) * gy;
                    nv.y -= ((double)qy.y - q1) * gy;
                    nw.x -= ((double)qz.x - q0) * gz;
                    nw.y -= ((double)qz.y - q1) * gz;
                    qc = qz;
                }
            } else {
                const f2 half = bc2(0.5f);
                du = mul2(half, add2(e1[0], du));
                dv = mul2(half, add2(e1[1], dv));
                dw = mul2(half, add2(e1[2], dw));
                if (pinc) {
                    du = fma2(K.ngx, sub2(pk2(qc.y, qE), qc), du);
                    dv = fma2(K.ngy, sub2(qy, qc), dv);
                    dw = fma2(bc2(P.nhw), sub2(qz, qc), dw);
                    qc = qz;
                }
            }
            if (inside) {
                if constexpr (!WIDE) {
                    nu = make_double2(u0.x + (double)du.x, u0.y + (double)du.y);
                    nv = make_double2(v0.x + (double)dv.x, v0.y + (double)dv.y);
                    nw = make_double2(w0.x + (double)dw.x, w0.y + (double)dw.y);
                }
                auto put = [&](double *f, size_t at, double x, double y) {
                    *reinterpret_cast<double2 *>(f + at + gA) = make_double2(x, y);
                };
                put(uo, pl, nu.x, nu.y);
                put(vo, pl, nv.x, nv.y);
                if (kq != p.nz || !p.whi) put(wo, pl, nw.x, nw.y);
                // imposeNoSlipBC
                if (p.wlo && kq == 1) {
                    put(uo, pl - sk, b2 - nu.x, b2 - nu.y);
                    put(vo, pl - sk, -nv.x, -nv.y);
                    put(wo, pl - sk, 0.0, 0.0);
                }
                if (p.whi && kq == p.nz) {
                    put(uo, pl + sk, b2 - nu.x, b2 - nu.y);
                    put(vo, pl + sk, -nv.x, -nv.y);
                    put(wo, pl, 0.0, 0.0);
                    put(wo, pl + sk, 0.0, 0.0);
                }
                su += (nu.x + nu.y) * pzl[kq];
            }
        } else if (kq == kbeg - 1) {
            // the bottom fluxes of stage 2's first plane: u1 plane kbeg in slot
            // a, and below it plane kbeg - 1 in slot b or, on the wall, the
            // image of plane 1; its prediction
            const MPlane P = m_plane(tab, kq);
            if (p.wlo && kq == 0) { // w1(0) = 0: no convection through the wall
                const float *n = sr + a * MSS + hxy0;
                const f2 u1 = ld2(n), v1 = ld2(n + MPS);
                s2.u = u1;
                s2.v = v1;
                s2.w = ld2(n + 2 * MPS);
                f2 ub = sub2(bc2(bcu2), u1);
                if constexpr (WIDE && CRF) ub = image32(q1[0], d1[0]); // the image in FP64
                s2.fu = top_flux2(P, bc2(0.f), ub, u1);
                s2.fv = top_flux2(P, bc2(0.f), make_float2(-v1.x, -v1.y), v1);
                s2.fw = w_flux2(P, bc2(0.f), ld2(n + 2 * MPS));
            } else {
                top_fluxes2(sr + b * MSS + hxy0, sr + a * MSS + hxy0, P, s2);
            }
            if (pinc && inside) qc = __ldg(reinterpret_cast<const float2 *>(pq + gA + sk * (kbeg - 1)));
        }
#pragma unroll
        for (int q = 0; q < 3; q++) {
            e1[q] = d1[q];
            e64[q] = q1[q];
        }
        __syncthreads();
    };
    const int stop = kend + 1;
    for (int mq = mstart;;) {
        march(std::integral_constant<int, 0>{}, mq);
        if (++mq > stop) break;
        march(std::integral_constant<int, 1>{}, mq);
        if (++mq > stop) break;
    }
    cp_async_wait<0>();
    mean_reduce(su, red);
}

// Grids that 32 x 16 tiles divide take the FP32 forms, the others the wide ones.
// The line is the one that the fused step has always had: grids that do not tile
// ran the two stage kernels, whose FP64 sums they keep.  RMS error of u, v, w after
// the RK phase against FP64, in units of the stage kernels': 0.37, 0.91, 0.81 wide,
// 0.58, 1.11, 0.88 with the FP32 forms (324x162x30); 324x162x150 0.223 ms
// wide, 0.168 with the FP32 forms, 0.622 as stage kernels.
static auto mixed_kernel(const StepParams &p)
{
    const bool wide = p.nx % MX != 0 || p.ny % MY != 0, crf = p.u_crf != 0.0;
    return wide ? (crf ? k_rk_mixed<true, true> : k_rk_mixed<false, true>)
                : (crf ? k_rk_mixed<true, false> : k_rk_mixed<false, false>);
}

static dim3 mixed_tiles(const StepParams &p) { return dim3((p.nx + MX - 1) / MX, (p.ny + MY - 1) / MY, 1); }

// an upper bound of the launch's CTA count (chunks of at least 2 planes)
int rk_mixed_blocks(const StepParams &p)
{
    const dim3 t = mixed_tiles(p);
    return (int)(t.x * t.y) * ((p.nz + 1) / 2);
}

static size_t mixed_smem()
{
    return sizeof(double2) * 3 * MPAIRS + sizeof(float) * 4 * MSS + (sizeof(float4) * 2 + sizeof(double)) * (MX_KCHUNK + 4);
}

int rk_mixed_prepare(const StepParams &p, RkLaunch *out)
{
    return rk_prepare((const void *)mixed_kernel(p), MT, mixed_smem(), mixed_tiles(p), p.nz, MX_KCHUNK, out);
}

int launch_rk_mixed(const double *u, const double *v, const double *w, double *uo, double *vo, double *wo,
                    const StepParams &p, const MeshDev &m, MeanState &ms, const float *pq, int pinc, const RkLaunch &l,
                    cudaStream_t st)
{
    if ((int)(l.grid.x * l.grid.y * l.grid.z) > ms.max_blocks) {
        set_error("mean buffer too small for the mixed fused RK kernel");
        return -1;
    }
    MConst K;
    auto both = [](double x) { return make_float2((float)x, (float)x); };
    K.nhx = both(-0.25 * p.dt * p.dx_inv);
    K.nhy = both(-0.25 * p.dt * p.dy_inv);
    K.ngx = both(-p.dt * p.dx_inv);
    K.ngy = both(-p.dt * p.dy_inv);
    K.cxx = both(p.dt * p.re_inv * p.dx_inv * p.dx_inv);
    K.cyy = both(p.dt * p.re_inv * p.dy_inv * p.dy_inv);
    K.ncc = both(-2.0 * p.dt * p.re_inv * (p.dx_inv * p.dx_inv + p.dy_inv * p.dy_inv));
    K.nucx = both(-0.5 * p.dt * p.u_crf * p.dx_inv);
    MeanRed r{ms.partial, ms.counter, ms.scalar, (double)p.nx, (double)p.ny, ms.vel_force};
    PL_CUDA_TRY(launch_chained(mixed_kernel(p), l.grid, dim3(MX, MT / MX), mixed_smem(), st, u, v, w, uo, vo, wo, p, m, K,
                               r, l.kchunk, pq, pinc));
    return 0;
}

} // namespace pl
