// rk_fused.cu -- both RK2 stages of timeIntVelRK1 / timeIntVelRK2
// (mod_calcVel.f90:52-146, 240-334) with their wall fills in one kernel, FP64
// flux form (the mixed path's kernel is rk_mixed.cu).
//
// 2.5D blocking: a CTA owns a 32 x 16 tile of (i, j), two y-adjacent points
// per thread, and marches up a chunk of k-planes.  Shared-memory rings hold
// three planes of u, v, w (halo 2 in x, y; cp.async, 16-byte pieces) and of
// the stage-1 field u1 = u + dt RHS(u) (halo 1), which never leaves the SM:
// HBM sees u, v, w read once and the new fields written once.
//
// What bounds it is on chip: the FP64 pipe (a warp instruction takes two
// cycles of a scheduler) and the shared-memory bandwidth (a warp's load of
// doubles is two wavefronts).  So the stencil is arranged to need few of both:
//   * convective edge products are formed once and serve the two equations
//     that share the edge (u north = v east, u top = w east, v top = w north),
//     and the southern products of a thread's upper point are the northern
//     ones of its lower point;
//   * the z flux of each component, convective and viscous together, is one
//     number per face, carried up the march: the plane below is never read;
//   * the point's own values of the next plane become its centre values one
//     plane later, in registers;
//   * per plane one barrier: stage 1 works on plane k, stage 2 on plane k-2,
//     and the copy of plane k+2 is in flight meanwhile.
// 67 FP64 operations and 14.5 shared loads per evaluation, against about 115
// and 27 for the reference's expressions point by point on a 32 x 8 tile with
// two barriers a plane: 512x384x256 1.503 -> 0.931 ms (40 % of the measured
// copy bandwidth at 48 B/point), 256x192x128 0.220 -> 0.129, 64x64x64 0.037 ->
// 0.020.  At 512x384x128 the FP64 pipe is 53 % busy and the shared-memory pipe
// 65 %, with 16 warps an SM (registers and shared memory both).
//
// Tiles may reach past the domain (their loads wrap, their stores are masked),
// so every even nx, ny takes this kernel: 324x162x150, 15 % of it masked,
// 0.638 ms as two stage kernels -> 0.193 ms.
//
// Every product that two points share is rounded on its own (no contraction
// into a neighbouring add), so the numbers do not depend on how the domain is
// cut into chunks or z slabs.
#include <type_traits>

#include "fft.cuh" // cp.async helpers
#include "stencil.cuh"
#include "stencil_rhs.cuh"

namespace pl {

namespace {

constexpr int FX = 32, FY = 16;       // tile; a thread owns the points (x, 2t) and (x, 2t+1)
constexpr int FT = 256;               // threads
constexpr int FW = 38, FH = FY + 4;   // ring plane: 36 columns used; a row pitch of 38 keeps rows on
                                      // 16-byte boundaries and spreads a column over the banks
constexpr int FPS = FW * FH;          // values per field and plane
constexpr int FSS = 3 * FPS;          // ring layout [slot][field][xy]
constexpr int F_KCHUNK = 64;          // longest z-chunk (planes)

// coefficients of a plane k, dt folded in where the term is added to the
// increment: the top face's interpolation (a q_k + b q_{k+1}, with the 1/4 of
// the convective term), its viscous factor rz = 1/Re / dzc(k), hz = dt / dzf(k);
// for w the cell k+1 above the face: rw = 1/Re / dzf(k+1), hw = dt / dzc(k)
struct FPlane {
    double a, b, rz, hz, rw, hw;
};
// hx, hy = dt/4 / dx, dy; gx, gy = dt / dx, dy; cxx, cyy = dt/Re / dx^2, dy^2
struct FConst {
    double hx, hy, gx, gy, cxx, cyy, ncc, ucx, fb[3];
};

__device__ __forceinline__ double mul(double a, double b) { return __dmul_rn(a, b); }

__device__ __forceinline__ FPlane f_plane(const double *tab, int k)
{
    const double2 *t = reinterpret_cast<const double2 *>(tab + 8 * k);
    const double2 x = t[0], y = t[1], z = t[2];
    return FPlane{x.x, x.y, y.x, y.y, z.x, z.y};
}

// convective edge product of the u (v) top face, a quarter of the reference's
__device__ __forceinline__ double top_edge(const FPlane &P, double q, double qz, double w2)
{
    return mul(fma(P.b, qz, mul(P.a, q)), w2);
}
// z flux of u (v) through the top face, from its edge product
__device__ __forceinline__ double top_flux(const FPlane &P, double e, double q, double qz)
{
    return fma(-P.rz, qz - q, e);
}
// z flux of w between the levels k and k+1
__device__ __forceinline__ double w_flux(const FPlane &P, double q, double qz)
{
    const double s = q + qz;
    return fma(mul(0.25, s), s, -mul(P.rw, qz - q));
}

// the three top fluxes of a point: c, p point at it in the planes k, k+1
__device__ __forceinline__ void top_fluxes(const double *c, const double *p, const FPlane &P, double &fu, double &fv,
                                           double &fw)
{
    const double *cw = c + 2 * FPS;
    fu = top_flux(P, top_edge(P, c[0], p[0], cw[0] + cw[1]), c[0], p[0]);
    fv = top_flux(P, top_edge(P, c[FPS], p[FPS], cw[0] + cw[FW]), c[FPS], p[FPS]);
    fw = w_flux(P, cw[0], p[2 * FPS]);
}

// what the march carries for a thread's two points: centre values and the
// fluxes through the bottom faces
struct Pair {
    double u[2], v[2], w[2], fu[2], fv[2], fw[2];
};

// x and y parts and the assembly of one component's increment.  sx, sy: sums
// of the two x, y neighbours; cx: the x flux difference; cy: the y one;
// dz: the z flux difference
template <bool CRF>
__device__ __forceinline__ double assemble(const FConst &K, double sx, double sy, double q, double hx, double cx,
                                           double hy, double cy, double hz, double dz, double dq, double fb)
{
    double r = fma(K.cxx, sx, fb);
    r = fma(K.cyy, sy, r);
    r = fma(K.ncc, q, r);
    r = fma(-hx, cx, r);
    r = fma(-hy, cy, r);
    r = fma(-hz, dz, r);
    if (CRF) r = fma(-K.ucx, dq, r);
    return r;
}

// dt * (momentum right-hand side) of the thread's two points A (at c, plane
// k) and B, one row up, p being A in plane k+1.  S: on entry the centres of
// plane k and the bottom fluxes; on return those of plane k+1.
template <bool CRF>
__device__ __forceinline__ void rhs_pair(const double *c, const double *p, const FPlane &P, const FConst &K, Pair &S,
                                         double *du, double *dv, double *dw)
{
    const double *cv = c + FPS, *cw = c + 2 * FPS, *pv = p + FPS, *pw = p + 2 * FPS;
    const double uA = S.u[0], uB = S.u[1], vA = S.v[0], vB = S.v[1], wA = S.w[0], wB = S.w[1];
    const double uS = c[-FW], uN = c[2 * FW], vS = cv[-FW], vN = cv[2 * FW], wS = cw[-FW], wN = cw[2 * FW];
    const double uwA = c[-1], uwB = c[FW - 1];
    const double veA = cv[1], veB = cv[FW + 1];
    const double uzA = p[0], uzB = p[FW], vzA = pv[0], vzB = pv[FW], wzA = pw[0], wzB = pw[FW];
    // (i+1/2, j+-1/2) edges: south of A, between A and B, north of B; and west of A, B
    const double nS = mul(uS + uA, vS + cv[1 - FW]), nA = mul(uA + uB, vA + veA), nB = mul(uB + uN, vB + veB);
    const double vwA = cv[-1], vwB = cv[FW - 1];
    const double wA1 = mul(uwA + uwB, vwA + vA), wB1 = mul(uwB + c[2 * FW - 1], vwB + vB);
    // (i+-1/2, k+1/2) edges
    const double weA = cw[1], weB = cw[FW + 1], wwA = cw[-1], wwB = cw[FW - 1];
    const double tA = top_edge(P, uA, uzA, wA + weA), tB = top_edge(P, uB, uzB, wB + weB);
    const double tWA = top_edge(P, uwA, p[-1], wwA + wA), tWB = top_edge(P, uwB, p[FW - 1], wwB + wB);
    // (j+-1/2, k+1/2) edges
    const double sS = top_edge(P, vS, pv[-FW], wS + wA), sA = top_edge(P, vA, vzA, wA + wB),
                 sB = top_edge(P, vB, vzB, wB + wN);
    { // u
        const double ueA = c[1], ueB = c[FW + 1];
        const double fA = top_flux(P, tA, uA, uzA), fB = top_flux(P, tB, uB, uzB);
        double sx = ueA + uwA, dx = ueA - uwA;
        du[0] = assemble<CRF>(K, sx, uS + uB, uA, K.hx, dx * fma(2.0, uA, sx), K.hy, nA - nS, P.hz, fA - S.fu[0], dx,
                              K.fb[0]);
        sx = ueB + uwB, dx = ueB - uwB;
        du[1] = assemble<CRF>(K, sx, uA + uN, uB, K.hx, dx * fma(2.0, uB, sx), K.hy, nB - nA, P.hz, fB - S.fu[1], dx,
                              K.fb[0]);
        S.fu[0] = fA;
        S.fu[1] = fB;
        S.u[0] = uzA;
        S.u[1] = uzB;
    }
    { // v
        const double fA = top_flux(P, sA, vA, vzA), fB = top_flux(P, sB, vB, vzB);
        double sy = vB + vS, dy = vB - vS;
        dv[0] = assemble<CRF>(K, veA + vwA, sy, vA, K.hx, nA - wA1, K.hy, dy * fma(2.0, vA, sy), P.hz, fA - S.fv[0],
                              veA - vwA, K.fb[1]);
        sy = vN + vA, dy = vN - vA;
        dv[1] = assemble<CRF>(K, veB + vwB, sy, vB, K.hx, nB - wB1, K.hy, dy * fma(2.0, vB, sy), P.hz, fB - S.fv[1],
                              veB - vwB, K.fb[1]);
        S.fv[0] = fA;
        S.fv[1] = fB;
        S.v[0] = vzA;
        S.v[1] = vzB;
    }
    { // w
        const double fA = w_flux(P, wA, wzA), fB = w_flux(P, wB, wzB);
        dw[0] = assemble<CRF>(K, weA + wwA, wS + wB, wA, K.gx, tA - tWA, K.gy, sA - sS, P.hw, fA - S.fw[0], weA - wwA,
                              K.fb[2]);
        dw[1] = assemble<CRF>(K, weB + wwB, wA + wN, wB, K.gx, tB - tWB, K.gy, sB - sA, P.hw, fB - S.fw[1], weB - wwB,
                              K.fb[2]);
        S.fw[0] = fA;
        S.fw[1] = fB;
        S.w[0] = wzA;
        S.w[1] = wzB;
    }
}

// the same for one point (the stage-1 halo); f: its carried fluxes
template <bool CRF>
__device__ __forceinline__ void rhs_one(const double *c, const double *p, const FPlane &P, const FConst &K, double *f,
                                        double &du, double &dv, double &dw)
{
    const double *cv = c + FPS, *cw = c + 2 * FPS, *pv = p + FPS, *pw = p + 2 * FPS;
    const double uc = c[0], vc = cv[0], wc = cw[0], uz = p[0], vz = pv[0], wz = pw[0];
    const double uS = c[-FW], uN = c[FW], uW = c[-1], uE = c[1];
    const double vS = cv[-FW], vN = cv[FW], vW = cv[-1], vE = cv[1];
    const double wS = cw[-FW], wN = cw[FW], wW = cw[-1], wE = cw[1];
    const double nS = mul(uS + uc, vS + cv[1 - FW]), nC = mul(uc + uN, vc + vE), nW = mul(uW + c[FW - 1], vW + vc);
    const double t = top_edge(P, uc, uz, wc + wE), tW = top_edge(P, uW, p[-1], wW + wc);
    const double s = top_edge(P, vc, vz, wc + wN), sS = top_edge(P, vS, pv[-FW], wS + wc);
    const double fu = top_flux(P, t, uc, uz), fv = top_flux(P, s, vc, vz), fw = w_flux(P, wc, wz);
    const double sx = uE + uW, dx = uE - uW, sy = vN + vS, dy = vN - vS;
    du = assemble<CRF>(K, sx, uS + uN, uc, K.hx, dx * fma(2.0, uc, sx), K.hy, nC - nS, P.hz, fu - f[0], dx, K.fb[0]);
    dv = assemble<CRF>(K, vE + vW, sy, vc, K.hx, nC - nW, K.hy, dy * fma(2.0, vc, sy), P.hz, fv - f[1], vE - vW,
                       K.fb[1]);
    dw = assemble<CRF>(K, wE + wW, wS + wN, wc, K.gx, t - tW, K.gy, s - sS, P.hw, fw - f[2], wE - wW, K.fb[2]);
    f[0] = fu;
    f[1] = fv;
    f[2] = fw;
}

} // namespace

template <bool CRF>
__global__ void __launch_bounds__(FT, 2) k_rk_fused(const double *__restrict__ u, const double *__restrict__ v,
                                                   const double *__restrict__ w, double *__restrict__ uo,
                                                   double *__restrict__ vo, double *__restrict__ wo, StepParams p,
                                                   MeshDev m, FConst K, MeanRed red, int kchunk)
{
    pdl_enter();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double *ur = reinterpret_cast<double *>(smem_raw); // u, v, w
    double *sr = ur + 3 * FSS;                         // u1, v1, w1
    double *tab = sr + 3 * FSS;                        // plane coefficients, 8 per plane
    const int lane = threadIdx.x, wid = threadIdx.y, tid = lane + FX * wid;
    const int i0 = blockIdx.x * FX, j0 = blockIdx.y * FY;
    const int kbeg = blockIdx.z * kchunk + 1, kend = min(kbeg + kchunk - 1, p.nz);
    const size_t sk = (size_t)p.nx * p.ny;
    const double bc2 = 2.0 * (0.0 - p.u_crf);

    // Copies: 20 rows of 18 aligned pairs per field and plane; thread t takes
    // pair t and, for t >= 152, pair t + 104 (warps 0-3 have the stage-1 halo
    // instead).  x and y wrap; nx is even, so a pair never straddles the wrap
    // and, i0 being even, starts on a 16-byte boundary.
    constexpr int FPAIR = FH * 18, PAIR2 = FT - (FPAIR - FT);
    int soff[2], pk[2];
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const int q = h == 0 ? tid : (tid >= PAIR2 ? tid + (FPAIR - FT) : 0);
        const int r = q / 18, c = q % 18;
        const int gx = (i0 - 2 + 2 * c + p.nx) % p.nx, gy = (j0 - 2 + r + p.ny) % p.ny;
        soff[h] = gy * p.nx + gx;
        pk[h] = r * FW + 2 * c;
    }
    const bool pv2 = tid >= PAIR2;
    auto issue = [&](int kq, int slot) { // u, v, w plane kq (>= -1: a slab's lower halo) into ring slot `slot`
        const long long off = (long long)sk * kq;
        double *d = ur + slot * FSS;
#pragma unroll
        for (int h = 0; h < 2; h++) {
            if (h == 0 || pv2) {
                const long long o = off + soff[h];
                cp_async_16(d + pk[h], u + o);
                cp_async_16(d + FPS + pk[h], v + o);
                cp_async_16(d + 2 * FPS + pk[h], w + o);
            }
        }
        cp_async_commit();
    };

    // stage 1 covers x 1..34, y 1..18 of the ring plane: the thread's pair,
    // and on warps 0-3 one point of the rim: rows 1 and 18 (warps 0, 1), the
    // columns 1 and 34 (warp 2 and 4 lanes of warp 3)
    const int hxy0 = (2 + 2 * wid) * FW + 2 + lane;
    const int he = (wid - 2) * 32 + lane;
    const int hxy1 = wid < 2 ? (wid == 0 ? 1 : 18) * FW + 2 + lane : (1 + he % 18) * FW + (he < 18 ? 1 : 34);
    const bool hval = wid < 3 || (wid == 3 && lane < 4);

    // the thread's points in the domain (the last tiles of a row or column of
    // tiles reach past it; ny is even, so a pair lies inside or outside)
    const int gi = i0 + lane, gj = j0 + 2 * wid;
    const bool inside = gi < p.nx && gj < p.ny;
    const size_t gA = (size_t)gi + (size_t)p.nx * gj;

    // stage 1 runs one plane beyond the chunk, but not on a wall plane; at a
    // slab interface it runs on the halo
    const int mstart = max(kbeg - 1, p.wlo ? 1 : 0), mend = min(kend + 1, p.whi ? p.nz : p.nz + 1);
    // slots: u plane k in (k - mstart + 1) % 3, u1 plane k in (k - mstart) % 3
    issue(mstart - 1, 0);
    issue(mstart, 1);
    issue(mstart + 1, 2);
    for (int k = mstart - 1 + tid; k <= mend; k += FT) {
        double *t = tab + 8 * (k - mstart + 1);
        const double ci = __ldg(m.dzc_inv + k);
        t[0] = 0.25 * (__ldg(m.dzf + k + 1) * ci);
        t[1] = 0.25 * (__ldg(m.dzf + k) * ci);
        t[2] = p.re_inv * ci;
        t[3] = p.dt * __ldg(m.dzf_inv + k);
        t[4] = p.re_inv * __ldg(m.dzf_inv + k + 1);
        t[5] = p.dt * ci;
        t[6] = __ldg(m.dzflzi + k);
    }
    tab -= 8 * (mstart - 1); // indexed by the plane
    cp_async_wait<0>();
    __syncthreads();

    Pair s1, s2 = {};
    double fh[3] = {0.0, 0.0, 0.0};
    {
        const FPlane P = f_plane(tab, mstart - 1);
#pragma unroll
        for (int q = 0; q < 2; q++) {
            const double *c = ur + hxy0 + q * FW, *n = c + FSS;
            top_fluxes(c, n, P, s1.fu[q], s1.fv[q], s1.fw[q]);
            s1.u[q] = n[0];
            s1.v[q] = n[FPS];
            s1.w[q] = n[2 * FPS];
        }
        if (hval) top_fluxes(ur + hxy1, ur + FSS + hxy1, P, fh[0], fh[1], fh[2]);
    }
    __syncthreads(); // slot 0 is free
    double su = 0.0;

    // one plane of the march: PH = (mq - mstart) % 3
    auto march = [&](auto PH, int mq) {
        constexpr int a = decltype(PH)::value, b = (a + 1) % 3, c = (a + 2) % 3;
        if (mq + 2 <= mend + 1) issue(mq + 2, a);
        if (mq <= mend) {
            const FPlane P = f_plane(tab, mq);
            const bool top = p.whi && mq == p.nz; // w1(nz) = 0, the wall
            double *o = sr + a * FSS;
            double du[2], dv[2], dw[2];
            const double cu[2] = {s1.u[0], s1.u[1]}, cv[2] = {s1.v[0], s1.v[1]}, cw[2] = {s1.w[0], s1.w[1]};
            rhs_pair<CRF>(ur + b * FSS + hxy0, ur + c * FSS + hxy0, P, K, s1, du, dv, dw);
#pragma unroll
            for (int q = 0; q < 2; q++) {
                o[hxy0 + q * FW] = cu[q] + du[q];
                o[hxy0 + q * FW + FPS] = cv[q] + dv[q];
                o[hxy0 + q * FW + 2 * FPS] = top ? 0.0 : cw[q] + dw[q];
            }
            if (hval) {
                const double *h = ur + b * FSS + hxy1;
                double eu, ev, ew;
                rhs_one<CRF>(h, ur + c * FSS + hxy1, P, K, fh, eu, ev, ew);
                o[hxy1] = h[0] + eu;
                o[hxy1 + FPS] = h[FPS] + ev;
                o[hxy1 + 2 * FPS] = top ? 0.0 : h[2 * FPS] + ew;
            }
        } else if (p.whi && mq == p.nz + 1) {
            // imposeNoSlipBC on the stage-1 field: plane nz+1 from plane nz
            double *o = sr + a * FSS;
            const double *n = sr + c * FSS;
            auto image = [&](int xy) {
                o[xy] = bc2 - n[xy];
                o[xy + FPS] = -n[xy + FPS];
                o[xy + 2 * FPS] = 0.0;
            };
            image(hxy0);
            image(hxy0 + FW);
            if (hval) image(hxy1);
        }
        const int kq = mq - 2; // u1 plane kq in slot b, kq + 1 in slot c
        if (kq >= kbeg && kq <= kend) {
            const size_t g = gA + sk * kq;
            double u0[2] = {0.0, 0.0}, v0[2] = {0.0, 0.0}, w0[2] = {0.0, 0.0};
            if (inside) {
                u0[0] = __ldg(u + g);
                u0[1] = __ldg(u + g + p.nx);
                v0[0] = __ldg(v + g);
                v0[1] = __ldg(v + g + p.nx);
                w0[0] = __ldg(w + g);
                w0[1] = __ldg(w + g + p.nx);
            }
            const FPlane P = f_plane(tab, kq);
            double du[2], dv[2], dw[2];
            const double cu[2] = {s2.u[0], s2.u[1]}, cv[2] = {s2.v[0], s2.v[1]}, cw[2] = {s2.w[0], s2.w[1]};
            rhs_pair<CRF>(sr + b * FSS + hxy0, sr + c * FSS + hxy0, P, K, s2, du, dv, dw);
            if (inside) {
                const double zl = tab[8 * kq + 6];
#pragma unroll
                for (int q = 0; q < 2; q++) {
                    const size_t gq = g + (size_t)q * p.nx;
                    const double nu = ((cu[q] + du[q]) + u0[q]) * 0.5, nv = ((cv[q] + dv[q]) + v0[q]) * 0.5,
                                 nw = ((cw[q] + dw[q]) + w0[q]) * 0.5;
                    uo[gq] = nu;
                    vo[gq] = nv;
                    if (kq != p.nz || !p.whi) wo[gq] = nw;
                    wall_fill<double>(uo, vo, wo, gq, kq, sk, p.nz, 0.0 - p.u_crf, nu, nv, p.wlo, p.whi);
                    su += nu * zl;
                }
            }
        } else if (kq == kbeg - 1) {
            // the bottom fluxes of stage 2's first plane: u1 plane kbeg in slot
            // c, and below it plane kbeg - 1 in slot b or, on the wall, the
            // image of plane 1
            const FPlane P = f_plane(tab, kq);
#pragma unroll
            for (int q = 0; q < 2; q++) {
                const double *n = sr + c * FSS + hxy0 + q * FW;
                s2.u[q] = n[0];
                s2.v[q] = n[FPS];
                s2.w[q] = n[2 * FPS];
                if (p.wlo && kq == 0) { // w1(0) = 0: no convection through the wall
                    s2.fu[q] = top_flux(P, 0.0, bc2 - s2.u[q], s2.u[q]);
                    s2.fv[q] = top_flux(P, 0.0, -s2.v[q], s2.v[q]);
                    s2.fw[q] = w_flux(P, 0.0, s2.w[q]);
                } else {
                    top_fluxes(sr + b * FSS + hxy0 + q * FW, n, P, s2.fu[q], s2.fv[q], s2.fw[q]);
                }
            }
        }
        cp_async_wait<0>();
        __syncthreads();
    };
    const int stop = kend + 2;
    for (int mq = mstart;;) {
        march(std::integral_constant<int, 0>{}, mq);
        if (++mq > stop) break;
        march(std::integral_constant<int, 1>{}, mq);
        if (++mq > stop) break;
        march(std::integral_constant<int, 2>{}, mq);
        if (++mq > stop) break;
    }
    mean_reduce(su, red);
}

static dim3 fused_tiles(const StepParams &p) { return dim3((p.nx + FX - 1) / FX, (p.ny + FY - 1) / FY, 1); }

// Planes per z-chunk: the count of waves of resident CTAs times a chunk's
// planes plus the few it recomputes or waits for, whichever chunk count gives
// least (a grid that does not fill the chip takes short chunks).
int rk_kchunk(long tiles, int nz, int most, int resident)
{
    int best = 0;
    long cost = 0;
    for (int kc = min(nz, most); kc >= 2; kc--) {
        const long ctas = tiles * ((nz + kc - 1) / kc);
        const long c = ((ctas + resident - 1) / resident) * (kc + 5);
        if (best == 0 || c < cost) {
            best = kc;
            cost = c;
        }
    }
    return best;
}

// an upper bound of the launch's CTA count (chunks of at least 2 planes)
int rk_fused_blocks(const StepParams &p)
{
    const dim3 t = fused_tiles(p);
    return (int)(t.x * t.y) * ((p.nz + 1) / 2);
}

static size_t fused_smem() { return sizeof(double) * (6 * FSS + 8 * (F_KCHUNK + 4)); }

int rk_prepare(const void *kern, int threads, size_t shm, dim3 tiles, int nz, int most, RkLaunch *out)
{
    PL_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)shm));
    // prefer the largest shared-memory carve-out: two CTAs per SM
    PL_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout,
                                     (int)cudaSharedmemCarveoutMaxShared));
    int per_sm = 0, dev = 0, nsm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, threads, shm) != cudaSuccess || per_sm < 1)
        per_sm = 1;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    out->kchunk = rk_kchunk((long)tiles.x * tiles.y, nz, most, per_sm * (nsm > 0 ? nsm : 1));
    out->grid = dim3(tiles.x, tiles.y, (nz + out->kchunk - 1) / out->kchunk);
    return 0;
}

// u_crf == 0 (the channel's usual frame) drops the frame-velocity terms
int rk_fused_prepare(const StepParams &p, RkLaunch *out)
{
    return rk_prepare(p.u_crf != 0.0 ? (const void *)k_rk_fused<true> : (const void *)k_rk_fused<false>, FT, fused_smem(),
                      fused_tiles(p), p.nz, F_KCHUNK, out);
}

int launch_rk_fused_fp64(const double *u, const double *v, const double *w, double *uo, double *vo, double *wo,
                         const StepParams &p, const MeshDev &m, MeanState &ms, const RkLaunch &l, cudaStream_t st)
{
    if ((int)(l.grid.x * l.grid.y * l.grid.z) > ms.max_blocks) {
        set_error("mean buffer too small for the fused RK kernel");
        return -1;
    }
    FConst K;
    K.hx = 0.25 * p.dt * p.dx_inv;
    K.hy = 0.25 * p.dt * p.dy_inv;
    K.gx = p.dt * p.dx_inv;
    K.gy = p.dt * p.dy_inv;
    K.cxx = p.dt * p.re_inv * p.dx_inv * p.dx_inv;
    K.cyy = p.dt * p.re_inv * p.dy_inv * p.dy_inv;
    K.ncc = -2.0 * (K.cxx + K.cyy);
    K.ucx = 0.5 * p.dt * p.u_crf * p.dx_inv;
    for (int q = 0; q < 3; q++) K.fb[q] = p.dt * p.fb[q];
    MeanRed r{ms.partial, ms.counter, ms.scalar, (double)p.nx, (double)p.ny, ms.vel_force};
    PL_CUDA_TRY(launch_chained(p.u_crf != 0.0 ? k_rk_fused<true> : k_rk_fused<false>, l.grid, dim3(FX, FT / FX),
                               fused_smem(), st, u, v, w, uo, vo, wo, p, m, K, r, l.kchunk));
    return 0;
}

} // namespace pl
