// adjoint.cu -- hand-written discrete adjoint of the FP64 RK2 projection step
// and the gradient of the kinetic energy after n steps with respect to the
// initial velocity and a uniform body force.
//
// The reference has no adjoint.  The forward map differentiated is the step of
// channel.cu, FP64 path, Thomas PPE (main.f90:137-208 plus the body force
// f added to the momentum right-hand side of both RK stages):
//   y1 = x + dt (R(E x) + f)                 RK1, E = wall/periodic fill
//   y2 = (y1 + dt (R(E y1) + f) + x) / 2     RK2
//   y3 = P y2                                calcRHS, PPE, correctVel
//   x' = y3 + (vel_force - Mean_h(y3)) e_x   forceVel
// Its adjoint, in reverse order:
//   forceVel^T : ybar3 = xbar' - (dzf_k / (lz nx ny)) sum(xbar'_u) e_x
//   P^T        : ybar2 = W P W^-1 ybar3, with W = dzf_k for u, v and dzc_k
//                for w: P is symmetric in the cell-volume inner product
//                (summation by parts of calcRHS against correctVel), so the
//                forward calcRHS + PPE + correctVel kernels apply it
//   RK2^T      : ybar1 = ybar2/2 + (dt/2) S(y1; ybar2)
//   RK1^T      : xbar  = ybar2/2 + ybar1 + dt S(x; ybar1)
//   fbar      += (dt/2) sum(ybar2) + dt sum(ybar1)     (per component)
// with S(q; r) = E^T J_R(E q)^T r, the transposed momentum stencil below.
// The degrees of freedom are u, v on levels 1..nz and w on levels 1..nz-1
// (w(nz) is the top wall).
//
// Checkpointing: the forward run stores the state every `every` steps; the
// reverse sweep recomputes each segment forward from its checkpoint, keeping
// the segment's states, and then runs the adjoint steps of the segment
// backwards.  Memory: ceil(n/every) + every states of 3 fields.
#include <algorithm>
#include <atomic>
#include <cmath>
#include <vector>

#include "channel.cuh"
#include "fft.cuh" // cp.async helpers
#include "stencil_rhs.cuh"

using namespace pl;

namespace {

constexpr int SUM_PARTS = MON_PARTS; // partial sums per level in the plane reductions

dim3 adj_block() { return dim3(64, 4, 1); }
dim3 adj_grid(const StepParams &p) { return dim3((p.nx + 63) / 64, (p.ny + 3) / 4, p.nz); }

// out = alpha r + beta S(q; r) + gamma e at every degree of freedom; the
// output's ghost planes are not written, and its w on level nz is zero.
// q: base state (BC-filled); r: adjoint fields with zero ghost planes and
// zero w on level nz.  Each flux of the momentum stencil shared by two
// equations (Pxy: y flux of u and x flux of v; Pxz: z flux of u and x flux
// of w; Pyz: z flux of v and y flux of w) gets one adjoint, the sum of the
// adjoints of its two uses; the adjoint of a flux difference
// -0.25 (F(o) - F(o-1)) h_o is -0.25 (h_o r(o) - h_{o+1} r(o+1)).
//
// 2.5D blocking as in the fused RK kernel: a CTA marches a 32 x 8 tile up a
// chunk of planes, with three-plane shared-memory rings of the six fields
// (halo 1 of 2 stored, so that copies are aligned pairs), one barrier per
// plane.  What a point needs of the plane below are the terms of the face
// between, which are those of that plane's upper face and stay in registers,
// as do the values above, the next plane's centre values: 30 shared loads a
// point.  A kernel of a point per thread, reading its 47 operands from L1 and
// L2, took 280 us at 256x192x128; this one takes 149, and 186 with the second
// operand e (3.0 and 3.2 TB/s at 72 and 96 B/point: six fields read and three
// written, and e).
constexpr int AX = 32, AY = 8, AW = AX + 4, AH = AY + 4, APS = AW * AH, AT = AX * AY, ASS = 6 * APS;

__global__ void __launch_bounds__(AT, 2) k_adj_rk(const double *__restrict__ u, const double *__restrict__ v,
                                                const double *__restrict__ w, const double *__restrict__ ru,
                                                const double *__restrict__ rv, const double *__restrict__ rw,
                                                const double *__restrict__ eu, const double *__restrict__ ev,
                                                const double *__restrict__ ew, double *__restrict__ ou,
                                                double *__restrict__ ov, double *__restrict__ ow, double alpha,
                                                double beta, double gamma, StepParams p, MeshDev m, int kchunk)
{
    extern __shared__ __align__(16) double ring[]; // [slot][u v w ru rv rw][xy]
    const int lane = threadIdx.x, wid = threadIdx.y, tid = lane + AX * wid;
    const int i0 = blockIdx.x * AX, j0 = blockIdx.y * AY;
    const int kbeg = blockIdx.z * kchunk + 1, kend = min(kbeg + kchunk - 1, p.nz);
    const size_t sk = (size_t)p.nx * p.ny;

    // copies: 12 rows of 18 aligned pairs per field and plane, a pair of each
    // field per thread; x and y wrap, nx is even
    constexpr int PAIRS = AH * (AW / 2);
    static_assert(PAIRS <= AT, "one pair per thread");
    const int cr = tid / (AW / 2), cc = tid % (AW / 2);
    const size_t soff = tid < PAIRS ? (size_t)((j0 - 2 + cr + p.ny) % p.ny) * p.nx + (i0 - 2 + 2 * cc + p.nx) % p.nx : 0;
    auto issue = [&](int k, int slot) {
        if (tid < PAIRS) {
            double *d = ring + slot * ASS + cr * AW + 2 * cc;
            const size_t o = sk * k + soff;
            cp_async_16(d, u + o);
            cp_async_16(d + APS, v + o);
            cp_async_16(d + 2 * APS, w + o);
            cp_async_16(d + 3 * APS, ru + o);
            cp_async_16(d + 4 * APS, rv + o);
            cp_async_16(d + 5 * APS, rw + o);
        }
        cp_async_commit();
    };
    const int i = i0 + lane, j = j0 + wid, xy = (2 + wid) * AW + 2 + lane;
    const bool inside = i < p.nx && j < p.ny;

    // plane k in slot (k - kbeg + 1) % 3
    issue(kbeg - 1, 0);
    issue(kbeg, 1);
    issue(kbeg + 1, 2);
    cp_async_wait<0>();
    __syncthreads();

    const double dxi = p.dx_inv, dyi = p.dy_inv, re = p.re_inv, q = 0.25;
    const double dxi2 = dxi * dxi, dyi2 = dyi * dyi, hc = 0.5 * p.u_crf * dxi;
    // mesh factors of the plane below, this plane and the plane above
    double f_m, f_c = __ldg(m.dzf + kbeg - 1), f_p = __ldg(m.dzf + kbeg);
    double ci_m, ci_c = __ldg(m.dzc_inv + kbeg - 1), ci_p = __ldg(m.dzc_inv + kbeg);
    double fi_c = __ldg(m.dzf_inv + kbeg - 1), fi_p = __ldg(m.dzf_inv + kbeg);
    // terms of the face below: the z differences of r, the products of the
    // base state with the flux adjoints
    double gu_m, gv_m, cw_m, tu_m, tv_m, zw_m;
    // centre values of plane k, and ru, u at x - 1, rv, v at y - 1
    double U, V, W, RU, RV, RW, Uxm, Vym, RUxm, RVym;
    auto above = [&](const double *n) { // n: the point in the plane above
        U = n[0];
        V = n[APS];
        W = n[2 * APS];
        RU = n[3 * APS];
        RV = n[4 * APS];
        RW = n[5 * APS];
        Uxm = n[-1];
        Vym = n[APS - AW];
        RUxm = n[3 * APS - 1];
        RVym = n[4 * APS - AW];
    };
    {
        const double *c = ring + xy, *n = c + ASS;
        gu_m = c[3 * APS] * fi_c - n[3 * APS] * fi_p;
        gv_m = c[4 * APS] * fi_c - n[4 * APS] * fi_p;
        cw_m = c[5 * APS] * ci_c - n[5 * APS] * ci_p;
        tu_m = (c[2 * APS] + c[2 * APS + 1]) * (-q * gu_m - q * dxi * (c[5 * APS] - c[5 * APS + 1]));
        tv_m = (c[2 * APS] + c[2 * APS + AW]) * (-q * gv_m - q * dyi * (c[5 * APS] - c[5 * APS + AW]));
        zw_m = (c[2 * APS] + n[2 * APS]) * (-q * cw_m);
        above(n);
    }
    int a = 1, b = 2, free = 0; // slots of the planes k, k + 1, k + 2
    for (int k = kbeg; k <= kend; k++) {
        __syncthreads(); // everyone is done with the slot of plane k - 1
        if (k < kend) issue(k + 2, free);
        f_m = f_c;
        f_c = f_p;
        f_p = __ldg(m.dzf + k + 1);
        ci_m = ci_c;
        ci_c = ci_p;
        ci_p = __ldg(m.dzc_inv + k + 1);
        fi_c = fi_p;
        fi_p = __ldg(m.dzf_inv + k + 1);
        const double *c = ring + a * ASS + xy, *n = ring + b * ASS + xy;
        const double *cv = c + APS, *cw = c + 2 * APS, *cru = c + 3 * APS, *crv = c + 4 * APS, *crw = c + 5 * APS;
        const double Uc = U, Vc = V, Wc = W, RUc = RU, RVc = RV, RWc = RW;
        const double Uxm_c = Uxm, Vym_c = Vym, RUxm_c = RUxm, RVym_c = RVym;
        above(n);
        const double Uxp = c[1], Uyp = c[AW], Uxmyp = c[AW - 1];
        const double Vxp = cv[1], Vyp = cv[AW], Vxpym = cv[1 - AW];
        const double Wxp = cw[1], Wyp = cw[AW];
        const double RUxp = cru[1], RUyp = cru[AW], RUym = cru[-AW], RUxmyp = cru[AW - 1];
        const double RVxp = crv[1], RVxm = crv[-1], RVyp = crv[AW], RVxpym = crv[1 - AW];
        const double RWxp = crw[1], RWxm = crw[-1], RWyp = crw[AW], RWym = crw[-AW];

        // z differences over the face above, here and at x - 1, y - 1
        const double gu = RUc * fi_c - RU * fi_p, gu_xm = RUxm_c * fi_c - RUxm * fi_p;
        const double gv = RVc * fi_c - RV * fi_p, gv_ym = RVym_c * fi_c - RVym * fi_p;
        const double cwz = RWc * ci_c - RW * ci_p;
        // flux adjoints
        const double Aux_c = -q * dxi * (RUc - RUxp), Aux_m = -q * dxi * (RUxm_c - RUc);
        const double Avy_c = -q * dyi * (RVc - RVyp), Avy_m = -q * dyi * (RVym_c - RVc);
        const double Pxy_c = -q * dyi * (RUc - RUyp) - q * dxi * (RVc - RVxp);
        const double Pxy_ym = -q * dyi * (RUym - RUc) - q * dxi * (RVym_c - RVxpym);
        const double Pxy_xm = -q * dyi * (RUxm_c - RUxmyp) - q * dxi * (RVxm - RVc);
        const double Pxz_c = -q * gu - q * dxi * (RWc - RWxp), Pxz_xm = -q * gu_xm - q * dxi * (RWxm - RWc);
        const double Pyz_c = -q * gv - q * dyi * (RWc - RWyp), Pyz_ym = -q * gv_ym - q * dyi * (RWym - RWc);
        const double tu = (Wc + Wxp) * Pxz_c, tv = (Wc + Wyp) * Pyz_c, zw = (Wc + W) * (-q * cwz);

        // convective part: flux adjoint times the derivative of the flux
        const double ut_c = (Uc * f_p + U * f_c) * ci_c, ut_xm = (Uxm_c * f_p + Uxm * f_c) * ci_c;
        const double vt_c = (Vc * f_p + V * f_c) * ci_c, vt_ym = (Vym_c * f_p + Vym * f_c) * ci_c;
        double su = 2.0 * (Uc + Uxp) * Aux_c + 2.0 * (Uxm_c + Uc) * Aux_m + (Vc + Vxp) * Pxy_c +
                    (Vym_c + Vxpym) * Pxy_ym + f_p * ci_c * tu + f_m * ci_m * tu_m;
        double sv = 2.0 * (Vc + Vyp) * Avy_c + 2.0 * (Vym_c + Vc) * Avy_m + (Uc + Uyp) * Pxy_c +
                    (Uxm_c + Uxmyp) * Pxy_xm + f_p * ci_c * tv + f_m * ci_m * tv_m;
        double sw = 2.0 * (zw + zw_m) + ut_c * Pxz_c + ut_xm * Pxz_xm + vt_c * Pyz_c + vt_ym * Pyz_ym;

        // u_crf advection: adjoint of -0.5 u_crf (q(i+1) - q(i-1)) dx_inv
        su -= hc * (RUxm_c - RUxp);
        sv -= hc * (RVxm - RVxp);
        sw -= hc * (RWxm - RWxp);

        // viscous part; the wall ghosts q(0) = 2bc - q(1), q(nz+1) = 2bc - q(nz)
        // of u and v double the wall-face coefficients
        const double ca = (k == 1) ? 2.0 : 1.0, cb = (k == p.nz) ? 2.0 : 1.0;
        su += re * ((RUxp - 2.0 * RUc + RUxm_c) * dxi2 + (RUyp - 2.0 * RUc + RUym) * dyi2) - cb * ci_c * re * gu +
              ca * ci_m * re * gu_m;
        sv += re * ((RVxp - 2.0 * RVc + RVxm) * dxi2 + (RVyp - 2.0 * RVc + RVym_c) * dyi2) - cb * ci_c * re * gv +
              ca * ci_m * re * gv_m;
        sw += re * ((RWxp - 2.0 * RWc + RWxm) * dxi2 + (RWyp - 2.0 * RWc + RWym) * dyi2) - fi_p * re * cwz +
              fi_c * re * cw_m;
        gu_m = gu;
        gv_m = gv;
        cw_m = cwz;
        tu_m = tu;
        tv_m = tv;
        zw_m = zw;

        if (inside) {
            const size_t g = (size_t)i + (size_t)p.nx * j + sk * k;
            double xu = alpha * RUc + beta * su, xv = alpha * RVc + beta * sv, xw = alpha * RWc + beta * sw;
            if (eu) {
                xu += gamma * __ldg(eu + g);
                xv += gamma * __ldg(ev + g);
                xw += gamma * __ldg(ew + g);
            }
            ou[g] = xu;
            ov[g] = xv;
            ow[g] = (k == p.nz) ? 0.0 : xw;
        }
        cp_async_wait<0>(); // plane k + 2
        const int t = a;
        a = b;
        b = free;
        free = t;
    }
}

int launch_adj_rk(const double *u, const double *v, const double *w, const double *ru, const double *rv,
                  const double *rw, const double *eu, const double *ev, const double *ew, double *ou, double *ov,
                  double *ow, double alpha, double beta, double gamma, const StepParams &p, const MeshDev &m,
                  const RkLaunch &l, cudaStream_t st)
{
    k_adj_rk<<<l.grid, dim3(AX, AY), sizeof(double) * 3 * ASS, st>>>(u, v, w, ru, rv, rw, eu, ev, ew, ou, ov, ow, alpha,
                                                                    beta, gamma, p, m, l.kchunk);
    PL_CHECK_LAUNCH();
    return 0;
}

// per-level partial sums of three fields over the degrees of freedom:
// MODE 0: sums of a, b, c; MODE 1: kinetic-energy terms dzf (a^2 + b^2) and
// dzc c^2.  part[((k-1) * SUM_PARTS + q) * 3 + comp], fixed summation order.
template <int MODE>
__global__ void __launch_bounds__(256) k_level_sums(const double *__restrict__ a, const double *__restrict__ b,
                                                    const double *__restrict__ c, StepParams p, MeshDev m,
                                                    double *__restrict__ part)
{
    __shared__ double sh[3][256];
    const int k = blockIdx.y + 1, q = blockIdx.x, t = threadIdx.x;
    const size_t sk = (size_t)p.nx * p.ny, n = sk;
    const size_t chunk = (n + SUM_PARTS - 1) / SUM_PARTS;
    const size_t beg = chunk * q, end = min(n, beg + chunk);
    double s0 = 0.0, s1 = 0.0, s2 = 0.0;
    const double *pa = a + sk * k, *pb = b + sk * k, *pc = c + sk * k;
    for (size_t x = beg + t; x < end; x += 256) {
        const double va = __ldg(pa + x), vb = __ldg(pb + x), vc = __ldg(pc + x);
        if (MODE == 0) {
            s0 += va;
            s1 += vb;
            s2 += vc;
        } else {
            s0 += va * va;
            s1 += vb * vb;
            s2 += vc * vc;
        }
    }
    if (k == p.nz) s2 = 0.0; // w(nz) is the wall
    sh[0][t] = s0;
    sh[1][t] = s1;
    sh[2][t] = s2;
    __syncthreads();
    for (int h = 128; h > 0; h >>= 1) {
        if (t < h) {
            sh[0][t] += sh[0][t + h];
            sh[1][t] += sh[1][t + h];
            sh[2][t] += sh[2][t + h];
        }
        __syncthreads();
    }
    if (t == 0) {
        double *o = part + ((size_t)(k - 1) * SUM_PARTS + q) * 3;
        if (MODE == 0) {
            o[0] = sh[0][0];
            o[1] = sh[1][0];
            o[2] = sh[2][0];
        } else {
            const double fz = __ldg(m.dzf + k), cz = 1.0 / __ldg(m.dzc_inv + k);
            o[0] = fz * sh[0][0];
            o[1] = fz * sh[1][0];
            o[2] = cz * sh[2][0];
        }
    }
}

// out[c] = (accumulate ? out[c] : 0) + coef * sum of the level partials, one
// component per block, as a tree of fixed order (three threads adding the
// 1,024 partials of 128 levels one after the other waited on every load)
__global__ void __launch_bounds__(256) k_sums_finish(const double *__restrict__ part, int nz, double coef,
                                                     int accumulate, double *__restrict__ out)
{
    __shared__ double sh[256];
    const int c = blockIdx.x, t = threadIdx.x;
    double s = 0.0;
    for (int x = t; x < nz * SUM_PARTS; x += 256) s += part[(size_t)x * 3 + c];
    sh[t] = s;
    __syncthreads();
    for (int h = 128; h > 0; h >>= 1) {
        if (t < h) sh[t] += sh[t + h];
        __syncthreads();
    }
    if (t == 0) out[c] = (accumulate ? out[c] : 0.0) + coef * sh[0];
}

// forceVel^T and division by the cell volumes: z = W^-1 (xbar - c_k S e_x),
// c_k = dzf_k / (lz nx ny), S = sum of xbar_u (scal[0]) when x is forced
__global__ void __launch_bounds__(256) k_adj_prep(const double *__restrict__ au, const double *__restrict__ av,
                                                  const double *__restrict__ aw, double *__restrict__ zu,
                                                  double *__restrict__ zv, double *__restrict__ zw,
                                                  const double *__restrict__ scal, int forced_x, StepParams p,
                                                  MeshDev m)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    const int k = blockIdx.z + 1;
    if (i >= p.nx || j >= p.ny) return;
    const size_t g = (size_t)i + (size_t)p.nx * j + (size_t)p.nx * p.ny * k;
    const double fi = __ldg(m.dzf_inv + k);
    double xu = au[g];
    if (forced_x) xu -= __ldg(m.dzflzi + k) / ((double)p.nx * p.ny) * scal[0];
    zu[g] = xu * fi;
    zv[g] = av[g] * fi;
    zw[g] = (k == p.nz) ? 0.0 : aw[g] * __ldg(m.dzc_inv + k);
}

// correctVel on z with the solved p, then multiplication by the cell
// volumes: ybar2 = W (z - dt G p), in place; p interior-only, p(nz+1) = p(nz)
__global__ void __launch_bounds__(256) k_adj_correct(const double *__restrict__ pp, double *zu, double *zv,
                                                     double *zw, StepParams p, MeshDev m)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    const int k = blockIdx.z + 1;
    if (i >= p.nx || j >= p.ny) return;
    const size_t sk = (size_t)p.nx * p.ny;
    const int ip = (i == p.nx - 1) ? 0 : i + 1, jp = (j == p.ny - 1) ? 0 : j + 1;
    const size_t g = (size_t)i + (size_t)p.nx * j + sk * k;
    const size_t c0 = (size_t)i + (size_t)p.nx * j + sk * (k - 1);
    const double p0 = __ldg(pp + c0);
    const double pxp = __ldg(pp + (size_t)ip + (size_t)p.nx * j + sk * (k - 1));
    const double pyp = __ldg(pp + (size_t)i + (size_t)p.nx * jp + sk * (k - 1));
    const double dt = p.dt, fz = __ldg(m.dzf + k);
    zu[g] = (zu[g] - (pxp - p0) * (dt * p.dx_inv)) * fz;
    zv[g] = (zv[g] - (pyp - p0) * (dt * p.dy_inv)) * fz;
    if (k == p.nz) {
        zw[g] = 0.0;
    } else {
        const double pzp = __ldg(pp + c0 + sk), ci = __ldg(m.dzc_inv + k);
        zw[g] = (zw[g] - (pzp - p0) * dt * ci) / ci;
    }
}

// seed of the reverse sweep: dJ/dx_N = dx dy W x_N
__global__ void __launch_bounds__(256) k_adj_seed(const double *__restrict__ u, const double *__restrict__ v,
                                                  const double *__restrict__ w, double *__restrict__ au,
                                                  double *__restrict__ av, double *__restrict__ aw, double dxdy,
                                                  StepParams p, MeshDev m)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    const int k = blockIdx.z + 1;
    if (i >= p.nx || j >= p.ny) return;
    const size_t g = (size_t)i + (size_t)p.nx * j + (size_t)p.nx * p.ny * k;
    const double fz = __ldg(m.dzf + k);
    au[g] = dxdy * fz * u[g];
    av[g] = dxdy * fz * v[g];
    aw[g] = (k == p.nz) ? 0.0 : dxdy / __ldg(m.dzc_inv + k) * w[g];
}

// The adjoint's device memory: one allocation of the nine adjoint fields, the
// checkpoints, the segment's states (three fields each) and the sums, kept with
// the channel for the next call (a program takes gradients one after the
// other: six steps at 256x192x128 take 8.93 ms, 9.55 with the 1.2 GB allocated
// and freed by the call).  What all channels of the process keep together is
// at most 1/32 of the device's memory: a call that would leave more frees its
// own on return, as one that allocates another size frees first.  The ghost
// planes of xa, y2 and y1 are zero from the allocation on.
std::atomic<size_t> g_adj_kept{0}; // bytes, all channels

struct AdjWork {
    double *xa = nullptr, *y2 = nullptr, *y1 = nullptr; // adjoint fields (3 fields each)
    double *ck = nullptr, *seg = nullptr;               // checkpoints, segment states (3 fields each)
    double *part = nullptr, *scal = nullptr, *fbar = nullptr;
    double *pool = nullptr;
    size_t bytes = 0, kept = 0; // of the pool; of it, what g_adj_kept counts
    size_t limit = 0;           // of g_adj_kept
    RkLaunch rk;                // of k_adj_rk
    void release()
    {
        g_adj_kept -= kept;
        cudaFree(pool);
        pool = nullptr;
        bytes = kept = 0;
    }
    bool reserve(size_t nck, size_t nseg, const pl_channel *c)
    {
        const size_t f3 = 3 * c->nf, sums = 3 * SUM_PARTS * (size_t)c->nz + 16;
        const size_t need = ((3 + nck + nseg) * f3 + sums) * sizeof(double);
        g_adj_kept -= kept; // in use
        kept = 0;
        if (bytes < need) {
            release();
            if (cudaMalloc(&pool, need) != cudaSuccess ||
                cudaMemsetAsync(pool, 0, 3 * f3 * sizeof(double), c->stream) != cudaSuccess)
                return false;
            bytes = need;
        }
        xa = pool;
        y2 = xa + f3;
        y1 = y2 + f3;
        ck = y1 + f3;
        seg = ck + nck * f3;
        part = seg + nseg * f3;
        scal = part + 3 * SUM_PARTS * (size_t)c->nz;
        fbar = scal + 4;
        return cudaMemsetAsync(scal, 0, 16 * sizeof(double), c->stream) == cudaSuccess;
    }
    // the call is over
    void keep()
    {
        if (!pool) return;
        kept = bytes;
        if ((g_adj_kept += kept) > limit) release();
    }
};

int level_sums(int mode, const double *a, const double *b, const double *c, const pl_channel *ch, double *part,
               double coef, int accumulate, double *out)
{
    dim3 g(SUM_PARTS, ch->nz);
    if (mode == 0)
        k_level_sums<0><<<g, 256, 0, ch->stream>>>(a, b, c, ch->sp, ch->m, part);
    else
        k_level_sums<1><<<g, 256, 0, ch->stream>>>(a, b, c, ch->sp, ch->m, part);
    PL_CHECK_LAUNCH();
    k_sums_finish<<<3, 256, 0, ch->stream>>>(part, ch->nz, coef, accumulate, out);
    PL_CHECK_LAUNCH();
    return 0;
}

int copy3(double *du, double *dv, double *dw, const double *su, const double *sv, const double *sw, size_t nf,
          cudaStream_t st)
{
    PL_CUDA_TRY(cudaMemcpyAsync(du, su, sizeof(double) * nf, cudaMemcpyDeviceToDevice, st));
    PL_CUDA_TRY(cudaMemcpyAsync(dv, sv, sizeof(double) * nf, cudaMemcpyDeviceToDevice, st));
    PL_CUDA_TRY(cudaMemcpyAsync(dw, sw, sizeof(double) * nf, cudaMemcpyDeviceToDevice, st));
    return 0;
}

// one adjoint step at base state x (3 fields): W.xa holds xbar_{n+1} on entry
// and xbar_n on return; fbar accumulates
int adjoint_step(pl_channel *c, const double *xu, const double *xv, const double *xw, AdjWork &W)
{
    const size_t nf = c->nf;
    const StepParams &p = c->sp;
    cudaStream_t st = c->stream;
    double *au = W.xa, *av = W.xa + nf, *aw = W.xa + 2 * nf;
    double *bu = W.y2, *bv = W.y2 + nf, *bw = W.y2 + 2 * nf;
    double *cu = W.y1, *cv = W.y1 + nf, *cw = W.y1 + 2 * nf;
    // stage-1 state y1 = RK1(x) (with its wall fill) into u1, v1, w1
    if (launch_rk1_fp64(xu, xv, xw, c->u1, c->v1, c->w1, p, c->m, st)) return -1;
    c->stage1_stale = false;
    // forceVel^T, W^-1
    const int fx = c->cfg.is_forced[0];
    if (fx && level_sums(0, au, av, aw, c, W.part, 1.0, 0, W.scal)) return -1;
    k_adj_prep<<<adj_grid(p), adj_block(), 0, st>>>(au, av, aw, bu, bv, bw, W.scal, fx, p, c->m);
    PL_CHECK_LAUNCH();
    // P, then W
    const int rc = ppe_xfwd_div<double>(&c->ppe, channel_div_in(c, bu, bv, bw), c->p, nullptr, st);
    if (rc < 0) return -1;
    if (rc > 0 ? launch_calc_rhs_fp64(bu, bv, bw, c->p, p, c->m, st) || ppe_solve_fp64(&c->ppe, c->p, st)
               : ppe_solve_fp64_from_x(&c->ppe, c->p, st))
        return -1;
    k_adj_correct<<<adj_grid(p), adj_block(), 0, st>>>(c->p, bu, bv, bw, p, c->m);
    PL_CHECK_LAUNCH();
    if (level_sums(0, bu, bv, bw, c, W.part, 0.5 * p.dt, 1, W.fbar)) return -1;
    // RK2^T at y1
    if (launch_adj_rk(c->u1, c->v1, c->w1, bu, bv, bw, nullptr, nullptr, nullptr, cu, cv, cw, 0.5, 0.5 * p.dt, 0.0, p,
                      c->m, W.rk, st))
        return -1;
    if (level_sums(0, cu, cv, cw, c, W.part, p.dt, 1, W.fbar)) return -1;
    // RK1^T at x
    return launch_adj_rk(xu, xv, xw, cu, cv, cw, bu, bv, bw, au, av, aw, 1.0, p.dt, 0.5, p, c->m, W.rk, st);
}

} // namespace

void pl::adjoint_free(pl_channel *c)
{
    if (!c->adj) return;
    static_cast<AdjWork *>(c->adj)->release();
    delete static_cast<AdjWork *>(c->adj);
    c->adj = nullptr;
}

extern "C" int pl_adjoint_release(pl_channel *c)
{
    adjoint_free(c);
    return 0;
}

extern "C" int pl_channel_set_body_force(pl_channel *c, const double f[3])
{
    if (c->cfg.precision != PL_FP64 && (f[0] != 0.0 || f[1] != 0.0 || f[2] != 0.0)) {
        set_error("pl_channel_set_body_force: the body force is defined for the FP64 path only");
        return -1;
    }
    for (int d = 0; d < 3; d++) c->sp.fb[d] = f[d];
    return 0;
}

extern "C" int pl_channel_kinetic_energy(pl_channel *c, double *ke)
{
    std::lock_guard<std::mutex> lk(c->mon_mu);
    double *out = c->d_mon;
    int rc = level_sums(1, c->u, c->v, c->w, c, c->d_mon + MON_OUT, 1.0, 0, out);
    double h[3] = {0, 0, 0};
    if (!rc && cudaMemcpyAsync(h, out, sizeof(h), cudaMemcpyDeviceToHost, c->stream) != cudaSuccess) rc = -1;
    if (!rc && cudaStreamSynchronize(c->stream) != cudaSuccess) rc = -1;
    if (rc) {
        set_error("pl_channel_kinetic_energy: device error");
        return -1;
    }
    const double dx = c->cfg.lx / c->nx, dy = c->cfg.ly / c->ny;
    *ke = 0.5 * dx * dy * (h[0] + h[1] + h[2]);
    return 0;
}

extern "C" int pl_adjoint_ke_gradient(pl_channel *c, int nsteps, int every, double *ke, double *d_gu, double *d_gv,
                                      double *d_gw, double grad_f[3])
{
    if (c->cfg.precision != PL_FP64) {
        set_error("pl_adjoint_ke_gradient: the adjoint is defined for the FP64 path");
        return -1;
    }
    if (c->cfg.trid_parts > 1) {
        set_error("pl_adjoint_ke_gradient: needs the Thomas PPE (trid_parts 0 or 1); PDD's truncated solve is "
                  "not an exact inverse, so the transposed projection differs from the forward one");
        return -1;
    }
    if (nsteps < 0 || every < 1) {
        set_error("pl_adjoint_ke_gradient: nsteps must be >= 0 and every >= 1");
        return -1;
    }
    const size_t nf = c->nf;
    const StepParams &p = c->sp;
    cudaStream_t st = c->stream;
    const int nck = (nsteps + every - 1) / every;
    const int nseg = std::min(every, std::max(nsteps, 1));
    if (!c->adj) {
        RkLaunch l;
        if (rk_prepare((const void *)k_adj_rk, AT, sizeof(double) * 3 * ASS,
                       dim3((c->nx + AX - 1) / AX, (c->ny + AY - 1) / AY, 1), c->nz, c->nz, &l))
            return -1;
        size_t free_bytes = 0, total = 0;
        PL_CUDA_TRY(cudaMemGetInfo(&free_bytes, &total));
        AdjWork *w = new AdjWork();
        w->limit = total / 32;
        w->rk = l;
        c->adj = w;
    }
    AdjWork &W = *static_cast<AdjWork *>(c->adj);
    struct Keep { // on every way out
        AdjWork &w;
        ~Keep() { w.keep(); }
    } keeper{W};
    if (!W.reserve(std::max(nck, 1), nseg, c)) {
        W.release();
        (void)cudaGetLastError();
        set_error("pl_adjoint_ke_gradient: out of device memory for checkpoints and adjoint fields");
        return -1;
    }
    auto state = [&](double *base, int slot) { return base + 3 * nf * (size_t)slot; };

    // forward sweep with checkpoints
    if (launch_fill_bc_vel(c->u, c->v, c->w, p, st)) return -1;
    if (copy3(state(W.ck, 0), state(W.ck, 0) + nf, state(W.ck, 0) + 2 * nf, c->u, c->v, c->w, nf, st)) return -1;
    for (int n = 0; n < nsteps; n++) {
        if (n % every == 0) {
            double *s = state(W.ck, n / every);
            if (copy3(s, s + nf, s + 2 * nf, c->u, c->v, c->w, nf, st)) return -1;
        }
        if (pl_channel_step(c, 1)) return -1;
    }
    double *keout = W.scal + 8;
    if (level_sums(1, c->u, c->v, c->w, c, W.part, 1.0, 0, keout)) return -1;
    double h[3];
    PL_CUDA_TRY(cudaMemcpyAsync(h, keout, sizeof(h), cudaMemcpyDeviceToHost, st));
    PL_CUDA_TRY(cudaStreamSynchronize(st));
    const double dx = c->cfg.lx / c->nx, dy = c->cfg.ly / c->ny;
    *ke = 0.5 * dx * dy * (h[0] + h[1] + h[2]);
    k_adj_seed<<<adj_grid(p), adj_block(), 0, st>>>(c->u, c->v, c->w, W.xa, W.xa + nf, W.xa + 2 * nf, dx * dy, p,
                                                    c->m);
    PL_CHECK_LAUNCH();

    // reverse sweep, segment by segment
    for (int s = nck - 1; s >= 0; s--) {
        const int n0 = s * every, n1 = std::min(nsteps, n0 + every);
        const double *ck = state(W.ck, s);
        if (copy3(c->u, c->v, c->w, ck, ck + nf, ck + 2 * nf, nf, st)) return -1;
        for (int n = n0; n < n1; n++) {
            double *x = state(W.seg, n - n0);
            if (copy3(x, x + nf, x + 2 * nf, c->u, c->v, c->w, nf, st)) return -1;
            if (n < n1 - 1 && pl_channel_step(c, 1)) return -1;
        }
        for (int n = n1 - 1; n >= n0; n--) {
            const double *x = state(W.seg, n - n0);
            if (adjoint_step(c, x, x + nf, x + 2 * nf, W)) return -1;
        }
    }

    // results; the fields are left at the initial state
    if (copy3(d_gu, d_gv, d_gw, W.xa, W.xa + nf, W.xa + 2 * nf, nf, st)) return -1;
    const double *x0 = state(W.ck, 0);
    if (copy3(c->u, c->v, c->w, x0, x0 + nf, x0 + 2 * nf, nf, st)) return -1;
    PL_CUDA_TRY(cudaMemcpyAsync(grad_f, W.fbar, 3 * sizeof(double), cudaMemcpyDeviceToHost, st));
    PL_CUDA_TRY(cudaStreamSynchronize(st));
    return 0;
}
