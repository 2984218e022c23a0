// plain_flux.cu -- FP64 parity form of the momentum right-hand side and the
// low-storage RK update.  Compiled with -fmad=false: every multiply and add
// is rounded separately, in the operation order of the reference, so the
// results agree with a plain FP64 build of the Fortran bit for bit.
//
//   tstle4_kon   src/flow/tstle4_mod.F90:139-265
//   tstle4_diff  src/flow/tstle4_mod.F90:268-458 (no LES: qc = st*0)
//   tstle4_gradp src/flow/tstle4_mod.F90:461-529
//   rkstep       src/core/rungekutta_mod.F90:315-333
//
// GB300 note: FP64 issues at a small fraction of the FP32 rate on this part,
// so this kernel is FP64-compute bound (~430 flop per cell, incl. divides);
// it is the reference-order baseline, the mixed form is the fast path.
#include "internal.h"

namespace mg {
MG_PLAIN_BEGIN
namespace {

struct GridPtrs {
    int kk, jj, ii;
    const double *dx, *dy, *dz, *ddx, *ddy, *ddz, *rdx, *rdy, *rdz, *rddx, *rddy, *rddz;
    const double *wx, *wy, *wz;   // ddx**(-cwb), ddy**(-cwb), ddz**(-cwb)
};

struct Spacing {
    const double *dx, *dy, *dz, *ddx, *ddy, *ddz, *rdx, *rdy, *rdz, *rddx, *rddy, *rddz;
    const double *wx, *wy, *wz;
};

// The Werner-Wengle constants (wernerwengle_mod.F90:13-28) and the face
// codes of one grid, for swcle3d on NOS (code 5) faces.
struct Wall {
    double rho, gmol, cpo4, cpo5, cpo6, cpo8;
    int bc[6];
    bool any;
    // G equal to one value g0 on every point tstle4_diff reads: each face
    // mean pair hm(g0, g0) + hm(g0, g0) is the same number h2
    bool guni;
    double h2;
};

#define IX(k, j, i) ((long long)((i) - 1) * kk * jj + (long long)((j) - 1) * kk + ((k) - 1))
#define A(a, k, j, i) a[IX(k, j, i)]

__device__ __forceinline__ double dmax(double a, double b) { return a < b ? b : a; }
// harmonic face mean of tstle4_diff: g*g'/MAX(g+g', gmol)
__device__ __forceinline__ double hm(double a, double b, double gmol) {
    return a * b / dmax(a + b, gmol);
}

// tauwin (wernerwengle_mod.F90:64-87) over rho and dds, swcle3d_one
// (tstle4_mod.F90:1832-1844); ddsb = dds**(-cwb) comes from the host.
__device__ double swcle3d_one(const Wall& q, double dds, double ddsb, double u) {
    const double vz = copysign(1.0, u);
    const double uquern = fabs(u);
    double tauwin;
    if (uquern >= q.cpo6 / dds)
        tauwin = vz * q.rho * pow(ddsb * (q.cpo4 * uquern + q.cpo5 / dds), q.cpo8);
    else
        tauwin = vz * 2.0 * q.gmol * uquern / dds;
    return tauwin / q.rho / dds;
}

// swcle3d (tstle4_mod.F90:1756-1829) at one point, per component in the
// reference's face order (front, back, right, left, bottom, top); each face
// acts on the layer next to the wall over its rows 2..n-1.
__device__ double wall_u(double x, int k, int j, int i, const GridPtrs& s, const Wall& q, double u) {
    if (!q.any) return x;
    const bool ik = i >= 2 && i <= s.ii - 1 && k >= 2 && k <= s.kk - 1;
    const bool ij = i >= 2 && i <= s.ii - 1 && j >= 2 && j <= s.jj - 1;
    if (q.bc[2] == 5 && j == 3 && ik) x = x - swcle3d_one(q, s.ddy[j], s.wy[j], u);
    if (q.bc[3] == 5 && j == s.jj - 2 && ik) x = x - swcle3d_one(q, s.ddy[j], s.wy[j], u);
    if (q.bc[4] == 5 && k == 3 && ij) x = x - swcle3d_one(q, s.ddz[k], s.wz[k], u);
    if (q.bc[5] == 5 && k == s.kk - 2 && ij) x = x - swcle3d_one(q, s.ddz[k], s.wz[k], u);
    return x;
}
__device__ double wall_v(double x, int k, int j, int i, const GridPtrs& s, const Wall& q, double v) {
    if (!q.any) return x;
    const bool jk = j >= 2 && j <= s.jj - 1 && k >= 2 && k <= s.kk - 1;
    const bool ij = i >= 2 && i <= s.ii - 1 && j >= 2 && j <= s.jj - 1;
    if (q.bc[0] == 5 && i == 3 && jk) x = x - swcle3d_one(q, s.ddx[i], s.wx[i], v);
    if (q.bc[1] == 5 && i == s.ii - 2 && jk) x = x - swcle3d_one(q, s.ddx[i], s.wx[i], v);
    if (q.bc[4] == 5 && k == 3 && ij) x = x - swcle3d_one(q, s.ddz[k], s.wz[k], v);
    if (q.bc[5] == 5 && k == s.kk - 2 && ij) x = x - swcle3d_one(q, s.ddz[k], s.wz[k], v);
    return x;
}
__device__ double wall_w(double x, int k, int j, int i, const GridPtrs& s, const Wall& q, double w) {
    if (!q.any) return x;
    const bool jk = j >= 2 && j <= s.jj - 1 && k >= 2 && k <= s.kk - 1;
    const bool ik = i >= 2 && i <= s.ii - 1 && k >= 2 && k <= s.kk - 1;
    if (q.bc[0] == 5 && i == 3 && jk) x = x - swcle3d_one(q, s.ddx[i], s.wx[i], w);
    if (q.bc[1] == 5 && i == s.ii - 2 && jk) x = x - swcle3d_one(q, s.ddx[i], s.wx[i], w);
    if (q.bc[2] == 5 && j == 3 && ik) x = x - swcle3d_one(q, s.ddy[j], s.wy[j], w);
    if (q.bc[3] == 5 && j == s.jj - 2 && ik) x = x - swcle3d_one(q, s.ddy[j], s.wy[j], w);
    return x;
}

// One output point of tstle4 for the U component (kon, swcle3d, diff, gradp).
__device__ double uo_point(int k, int j, int i, int kk, int jj, const double* u, const double* v,
                           const double* w, const double* ut, const double* vt, const double* wt,
                           const double* p, const double* gg, const GridPtrs& s, const Wall& wl,
                           double gmol, double rho, double iles, double gpx) {
    const double *dx = s.dx, *dy = s.dy, *ddx = s.ddx, *ddy = s.ddy, *ddz = s.ddz;
    const double *rdx = s.rdx, *rdy = s.rdy, *rdz = s.rdz, *rddx = s.rddx, *rddy = s.rddy,
                 *rddz = s.rddz;
    double uo;
    {
        double ax = ddy[j] * ddz[k], ay = dx[i] * ddz[k], az = dx[i] * ddy[j];
        double fe = ax * (A(ut, k, j, i) + (A(ut, k, j, i + 1) - A(ut, k, j, i)) * 0.5 * dx[i] / ddx[i + 1]);
        double fw = ax * (A(ut, k, j, i - 1) + (A(ut, k, j, i) - A(ut, k, j, i - 1)) * 0.5 * dx[i - 1] / ddx[i]);
        double fn = ay * (A(vt, k, j, i) + A(vt, k, j, i + 1)) * 0.5;
        double fs = ay * (A(vt, k, j - 1, i) + A(vt, k, j - 1, i + 1)) * 0.5;
        double ft = az * (A(wt, k, j, i) + A(wt, k, j, i + 1)) * 0.5;
        double fb = az * (A(wt, k - 1, j, i) + A(wt, k - 1, j, i + 1)) * 0.5;
        double qe = 0.5 * fe * (A(u, k, j, i) + A(u, k, j, i + 1));
        double qw = 0.5 * fw * (A(u, k, j, i - 1) + A(u, k, j, i));
        double qn = 0.5 * fn * (A(u, k, j, i) + A(u, k, j + 1, i));
        double qs = 0.5 * fs * (A(u, k, j - 1, i) + A(u, k, j, i));
        double qt = 0.5 * ft * (A(u, k, j, i) + A(u, k + 1, j, i));
        double qb = 0.5 * fb * (A(u, k - 1, j, i) + A(u, k, j, i));
        uo = -(qe - qw + qn - qs + qt - qb) * rdx[i] * rddy[j] * rddz[k];
    }
    uo = wall_u(uo, k, j, i, s, wl, A(u, k, j, i));
    {
        double ax = ddy[j] * ddz[k], ay = dx[i] * ddz[k], az = dx[i] * ddy[j];
        double ge = A(gg, k, j, i + 1);
        double gw = A(gg, k, j, i);
        double gn = wl.guni ? wl.h2 : hm(A(gg, k, j, i), A(gg, k, j + 1, i), gmol) + hm(A(gg, k, j, i + 1), A(gg, k, j + 1, i + 1), gmol);
        double gs = wl.guni ? wl.h2 : hm(A(gg, k, j - 1, i), A(gg, k, j, i), gmol) + hm(A(gg, k, j - 1, i + 1), A(gg, k, j, i + 1), gmol);
        double gt = wl.guni ? wl.h2 : hm(A(gg, k, j, i), A(gg, k + 1, j, i), gmol) + hm(A(gg, k, j, i + 1), A(gg, k + 1, j, i + 1), gmol);
        double gb = wl.guni ? wl.h2 : hm(A(gg, k - 1, j, i), A(gg, k, j, i), gmol) + hm(A(gg, k - 1, j, i + 1), A(gg, k, j, i + 1), gmol);
        double qe = -ge * ax * rddx[i + 1] * (A(u, k, j, i + 1) - A(u, k, j, i));
        double qw = -gw * ax * rddx[i] * (A(u, k, j, i) - A(u, k, j, i - 1));
        double qn = -gn * ay * rdy[j] * (A(u, k, j + 1, i) - A(u, k, j, i));
        double qs = -gs * ay * rdy[j - 1] * (A(u, k, j, i) - A(u, k, j - 1, i));
        double qt = -gt * az * rdz[k] * (A(u, k + 1, j, i) - A(u, k, j, i));
        double qb = -gb * az * rdz[k - 1] * (A(u, k, j, i) - A(u, k - 1, j, i));
        double st = ((ge * (A(u, k, j, i + 1) - A(u, k, j, i)) * rddx[i + 1]) -
                     (gw * (A(u, k, j, i) - A(u, k, j, i - 1)) * rddx[i])) * ax +
                    ((gn * (A(v, k, j, i + 1) - A(v, k, j, i))) -
                     (gs * (A(v, k, j - 1, i + 1) - A(v, k, j - 1, i)))) * ddz[k] +
                    ((gt * (A(w, k, j, i + 1) - A(w, k, j, i))) -
                     (gb * (A(w, k - 1, j, i + 1) - A(w, k - 1, j, i)))) * ddy[j];
        double qc = st * iles;   // the LES cross term (iles = 0 without LES model)
        double fak = 1.0 / rho * rddy[j] * rdx[i] * rddz[k];
        uo = uo - fak * (qe - qw + qn - qs + qt - qb - qc);
    }
    uo = uo - 1.0 / (rho * dx[i]) * (A(p, k, j, i + 1) - A(p, k, j, i) + gpx * dx[i]);
    return uo;
}

__device__ double vo_point(int k, int j, int i, int kk, int jj, const double* u, const double* v,
                           const double* w, const double* ut, const double* vt, const double* wt,
                           const double* p, const double* gg, const GridPtrs& s, const Wall& wl,
                           double gmol, double rho, double iles, double gpy) {
    const double *dy = s.dy, *ddx = s.ddx, *ddy = s.ddy, *ddz = s.ddz;
    const double *rdx = s.rdx, *rdy = s.rdy, *rdz = s.rdz, *rddx = s.rddx, *rddy = s.rddy,
                 *rddz = s.rddz;
    double vo;
    {
        double ax = dy[j] * ddz[k], ay = ddx[i] * ddz[k], az = ddx[i] * dy[j];
        double fe = ax * (A(ut, k, j, i) + A(ut, k, j + 1, i)) * 0.5;
        double fw = ax * (A(ut, k, j, i - 1) + A(ut, k, j + 1, i - 1)) * 0.5;
        double fn = ay * (A(vt, k, j, i) + (A(vt, k, j + 1, i) - A(vt, k, j, i)) * 0.5 * dy[j] / ddy[j + 1]);
        double fs = ay * (A(vt, k, j - 1, i) + (A(vt, k, j, i) - A(vt, k, j - 1, i)) * 0.5 * dy[j - 1] / ddy[j]);
        double ft = az * (A(wt, k, j, i) + A(wt, k, j + 1, i)) * 0.5;
        double fb = az * (A(wt, k - 1, j, i) + A(wt, k - 1, j + 1, i)) * 0.5;
        double qe = 0.5 * fe * (A(v, k, j, i) + A(v, k, j, i + 1));
        double qw = 0.5 * fw * (A(v, k, j, i - 1) + A(v, k, j, i));
        double qn = 0.5 * fn * (A(v, k, j, i) + A(v, k, j + 1, i));
        double qs = 0.5 * fs * (A(v, k, j - 1, i) + A(v, k, j, i));
        double qt = 0.5 * ft * (A(v, k, j, i) + A(v, k + 1, j, i));
        double qb = 0.5 * fb * (A(v, k - 1, j, i) + A(v, k, j, i));
        vo = -(qe - qw + qn - qs + qt - qb) * rddx[i] * rdy[j] * rddz[k];
    }
    vo = wall_v(vo, k, j, i, s, wl, A(v, k, j, i));
    {
        double ax = dy[j] * ddz[k], ay = ddx[i] * ddz[k], az = ddx[i] * dy[j];
        double ge = wl.guni ? wl.h2 : hm(A(gg, k, j, i), A(gg, k, j, i + 1), gmol) + hm(A(gg, k, j + 1, i), A(gg, k, j + 1, i + 1), gmol);
        double gw = wl.guni ? wl.h2 : hm(A(gg, k, j, i - 1), A(gg, k, j, i), gmol) + hm(A(gg, k, j + 1, i - 1), A(gg, k, j + 1, i), gmol);
        double gn = A(gg, k, j + 1, i);
        double gs = A(gg, k, j, i);
        double gt = wl.guni ? wl.h2 : hm(A(gg, k, j, i), A(gg, k + 1, j, i), gmol) + hm(A(gg, k, j + 1, i), A(gg, k + 1, j + 1, i), gmol);
        double gb = wl.guni ? wl.h2 : hm(A(gg, k - 1, j, i), A(gg, k, j, i), gmol) + hm(A(gg, k - 1, j + 1, i), A(gg, k, j + 1, i), gmol);
        double qe = -ge * ax * rdx[i] * (A(v, k, j, i + 1) - A(v, k, j, i));
        double qw = -gw * ax * rdx[i - 1] * (A(v, k, j, i) - A(v, k, j, i - 1));
        double qn = -gn * ay * rddy[j + 1] * (A(v, k, j + 1, i) - A(v, k, j, i));
        double qs = -gs * ay * rddy[j] * (A(v, k, j, i) - A(v, k, j - 1, i));
        double qt = -gt * az * rdz[k] * (A(v, k + 1, j, i) - A(v, k, j, i));
        double qb = -gb * az * rdz[k - 1] * (A(v, k, j, i) - A(v, k - 1, j, i));
        double st = ((ge * (A(u, k, j + 1, i) - A(u, k, j, i))) -
                     (gw * (A(u, k, j + 1, i - 1) - A(u, k, j, i - 1)))) * ddz[k] +
                    ((gn * (A(v, k, j + 1, i) - A(v, k, j, i)) * rddy[j + 1]) -
                     (gs * (A(v, k, j, i) - A(v, k, j - 1, i)) * rddy[j])) * ay +
                    ((gt * (A(w, k, j + 1, i) - A(w, k, j, i))) -
                     (gb * (A(w, k - 1, j + 1, i) - A(w, k - 1, j, i)))) * ddx[i];
        double qc = st * iles;
        double fak = 1.0 / rho * rddx[i] * rdy[j] * rddz[k];
        vo = vo - fak * (qe - qw + qn - qs + qt - qb - qc);
    }
    vo = vo - 1.0 / (rho * dy[j]) * (A(p, k, j + 1, i) - A(p, k, j, i) + gpy * dy[j]);
    return vo;
}

__device__ double wo_point(int k, int j, int i, int kk, int jj, const double* u, const double* v,
                           const double* w, const double* ut, const double* vt, const double* wt,
                           const double* p, const double* gg, const GridPtrs& s, const Wall& wl,
                           double gmol, double rho, double iles, double gpz) {
    const double *dz = s.dz, *ddx = s.ddx, *ddy = s.ddy, *ddz = s.ddz;
    const double *rdx = s.rdx, *rdy = s.rdy, *rdz = s.rdz, *rddx = s.rddx, *rddy = s.rddy,
                 *rddz = s.rddz;
    double wo;
    {
        double ax = ddy[j] * dz[k], ay = ddx[i] * dz[k], az = ddx[i] * ddy[j];
        double fe = ax * (A(ut, k, j, i) + A(ut, k + 1, j, i)) * 0.5;
        double fw = ax * (A(ut, k, j, i - 1) + A(ut, k + 1, j, i - 1)) * 0.5;
        double fn = ay * (A(vt, k, j, i) + A(vt, k + 1, j, i)) * 0.5;
        double fs = ay * (A(vt, k, j - 1, i) + A(vt, k + 1, j - 1, i)) * 0.5;
        double ft = az * (A(wt, k, j, i) + (A(wt, k + 1, j, i) - A(wt, k, j, i)) * 0.5 * dz[k] / ddz[k + 1]);
        double fb = az * (A(wt, k - 1, j, i) + (A(wt, k, j, i) - A(wt, k - 1, j, i)) * 0.5 * dz[k - 1] / ddz[k]);
        double qe = 0.5 * fe * (A(w, k, j, i) + A(w, k, j, i + 1));
        double qw = 0.5 * fw * (A(w, k, j, i - 1) + A(w, k, j, i));
        double qn = 0.5 * fn * (A(w, k, j, i) + A(w, k, j + 1, i));
        double qs = 0.5 * fs * (A(w, k, j - 1, i) + A(w, k, j, i));
        double qt = 0.5 * ft * (A(w, k, j, i) + A(w, k + 1, j, i));
        double qb = 0.5 * fb * (A(w, k - 1, j, i) + A(w, k, j, i));
        wo = -(qe - qw + qn - qs + qt - qb) * rddx[i] * rddy[j] * rdz[k];
    }
    wo = wall_w(wo, k, j, i, s, wl, A(w, k, j, i));
    {
        double ax = ddy[j] * dz[k], ay = ddx[i] * dz[k], az = ddx[i] * ddy[j];
        double ge = wl.guni ? wl.h2 : hm(A(gg, k, j, i), A(gg, k, j, i + 1), gmol) + hm(A(gg, k + 1, j, i), A(gg, k + 1, j, i + 1), gmol);
        double gw = wl.guni ? wl.h2 : hm(A(gg, k, j, i - 1), A(gg, k, j, i), gmol) + hm(A(gg, k + 1, j, i - 1), A(gg, k + 1, j, i), gmol);
        double gn = wl.guni ? wl.h2 : hm(A(gg, k, j, i), A(gg, k, j + 1, i), gmol) + hm(A(gg, k + 1, j, i), A(gg, k + 1, j + 1, i), gmol);
        double gs = wl.guni ? wl.h2 : hm(A(gg, k, j - 1, i), A(gg, k, j, i), gmol) + hm(A(gg, k + 1, j - 1, i), A(gg, k + 1, j, i), gmol);
        double gt = A(gg, k + 1, j, i);
        double gb = A(gg, k, j, i);
        double qe = -ge * ax * rdx[i] * (A(w, k, j, i + 1) - A(w, k, j, i));
        double qw = -gw * ax * rdx[i - 1] * (A(w, k, j, i) - A(w, k, j, i - 1));
        double qn = -gn * ay * rdy[j] * (A(w, k, j + 1, i) - A(w, k, j, i));
        double qs = -gs * ay * rdy[j - 1] * (A(w, k, j, i) - A(w, k, j - 1, i));
        double qt = -gt * az * rddz[k + 1] * (A(w, k + 1, j, i) - A(w, k, j, i));
        double qb = -gb * az * rddz[k] * (A(w, k, j, i) - A(w, k - 1, j, i));
        double st = ((ge * (A(u, k + 1, j, i) - A(u, k, j, i))) -
                     (gw * (A(u, k + 1, j, i - 1) - A(u, k, j, i - 1)))) * ddy[j] +
                    ((gn * (A(v, k + 1, j, i) - A(v, k, j, i))) -
                     (gs * (A(v, k + 1, j - 1, i) - A(v, k, j - 1, i)))) * ddx[i] +
                    ((gt * (A(w, k + 1, j, i) - A(w, k, j, i)) * rddz[k + 1]) -
                     (gb * (A(w, k, j, i) - A(w, k - 1, j, i)) * rddz[k])) * az;
        double qc = st * iles;
        double fak = 1.0 / rho * rddx[i] * rddy[j] * rdz[k];
        wo = wo - fak * (qe - qw + qn - qs + qt - qb - qc);
    }
    wo = wo - 1.0 / (rho * dz[k]) * (A(p, k + 1, j, i) - A(p, k, j, i) + gpz * dz[k]);
    return wo;
}

__device__ __forceinline__ bool all_connected(const DevGrid& G) {
    bool r = true;
    for (int f = 0; f < 6; ++f) r = r && G.bc[f] == 7;
    return r;
}

// tstle4 over the full box of every grid: points outside the reference's
// loop ranges get 0, as tstle4 zeroes uo, vo, wo before its loops.
__global__ void __launch_bounds__(256) k_tstle4(const DevGrid* __restrict__ grids, Spacing sp,
                                                double* __restrict__ uo, double* __restrict__ vo,
                                                double* __restrict__ wo, const double* __restrict__ U,
                                                const double* __restrict__ V, const double* __restrict__ W,
                                                const double* __restrict__ UT, const double* __restrict__ VT,
                                                const double* __restrict__ WT,
                                                const double* __restrict__ P, const double* __restrict__ Gf,
                                                Wall wl, double iles, double gx, double gy, double gz,
                                                const double* __restrict__ FX, const double* __restrict__ FY,
                                                const double* __restrict__ FZ, const double* __restrict__ GU,
                                                const double* __restrict__ redo) {
    const int gi = blockIdx.y;
    const DevGrid G = grids[gi];
    if (redo && redo[gi] == 0.0) return;   // k_tstle4_march has done it
    const int kk = G.kk, jj = G.jj, ii = G.ii;
    const int npts = kk * jj * ii;
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= npts) return;
    const int k = t % kk + 1;
    const int j = (t / kk) % jj + 1;
    const int i = t / (kk * jj) + 1;
    if (GU) {
        wl.guni = GU[2 * gi] != 0.0;
        wl.h2 = GU[2 * gi + 1];
    }
    GridPtrs s;
    s.kk = kk; s.jj = jj; s.ii = ii;
    s.dx = sp.dx + G.ipx - 1; s.dy = sp.dy + G.ipy - 1; s.dz = sp.dz + G.ipz - 1;
    s.ddx = sp.ddx + G.ipx - 1; s.ddy = sp.ddy + G.ipy - 1; s.ddz = sp.ddz + G.ipz - 1;
    s.rdx = sp.rdx + G.ipx - 1; s.rdy = sp.rdy + G.ipy - 1; s.rdz = sp.rdz + G.ipz - 1;
    s.rddx = sp.rddx + G.ipx - 1; s.rddy = sp.rddy + G.ipy - 1; s.rddz = sp.rddz + G.ipz - 1;
    s.wx = sp.wx + G.ipx - 1; s.wy = sp.wy + G.ipy - 1; s.wz = sp.wz + G.ipz - 1;
    const long long o = G.ip3;
    const double *u = U + o, *v = V + o, *w = W + o, *p = P + o, *g = Gf + o;
    const double *ut = UT + o, *vt = VT + o, *wt = WT + o;
    const int nfro = G.bc[0], nbac = G.bc[1], nrgt = G.bc[2], nlft = G.bc[3], nbot = G.bc[4],
              ntop = G.bc[5];
    const int nbu = (nbac == 7 || nbac == 3) ? 1 : 0;
    const int nlv = (nlft == 7 || nlft == 3) ? 1 : 0;
    const int ntw = (ntop == 7 || ntop == 3) ? 1 : 0;
    const int nfu = nfro == 3 ? 1 : 0, nrv = nrgt == 3 ? 1 : 0, nbw = nbot == 3 ? 1 : 0;
    const double gfl = (double)G.gradpflag;
    const bool jin = j >= 3 && j <= jj - 2, kin = k >= 3 && k <= kk - 2, iin = i >= 3 && i <= ii - 2;
    for (int f = 0; f < 6; ++f) wl.bc[f] = G.bc[f];
    wl.any = nfro == 5 || nbac == 5 || nrgt == 5 || nlft == 5 || nbot == 5 || ntop == 5;
    const double gmol = wl.gmol, rho = wl.rho;
    // outside the flux ranges uo, vo, wo are zero apart from swcle3d's rows
    double ru, rv, rw;
    // the steady body force FX, FY, FZ (when set) follows gradp
    if (i >= 3 - nfu && i <= ii - 3 + nbu && jin && kin) {
        ru = uo_point(k, j, i, kk, jj, u, v, w, ut, vt, wt, p, g, s, wl, gmol, rho, iles, gx * gfl);
        if (FX) ru = ru + FX[o + t];
    } else {
        ru = wall_u(0.0, k, j, i, s, wl, u[t]);
    }
    if (iin && j >= 3 - nrv && j <= jj - 3 + nlv && kin) {
        rv = vo_point(k, j, i, kk, jj, u, v, w, ut, vt, wt, p, g, s, wl, gmol, rho, iles, gy * gfl);
        if (FY) rv = rv + FY[o + t];
    } else {
        rv = wall_v(0.0, k, j, i, s, wl, v[t]);
    }
    if (iin && jin && k >= 3 - nbw && k <= kk - 3 + ntw) {
        rw = wo_point(k, j, i, kk, jj, u, v, w, ut, vt, wt, p, g, s, wl, gmol, rho, iles, gz * gfl);
        if (FZ) rw = rw + FZ[o + t];
    } else {
        rw = wall_w(0.0, k, j, i, s, wl, w[t]);
    }
    uo[o + t] = ru;
    vo[o + t] = rv;
    wo[o + t] = rw;
}

// ---- tstle4 of grids between other grids -------------------------------------
// Most grids have six connected faces, one value of G and no model term.  There a
// face flux of one cell is, operation for operation, that of its neighbour across the
// face (qe(i) = qw(i+1), ...), so each is computed once: a thread keeps a column
// (k, j) and marches in i, the fluxes through its i face stay in registers, those
// through its j and k faces reach the neighbours through shared memory.  The model
// term st*0 is zero for finite fields and falls away; a grid with a result that is not
// finite is left to k_tstle4, as one with several values of G is.
// Bound by the FP64 pipe (ncu: busy all the time on the SMs with a CTA): 526
// instructions a cell in k_tstle4, 195 here (343 grids of 24^3, with the faces that two
// CTAs compute and the idle lanes of partial warps).  512 grids of 24^3
// contracted 6.15 -> 2.72 ms, 64 grids uncontracted 0.95 -> 0.45, 216 of 20^3 1.84 ->
// 0.74.

// (a comparison of doubles is an FP64 instruction, one of their words is not)
__device__ __forceinline__ bool is_zero(double x) {
    return ((__double2hiint(x) & 0x7fffffff) | __double2loint(x)) == 0;
}
__device__ __forceinline__ bool is_finite(double x) { return (__double2hiint(x) & 0x7ff00000) != 0x7ff00000; }

// x / 2: the exponent less one, an integer operation, where that is exact
__device__ __forceinline__ double half_of(double x) {
    const int hi = __double2hiint(x), lo = __double2loint(x), e = hi & 0x7ff00000;
    if (e > 0x00100000 && e < 0x7ff00000) return __hiloint2double(hi - 0x00100000, lo);
    return is_zero(x) ? x : x * 0.5;
}

// x / d with r = RN(1 / d): Markstein's correction (P. Markstein, IBM J. Res. Dev. 34,
// 1990) -- after one step the quotient is within an ulp, after the second it is the
// correctly rounded one, for operands whose products stay normal.  mid: d is one of
// them.
__device__ __forceinline__ bool mid_range(double x) {
    return (unsigned)((__double2hiint(x) >> 20) & 0x7ff) - 523u < 1000u;   // 2^-500 .. 2^499
}
__device__ __forceinline__ double div_by(double x, double d, double r, bool mid) {
    if (is_zero(x)) return x;   // (d > 0)
    if (!mid || !mid_range(x)) return x / d;
    double q = __dmul_rn(x, r);
    q = __fma_rn(__fma_rn(-d, q, x), r, q);
    return __fma_rn(__fma_rn(-d, q, x), r, q);
}

struct MarchArgs {
    const DevGrid* grids;
    Spacing sp;
    double *uo, *vo, *wo;
    const double *U, *V, *W, *P, *G, *FX, *FY, *FZ, *GU;
    Wall wl;
    double* redo;                  // [ngrid] not 0: k_tstle4 does the grid
    double gx, gy, gz;
    int rows, nrow, len, nchunk;   // rows and planes of a CTA; CTAs along j and i
};

// what a plane of constant i needs
struct MarchPlane {
    double dx, ddx, rdx, rddx;
    double ddxe, rddxe, rcp;       // ddx and rddx at i+1, 1 / ddx(i+1)
    double pu, gdx;                // 1/(rho dx), gpx dx
};
// products of a plane with a row k or j: face areas, and with the viscosity
struct MarchK {
    double ayu, ayv, ayw, nyu, nyv, nyw;
};
struct MarchJ {
    double azu, azv, azw, nzu, nzv, nzw, fu, fv, fw;   // f: 1/rho and the spacings but k's
};

constexpr int kMarchThreads = 640;

__device__ __forceinline__ GridPtrs march_spacing(const MarchArgs& a, const DevGrid& G) {
    GridPtrs s;
    s.kk = G.kk; s.jj = G.jj; s.ii = G.ii;
    s.dx = a.sp.dx + G.ipx - 1; s.dy = a.sp.dy + G.ipy - 1; s.dz = a.sp.dz + G.ipz - 1;
    s.ddx = a.sp.ddx + G.ipx - 1; s.ddy = a.sp.ddy + G.ipy - 1; s.ddz = a.sp.ddz + G.ipz - 1;
    s.rdx = a.sp.rdx + G.ipx - 1; s.rdy = a.sp.rdy + G.ipy - 1; s.rdz = a.sp.rdz + G.ipz - 1;
    s.rddx = a.sp.rddx + G.ipx - 1; s.rddy = a.sp.rddy + G.ipy - 1; s.rddz = a.sp.rddz + G.ipz - 1;
    return s;
}

__global__ void __launch_bounds__(kMarchThreads) k_tstle4_march(const __grid_constant__ MarchArgs a) {
    const int gi = blockIdx.y;
    const DevGrid G = a.grids[gi];
    if (!all_connected(G) || a.GU[2 * gi] == 0.0) return;
    extern __shared__ __align__(16) unsigned char msm[];
    const int kk = G.kk, jj = G.jj, ii = G.ii, nt = blockDim.x, tid = threadIdx.x;
    const int row = blockIdx.x % a.nrow, chunk = blockIdx.x / a.nrow;
    const int ja = 3 + row * a.rows, je = min(ja + a.rows - 1, jj - 2);
    const int ia = 3 + chunk * a.len, ie = min(ia + a.len - 1, ii - 2);
    const long long o = G.ip3;
    double *uo = a.uo + o, *vo = a.vo + o, *wo = a.wo + o;
    const double *u = a.U + o, *v = a.V + o, *w = a.W + o, *p = a.P + o;
    const GridPtrs s = march_spacing(a, G);
    const double gfl = (double)G.gradpflag, rho = a.wl.rho;
    const double gx = a.gx * gfl, gy = a.gy * gfl, gz = a.gz * gfl;
    // the ghost layers: zero (tstle4 zeroes uo, vo, wo before its loops)
    {
        const int j0 = ja == 3 ? 1 : ja, j1 = je == jj - 2 ? jj : je;
        const int i0 = ia == 3 ? 1 : ia, i1 = ie == ii - 2 ? ii : ie;
        for (int t = tid; t < (j1 - j0 + 1) * kk; t += nt) {
            const int k = t % kk + 1, j = t / kk + j0;
            const bool shell = k < 3 || k > kk - 2 || j < 3 || j > jj - 2;
            for (int i = i0; i <= i1; ++i)
                if (shell || i < 3 || i > ii - 2) {
                    const long long c = IX(k, j, i);
                    uo[c] = 0.0;
                    vo[c] = 0.0;
                    wo[c] = 0.0;
                }
        }
    }
    const int nk1 = kk - 3;
    const int k = 2 + tid % nk1, j = ja - 1 + tid / nk1;
    const bool on = j <= je, out = on && k >= 3 && j >= ja;
    const double g0 = A((a.G + o), 3, 3, 3), h2 = a.GU[2 * gi + 1], ir = 1.0 / rho;
    // faces: [2][12][nt]; planes ia-1 .. ie
    double* face = reinterpret_cast<double*>(msm);
    MarchPlane* pl = reinterpret_cast<MarchPlane*>(face + 24 * nt);
    bool mid = true;
    for (int q = tid; q <= ie - ia + 1; q += nt) {
        const int i = ia - 1 + q;
        MarchPlane m;
        m.dx = s.dx[i]; m.ddx = s.ddx[i]; m.rdx = s.rdx[i]; m.rddx = s.rddx[i];
        m.ddxe = s.ddx[i + 1]; m.rddxe = s.rddx[i + 1];
        m.rcp = 1.0 / m.ddxe;
        m.pu = 1.0 / (rho * m.dx);
        m.gdx = gx * m.dx;
        mid = mid && mid_range(m.ddxe);
        pl[q] = m;
    }
    MarchK* pk = reinterpret_cast<MarchK*>(pl + a.len + 1);
    MarchJ* pj = reinterpret_cast<MarchJ*>(pk + (a.len + 1) * nk1);
    const int nj1 = je - ja + 2;
    for (int t = tid; t < (ie - ia + 2) * nk1; t += nt) {
        const int i = ia - 1 + t / nk1, kq = 2 + t % nk1;
        MarchK m;
        m.ayu = s.dx[i] * s.ddz[kq]; m.nyu = -h2 * m.ayu;
        m.ayv = s.ddx[i] * s.ddz[kq]; m.nyv = -g0 * m.ayv;
        m.ayw = s.ddx[i] * s.dz[kq]; m.nyw = -h2 * m.ayw;
        pk[t] = m;
    }
    for (int t = tid; t < (ie - ia + 2) * nj1; t += nt) {
        const int i = ia - 1 + t / nj1, jq = ja - 1 + t % nj1;
        MarchJ m;
        m.azu = s.dx[i] * s.ddy[jq]; m.nzu = -h2 * m.azu;
        m.azv = s.ddx[i] * s.dy[jq]; m.nzv = -h2 * m.azv;
        m.azw = s.ddx[i] * s.ddy[jq]; m.nzw = -g0 * m.azw;
        m.fu = ir * s.rddy[jq] * s.rdx[i];
        m.fv = ir * s.rddx[i] * s.rdy[jq];
        m.fw = ir * s.rddx[i] * s.rddy[jq];
        pj[t] = m;
    }
    double dy = 1.0, ddy = 1.0, rdy = 1.0, rddy = 1.0, ddyn = 1.0, rddyn = 1.0;
    double dz = 1.0, ddz = 1.0, rdz = 1.0, rddz = 1.0, ddzt = 1.0, rddzt = 1.0;
    if (on) {
        dy = s.dy[j]; ddy = s.ddy[j]; rdy = s.rdy[j]; rddy = s.rddy[j]; ddyn = s.ddy[j + 1]; rddyn = s.rddy[j + 1];
        dz = s.dz[k]; ddz = s.ddz[k]; rdz = s.rdz[k]; rddz = s.rddz[k]; ddzt = s.ddz[k + 1]; rddzt = s.rddz[k + 1];
        mid = mid && mid_range(ddyn) && mid_range(ddzt);
    }
    mid = __syncthreads_and(mid);
    const double rcpy = 1.0 / ddyn, rcpz = 1.0 / ddzt;
    const double pv = 1.0 / (rho * dy), pw = 1.0 / (rho * dz), gdy = gy * dy, gdz = gz * dz;
    const double axu = ddy * ddz, axv = dy * ddz, axw = ddy * dz;
    const double eu = -g0 * axu, ev = -h2 * axv, ew = -h2 * axw;
    double u0 = 0.0, v0 = 0.0, w0 = 0.0, p0 = 0.0;
    long long c = IX(k, j, ia - 1);
    const int sj = kk, si = kk * jj;
    if (on) {
        u0 = u[c]; v0 = v[c]; w0 = w[c];
        p0 = p[c + si];
    }
    double cw[3] = {0.0, 0.0, 0.0}, dw[3] = {0.0, 0.0, 0.0};   // through the face before
    for (int q = 0; q <= ie - ia + 1; ++q) {
        const MarchPlane& m = pl[q];
        const MarchK& mk = pk[q * nk1 + k - 2];
        const MarchJ& mj = pj[q * nj1 + min(j - ja + 1, nj1 - 1)];
        double ce[3], de[3], u1 = 0.0, v1 = 0.0, w1 = 0.0;
        if (on) {
            const double un = u[c + sj], uk = u[c + 1], vk = v[c + 1], vn = v[c + sj], wn = w[c + sj], wk = w[c + 1];
            u1 = u[c + si]; v1 = v[c + si]; w1 = w[c + si];
            double f;
            // i face
            f = axu * (u0 + div_by(half_of(u1 - u0) * m.dx, m.ddxe, m.rcp, mid));
            ce[0] = half_of(f) * (u0 + u1);
            f = half_of(axv * (u0 + un));
            ce[1] = half_of(f) * (v0 + v1);
            f = half_of(axw * (u0 + uk));
            ce[2] = half_of(f) * (w0 + w1);
            de[0] = eu * m.rddxe * (u1 - u0);
            de[1] = ev * m.rdx * (v1 - v0);
            de[2] = ew * m.rdx * (w1 - w0);
            if (q > 0) {
                double* x = face + (q & 1) * 12 * nt + tid;
                f = half_of(mk.ayu * (v0 + v1));
                x[0] = half_of(f) * (u0 + un);
                x[nt] = mk.nyu * rdy * (un - u0);
                f = half_of(mj.azu * (w0 + w1));
                x[2 * nt] = half_of(f) * (u0 + uk);
                x[3 * nt] = mj.nzu * rdz * (uk - u0);
                f = mk.ayv * (v0 + div_by(half_of(vn - v0) * dy, ddyn, rcpy, mid));
                x[4 * nt] = half_of(f) * (v0 + vn);
                x[5 * nt] = mk.nyv * rddyn * (vn - v0);
                f = half_of(mj.azv * (w0 + wn));
                x[6 * nt] = half_of(f) * (v0 + vk);
                x[7 * nt] = mj.nzv * rdz * (vk - v0);
                f = half_of(mk.ayw * (v0 + vk));
                x[8 * nt] = half_of(f) * (w0 + wn);
                x[9 * nt] = mk.nyw * rdy * (wn - w0);
                f = mj.azw * (w0 + div_by(half_of(wk - w0) * dz, ddzt, rcpz, mid));
                x[10 * nt] = half_of(f) * (w0 + wk);
                x[11 * nt] = mj.nzw * rddzt * (wk - w0);
            }
        }
        __syncthreads();
        if (out && q > 0) {
            const double* x = face + (q & 1) * 12 * nt + tid;
            // fluxes through the faces: e w (this thread), n s (row before), t b (k before)
            auto sum = [&](int f, double e, double ww) {
                return e - ww + x[f * nt] - x[f * nt - nk1] + x[(f + 2) * nt] - x[(f + 2) * nt - 1];
            };
            double ru = -sum(0, ce[0], cw[0]) * m.rdx * rddy * rddz;
            ru = ru - mj.fu * rddz * sum(1, de[0], dw[0]);
            ru = ru - m.pu * (p[c + si] - p0 + m.gdx);
            double rv = -sum(4, ce[1], cw[1]) * m.rddx * rdy * rddz;
            rv = rv - mj.fv * rddz * sum(5, de[1], dw[1]);
            rv = rv - pv * (p[c + sj] - p0 + gdy);
            double rw = -sum(8, ce[2], cw[2]) * m.rddx * rddy * rdz;
            rw = rw - mj.fw * rdz * sum(9, de[2], dw[2]);
            rw = rw - pw * (p[c + 1] - p0 + gdz);
            if (!is_finite(ru) || !is_finite(rv) || !is_finite(rw)) a.redo[gi] = 1.0;
            // the steady body force (when set) follows gradp
            uo[c] = a.FX ? ru + a.FX[o + c] : ru;
            vo[c] = a.FY ? rv + a.FY[o + c] : rv;
            wo[c] = a.FZ ? rw + a.FZ[o + c] : rw;
            p0 = p[c + si];
        }
        u0 = u1; v0 = v1; w0 = w1;
#pragma unroll
        for (int f = 0; f < 3; ++f) {
            cw[f] = ce[f];
            dw[f] = de[f];
        }
        c += si;
    }
}

// rkstep: dp = frhs*dp + rhs; p = p + dtfu*dp over the whole flat array.
__global__ void k_rkstep(double* __restrict__ p, double* __restrict__ dp,
                         const double* __restrict__ rhs, double frhs, double dtfu, long long n) {
    long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (; t < n; t += stride) {
        double d = frhs * dp[t] + rhs[t];
        dp[t] = d;
        p[t] = p[t] + dtfu * d;
    }
}

}  // namespace

static Spacing spacing(Ctx* c) {
    Spacing s;
    s.dx = c->L("DX"); s.dy = c->L("DY"); s.dz = c->L("DZ");
    s.ddx = c->L("DDX"); s.ddy = c->L("DDY"); s.ddz = c->L("DDZ");
    s.rdx = c->L("RDX"); s.rdy = c->L("RDY"); s.rdz = c->L("RDZ");
    s.rddx = c->L("RDDX"); s.rddy = c->L("RDDY"); s.rddz = c->L("RDDZ");
    s.wx = c->L("WWX"); s.wy = c->L("WWY"); s.wz = c->L("WWZ");
    return s;
}

// Per grid {1, h2} when G holds one value g0 on the box 2..n-1 in every
// direction (all points of G that tstle4_diff reads), else {0, 0}; h2 is
// hm(g0, g0) + hm(g0, g0) by the same operations, so the shortcut keeps the
// bits.  Without an LES model G is gmol there on grids without walls.
__global__ void k_g_uniform(const DevGrid* __restrict__ grids, const double* __restrict__ Gf, double gmol,
                            double* __restrict__ out) {
    const DevGrid G = grids[blockIdx.x];   // (behind the pairs: 1 where k_tstle4 has to run)
    const int kk = G.kk, jj = G.jj, ii = G.ii;
    const int nk = kk - 2, nj = jj - 2, ni = ii - 2;
    const double* g = Gf + G.ip3;
    const double g0 = A(g, 2, 2, 2);
    int bad = 0;
    for (int t = threadIdx.x; t < ni * nj * nk; t += blockDim.x) {
        const int k = t % nk + 2, j = (t / nk) % nj + 2, i = t / (nk * nj) + 2;
        bad |= !(A(g, k, j, i) == g0);
    }
    bad = __syncthreads_or(bad);
    if (threadIdx.x == 0) {
        const double h = hm(g0, g0, gmol);
        out[2 * gridDim.x + blockIdx.x] = bad || !all_connected(G) ? 1.0 : 0.0;
        out[2 * blockIdx.x] = bad ? 0.0 : 1.0;
        out[2 * blockIdx.x + 1] = bad ? 0.0 : h + h;
    }
}

// Per grid {1, h2} where G is one value on the box 2..n-1 (see k_g_uniform)
// into the context's d_guni.
int launch_g_uniform(Ctx* c) {
    k_g_uniform<<<c->ngrid, 256, 0, c->stream>>>(c->d_grids, c->F("G"), c->prm.gmol, c->d_guni);
    MG_LAUNCHED(c);
    return 0;
}

static int max_points(Ctx* c) {
    int m = 0;
    for (const DevGrid& g : c->grids) m = std::max(m, g.kk * g.jj * g.ii);
    return m;
}

// Threads of k_tstle4_march: rows + 1 rows of k = 2 .. kk-2
static int march_threads(int rows, int kk) { return ((rows + 1) * (kk - 3) + 31) / 32 * 32; }

static size_t march_smem(int rows, int len, int kk) {
    return (size_t)24 * march_threads(rows, kk) * sizeof(double) +
           (len + 1) * (sizeof(MarchPlane) + (kk - 3) * sizeof(MarchK) + (rows + 1) * sizeof(MarchJ));
}
constexpr size_t kMarchSmem = 220 * 1024;

// How k_tstle4_march cuts the grids: rows (the row before a CTA's first is computed
// twice) and planes (the fluxes through its first i face twice) so that the largest
// share of an SM in FP64 work, whole warps times planes, is least.  Returns the grids it takes:
// equal dimensions, all six faces connected.
static int march_shape(Ctx* c, MarchArgs* m) {
    int n = 0;
    for (const DevGrid& G : c->grids) {
        bool con = true;
        for (int f = 0; f < 6; ++f) con = con && G.bc[f] == 7;
        n += con;
    }
    const DevGrid& G = c->grids[0];
    const int nk1 = G.kk - 3, nj = G.jj - 4, ni = G.ii - 4;
    if (!c->uniform || n == 0 || 2 * nk1 > kMarchThreads) return 0;
    const int most = std::min(nj, kMarchThreads / nk1 - 1);
    double best = 0.0;
    for (int rows = most; rows >= 1; --rows)
        for (int len = 1; len <= ni; ++len) {
            if (march_smem(rows, len, G.kk) > kMarchSmem) break;
            const int nrow = (nj + rows - 1) / rows, nchunk = (ni + len - 1) / len;
            const long long waves = ((long long)n * nrow * nchunk + 151) / 152;
            const double t = (double)waves * (len + 0.5) * (march_threads(rows, G.kk) / 32);
            if (best == 0.0 || t < best) {
                best = t;
                m->rows = rows;
                m->nrow = nrow;
                m->len = len;
                m->nchunk = nchunk;
            }
        }
    if (best == 0.0) return 0;
    return n;
}

int launch_tstle4(Ctx* c, double* uo, double* vo, double* wo, const double* u, const double* v,
                  const double* w, const double* ut, const double* vt, const double* wt,
                  const double* p, const double* g) {
    ProfScope ps_(c, "tstle4");
    dim3 grid((max_points(c) + 255) / 256, c->ngrid);
    k_g_uniform<<<c->ngrid, 256, 0, c->stream>>>(c->d_grids, g, c->prm.gmol, c->d_guni);
    MG_LAUNCHED(c);
    // wernerwengle_mod.F90:13-28 init_wernerwengle
    Wall wl = {};
    const double gmol = c->prm.gmol, rho = c->prm.rho, cwa = 8.3, cwb = 1.0 / 7.0;
    const double cpo1 = 1.0 - cwb, cpo2 = 1.0 + cwb;
    wl.rho = rho;
    wl.gmol = gmol;
    wl.cpo4 = cpo2 / cwa * std::pow(gmol / rho, cwb);
    wl.cpo5 = 0.5 * cpo1 * std::pow(cwa, cpo2 / cpo1) * std::pow(gmol / rho, cpo2);
    wl.cpo6 = 0.5 * gmol / rho * std::pow(cwa, 2.0 / cpo1);
    wl.cpo8 = 2.0 / cpo2;
    MarchArgs m{};
    if (int n = march_shape(c, &m); n > 0 && u == ut && v == vt && w == wt && !c->ilesmodel) {
        m.grids = c->d_grids;
        m.sp = spacing(c);
        m.uo = uo; m.vo = vo; m.wo = wo;
        m.U = u; m.V = v; m.W = w; m.P = p; m.G = g;
        if (c->bodyforce) {
            m.FX = c->F("FBX"); m.FY = c->F("FBY"); m.FZ = c->F("FBZ");
        }
        m.GU = c->d_guni;
        m.redo = c->d_guni + 2 * c->ngrid;
        m.wl = wl;
        m.gx = c->prm.gradp[0]; m.gy = c->prm.gradp[1]; m.gz = c->prm.gradp[2];
        const int threads = march_threads(m.rows, c->grids[0].kk);
        const size_t smem = march_smem(m.rows, m.len, c->grids[0].kk);
        MG_CUDA(cudaFuncSetAttribute(k_tstle4_march, cudaFuncAttributeMaxDynamicSharedMemorySize, kMarchSmem));
        k_tstle4_march<<<dim3(m.nrow * m.nchunk, c->ngrid), threads, smem, c->stream>>>(m);
        MG_LAUNCHED(c);
    }
    k_tstle4<<<grid, 256, 0, c->stream>>>(c->d_grids, spacing(c), uo, vo, wo, u, v, w, ut, vt, wt, p, g,
                                          wl, c->ilesmodel ? 1.0 : 0.0, c->prm.gradp[0], c->prm.gradp[1],
                                          c->prm.gradp[2],
                                          c->bodyforce ? c->F("FBX") : nullptr,
                                          c->bodyforce ? c->F("FBY") : nullptr,
                                          c->bodyforce ? c->F("FBZ") : nullptr, c->d_guni, m.redo);
    MG_LAUNCHED(c);
    // tstle4_mod.F90:114: tstle4_par after kon, diff and gradp (PAR faces)
    return launch_tstle4_par(c, uo, vo, wo, u, v, w, ut, vt, wt);
}

int launch_rkstep(Ctx* c, double* p, double* dp, const double* rhs, double frhs, double dtfu) {
    ProfScope ps_(c, "rkstep");
    long long n = c->idim3d;
    int blocks = (int)std::min<long long>((n + 255) / 256, 152LL * 16);
    k_rkstep<<<blocks, 256, 0, c->stream>>>(p, dp, rhs, frhs, dtfu, n);
    MG_LAUNCHED(c);
    return 0;
}

MG_PLAIN_END
}  // namespace mg
