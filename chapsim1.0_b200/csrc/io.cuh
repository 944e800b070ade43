// Main-domain (IO, x-periodic) substep, SOLVERRK3_MOM_io
// (src/SOLVERRK3_MOM_IO.f90:11-120) with explicit (iVisScheme = 0) or
// Crank-Nicolson (iVisScheme = 1, sweeps in io_cn.cuh) viscous terms, for a
// flow whose property fields (DENSITY0, Viscousity0, Viscousity) are given
// and held fixed unless the thermal solver (thermal.cuh) updates them.
//
//   k_io_props     DENSITY_Staggered + MU_Staggered (src/MASSFLUX_CALC_IO.f90:155-329), once per upload
//   k_io_divu      DIVG_U_io (src/DIVG.f90:140-246): DivU = div(u)/3
//   k_io_rhs_tile<CN> (FP64), k_io_rhs<CN> (FP32 storage)
//                  CONVECTION_X/Y/Z_io, VISCOUS_ALL_EXPLT_X/Y/Z_io (or VISCOUS_PAR_EXPLT_*), RHS_MOM_EXPLICIT_io
//                  (RK combination, EXPLT0 update, pressure gradient, grid sum of the
//                  bulk-forcing integrand), all components at once
//   k_io_massflux  bulk forcing subtraction + MASSFLUX_CALC_io (G += RHS)
//   k_io_div_fftx  DIVG_io (src/DIVG.f90:54-137) + forward x transform
//   (shared)       k_fftz / y-solve / k_fftz / k_fftx_inv of poisson.cuh: the
//                  discrete problem of FISHPACK_POIS3D_SIMPLE (same AMPH/ACPH/APPH operator
//                  and x/z eigenvalues); its singular kx = kz = 0 mode is fixed at
//                  phi_hat(y_1) = 0, which shifts DPH and PR by a constant only
//   k_io_correct   PRCALC_io (PR += DPH, minus BE*RHSLLPHI under CN), MASSFLUX_UPDATE_io
//                  (src/VELO_CORRECTION.f90:103-179), VELOCITY_CALC_io (Q = G/D_STG)
//   k_io_cfl       CFL_io (src/CFL.f90:55-107), including the viscous number
#pragma once
#include "common.cuh"
#include "fft.cuh"
#include "poisson.cuh"

#define IO_NT 256

// RHO is DENSITY0 and DEN is DENSITY (the same array while the thermal
// solver is off); MU0 is Viscousity0 and MU is Viscousity.
// PR0A/PR0B: PR0_io(:,:,:,1) and PR0_io(:,:,:,2) of iWeightedPre = 1 (NULL when
// off).  igrav/fa: iGravity and F_A of thermal_gravity (src/Flow_State.f90:95-125).
// F is the storage type of the flow fields G, Q, PR, EXPLT0, RHS, D_STG, MU_STG
// and DivU (NULL in FP64, whose right-hand side forms it): double, or float in the mixed-precision step.  The property
// fields (DENSITY, DENSITY0, Viscousity, Viscousity0) stay FP64 (they come
// from the FP64 property update), and the kernels evaluate in FP64.
template <typename F>
struct IoFieldsT {
    F *G, *Q, *PR, *EX0, *RHS;
    double *RHO, *MU0, *MU;
    F *DST, *MST, *DIVU;
    double* DEN;
    const double *PR0A = nullptr, *PR0B = nullptr;
    double fa = 0.0;
    int igrav = 0;
};
using IoFields = IoFieldsT<double>;

// iWeightedPre: pres_epslon (src/modules.f90:483)
#define IO_PRES_EPSLON 0.001

// PGM of RHS_MOM_EXPLICIT_io (src/RHS_MOM_EXPLICIT_io.f90:103-159): the
// pressure difference between point c and its lower neighbour cm times coe,
// blended with the two PR0_io layers when iWeightedPre = 1
template <typename F>
__device__ __forceinline__ double io_pgm(const IoFieldsT<F>& f, long long c, long long cm, double pc, double pm,
                                         double coe) {
    if (f.PR0A)
        return ((f.PR0B[c] - f.PR0B[cm]) * (0.25 - IO_PRES_EPSLON) + (f.PR0A[c] - f.PR0A[cm]) * 0.5 +
                (pc - pm) * (0.25 + IO_PRES_EPSLON)) * coe;
    return (pc - pm) * coe;
}


// ---------------------------------------------------------------------------
// DENSITY_Staggered and MU_Staggered at one point; d1, d2, d3 receive the point's D_STG as stored
template <typename F>
__device__ __forceinline__ void io_props_point(const Geo& g, const IoFieldsT<F>& f, int i, int j, int k, F& d1, F& d2, F& d3) {
    const int im = xmn(g, i), km = wrapm(k, g.N);
    const long long c = pidx(g, i, j, k);
    const double* R = f.RHO;
    const double* U0 = f.MU0;
    d1 = (F)((R[c] + R[pidx(g, im, j, k)]) * 0.5);
    d3 = (F)((R[c] + R[pidx(g, i, j, km)]) * 0.5);
    d2 = (F)(j >= 2 ? g.wff[j] * R[c] + g.wfb[j] * R[pidx(g, i, j - 1, k)] : R[pidx(g, i, 0, k)]);
    F m1, m3;
    if (j >= 2) {
        m1 = (F)(((U0[c] + U0[pidx(g, im, j, k)]) * g.wff[j] + (U0[pidx(g, i, j - 1, k)] + U0[pidx(g, im, j - 1, k)]) * g.wfb[j]) * 0.5);
        m3 = (F)(((U0[pidx(g, i, j, km)] + U0[c]) * g.wff[j] + (U0[pidx(g, i, j - 1, km)] + U0[pidx(g, i, j - 1, k)]) * g.wfb[j]) * 0.5);
    } else {
        m1 = m3 = (F)U0[pidx(g, i, 0, k)];
    }
    const F m2 = (F)((U0[c] + U0[pidx(g, im, j, k)] + U0[pidx(g, i, j, km)] + U0[pidx(g, im, j, km)]) * 0.5 * 0.5);
    f.DST[c] = d1;
    f.DST[c + g.FS] = d2;
    f.DST[c + 2 * g.FS] = d3;
    f.MST[c] = m1;
    f.MST[c + g.FS] = m2;
    f.MST[c + 2 * g.FS] = m3;
    if (j == g.M) {
        const long long ct = pidx(g, i, g.M + 1, k);
        f.DST[ct + g.FS] = (F)R[ct];
        f.MST[ct] = (F)U0[ct];
        f.MST[ct + 2 * g.FS] = (F)U0[ct];
    }
}

template <typename F>
__global__ void __launch_bounds__(IO_NT) k_io_props(Geo g, IoFieldsT<F> f) {
    const long long tot = io_points(g);
    for (long long t = (long long)blockIdx.x * IO_NT + threadIdx.x; t < tot; t += (long long)gridDim.x * IO_NT) {
        int i, j, k;
        io_decode(g, t, i, j, k);
        F d1, d2, d3;
        io_props_point(g, f, i, j, k, d1, d2, d3);
    }
}

// DIVG_U_io; also VELOCITY_CALC_io of the upload (Q = G / D_STG) when vel != 0
template <typename F>
__global__ void __launch_bounds__(IO_NT) k_io_velocity(Geo g, IoFieldsT<F> f) {
    const long long tot = io_points(g);
    for (long long t = (long long)blockIdx.x * IO_NT + threadIdx.x; t < tot; t += (long long)gridDim.x * IO_NT) {
        int i, j, k;
        io_decode(g, t, i, j, k);
        const long long c = pidx(g, i, j, k);
        const double g1 = f.G[c], g3 = f.G[c + 2 * g.FS], d1 = f.DST[c], d3 = f.DST[c + 2 * g.FS];
        f.Q[c] = (F)(g1 / d1);
        f.Q[c + 2 * g.FS] = (F)(g3 / d3);
        if (j >= 2) f.Q[c + g.FS] = (F)((double)f.G[c + g.FS] / (double)f.DST[c + g.FS]);
    }
}

template <typename F>
__global__ void __launch_bounds__(IO_NT) k_io_divu(Geo g, IoFieldsT<F> f) {
    const int L = g.L, N = g.N;  // L: row stride
    const long long tot = io_points(g);
    for (long long t = (long long)blockIdx.x * IO_NT + threadIdx.x; t < tot; t += (long long)gridDim.x * IO_NT) {
        int i, j, k;
        io_decode(g, t, i, j, k);
        const long long c = pidx(g, i, j, k);
        const F* Q = f.Q;
        const double u = Q[c], up = Q[pidx(g, xpn(g, i), j, k)];
        const double v = Q[c + g.FS], vp = Q[c + g.FS + L];
        const double w = Q[c + 2 * g.FS], wp = Q[pidx(g, i, j, wrapp(k, N)) + 2 * g.FS];
        const double DIVX = (up - u) * g.dxi;
        const double DIVY = (vp - v) * (g.dyfi[j] * 1.0);
        const double DIVZ = (wp - w) * (g.dzi * 1.0);
        f.DIVU[c] = (F)((DIVX + DIVY + DIVZ) / 3.0);
    }
}

// ---------------------------------------------------------------------------
// CONVECTION_X/Y/Z_io + the viscous terms + RHS_MOM_EXPLICIT_io, all three
// components per point.
//   CN = false (VisExplicit): VISCOUS_ALL_EXPLT_X/Y/Z_io, RHS = RK combination.
//   CN = true  (VisImplicit): VISCOUS_PAR_EXPLT_X/Y/Z_io
//     (src/VISCOUS_X_EXPLICIT_io.f90:131-293, VISCOUS_Y_EXPLICIT_io.f90:278-443,
//     VISCOUS_Z_EXPLICIT_io.f90:300-465): the explicit part joins the
//     convection term, the implicit part enters with alpha*dt
//     (RHS_MOM_EXPLICIT_io.f90:87-99).  The density-correction part
//     (DIVU_io, weight alpha*dt/2) is identically zero: it differentiates
//     G * DRHOI_STG, and DRHOI_STG = 1/D_STG - 1/(the same average of
//     DENSITY0) is 0 in every entry because DENSITY_IMPLICIT_add runs right
//     after DENSITY_Staggered on the same DENSITY0 (src/SOLVE.f90:123-127,
//     src/MASSFLUX_CALC_IO.f90:332-416), and 0 before that (MEMALLOCT.f90:209).
//     It is therefore not computed.  The v row j = 1 is left unwritten; the
//     Crank-Nicolson sweeps treat it as zero.
// The convection and viscous terms of one point: ex the explicit part, im the implicit one (CN only).
// A gives the fields at the point's neighbours: q, g, ms (component, di, dj, dk), u0, u, dv (di, dj, dk).
struct IoRow { double wffj, wfbj, wffp, wfbp, dyfij, dyfim, dycij, dycip; };  // y coefficients of row j
__device__ __forceinline__ IoRow io_row(const Geo& g, int j) {
    return {g.wff[j], g.wfb[j], g.wff[j + 1], g.wfb[j + 1], g.dyfi[j], g.dyfi[j - 1], g.dyci[j], g.dyci[j + 1]};
}
template <bool CN, class A>
__device__ __forceinline__ void io_rhs_terms(const Geo& g, const IoRow& y, const A& a, int j, double& ex1, double& ex2, double& ex3,
                                             double& im1, double& im2, double& im3) {
    const double cv = g.cvisc;
    const double wffj = y.wffj, wfbj = y.wfbj, wffp = y.wffp, wfbp = y.wfbp;
    const double dyfij = y.dyfij, dyfim = y.dyfim, dycij = y.dycij, dycip = y.dycip;
    ex2 = im1 = im2 = im3 = 0.0;
    // -------- x momentum: CONVECTION_X_io + viscous terms --------
    {
        const double H11F = (a.g(0, 1, 0, 0) + a.g(0, 0, 0, 0)) * (a.q(0, 1, 0, 0) + a.q(0, 0, 0, 0));
        const double H11B = (a.g(0, 0, 0, 0) + a.g(0, -1, 0, 0)) * (a.q(0, 0, 0, 0) + a.q(0, -1, 0, 0));
        const double H11 = (H11F - H11B) * (g.dxi * 0.5 * 0.5);
        const double H12F = (a.g(1, 0, 1, 0) + a.g(1, -1, 1, 0)) * (wffp * a.q(0, 0, 1, 0) + wfbp * a.q(0, 0, 0, 0));
        const double H12B = (a.g(1, 0, 0, 0) + a.g(1, -1, 0, 0)) * (wffj * a.q(0, 0, 0, 0) + wfbj * a.q(0, 0, -1, 0));
        const double H12 = (H12F - H12B) * (dyfij * 0.5 * 1.0);
        const double H13F = (a.g(2, 0, 0, 1) + a.g(2, -1, 0, 1)) * (a.q(0, 0, 0, 1) + a.q(0, 0, 0, 0));
        const double H13B = (a.g(2, 0, 0, 0) + a.g(2, -1, 0, 0)) * (a.q(0, 0, 0, 0) + a.q(0, 0, 0, -1));
        const double H13 = (H13F - H13B) * ((g.dzi * 0.5 * 0.5) * 1.0);
        ex1 = -(H11 + H12 + H13);
        if constexpr (!CN) {
            double DUDX = (a.q(0, 1, 0, 0) - a.q(0, 0, 0, 0)) * g.dxi;
            const double T11F = 0.5 * (a.u0(0, 0, 0) + a.u0(0, 0, 0)) * (DUDX - a.dv(0, 0, 0));
            DUDX = (a.q(0, 0, 0, 0) - a.q(0, -1, 0, 0)) * g.dxi;
            const double T11B = 0.5 * (a.u0(-1, 0, 0) + a.u0(-1, 0, 0)) * (DUDX - a.dv(-1, 0, 0));
            const double D11 = (T11F - T11B) * (2.0 * g.dxi * cv);
            double DUDY = (a.q(0, 0, 1, 0) - a.q(0, 0, 0, 0)) * dycip / 1.0;
            double DVDX = (a.q(1, 0, 1, 0) - a.q(1, -1, 1, 0)) * g.dxi;
            const double T12F = a.ms(0, 0, 1, 0) * (DUDY + DVDX);
            DUDY = (a.q(0, 0, 0, 0) - a.q(0, 0, -1, 0)) * dycij / 1.0;
            DVDX = (a.q(1, 0, 0, 0) - a.q(1, -1, 0, 0)) * g.dxi;
            const double T12B = a.ms(0, 0, 0, 0) * (DUDY + DVDX);
            const double D12 = (T12F - T12B) * (dyfij * cv * 1.0);
            double DUDZ = (a.q(0, 0, 0, 1) - a.q(0, 0, 0, 0)) * g.dzi;
            double DWDX = (a.q(2, 0, 0, 1) - a.q(2, -1, 0, 1)) * g.dxi;
            const double T13F = a.ms(1, 0, 0, 1) * (DUDZ + DWDX);
            DUDZ = (a.q(0, 0, 0, 0) - a.q(0, 0, 0, -1)) * g.dzi;
            DWDX = (a.q(2, 0, 0, 0) - a.q(2, -1, 0, 0)) * g.dxi;
            const double T13B = a.ms(1, 0, 0, 0) * (DUDZ + DWDX);
            const double D13 = (T13F - T13B) * ((g.dzi * cv) * 1.0);
            ex1 = ex1 + D11 + D12 + D13;
        } else {
            const double coe1 = -2.0 / 3.0 * g.dxi * cv;
            double DUDX = (a.q(0, 1, 0, 0) - a.q(0, 0, 0, 0)) * g.dxi;
            double DVDY = (a.q(1, 0, 1, 0) - a.q(1, 0, 0, 0)) * dyfij * 1.0;
            double DWDZ = (a.q(2, 0, 0, 1) - a.q(2, 0, 0, 0)) * g.dzi * 1.0;
            const double F_EX11 = a.u(0, 0, 0) * (DVDY + DWDZ), F_IM11 = a.u(0, 0, 0) * DUDX;
            DUDX = (a.q(0, 0, 0, 0) - a.q(0, -1, 0, 0)) * g.dxi;
            DVDY = (a.q(1, -1, 1, 0) - a.q(1, -1, 0, 0)) * dyfij * 1.0;
            DWDZ = (a.q(2, -1, 0, 1) - a.q(2, -1, 0, 0)) * g.dzi * 1.0;
            const double B_EX11 = a.u(-1, 0, 0) * (DVDY + DWDZ), B_IM11 = a.u(-1, 0, 0) * DUDX;
            const double D11_EX = (F_EX11 - B_EX11) * coe1;
            const double D11_IM = (F_IM11 - B_IM11) * coe1 * (-2.0);
            const double coe2 = dyfij * cv * 1.0;
            double DVDX = (a.q(1, 0, 1, 0) - a.q(1, -1, 1, 0)) * g.dxi;
            double DUDY = (a.q(0, 0, 1, 0) - a.q(0, 0, 0, 0)) * dycip / 1.0;
            const double F_EX12 = a.ms(0, 0, 1, 0) * DVDX, F_IM12 = a.ms(0, 0, 1, 0) * DUDY;
            DUDY = (a.q(0, 0, 0, 0) - a.q(0, 0, -1, 0)) * dycij / 1.0;
            DVDX = (a.q(1, 0, 0, 0) - a.q(1, -1, 0, 0)) * g.dxi;
            const double B_EX12 = a.ms(0, 0, 0, 0) * DVDX, B_IM12 = a.ms(0, 0, 0, 0) * DUDY;
            const double D12_EX = (F_EX12 - B_EX12) * coe2;
            const double D12_IM = (F_IM12 - B_IM12) * coe2;
            const double coe32 = (g.dzi * cv) * 1.0;
            double DUDZ = (a.q(0, 0, 0, 1) - a.q(0, 0, 0, 0)) * g.dzi;
            double DWDX = (a.q(2, 0, 0, 1) - a.q(2, -1, 0, 1)) * g.dxi;
            const double F_EX13 = a.ms(1, 0, 0, 1) * DWDX, F_IM13 = a.ms(1, 0, 0, 1) * DUDZ;
            DUDZ = (a.q(0, 0, 0, 0) - a.q(0, 0, 0, -1)) * g.dzi;
            DWDX = (a.q(2, 0, 0, 0) - a.q(2, -1, 0, 0)) * g.dxi;
            const double B_EX13 = a.ms(1, 0, 0, 0) * DWDX, B_IM13 = a.ms(1, 0, 0, 0) * DUDZ;
            const double D13_EX = (F_EX13 - B_EX13) * coe32;
            const double D13_IM = (F_IM13 - B_IM13) * coe32;
            ex1 = D11_EX + D12_EX + D13_EX + ex1;
            im1 = D11_IM + D12_IM + D13_IM;
        }
    }
    // -------- y momentum (j >= 2) --------
    if (j >= 2) {
        const double H21F = (wffj * a.g(0, 1, 0, 0) + wfbj * a.g(0, 1, -1, 0)) * (a.q(1, 1, 0, 0) + a.q(1, 0, 0, 0));
        const double H21B = (wffj * a.g(0, 0, 0, 0) + wfbj * a.g(0, 0, -1, 0)) * (a.q(1, 0, 0, 0) + a.q(1, -1, 0, 0));
        const double H21 = (H21F - H21B) * (g.dxi * 0.5);
        const double H22F = (a.g(1, 0, 1, 0) + a.g(1, 0, 0, 0)) * (a.q(1, 0, 1, 0) * 1.0 + a.q(1, 0, 0, 0) * 1.0);
        const double H22B = (a.g(1, 0, 0, 0) + a.g(1, 0, -1, 0)) * (a.q(1, 0, 0, 0) * 1.0 + a.q(1, 0, -1, 0) * 1.0);
        const double H22 = (H22F - H22B) * (dycij * 0.5 * 0.5);
        const double H23F = (wffj * a.g(2, 0, 0, 1) * 1.0 + wfbj * a.g(2, 0, -1, 1) * 1.0) * (a.q(1, 0, 0, 1) + a.q(1, 0, 0, 0));
        const double H23B = (wffj * a.g(2, 0, 0, 0) * 1.0 + wfbj * a.g(2, 0, -1, 0) * 1.0) * (a.q(1, 0, 0, 0) + a.q(1, 0, 0, -1));
        const double H23 = (H23F - H23B) * ((g.dzi * 0.5) * 1.0);
        ex2 = -(H21 + H22 + H23);
        if constexpr (!CN) {
            double DVDY = (a.q(1, 0, 1, 0) - a.q(1, 0, 0, 0)) * dyfij;
            const double T22F = 0.5 * (a.u0(0, 0, 0) + a.u0(0, 0, 0)) * (DVDY - a.dv(0, 0, 0));
            DVDY = (a.q(1, 0, 0, 0) - a.q(1, 0, -1, 0)) * dyfim;
            const double T22B = 0.5 * (a.u0(0, -1, 0) + a.u0(0, -1, 0)) * (DVDY - a.dv(0, -1, 0));
            const double D22 = (T22F - T22B) * (2.0 * dycij * cv);
            double DVDX = (a.q(1, 1, 0, 0) - a.q(1, 0, 0, 0)) * g.dxi;
            double DUDY = (a.q(0, 1, 0, 0) - a.q(0, 1, -1, 0)) * dycij;
            const double T21F = a.ms(0, 1, 0, 0) * (DVDX + DUDY);
            DVDX = (a.q(1, 0, 0, 0) - a.q(1, -1, 0, 0)) * g.dxi;
            DUDY = (a.q(0, 0, 0, 0) - a.q(0, 0, -1, 0)) * dycij;
            const double T21B = a.ms(0, 0, 0, 0) * (DVDX + DUDY);
            const double D21 = (T21F - T21B) * (g.dxi * cv);
            double DVDZ = (a.q(1, 0, 0, 1) - a.q(1, 0, 0, 0)) * g.dzi;
            double DWDY = (a.q(2, 0, 0, 1) - a.q(2, 0, -1, 1)) * dycij;
            const double T23F = a.ms(2, 0, 0, 1) * (DVDZ + DWDY);
            DVDZ = (a.q(1, 0, 0, 0) - a.q(1, 0, 0, -1)) * g.dzi;
            DWDY = (a.q(2, 0, 0, 0) - a.q(2, 0, -1, 0)) * dycij;
            const double T23B = a.ms(2, 0, 0, 0) * (DVDZ + DWDY);
            const double D23 = (T23F - T23B) * (g.dzi * cv);
            ex2 = ex2 + D21 + D22 + D23;
        } else {
            const double coe2 = -2.0 / 3.0 * dycij * cv;
            double DUDX = (a.q(0, 1, 0, 0) - a.q(0, 0, 0, 0)) * g.dxi;
            double DVDY = (a.q(1, 0, 1, 0) - a.q(1, 0, 0, 0)) * dyfij;
            double DWDZ = (a.q(2, 0, 0, 1) - a.q(2, 0, 0, 0)) * g.dzi;
            const double F_EX22 = a.u(0, 0, 0) * (DUDX + DWDZ), F_IM22 = a.u(0, 0, 0) * DVDY;
            DUDX = (a.q(0, 1, -1, 0) - a.q(0, 0, -1, 0)) * g.dxi;
            DVDY = (a.q(1, 0, 0, 0) - a.q(1, 0, -1, 0)) * dyfim;
            DWDZ = (a.q(2, 0, -1, 1) - a.q(2, 0, -1, 0)) * g.dzi;
            const double B_EX22 = a.u(0, -1, 0) * (DUDX + DWDZ), B_IM22 = a.u(0, -1, 0) * DVDY;
            const double D22_EX = (F_EX22 - B_EX22) * coe2;
            const double D22_IM = (F_IM22 - B_IM22) * coe2 * (-2.0);
            const double coe1 = g.dxi * cv;
            double DVDX = (a.q(1, 1, 0, 0) - a.q(1, 0, 0, 0)) * g.dxi;
            double DUDY = (a.q(0, 1, 0, 0) - a.q(0, 1, -1, 0)) * dycij;
            const double F_EX21 = a.ms(0, 1, 0, 0) * DUDY, F_IM21 = a.ms(0, 1, 0, 0) * DVDX;
            DVDX = (a.q(1, 0, 0, 0) - a.q(1, -1, 0, 0)) * g.dxi;
            DUDY = (a.q(0, 0, 0, 0) - a.q(0, 0, -1, 0)) * dycij;
            const double B_EX21 = a.ms(0, 0, 0, 0) * DUDY, B_IM21 = a.ms(0, 0, 0, 0) * DVDX;
            const double D21_EX = (F_EX21 - B_EX21) * coe1;
            const double D21_IM = (F_IM21 - B_IM21) * coe1;
            const double coe3 = g.dzi * cv;
            double DVDZ = (a.q(1, 0, 0, 1) - a.q(1, 0, 0, 0)) * g.dzi;
            double DWDY = (a.q(2, 0, 0, 1) - a.q(2, 0, -1, 1)) * dycij;
            const double F_EX23 = a.ms(2, 0, 0, 1) * DWDY, F_IM23 = a.ms(2, 0, 0, 1) * DVDZ;
            DVDZ = (a.q(1, 0, 0, 0) - a.q(1, 0, 0, -1)) * g.dzi;
            DWDY = (a.q(2, 0, 0, 0) - a.q(2, 0, -1, 0)) * dycij;
            const double B_EX23 = a.ms(2, 0, 0, 0) * DWDY, B_IM23 = a.ms(2, 0, 0, 0) * DVDZ;
            const double D23_EX = (F_EX23 - B_EX23) * coe3;
            const double D23_IM = (F_IM23 - B_IM23) * coe3;
            ex2 = D21_EX + D22_EX + D23_EX + ex2;
            im2 = D21_IM + D22_IM + D23_IM;
        }
    }
    // -------- z momentum --------
    {
        const double H31F = (a.g(0, 1, 0, 0) + a.g(0, 1, 0, -1)) * (a.q(2, 1, 0, 0) + a.q(2, 0, 0, 0));
        const double H31B = (a.g(0, 0, 0, 0) + a.g(0, 0, 0, -1)) * (a.q(2, 0, 0, 0) + a.q(2, -1, 0, 0));
        const double H31 = (H31F - H31B) * (g.dxi * 0.5 * 0.5);
        const double H32F = (a.g(1, 0, 1, 0) + a.g(1, 0, 1, -1)) * (wffp * a.q(2, 0, 1, 0) * 1.0 + wfbp * a.q(2, 0, 0, 0) * 1.0);
        const double H32B = (a.g(1, 0, 0, 0) + a.g(1, 0, 0, -1)) * (wffj * a.q(2, 0, 0, 0) * 1.0 + wfbj * a.q(2, 0, -1, 0) * 1.0);
        const double H32 = (H32F - H32B) * (dyfij * 0.5);
        const double H33F = (a.g(2, 0, 0, 1) + a.g(2, 0, 0, 0)) * (a.q(2, 0, 0, 1) + a.q(2, 0, 0, 0));
        const double H33B = (a.g(2, 0, 0, 0) + a.g(2, 0, 0, -1)) * (a.q(2, 0, 0, 0) + a.q(2, 0, 0, -1));
        const double H33 = (H33F - H33B) * ((g.dzi * 0.5 * 0.5) * 1.0);
        ex3 = -(H31 + H32 + H33);
        if constexpr (!CN) {
            double DWDZ = (a.q(2, 0, 0, 1) - a.q(2, 0, 0, 0)) * g.dzi;
            const double T33F = 0.5 * (a.u0(0, 0, 0) + a.u0(0, 0, 0)) * (DWDZ - a.dv(0, 0, 0));
            DWDZ = (a.q(2, 0, 0, 0) - a.q(2, 0, 0, -1)) * g.dzi;
            const double T33B = 0.5 * (a.u0(0, 0, -1) + a.u0(0, 0, -1)) * (DWDZ - a.dv(0, 0, -1));
            const double D33 = (T33F - T33B) * (2.0 * g.dzi * cv);
            double DWDX = (a.q(2, 1, 0, 0) - a.q(2, 0, 0, 0)) * g.dxi;
            double DUDZ = (a.q(0, 1, 0, 0) - a.q(0, 1, 0, -1)) * g.dzi;
            const double T31F = a.ms(1, 1, 0, 0) * (DWDX + DUDZ);
            DWDX = (a.q(2, 0, 0, 0) - a.q(2, -1, 0, 0)) * g.dxi;
            DUDZ = (a.q(0, 0, 0, 0) - a.q(0, 0, 0, -1)) * g.dzi;
            const double T31B = a.ms(1, 0, 0, 0) * (DWDX + DUDZ);
            const double D31 = (T31F - T31B) * (g.dxi * cv);
            double DWDY = (a.q(2, 0, 1, 0) - a.q(2, 0, 0, 0)) * dycip;
            double DVDZ = (a.q(1, 0, 1, 0) - a.q(1, 0, 1, -1)) * g.dzi;
            const double T32F = a.ms(2, 0, 1, 0) * (DWDY + DVDZ);
            DWDY = (a.q(2, 0, 0, 0) - a.q(2, 0, -1, 0)) * dycij;
            DVDZ = (a.q(1, 0, 0, 0) - a.q(1, 0, 0, -1)) * g.dzi;
            const double T32B = a.ms(2, 0, 0, 0) * (DWDY + DVDZ);
            const double D32 = (T32F - T32B) * (dyfij * cv);
            ex3 = ex3 + D31 + D32 + D33;
        } else {
            const double coe3 = -2.0 / 3.0 * g.dzi * cv;
            double DUDX = (a.q(0, 1, 0, 0) - a.q(0, 0, 0, 0)) * g.dxi;
            double DVDY = (a.q(1, 0, 1, 0) - a.q(1, 0, 0, 0)) * dyfij;
            double DWDZ = (a.q(2, 0, 0, 1) - a.q(2, 0, 0, 0)) * g.dzi;
            const double F_EX33 = a.u(0, 0, 0) * (DUDX + DVDY), F_IM33 = a.u(0, 0, 0) * DWDZ;
            DUDX = (a.q(0, 1, 0, -1) - a.q(0, 0, 0, -1)) * g.dxi;
            DVDY = (a.q(1, 0, 1, -1) - a.q(1, 0, 0, -1)) * dyfij;
            DWDZ = (a.q(2, 0, 0, 0) - a.q(2, 0, 0, -1)) * g.dzi;
            const double B_EX33 = a.u(0, 0, -1) * (DUDX + DVDY), B_IM33 = a.u(0, 0, -1) * DWDZ;
            const double D33_EX = (F_EX33 - B_EX33) * coe3;
            const double D33_IM = (F_IM33 - B_IM33) * coe3 * (-2.0);
            const double coe1 = g.dxi * cv;
            double DWDX = (a.q(2, 1, 0, 0) - a.q(2, 0, 0, 0)) * g.dxi;
            double DUDZ = (a.q(0, 1, 0, 0) - a.q(0, 1, 0, -1)) * g.dzi;
            const double F_EX31 = a.ms(1, 1, 0, 0) * DUDZ, F_IM31 = a.ms(1, 1, 0, 0) * DWDX;
            DWDX = (a.q(2, 0, 0, 0) - a.q(2, -1, 0, 0)) * g.dxi;
            DUDZ = (a.q(0, 0, 0, 0) - a.q(0, 0, 0, -1)) * g.dzi;
            const double B_EX31 = a.ms(1, 0, 0, 0) * DUDZ, B_IM31 = a.ms(1, 0, 0, 0) * DWDX;
            const double D31_EX = (F_EX31 - B_EX31) * coe1;
            const double D31_IM = (F_IM31 - B_IM31) * coe1;
            const double coe2 = dyfij * cv;
            double DWDY = (a.q(2, 0, 1, 0) - a.q(2, 0, 0, 0)) * dycip;
            double DVDZ = (a.q(1, 0, 1, 0) - a.q(1, 0, 1, -1)) * g.dzi;
            const double F_EX32 = a.ms(2, 0, 1, 0) * DVDZ, F_IM32 = a.ms(2, 0, 1, 0) * DWDY;
            DWDY = (a.q(2, 0, 0, 0) - a.q(2, 0, -1, 0)) * dycij;
            DVDZ = (a.q(1, 0, 0, 0) - a.q(1, 0, 0, -1)) * g.dzi;
            const double B_EX32 = a.ms(2, 0, 0, 0) * DVDZ, B_IM32 = a.ms(2, 0, 0, 0) * DWDY;
            const double D32_EX = (F_EX32 - B_EX32) * coe2;
            const double D32_IM = (F_IM32 - B_IM32) * coe2;
            ex3 = D31_EX + D32_EX + D33_EX + ex3;
            im3 = D31_IM + D32_IM + D33_IM;
        }
    }
}

// RHS_MOM_EXPLICIT_io at one point (c, ii: its padded and interior index; pc, pim, pjm, pkm: the pressure there
// and at its lower neighbours; e0: the three EXPLT0 values): writes EXPLT0 and RHS, returns the point's x
// right-hand side for the bulk forcing (0 at a fixed inlet face).
template <bool CN, typename F>
__device__ __forceinline__ double io_rhs_combine(const Geo& g, const IoFieldsT<F>& f, int i, int j, int k, long long c, long long ii,
                                                 double dycij, int ns, double dt, double ex1, double ex2, double ex3, double im1, double im2, double im3,
                                                 double pc, double pim, double pjm, double pkm, double e01, double e02, double e03) {
    const long long FS = g.FS;
    const long long cim = c + (xmn(g, i) - i), cjm = c - g.L, ckm = c + (wrapm(k, g.N) - k) * g.P;
    const double tg = g.tgam[ns], tr = g.troh[ns], ta = g.talp[ns];
    // with inflow the inlet face u(1) is a boundary value: its x-momentum RHS, EXPLT0 and
    // G are left alone (NXI = 2, src/RHS_MOM_EXPLICIT_io.f90:35)
    const bool ux = !(g.xo && i == 1);
    const double coa = ta * dt;
    // buoyancy (:161-226): D_STG * TALP*DT*F_A on the component |iGravity| (1/RNDI1 = 1/RCCI1 = 1)
    const int ig = f.igrav < 0 ? -f.igrav : f.igrav;
    const double cob = ta * dt * f.fa;
    double r1 = (tg * ex1 + tr * e01) * dt;
    if constexpr (CN) r1 = r1 + coa * im1;
    r1 = r1 - io_pgm(f, c, cim, pc, pim, ta * dt * g.dxi);
    if (ig == 1) r1 = r1 + f.DST[c] * cob;
    double r3 = (tg * ex3 + tr * e03) * dt;
    if constexpr (CN) r3 = r3 + coa * im3;
    r3 = r3 - io_pgm(f, c, ckm, pc, pkm, ta * dt * g.dzi);
    if (ig == 3) r3 = r3 + f.DST[c + 2 * FS] * (cob / 1.0);
    if (ux) {
        f.EX0[ii] = (F)ex1;
        f.RHS[ii] = (F)r1;
    }
    f.EX0[ii + 2 * g.FI] = (F)ex3;
    f.RHS[ii + 2 * g.FI] = (F)r3;
    if (j >= 2) {
        double r2 = (tg * ex2 + tr * e02) * dt;
        if constexpr (CN) r2 = r2 + coa * im2;
        r2 = r2 - io_pgm(f, c, cjm, pc, pjm, ta * dt * dycij / 1.0);
        if (ig == 2) r2 = r2 + f.DST[c + FS] * (cob / 1.0);
        f.EX0[ii + g.FI] = (F)ex2;
        f.RHS[ii + g.FI] = (F)r2;
    }
    return ux ? r1 : 0.0;
}

// Grid sum of the bulk-forcing integrand: block partials, added by the last block to finish, in order
template <int NT>
__device__ __forceinline__ void io_rhs_bulk(double bulk, double* sred, double* __restrict__ partial, DevState* __restrict__ st) {
    __shared__ int is_last;
    double s = block_sum<NT>(bulk, sred);
    if (threadIdx.x == 0) {
        partial[blockIdx.x] = s;
        __threadfence();
        const unsigned prev = atomicAdd(&st->ctr, 1u);
        is_last = (prev == gridDim.x - 1);
    }
    __syncthreads();
    if (is_last) {
        __threadfence();
        double a = 0.0;
        for (int t = threadIdx.x; t < (int)gridDim.x; t += NT) a += __ldcg(partial + t);
        a = block_sum<NT>(a, sred);
        if (threadIdx.x == 0) {
            st->bulksum = a;
            st->ctr = 0u;
        }
    }
}

// neighbours of one point in global memory
template <typename F>
struct IoGlobal {
    const F *Q, *G, *MS, *DV;
    const double *U0, *U;
    long long FS, c, dip, dim, djp, djm, dkp, dkm;
    __device__ __forceinline__ long long at(int di, int dj, int dk) const {
        return c + (di > 0 ? dip : di < 0 ? dim : 0) + (dj > 0 ? djp : dj < 0 ? djm : 0) + (dk > 0 ? dkp : dk < 0 ? dkm : 0);
    }
    __device__ __forceinline__ F q(int n, int di, int dj, int dk) const { return Q[at(di, dj, dk) + n * FS]; }
    __device__ __forceinline__ F g(int n, int di, int dj, int dk) const { return G[at(di, dj, dk) + n * FS]; }
    __device__ __forceinline__ F ms(int n, int di, int dj, int dk) const { return MS[at(di, dj, dk) + n * FS]; }
    __device__ __forceinline__ double u0(int di, int dj, int dk) const { return U0[at(di, dj, dk)]; }
    __device__ __forceinline__ double u(int di, int dj, int dk) const { return U[at(di, dj, dk)]; }
    __device__ __forceinline__ F dv(int di, int dj, int dk) const { return DV[at(di, dj, dk)]; }
};

// FP32 storage: one thread per point in flat order.  (The order of the bulk sum decides the last bit of the
// forcing, and with FP32 storage a changed last bit of an FP64 value is a changed stored value now and
// then, so this form keeps its order.)
template <bool CN, typename F>
__global__ void __launch_bounds__(IO_NT, 2) k_io_rhs(Geo g, IoFieldsT<F> f, double* __restrict__ partial, DevState* __restrict__ st,
                                                  int ns) {
    __shared__ double sred[32];
    const int N = g.N;
    const long long tot = io_points(g);
    const double dt = st->dt;
    double bulk = 0.0;
    for (long long t = (long long)blockIdx.x * IO_NT + threadIdx.x; t < tot; t += (long long)gridDim.x * IO_NT) {
        int i, j, k;
        io_decode(g, t, i, j, k);
        const long long c = pidx(g, i, j, k), cim = pidx(g, xmn(g, i), j, k), ckm = pidx(g, i, j, wrapm(k, N));
        const IoGlobal<F> a{f.Q, f.G, f.MST, f.DIVU, f.MU0, f.MU, g.FS, c, pidx(g, xpn(g, i), j, k) - c, cim - c, g.L, -g.L,
                            pidx(g, i, j, wrapp(k, N)) - c, ckm - c};
        double ex1, ex2, ex3, im1, im2, im3;
        io_rhs_terms<CN>(g, io_row(g, j), a, j, ex1, ex2, ex3, im1, im2, im3);
        const long long ii = io_iidx(g, i, j, k);
        const double e01 = f.EX0[ii], e02 = f.EX0[ii + g.FI], e03 = f.EX0[ii + 2 * g.FI];
        bulk += io_rhs_combine<CN>(g, f, i, j, k, c, ii, g.dyci[j], ns, dt, ex1, ex2, ex3, im1, im2, im3, f.PR[c], f.PR[cim], f.PR[c - g.L],
                                   f.PR[ckm], e01, e02, e03) / g.dyfi[j] / 1.0;
    }
    io_rhs_bulk<IO_NT>(bulk, sred, partial, st);
}

// FP64: a block of 32 x 16 threads owns 32 (i) x 16 (j) columns and marches over `chunk` planes in k.  The
// planes of the fields, tile and one-point halo, are in shared memory (rings of four planes for Q and G,
// three for MU_STG, the viscosity and PR), the next one arriving by asynchronous copies while a plane is
// computed.  The flat form reads about 75 neighbour values per point from L1 and L2 with 16 warps per SM
// to wait for them, in 900 instructions, half of them addresses; here every neighbour is a
// shared-memory read at a constant offset and each field is fetched once per tile.  The explicit scheme's
// DivU is formed from Q in shared memory (DIVG_U_io's pass over the fields is not needed).  One block per
// SM by shared memory; bound by the latencies of its 16 warps (issue slots a third busy).  Per step (three
// launches): Crank-Nicolson at 256 x 192 x 128 1.55 -> 1.08 ms, explicit with DivU at 128^3 0.55 -> 0.41.
constexpr int IT_I = 32, IT_J = 16, IT_NT = IT_I * IT_J;
constexpr int IT_HI = IT_I + 2, IT_PL = IT_HI * (IT_J + 2);      // row and plane of a tile with its halo
constexpr int IT_SMEM = (6 * 4 + 3 * 3 + 2 * 3) * IT_PL * 8;     // bytes

// planes per block: the split of N that gives the least time, counted in planes loaded by the busiest SM (one
// block per SM; each block loads three more planes than it computes)
inline int io_tile_chunk(const Geo& g, int nsm) {
    const int tiles = ((g.LI + IT_I - 1) / IT_I) * (g.M / IT_J);
    int best = g.N;
    long long cost = -1;
    for (int n = 1; n <= g.N / 8; ++n) {
        const int chunk = (g.N + n - 1) / n;
        const int nb = (g.N + chunk - 1) / chunk;
        const long long t = (long long)((tiles * nb + nsm - 1) / nsm) * (chunk + 3);
        if (cost < 0 || t < cost) { cost = t; best = chunk; }
    }
    return best;
}
inline int io_tile_blocks(const Geo& g, int chunk) {
    return ((g.LI + IT_I - 1) / IT_I) * (g.M / IT_J) * ((g.N + chunk - 1) / chunk);
}

struct IoTileAcc {  // neighbours of one point in the tile's planes
    const double *qm, *qc, *qp, *mc, *mp, *vm, *vc;  // Q and G, MU_STG, viscosity and PR at planes k - 1, k, k + 1
    double dxi, dzi, dyfij, dyfim;
    static __device__ __forceinline__ int o(int di, int dj) { return di + IT_HI * dj; }
    __device__ __forceinline__ double q(int n, int di, int dj, int dk) const { return (dk > 0 ? qp : dk < 0 ? qm : qc)[n * IT_PL + o(di, dj)]; }
    __device__ __forceinline__ double g(int n, int di, int dj, int dk) const { return q(3 + n, di, dj, dk); }
    __device__ __forceinline__ double ms(int n, int di, int dj, int dk) const { return (dk > 0 ? mp : mc)[n * IT_PL + o(di, dj)]; }
    __device__ __forceinline__ double u0(int di, int dj, int dk) const { return (dk < 0 ? vm : vc)[o(di, dj)]; }
    __device__ __forceinline__ double u(int di, int dj, int dk) const { return u0(di, dj, dk); }
    __device__ __forceinline__ double pr(int di, int dj, int dk) const { return (dk < 0 ? vm : vc)[IT_PL + o(di, dj)]; }
    // DIVG_U_io at the point (0 0 0) or its lower neighbour in one direction
    __device__ __forceinline__ double dv(int di, int dj, int dk) const {
        const double dx = (q(0, di + 1, dj, dk) - q(0, di, dj, dk)) * dxi;
        const double dy = (q(1, di, dj + 1, dk) - q(1, di, dj, dk)) * (dj < 0 ? dyfim : dyfij);
        const double dz = (q(2, di, dj, dk + 1) - q(2, di, dj, dk)) * dzi;
        // the quotient by 3, correctly rounded as in DIVG_U_io: a product by the rounded reciprocal and its correction
        // (Markstein, see io_cn.cuh); the product alone has 1.2 times the rounding error where div(u) is not small
        const double sum = dx + dy + dz, q3 = sum * (1.0 / 3.0);
        return fma(fma(-3.0, q3, sum), 1.0 / 3.0, q3);
    }
};

template <bool CN>
__global__ void __launch_bounds__(IT_NT, 1) k_io_rhs_tile(Geo g, IoFields f, double* __restrict__ partial, DevState* __restrict__ st,
                                                         int ns, int chunk) {
    extern __shared__ __align__(16) double smt[];
    __shared__ double sred[32];
    // the rows' y coefficients: in shared memory, as the L1 left beside the rings is small and the planes
    // stream through it
    __shared__ IoRow srow[IT_J];
    const int N = g.N, nti = (g.LI + IT_I - 1) / IT_I, ntj = g.M / IT_J;
    const int b = blockIdx.x, r = b / nti, kc = r / ntj;
    const int i0 = IT_I * (b - r * nti) + g.xo, j0 = 1 + IT_J * (r - kc * ntj);
    const int k0 = kc * chunk, k1 = min(N, k0 + chunk);
    const int i = i0 + (threadIdx.x & 31), j = j0 + (threadIdx.x >> 5);
    const bool on = i - g.xo < g.LI;
    const double dt = st->dt;
    double* const smq = smt;                     // 4 planes of Q, G
    double* const smm = smq + 4 * 6 * IT_PL;     // 3 planes of MU_STG
    double* const smv = smm + 3 * 3 * IT_PL;     // 3 planes of the viscosity and PR
    // this thread's points of a plane: padded offsets at k = 0 (columns past the row's last storage column
    // repeat it; they feed only threads that are off)
    constexpr int NE = (IT_PL + IT_NT - 1) / IT_NT;
    long long eo[NE];
#pragma unroll
    for (int e = 0; e < NE; ++e) {
        const int q = threadIdx.x + e * IT_NT, jj = q / IT_HI;
        int ii = i0 - 1 + (q - jj * IT_HI);
        if (g.xo) ii = min(ii, g.L - 1);
        else ii = ii < 0 ? ii + g.L : ii >= g.L ? ii - g.L : ii;
        eo[e] = q < IT_PL ? pidx(g, ii, j0 - 1 + jj, 0) : -1;
    }
    auto wrap = [&](int k) { return k < 0 ? k + N : k >= N ? k - N : k; };
    auto load_q = [&](int k, double* dst) {
        const long long ko = g.P * wrap(k);
#pragma unroll
        for (int e = 0; e < NE; ++e)
            if (eo[e] >= 0) {
                double* d = dst + threadIdx.x + e * IT_NT;
                const long long o = eo[e] + ko;
#pragma unroll
                for (int n = 0; n < 3; ++n) {
                    cp_async8(d + n * IT_PL, f.Q + o + n * g.FS);
                    cp_async8(d + (3 + n) * IT_PL, f.G + o + n * g.FS);
                }
            }
    };
    auto load_m = [&](int k, double* dst) {
        const long long ko = g.P * wrap(k);
#pragma unroll
        for (int e = 0; e < NE; ++e)
            if (eo[e] >= 0) {
#pragma unroll
                for (int n = 0; n < 3; ++n) cp_async8(dst + threadIdx.x + e * IT_NT + n * IT_PL, f.MST + eo[e] + ko + n * g.FS);
            }
    };
    auto load_v = [&](int k, double* dst) {
        const long long ko = g.P * wrap(k);
        const double* U = CN ? f.MU : f.MU0;
#pragma unroll
        for (int e = 0; e < NE; ++e)
            if (eo[e] >= 0) {
                double* d = dst + threadIdx.x + e * IT_NT;
                cp_async8(d, U + eo[e] + ko);
                cp_async8(d + IT_PL, f.PR + eo[e] + ko);
            }
    };
    constexpr int QS = 6 * IT_PL, MSZ = 3 * IT_PL, VS = 2 * IT_PL;
    int sq = 1, sm = 0, sv = 1;  // ring slots of plane k
    load_q(k0 - 1, smq); load_q(k0, smq + QS); load_q(k0 + 1, smq + 2 * QS);
    load_m(k0, smm); load_m(k0 + 1, smm + MSZ);
    load_v(k0 - 1, smv); load_v(k0, smv + VS);
    const int cc = (threadIdx.x >> 5) * IT_HI + IT_HI + (threadIdx.x & 31) + 1;  // this point inside a plane
    if (threadIdx.x < IT_J) srow[threadIdx.x] = io_row(g, j0 + threadIdx.x);
    const IoRow& y = srow[threadIdx.x >> 5];
    long long c = pidx(g, i, j, k0), ii = io_iidx(g, i, j, k0);
    double bulk = 0.0;
#pragma unroll 1
    for (int k = k0; k < k1; ++k, c += g.P, ii += g.PI_) {
        const int sqp = (sq + 1) & 3, sqm = (sq + 3) & 3, smp = sm == 2 ? 0 : sm + 1, svm = sv == 0 ? 2 : sv - 1;
        cp_async_wait_all();
        __syncthreads();  // planes k - 1 .. k + 1 are here, and every thread is done with the slots filled next
        if (k + 1 < k1) {
            load_q(k + 2, smq + ((sq + 2) & 3) * QS);
            load_m(k + 2, smm + (sm == 0 ? 2 : sm - 1) * MSZ);
            load_v(k + 1, smv + (sv == 2 ? 0 : sv + 1) * VS);
        }
        if (on) {
            const double e01 = f.EX0[ii], e02 = f.EX0[ii + g.FI], e03 = f.EX0[ii + 2 * g.FI];
            const IoTileAcc a{smq + sqm * QS + cc, smq + sq * QS + cc, smq + sqp * QS + cc, smm + sm * MSZ + cc, smm + smp * MSZ + cc,
                              smv + svm * VS + cc, smv + sv * VS + cc, g.dxi, g.dzi, y.dyfij, y.dyfim};
            double ex1, ex2, ex3, im1, im2, im3;
            io_rhs_terms<CN>(g, y, a, j, ex1, ex2, ex3, im1, im2, im3);
            bulk += io_rhs_combine<CN>(g, f, i, j, k, c, ii, y.dycij, ns, dt, ex1, ex2, ex3, im1, im2, im3, a.pr(0, 0, 0), a.pr(-1, 0, 0),
                                       a.pr(0, -1, 0), a.pr(0, 0, -1), e01, e02, e03);
        }
        sq = sqp; sm = smp; sv = sv == 2 ? 0 : sv + 1;
    }
    io_rhs_bulk<IT_NT>(bulk / g.dyfi[j], sred, partial, st);  // one row per thread
}

// bulk forcing (RHS_MOM_EXPLICIT_io :228-265) + MASSFLUX_CALC_io
template <typename F>
__global__ void __launch_bounds__(IO_NT) k_io_massflux(Geo g, IoFieldsT<F> f, const DevState* __restrict__ st, int ns) {
    const long long tot = io_points(g);
    double dpg = 0.0;
    if (g.iflowdriven == 1) dpg = st->bulksum / g.volm;
    else if (g.iflowdriven == 2) dpg = -0.5 * g.cf_given * (g.talp[ns] * st->dt);
    for (long long t = (long long)blockIdx.x * IO_NT + threadIdx.x; t < tot; t += (long long)gridDim.x * IO_NT) {
        int i, j, k;
        io_decode(g, t, i, j, k);
        const long long c = pidx(g, i, j, k), ii = io_iidx(g, i, j, k);
        const double g1 = f.G[c], g2 = f.G[c + g.FS], g3 = f.G[c + 2 * g.FS];
        const double r1 = f.RHS[ii] - dpg, r3 = f.RHS[ii + 2 * g.FI];
        if (!(g.xo && i == 1)) f.G[c] = (F)(g1 + r1);  // NXI = 2 with inflow
        f.G[c + 2 * g.FS] = (F)(g3 + r3);
        if (j >= 2) f.G[c + g.FS] = (F)(g2 + (double)f.RHS[ii + g.FI]);
    }
}

// DIVG_io + forward x transform (same tiling as k_div_fftx)
// DRHO: DrhoDtP of the thermal solver, or NULL (zero) while it is off;
// the divergence is divided by wdiv (DIVG.f90:78-82)
template <int N1, int N2, typename F>
__global__ void __launch_bounds__(PX_NT, PX_MINB) k_io_div_fftx(Geo g, const F* __restrict__ G, double* __restrict__ RHSLL,
                                                       double2* __restrict__ SP, const DevState* __restrict__ st, int ns,
                                                       const double* __restrict__ DRHO, double wdiv) {
    extern __shared__ double2 smc[];
    constexpr int L = N1 * N2, LH = L / 2 + 1, LD = L + N2 + 1, NP = PX_TJ / 2;
    const int M = g.M, N = g.N;
    const int j0 = 1 + blockIdx.x * PX_TJ;
    const int k = blockIdx.y;
    const int kp = wrapp(k, N);
    // wdiv: 0.25 + pres_epslon with iWeightedPre = 1, else 1 (an exact division)
    const double coe0 = 1.0 / st->dt / g.talp[ns] / wdiv;
    const double coe1 = g.dxi / 1.0;
    // one item = two consecutive points of both rows of a packed pair, by vector loads (rows start at multiples
    // of L, which is a multiple of 32; M is one too, so every row of the tile exists): twice the bytes in
    // flight of single loads, and both rows' loads issued together: 0.32 -> 0.23 ms per step at
    // 256 x 192 x 128 (FP32 storage 0.31 -> 0.20)
    auto ld2 = [](const F* p, double (&o)[2]) {
        if constexpr (sizeof(F) == 8) {
            const double2 v = *reinterpret_cast<const double2*>(p);
            o[0] = v.x; o[1] = v.y;
        } else {
            const float2 v = *reinterpret_cast<const float2*>(p);
            o[0] = v.x; o[1] = v.y;
        }
    };
    constexpr int LV = L / 2, NI = NP * LV;
    static_assert(NI % PX_NT == 0, "whole items per thread");
#pragma unroll 2
    for (int t = 0; t < NI / PX_NT; ++t) {
        const int p = threadIdx.x + t * PX_NT;
        const int pair = p / LV, i0 = (p - pair * LV) * 2;
        const int j = j0 + 2 * pair;
        const long long c = pidx(g, i0, j, k), cp = pidx(g, i0, j, kp) + 2 * g.FS;
        const int dn = i0 + 2 == L ? 2 - L : 2;  // u at i0 + 2 (periodic)
        double u[2][2], v[3][2], w[2][2], wp[2][2], un[2], dr[2][2];
#pragma unroll
        for (int part = 0; part < 2; ++part) {
            ld2(G + c + part * L, u[part]);
            ld2(G + c + g.FS + part * L, v[part]);
            ld2(G + c + 2 * g.FS + part * L, w[part]);
            ld2(G + cp + part * L, wp[part]);
            un[part] = G[c + part * L + dn];
        }
        ld2(G + c + g.FS + 2 * L, v[2]);
#pragma unroll
        for (int part = 0; part < 2; ++part) {
            dr[part][0] = dr[part][1] = 0.0;
            if (DRHO) {
                const double2 d = *reinterpret_cast<const double2*>(DRHO + c + part * L);
                dr[part][0] = d.x / 1.0; dr[part][1] = d.y / 1.0;
            }
        }
        double val[2][2];
#pragma unroll
        for (int part = 0; part < 2; ++part) {
            const double coe2 = g.dyfi[j + part] / 1.0;
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const double up = e == 0 ? u[part][1] : un[part];
                const double DIVX = (up - u[part][e]) * coe1, DIVY = (v[part + 1][e] - v[part][e]) * coe2,
                             DIVZ = (wp[part][e] - w[part][e]) * g.dzi;
                const double DQ = DIVX + DIVY + DIVZ + dr[part][e];
                val[part][e] = DQ * coe0;
            }
            *reinterpret_cast<double2*>(RHSLL + iidx(g, i0, j + part, k)) = make_double2(val[part][0], val[part][1]);
        }
        double2* line = smc + pair * LD + i0;
        line[0] = make_double2(val[0][0], val[1][0]);
        line[1] = make_double2(val[0][1], val[1][1]);
    }
    block_fft4s<N1, N2, -1>(smc, NP, LD, g.twx);
    const double sc = 0.5 / (double)L;
    for (int p = threadIdx.x; p < NP * LH; p += PX_NT) {
        const int pair = p / LH, kx = p - pair * LH;
        const double2* line = smc + pair * LD;
        const double2 z = line[kx];
        const double2 zc = line[kx == 0 ? 0 : L - kx];
        double2* sp = SP + kx + (long long)LH * ((j0 + 2 * pair - 1) + (long long)M * k);
        sp[0] = make_double2((z.x + zc.x) * sc, (z.y - zc.y) * sc);
        sp[LH] = make_double2((z.y + zc.y) * sc, (zc.x - z.x) * sc);
    }
}

// PRCALC_io + MASSFLUX_UPDATE_io + VELOCITY_CALC_io.  RHSLL == NULL: the
// explicit scheme's PR += DPH; otherwise the Crank-Nicolson scheme's
// PR += DPH - BE * RHSLLPHI_io, BE = alpha*dt/(2 Re) (src/PRESSURE_CORRECTION.f90:113-123).
// VEL = false leaves the velocity out: inside a captured step with the thermal solver the next substep's
// k_eng_state forms it from the same G and the new densities before anything reads it (10 words per point
// instead of 16; 0.40 -> 0.34 ms per step at 256 x 192 x 128, FP32 storage 0.33 -> 0.25).
template <bool VEL, typename F>
__global__ void __launch_bounds__(IO_NT) k_io_correct(Geo g, IoFieldsT<F> f, const double* __restrict__ DPH,
                                                      const DevState* __restrict__ st, int ns,
                                                      const double* __restrict__ RHSLL) {
    const int M = g.M, N = g.N;
    const long long tot = io_points(g);
    const double dt = st->dt, ta = g.talp[ns];
    const double be = 0.50 * ta * dt * g.cvisc;
    for (long long t = (long long)blockIdx.x * IO_NT + threadIdx.x; t < tot; t += (long long)gridDim.x * IO_NT) {
        int i, j, k;
        io_decode(g, t, i, j, k);
        const long long c = pidx(g, i, j, k);
        const double ph = DPH[c];
        const double phim = DPH[pidx(g, xmn(g, i), j, k)];
        const double phkm = DPH[pidx(g, i, j, wrapm(k, N))];
        const double phjm = j >= 2 ? DPH[pidx(g, i, j - 1, k)] : 0.0;
        const double g1 = f.G[c], g2 = f.G[c + g.FS], g3 = f.G[c + 2 * g.FS], pr = f.PR[c];
        double d1 = 1.0, d2 = 1.0, d3 = 1.0;
        if constexpr (VEL) { d1 = f.DST[c]; d2 = f.DST[c + g.FS]; d3 = f.DST[c + 2 * g.FS]; }
        const double pn = RHSLL ? pr + ph - be * RHSLL[io_iidx(g, i, j, k)] : pr + ph;
        f.PR[c] = (F)pn;
        if (j == 1) f.PR[pidx(g, i, 0, k)] = (F)pn;
        if (j == M) f.PR[pidx(g, i, M + 1, k)] = (F)pn;
        // u faces NXI..NXE: 1..L, or 2..L+1 with inflow (MASSFLUX_UPDATE_io, src/VELO_CORRECTION.f90:121-137);
        // VELOCITY_CALC_io still divides the fixed inlet face, and leaves the outlet face's Q alone
        const double n1 = (g.xo && i == 1) ? g1 : g1 - (ph - phim) * (dt * ta * g.dxi);
        const double n3 = g3 - (ph - phkm) * (dt * ta * g.dzi);
        f.G[c] = (F)n1;
        if (g.xo && i == g.LI) {
            const double go = f.G[c + 1];
            f.G[c + 1] = (F)(go - (DPH[c + 1] - ph) * (dt * ta * g.dxi));
        }
        f.G[c + 2 * g.FS] = (F)n3;
        if constexpr (VEL) {
            f.Q[c] = (F)(n1 / d1);
            f.Q[c + 2 * g.FS] = (F)(n3 / d3);
        }
        if (j >= 2) {
            const double n2 = g2 - (ph - phjm) * (dt * ta * g.dyci[j] / 1.0);
            f.G[c + g.FS] = (F)n2;
            if constexpr (VEL) f.Q[c + g.FS] = (F)(n2 / d2);
        }
    }
}

template <typename F>
__global__ void __launch_bounds__(IO_NT) k_io_cfl(Geo g, IoFieldsT<F> f, double* __restrict__ partial, DevState* __restrict__ st) {
    __shared__ double sred[32];
    const int L = g.L, N = g.N;  // L: row stride
    const long long tot = io_points(g);
    double mx = 0.0;
    bool bad = false;
    for (long long t = (long long)blockIdx.x * IO_NT + threadIdx.x; t < tot; t += (long long)gridDim.x * IO_NT) {
        int i, j, k;
        io_decode(g, t, i, j, k);
        const long long c = pidx(g, i, j, k);
        const F* Q = f.Q;
        double q = (fabs(((double)Q[c] + (double)Q[pidx(g, xpn(g, i), j, k)]) * g.dxi) +
                    fabs(((double)Q[c + g.FS] + (double)Q[c + g.FS + L]) * g.dyfi[j] * 1.0) +
                    fabs(((double)Q[c + 2 * g.FS] + (double)Q[pidx(g, i, j, wrapp(k, N)) + 2 * g.FS]) * g.dzi * 1.0)) * 0.5;
        const double vcf = 2.0 * g.cvisc * (g.dxqi + g.dzqi * 1.0 + g.dyfi[j] * g.dyfi[j]) * f.MU[c] / f.DEN[c];
        if (!(q == q) || !(vcf == vcf)) bad = true;
        q = fmax(q, vcf);
        mx = fmax(mx, q);
    }
    if (bad) atomicOr(&st->err, CHS_EBIT_NAN);
    if (blockIdx.x == 0 && threadIdx.x == 0) st->dtprev = st->dt;
    double r = block_max<IO_NT>(mx, sred);
    if (threadIdx.x == 0) partial[blockIdx.x] = r;
}

// DIVGCK_io (src/DIVGCK.f90:60-121 with DIVGCK_Comm_io :125-184), x-periodic
// main domain: max over the interior of |div G + DrhoDtP| (all three ranges of
// MAXDIVGV_io coincide).  Per-block maxima; k_maxdiv_final reduces them.  DRHO
// is NULL while the thermal solver is off (DrhoDtP = 0).
template <typename F>
__global__ void __launch_bounds__(IO_NT) k_io_divgck(Geo g, const F* __restrict__ G,
                                                     const double* __restrict__ DRHO, double* __restrict__ partial) {
    __shared__ double sred[32];
    const int L = g.L, N = g.N;  // L: row stride
    const long long tot = io_points(g);
    double mx = 0.0;
    for (long long t = (long long)blockIdx.x * IO_NT + threadIdx.x; t < tot; t += (long long)gridDim.x * IO_NT) {
        int i, j, k;
        io_decode(g, t, i, j, k);
        const long long c = pidx(g, i, j, k);
        const double DIVX = ((double)G[pidx(g, xpn(g, i), j, k)] - (double)G[c]) * g.dxi;
        const double DIVY = ((double)G[c + g.FS + L] - (double)G[c + g.FS]) * (g.dyfi[j] * 1.0);
        const double DIVZ = ((double)G[pidx(g, i, j, wrapp(k, N)) + 2 * g.FS] - (double)G[c + 2 * g.FS]) * (g.dzi * 1.0);
        const double DTRHO = DRHO ? DRHO[c] : 0.0;
        const double DQCAP = DIVX + DIVY + DIVZ + DTRHO;
        mx = fmax(fabs(DQCAP), mx);
    }
    const double r = block_max<IO_NT>(mx, sred);
    if (threadIdx.x == 0) partial[blockIdx.x] = r;
}
