// Thermal solver of the main (IO) domain, run before the momentum part of
// each RK3 substep (src/SOLVE.f90:119-128):
//   k_eng_rhs, k_eng_rhs_tile  SOLVERRK3_ENG_io (src/SOLVERRK3_ENG_IO.f90:11-82) with
//                RHS_ENERGY_EXPLICIT (src/RHS_ENERGY_EXPLICIT.f90:11-155):
//                rho*h += TGAM dt RHS + TROH dt RHS0, clipped to the table's
//                [DHmin, DHmax] (search-table limiter), RHS0 = RHS; constant
//                wall heat flux on both walls
//   k_eng_props  THERM_PROP_UPDATE(IMAIND) by table search on rows 1..M; the
//                old DENSITY and Viscousity are kept as DENSITY0 and
//                Viscousity0 point by point before being overwritten (the
//                whole-field copies at the top of SOLVERRK3_ENG_io)
//   k_eng_bc     BC_WALL_Isoflux (src/BC_WALL.f90:541-619): ghost rho*h
//                extrapolated from rows 1, 2 (M, M-1), then its properties
//   k_eng_state  DENSITY_TIME_DERIVATION (src/DIVG.f90:249-317):
//                DrhoDtP = -TGAM div(G) - TROH div(G0); DENSITY_Staggered and
//                MU_Staggered from DENSITY0 and Viscousity0; G0 = G and
//                VELOCITY_CALC_io, with which the momentum substep starts
// Plane channel: RCCI1 = RCCI2 = RNDI1 = 1.
#pragma once
#include "common.cuh"
#include "io.cuh"
#include "thermo.cuh"

#ifndef CHS_EBIT_TABLE
#define CHS_EBIT_TABLE 4u  // a point (or its h) left the property table
#endif

struct ThermoFields {
    double *DH, *ENTH, *TEMP, *KAP, *HCP, *RHSE0, *DIVG0, *DRHO;  // DIVG0: div(G0_io)
};
struct ThermoParams {
    double wf_bot, wf_top;  // WALLFLUX of the bottom (+q) and top (-q) walls (src/Flow_State.f90:150-175)
    double cthecd;          // 1 / (REN PRT0)
    double dhmin, dhmax;    // LIST_DH at IMIN_DH, IMAX_DH
    // BC_Fixed_Temperature walls (0 bottom, 1 top): the wall state T, H, D, M, K held in the ghost
    // row (BC_WALL_IsoTHERMAL, src/BC_WALL.f90:484-538); 0 = constant heat flux
    int iso[2];
    double wv[2][5];
};

// One thread per point, every neighbour from memory: with FP32 storage, whose fields stay the same to the bit
// in this order of operations (FP64: k_eng_rhs_tile)
template <typename F>
__global__ void __launch_bounds__(IO_NT, 4) k_eng_rhs(Geo g, IoFieldsT<F> f, ThermoFields t, ThermoParams tp,
                                                   const DevState* __restrict__ st, int ns) {
    const int M = g.M, N = g.N;
    const long long tot = io_points(g);
    const double dt = st->dt;
    const double coe1n = g.tgam[ns] * dt, coe0n = g.troh[ns] * dt;
    const double XND2CL = 0.5, ZND2CL = 0.5;
    const double COE1 = g.dxi * XND2CL * 0.5;
    const double COE11 = g.dxqi * XND2CL * tp.cthecd;
    const double* Hh = t.ENTH;
    const double* T = t.TEMP;
    const double* K = t.KAP;
    const F* G1 = f.G;
    const F* G2 = f.G + g.FS;
    const F* G3 = f.G + 2 * g.FS;
    for (long long q = (long long)blockIdx.x * IO_NT + threadIdx.x; q < tot; q += (long long)gridDim.x * IO_NT) {
        int i, j, k;
        io_decode(g, q, i, j, k);
        const int ip = xpn(g, i), im = xmn(g, i), kp = wrapp(k, N), km = wrapm(k, N);
        const int jp = j + 1, jm = j - 1;
        const long long c = pidx(g, i, j, k);
        const long long cip = pidx(g, ip, j, k), cim = pidx(g, im, j, k);
        const long long cjp = pidx(g, i, jp, k), cjm = pidx(g, i, jm, k);
        const long long ckp = pidx(g, i, j, kp), ckm = pidx(g, i, j, km);
        const double COE2 = g.dyfi[j] * 1.0 * 0.5;
        const double COE3 = g.dzi * ZND2CL * 1.0 * 0.5;
        const double COE33 = g.dzqi * ZND2CL * 1.0 * tp.cthecd;
        const double COE22 = g.dyfi[j] * 1.0 * tp.cthecd;
        double COE221, COE222;
        if (j == 1) {  // src/RHS_ENERGY_EXPLICIT.f90:50-77: the wall face of an isothermal wall keeps DYCI
            COE221 = g.dyci[jp] / 1.0;
            COE222 = tp.iso[0] ? g.dyci[j] / 1.0 : 1.0 / 1.0;
        } else if (j == M) {
            COE222 = g.dyci[j] / 1.0;
            COE221 = tp.iso[1] ? g.dyci[jp] / 1.0 : 1.0 / 1.0;
        } else {
            COE221 = g.dyci[jp] / 1.0;
            COE222 = g.dyci[j] / 1.0;
        }
        const double hc = Hh[c], tc = T[c], kc = K[c];
        double DX_DHU = (Hh[cip] + hc) * (G1[cip] + G1[cip]) - (hc + Hh[cim]) * (G1[c] + G1[c]);
        DX_DHU = DX_DHU * COE1;
        double DY_DHV = (g.wff[jp] * Hh[cjp] + g.wfb[jp] * hc) * (G2[cjp] + G2[cjp]) -
                        (g.wff[j] * hc + g.wfb[j] * Hh[cjm]) * (G2[c] + G2[c]);
        DY_DHV = DY_DHV * COE2;
        double DZ_DHW = (Hh[ckp] + hc) * (G3[ckp] + G3[ckp]) - (hc + Hh[ckm]) * (G3[c] + G3[c]);
        DZ_DHW = DZ_DHW * COE3;
        double DX_KDT = (K[cip] + kc) * (T[cip] - tc) - (kc + K[cim]) * (tc - T[cim]);
        DX_KDT = DX_KDT * COE11;
        double KDTy1 = (g.wff[jp] * K[cjp] + g.wfb[jp] * kc) * (T[cjp] - tc) * COE221;
        double KDTy2 = (g.wff[j] * kc + g.wfb[j] * K[cjm]) * (tc - T[cjm]) * COE222;
        if (j == 1 && !tp.iso[0]) KDTy2 = -tp.wf_bot * COE222;
        else if (j == M && !tp.iso[1]) KDTy1 = -tp.wf_top * COE221;
        const double DY_KDT = (KDTy1 - KDTy2) * COE22;
        double DZ_KDT = (K[ckp] + kc) * (T[ckp] - tc) - (K[ckm] + kc) * (tc - T[ckm]);
        DZ_KDT = DZ_KDT * COE33;
        const double rhs = -DX_DHU - DY_DHV - DZ_DHW + DX_KDT + DY_KDT + DZ_KDT;
        double d = t.DH[c] + coe1n * rhs + coe0n * t.RHSE0[c];
        d = fmin(tp.dhmax - 1.0e-14, d);
        d = fmax(tp.dhmin + 1.0e-14, d);
        t.DH[c] = d;
        t.RHSE0[c] = rhs;
    }
}

// RHS_ENERGY_EXPLICIT's y coefficients of a row
struct EngRow { double COE2, COE22, COE221, COE222, wffp, wfbp, wff, wfb; };
__device__ __forceinline__ EngRow eng_row(const Geo& g, const ThermoParams& tp, int j) {
    const int jp = j + 1;
    EngRow r;
    r.COE2 = g.dyfi[j] * 1.0 * 0.5;
    r.COE22 = g.dyfi[j] * 1.0 * tp.cthecd;
    if (j == 1) {  // src/RHS_ENERGY_EXPLICIT.f90:50-77: the wall face of an isothermal wall keeps DYCI
        r.COE221 = g.dyci[jp] / 1.0;
        r.COE222 = tp.iso[0] ? g.dyci[j] / 1.0 : 1.0 / 1.0;
    } else if (j == g.M) {
        r.COE222 = g.dyci[j] / 1.0;
        r.COE221 = tp.iso[1] ? g.dyci[jp] / 1.0 : 1.0 / 1.0;
    } else {
        r.COE221 = g.dyci[jp] / 1.0;
        r.COE222 = g.dyci[j] / 1.0;
    }
    r.wffp = g.wff[jp]; r.wfbp = g.wfb[jp];
    r.wff = g.wff[j]; r.wfb = g.wfb[j];
    return r;
}

// Energy right-hand side and DH update.  Tiles of 32 x 16 points march through chunk planes of z (as
// k_io_rhs_tile): H, T and kappa of planes k, k + 1 and, in flight, k + 2 sit in a ring in shared memory
// with the tile's halo, plane k - 1 of the own column and G3 at k in registers, so a point loads 3.6 words of
// those fields instead of 21.  Two blocks of 512 threads per SM; the own point's other words are asked for before the
// plane's barrier.  10 words in and out are 76 us of memory time at 256 x 192 x 128; one thread per point took 157 us
// there (L2 bandwidth: 22 words a point beyond the row's own), this 118; 128 x 96 x 128 41 -> 36 us.
constexpr int ET_R = 3;  // planes in the ring
__global__ void __launch_bounds__(IT_NT, 2) k_eng_rhs_tile(Geo g, IoFields f, ThermoFields t, ThermoParams tp,
                                                           const DevState* __restrict__ st, int ns, int chunk) {
    __shared__ double ring[ET_R * 3 * IT_PL];
    __shared__ EngRow srow[IT_J];
    const int N = g.N, nti = (g.LI + IT_I - 1) / IT_I, ntj = g.M / IT_J;
    const int b = blockIdx.x, r = b / nti, kc = r / ntj;
    const int i0 = IT_I * (b - r * nti) + g.xo, j0 = 1 + IT_J * (r - kc * ntj);
    const int k0 = kc * chunk, k1 = min(N, k0 + chunk);
    const int i = i0 + (threadIdx.x & 31), j = j0 + (threadIdx.x >> 5);
    const bool on = i - g.xo < g.LI;
    const double dt = st->dt;
    const double coe1n = g.tgam[ns] * dt, coe0n = g.troh[ns] * dt;
    const double XND2CL = 0.5, ZND2CL = 0.5;
    const double COE1 = g.dxi * XND2CL * 0.5;
    const double COE11 = g.dxqi * XND2CL * tp.cthecd;
    const double COE3 = g.dzi * ZND2CL * 1.0 * 0.5;
    const double COE33 = g.dzqi * ZND2CL * 1.0 * tp.cthecd;
    // this thread's points of a plane: padded offsets at k = 0 (columns past the row's last storage column
    // repeat it; they feed only threads that are off)
    constexpr int NE = (IT_PL + IT_NT - 1) / IT_NT;
    int eo[NE];
#pragma unroll
    for (int e = 0; e < NE; ++e) {
        const int q = threadIdx.x + e * IT_NT, jj = q / IT_HI;
        int ii = i0 - 1 + (q - jj * IT_HI);
        if (g.xo) ii = min(ii, g.L - 1);
        else ii = ii < 0 ? ii + g.L : ii >= g.L ? ii - g.L : ii;
        eo[e] = q < IT_PL ? (int)pidx(g, ii, j0 - 1 + jj, 0) : -1;
    }
    auto load = [&](int k, double* dst) {
        const long long ko = g.P * (k >= N ? k - N : k);
#pragma unroll
        for (int e = 0; e < NE; ++e)
            if (eo[e] >= 0) {
                double* d = dst + threadIdx.x + e * IT_NT;
                const long long o = eo[e] + ko;
                cp_async8(d, t.ENTH + o);
                cp_async8(d + IT_PL, t.TEMP + o);
                cp_async8(d + 2 * IT_PL, t.KAP + o);
            }
    };
    constexpr int PS = 3 * IT_PL;
    load(k0, ring);
    load(k0 + 1, ring + PS);
    if (threadIdx.x < IT_J) srow[threadIdx.x] = eng_row(g, tp, j0 + threadIdx.x);
    const EngRow& y = srow[threadIdx.x >> 5];
    const int cc = (threadIdx.x >> 5) * IT_HI + IT_HI + (threadIdx.x & 31) + 1;  // this point inside a plane
    const double* G1 = f.G;
    const double* G2 = f.G + g.FS;
    const double* G3 = f.G + 2 * g.FS;
    long long c = pidx(g, i, j, k0);
    const int ip = on ? xpn(g, i) - i : 0;
    double hm = 0.0, tm = 0.0, km = 0.0, g3 = 0.0;
    if (on) {
        const long long cm = pidx(g, i, j, wrapm(k0, N));
        hm = t.ENTH[cm]; tm = t.TEMP[cm]; km = t.KAP[cm];
        g3 = G3[c];
    }
    int sk = 0;
#pragma unroll 1
    for (int k = k0; k < k1; ++k, c += g.P) {
        const int sp = sk == ET_R - 1 ? 0 : sk + 1;
        double g1 = 0.0, g1p = 0.0, g2 = 0.0, g2p = 0.0, g3p = 0.0, dh = 0.0, e0 = 0.0;
        if (on) {
            g1 = G1[c]; g1p = G1[c + ip];
            g2 = G2[c]; g2p = G2[c + g.L];
            g3p = G3[k + 1 == N ? pidx(g, i, j, 0) : c + g.P];
            dh = t.DH[c]; e0 = t.RHSE0[c];
        }
        cp_async_wait_all();
        __syncthreads();  // planes k and k + 1 are here, and every thread is done with the slot filled next
        if (k + 1 < k1) load(k + 2, ring + (sp == ET_R - 1 ? 0 : sp + 1) * PS);
        if (on) {
            const double *Hh = ring + sk * PS + cc, *T = Hh + IT_PL, *K = T + IT_PL;
            const double *Hp = ring + sp * PS + cc, *Tp = Hp + IT_PL, *Kp = Tp + IT_PL;
            const double hc = Hh[0], tc = T[0], kc = K[0];
            double DX_DHU = (Hh[1] + hc) * (g1p + g1p) - (hc + Hh[-1]) * (g1 + g1);
            DX_DHU = DX_DHU * COE1;
            double DY_DHV = (y.wffp * Hh[IT_HI] + y.wfbp * hc) * (g2p + g2p) - (y.wff * hc + y.wfb * Hh[-IT_HI]) * (g2 + g2);
            DY_DHV = DY_DHV * y.COE2;
            double DZ_DHW = (Hp[0] + hc) * (g3p + g3p) - (hc + hm) * (g3 + g3);
            DZ_DHW = DZ_DHW * COE3;
            double DX_KDT = (K[1] + kc) * (T[1] - tc) - (kc + K[-1]) * (tc - T[-1]);
            DX_KDT = DX_KDT * COE11;
            double KDTy1 = (y.wffp * K[IT_HI] + y.wfbp * kc) * (T[IT_HI] - tc) * y.COE221;
            double KDTy2 = (y.wff * kc + y.wfb * K[-IT_HI]) * (tc - T[-IT_HI]) * y.COE222;
            if (j == 1 && !tp.iso[0]) KDTy2 = -tp.wf_bot * y.COE222;
            else if (j == g.M && !tp.iso[1]) KDTy1 = -tp.wf_top * y.COE221;
            const double DY_KDT = (KDTy1 - KDTy2) * y.COE22;
            double DZ_KDT = (Kp[0] + kc) * (Tp[0] - tc) - (km + kc) * (tc - tm);
            DZ_KDT = DZ_KDT * COE33;
            const double rhs = -DX_DHU - DY_DHV - DZ_DHW + DX_KDT + DY_KDT + DZ_KDT;
            double d = dh + coe1n * rhs + coe0n * e0;
            d = fmin(tp.dhmax - 1.0e-14, d);
            d = fmax(tp.dhmin + 1.0e-14, d);
            t.DH[c] = d;
            t.RHSE0[c] = rhs;
            hm = hc; tm = tc; km = kc;
            g3 = g3p;
        }
        sk = sp;
    }
}
// planes per block of k_eng_rhs_tile: the split of N that gives the least time, counted in planes loaded by the
// busiest SM (two blocks per SM; each block loads two more planes than it computes)
inline int eng_tile_chunk(const Geo& g, int nsm) {
    const int tiles = ((g.LI + IT_I - 1) / IT_I) * (g.M / IT_J);
    int best = g.N;
    long long cost = -1;
    for (int n = 1; n <= g.N / 4; ++n) {
        const int chunk = (g.N + n - 1) / n;
        const int nb = (g.N + chunk - 1) / chunk;
        const long long t = (long long)((tiles * nb + 2 * nsm - 1) / (2 * nsm)) * (chunk + 2);
        if (cost < 0 || t < cost) { cost = t; best = chunk; }
    }
    return best;
}

// Properties of one padded point from its rho*h; the old DENSITY and
// Viscousity are kept in DENSITY0 (f.RHO) and Viscousity0 (f.MU0) first.
template <typename F>
__device__ __forceinline__ void eng_point(const PropTab& tb, const double* xdh, const double* xh, const IoFieldsT<F>& f,
                                          const ThermoFields& t, long long p, DevState* st) {
    f.RHO[p] = f.DEN[p];
    f.MU0[p] = f.MU[p];
    double o[6];
    if (!prop_point(tb, xdh, xh, t.DH[p], o)) atomicOr(&st->err, CHS_EBIT_TABLE);
    t.ENTH[p] = o[0];
    t.TEMP[p] = o[1];
    f.DEN[p] = o[2];
    f.MU[p] = o[3];
    t.KAP[p] = o[4];
    t.HCP[p] = o[5];
}

__device__ __forceinline__ void stage_keys(const PropTab& tb, double* keys, const double*& xdh, const double*& xh) {
    for (int r = threadIdx.x; r < tb.n; r += blockDim.x) {
        keys[r] = tb.xdh[r];
        keys[tb.n + r] = tb.xh[r];
    }
    __syncthreads();
    xdh = keys;
    xh = keys + tb.n;
}

template <bool SMEM, typename F>
__global__ void __launch_bounds__(PROP_NT) k_eng_props(PropTab tb, Geo g, IoFieldsT<F> f, ThermoFields t, DevState* st) {
    extern __shared__ double keys[];
    const double* xdh = tb.xdh;
    const double* xh = tb.xh;
    if (SMEM) stage_keys(tb, keys, xdh, xh);
    const long long tot = io_points(g);
    for (long long q = (long long)blockIdx.x * PROP_NT + threadIdx.x; q < tot; q += (long long)gridDim.x * PROP_NT) {
        int i, j, k;
        io_decode(g, q, i, j, k);
        eng_point(tb, xdh, xh, f, t, pidx(g, i, j, k), st);
    }
}

// ghost rows j = 0 (bottom) and j = M+1 (top), every i and k
template <bool SMEM, typename F>
__global__ void __launch_bounds__(PROP_NT) k_eng_bc(PropTab tb, Geo g, IoFieldsT<F> f, ThermoFields t, ThermoParams tp,
                                                  DevState* st) {
    extern __shared__ double keys[];
    const double* xdh = tb.xdh;
    const double* xh = tb.xh;
    if (SMEM) stage_keys(tb, keys, xdh, xh);
    const int L = g.L, M = g.M;
    const long long plane = (long long)L * g.N;
    for (long long q = (long long)blockIdx.x * PROP_NT + threadIdx.x; q < 2 * plane; q += (long long)gridDim.x * PROP_NT) {
        const bool top = q >= plane;
        const long long r = top ? q - plane : q;
        const int i = (int)(r % L), k = (int)(r / L);
        long long p;
        const int w = top ? 1 : 0;
        if (tp.iso[w]) {  // BC_WALL_IsoTHERMAL: the wall state, DH = H * D (DENSITY0, Viscousity0 keep the old row)
            p = pidx(g, i, top ? M + 1 : 0, k);
            f.RHO[p] = f.DEN[p];
            f.MU0[p] = f.MU[p];
            t.TEMP[p] = tp.wv[w][0];
            t.ENTH[p] = tp.wv[w][1];
            f.DEN[p] = tp.wv[w][2];
            f.MU[p] = tp.wv[w][3];
            t.KAP[p] = tp.wv[w][4];
            t.DH[p] = t.ENTH[p] * f.DEN[p];
            continue;
        }
        if (top) {
            p = pidx(g, i, M + 1, k);
            t.DH[p] = 2.0 * t.DH[pidx(g, i, M, k)] - g.wff[M] * t.DH[pidx(g, i, M, k)] - g.wfb[M] * t.DH[pidx(g, i, M - 1, k)];
        } else {
            p = pidx(g, i, 0, k);
            t.DH[p] = 2.0 * t.DH[pidx(g, i, 1, k)] - g.wff[2] * t.DH[pidx(g, i, 2, k)] - g.wfb[2] * t.DH[pidx(g, i, 1, k)];
        }
        eng_point(tb, xdh, xh, f, t, p, st);
    }
}

// div(G) at a point, as DENSITY_TIME_DERIVATION forms it
template <typename F>
__device__ __forceinline__ double eng_divg(const Geo& g, const F* G, int i, int j, int k, double g1, double g2, double g3) {
    const long long cip = pidx(g, xpn(g, i), j, k), ckp = pidx(g, i, j, wrapp(k, g.N)), cjp = pidx(g, i, j + 1, k);
    const double COE2 = g.dyfi[j] * 1.0, COE3 = g.dzi * 1.0;
    const double DIVX = ((double)G[cip] - g1) * g.dxi;
    const double DIVY = ((double)G[cjp + g.FS] - g2) * COE2;
    const double DIVZ = ((double)G[ckp + 2 * g.FS] - g3) * COE3;
    return DIVX + DIVY + DIVZ;
}

// The point-wise work between the property update and the momentum step, in one pass over the points:
// DENSITY_TIME_DERIVATION, DENSITY_Staggered and MU_Staggered, then G0_io = G_io and VELOCITY_CALC_io.
// Of G0 only its divergence is ever used, and it is the div(G) of the previous call (G does not change between
// DENSITY_TIME_DERIVATION and G0_io = G_io): DIVG0 holds that, one word per point read and written where
// the three-component copy took three of each.  17 words per point instead of the 27 of three
// kernels; 1.10 -> 0.59 ms per step at 256 x 192 x 128 (FP64), and 0.53 with four blocks per SM (64
// registers instead of 78; FP32 storage 0.54 -> 0.42).
// mpart (inflow/outflow domain, else NULL): per-block sums of DrhoDtP / DYFI for the interior mass
// rate of CHK_MassConsv_io (src/processing/CHK_conservation.f90:41-53)
template <typename F>
__global__ void __launch_bounds__(IO_NT, 4) k_eng_state(Geo g, IoFieldsT<F> f, ThermoFields t, int ns, double* __restrict__ mpart) {
    __shared__ double sred[32];
    const long long tot = io_points(g);
    double ms = 0.0;
    const double tgam = g.tgam[ns], troh = g.troh[ns];
    for (long long q = (long long)blockIdx.x * IO_NT + threadIdx.x; q < tot; q += (long long)gridDim.x * IO_NT) {
        int i, j, k;
        io_decode(g, q, i, j, k);
        const long long c = pidx(g, i, j, k);
        const double g1 = f.G[c], g2 = f.G[c + g.FS], g3 = f.G[c + 2 * g.FS], div0 = t.DIVG0[c];
        const double div = eng_divg(g, f.G, i, j, k, g1, g2, g3);
        F d1, d2, d3;
        io_props_point(g, f, i, j, k, d1, d2, d3);
        const double dr = -tgam * div - troh * div0;
        t.DRHO[c] = dr;
        t.DIVG0[c] = div;
        f.Q[c] = (F)(g1 / (double)d1);
        f.Q[c + 2 * g.FS] = (F)(g3 / (double)d3);
        if (j >= 2) f.Q[c + g.FS] = (F)(g2 / (double)d2);
        if (mpart) ms += dr * (1.0 / g.dyfi[j] / 1.0);
    }
    if (mpart) {
        const double b = block_sum<IO_NT>(ms, sred);
        if (threadIdx.x == 0) mpart[blockIdx.x] = b;
    }
}

// DIVG0 of the thermal solver's start, where G0_io = G_io
template <typename F>
__global__ void __launch_bounds__(IO_NT) k_eng_divg0(Geo g, IoFieldsT<F> f, ThermoFields t) {
    const long long tot = io_points(g);
    for (long long q = (long long)blockIdx.x * IO_NT + threadIdx.x; q < tot; q += (long long)gridDim.x * IO_NT) {
        int i, j, k;
        io_decode(g, q, i, j, k);
        const long long c = pidx(g, i, j, k);
        t.DIVG0[c] = eng_divg(g, f.G, i, j, k, f.G[c], f.G[c + g.FS], f.G[c + 2 * g.FS]);
    }
}
