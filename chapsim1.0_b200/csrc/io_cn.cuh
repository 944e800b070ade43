// Crank-Nicolson sweeps of the main-domain momentum step (iVisScheme = 1):
// MOMFA_io(NS, IDR) (src/MOMFA_io.f90:18-406) for the three components at
// once, after k_io_rhs<true> has formed the right-hand sides.
//
//   k_io_cn_xsweep<S>  MOMFA1_X_io (:79-172): cyclic in x, per-point
//                      coefficients; subtracts the bulk forcing DPGRNS from the
//                      u right-hand side on load (RHS_MOM_EXPLICIT_io.f90:228-265)
//   k_io_cn_zsweep<S>  MOMFA2_Z_io (:175-261): cyclic in z
//   k_io_cn_ysweep<S>  MOMFA3_Y_io (:264-406): non-cyclic in y with the wall
//                      rows of the u and w equations built from AMVR1 / APVRN
//                      and the half-sum of the cell and ghost viscosity; then
//                      G += RHS for j >= N2I (:38-44)
//
// The operator of component IDR is (1 - A) dG with A's rows
// (amu/rho_m, -(amu+apu)/rho_c, apu/rho_p): it acts on dG/rho.  The
// viscosities are Viscousity (cell), MU_STG (edges, from Viscousity0) and the
// densities D_STG of the component, all fixed during the substep.  Each
// coefficient is evaluated with the reference's operand order.  Two details
// of the reference are kept: the v rows divide the coupling to row j+1 by
// D_STG at row j, and the v row j = 1 (the wall face) is the identity with a
// zero right-hand side (AMVR(1,2) = APVR(1,2) = 0; its sweeps in x and z are
// skipped, N2I = 2), so its value stays 0 and the G update starts at j = 2.
//
// A line of n = W S rows is split into W segments of S rows, one thread each, solved as warp_tdma of
// tdma.cuh does: Thomas elimination of a segment's inner rows in registers, its two interface rows
// folded into one unknown per segment, parallel cyclic reduction over the W segments, back
// substitution.  z and y: thread (il, seg) of a block owns segment seg of line il, TI lines being
// consecutive i, so every global access is a row piece of TI values and the right-hand sides and
// property fields go from global memory straight into registers; the interface rows change over through
// shared memory to one lane per segment, where the reduction runs on shuffles.  x lines are
// contiguous: their rows are staged in shared memory by asynchronous copies and each lane reads its
// segment.
//
// Divisions were half of the sweeps' instructions (three quotients by densities per row, two per
// reduction step).  Here each density and each pivot is inverted once.  FP64 (W = 16: longer segments,
// two lines per warp in the reduction, 1.25 instead of 3 inversions per row) multiplies by the
// inverse.  With FP32 storage (W = 32) the quotients are the correctly rounded ones of a division
// (Markstein's correction of a product by the rounded reciprocal, IBM J. Res. Dev. 34 (1990) 111) and
// every operation keeps its order, so that the mixed-precision step gives the same fields to the
// bit: its FP32 rounding turns any change of the last FP64 bit into one of the stored value.
//
// Measured at 256 x 192 x 128 (three launches each): FP64 z + y 2.71 -> 0.75 ms and x 1.07 -> 0.35 ms per
// step (floors of their 27 and 12 words per point at the measured copy bandwidth: 0.63 and 0.28);
// FP32 storage 2.56 -> 1.07 and 0.99 -> 0.39.
#pragma once
#include "common.cuh"
#include "tdma.cuh"
#include "io.cuh"

// DPGRNS of RHS_MOM_EXPLICIT_io (:231-263)
__device__ __forceinline__ double cn_dpgrns(const Geo& g, const DevState* st, int ns) {
    if (g.iflowdriven == 1) return st->bulksum / g.volm;
    if (g.iflowdriven == 2) return -0.5 * g.cf_given * (g.talp[ns] * st->dt);
    return 0.0;
}

// segments per line, lines per z or y block, and lines per x block for the storage type F
template <typename F> __host__ __device__ constexpr int cn_w() { return sizeof(F) == 8 ? 16 : 32; }
template <typename F> __host__ __device__ constexpr int cn_ti() { return 256 / cn_w<F>(); }
#define CN_NT 256
#define CN_XNT 128
template <typename F> __host__ __device__ constexpr int cn_xlines() { return CN_XNT / cn_w<F>(); }

// a / d from r = 1 / d
template <bool EXACT>
__device__ __forceinline__ double cn_div(double a, double d, double r) {
    const double q = a * r;
    if constexpr (!EXACT) return q;
    return fma(fma(-q, d, a), r, q);
}

struct CnEnds { double A0, B0, C0, D0, A1, B1, C1, D1; };  // a segment's two interface rows

// Forward elimination of a segment.  coef(k, a, b, c) gives row k's coefficients, d the right-hand
// sides; leaves the inner rows as y_k = d_k - ap_k y_0 - cq_k y_{S-1}.
template <int S, class Coef>
__device__ __forceinline__ CnEnds cn_forward(double (&d)[S], double (&ap)[S], double (&cq)[S], const Coef& coef) {
    CnEnds e;
    if constexpr (S <= 2) {
        coef(0, e.A0, e.B0, e.C0);
        e.D0 = d[0];
        if constexpr (S == 2) {
            coef(1, e.A1, e.B1, e.C1);
            e.D1 = d[1];
        } else {
            e.A1 = e.B1 = e.C1 = e.D1 = 0.0;
        }
    } else {
        double a0, b0, c0, ak, bk, ck;
        coef(0, a0, b0, c0);
        coef(1, ak, bk, ck);
        {
            const double r = 1.0 / bk;
            ap[1] = ak * r;
            cq[1] = ck * r;
            d[1] *= r;
        }
#pragma unroll
        for (int k = 2; k <= S - 2; ++k) {
            coef(k, ak, bk, ck);
            const double r = 1.0 / (bk - ak * cq[k - 1]);
            d[k] = (d[k] - ak * d[k - 1]) * r;
            ap[k] = -ak * ap[k - 1] * r;
            cq[k] = ck * r;
        }
#pragma unroll
        for (int k = S - 3; k >= 1; --k) {
            d[k] = d[k] - cq[k] * d[k + 1];
            ap[k] = ap[k] - cq[k] * ap[k + 1];
            cq[k] = -cq[k] * cq[k + 1];
        }
        double aL, bL, cL;
        coef(S - 1, aL, bL, cL);
        e.A0 = a0;
        e.B0 = b0 - c0 * ap[1];
        e.C0 = -c0 * cq[1];
        e.D0 = d[0] - c0 * d[1];
        e.A1 = -aL * ap[S - 2];
        e.B1 = bL - aL * cq[S - 2];
        e.C1 = cL;
        e.D1 = d[S - 1] - aL * d[S - 2];
    }
    return e;
}

// The W interface unknowns of a line, lane l of a W-wide group holding segment l's rows: u = y_{S-1}
// and y0 = y_0 of the segment.
template <int S, int W, bool CYCLIC, bool EXACT>
__device__ __forceinline__ void cn_reduce(CnEnds e, int lane, double& u, double& y0) {
    auto sh = [](double v, int src) { return __shfl_sync(0xffffffffu, v, src & (W - 1), W); };
    if constexpr (!CYCLIC) {
        if (lane == 0) e.A0 = 0.0;
        if (lane == W - 1) { if constexpr (S == 1) e.C0 = 0.0; else e.C1 = 0.0; }
    }
    Row4 row;
    double iB0 = 0.0;
    if constexpr (S == 1) {
        row.al = e.A0; row.be = e.B0; row.ga = e.C0; row.de = e.D0;
    } else {
        iB0 = 1.0 / e.B0;
        const double A0n = sh(e.A0, lane + 1), C0n = sh(e.C0, lane + 1), D0n = sh(e.D0, lane + 1), iB0n = sh(iB0, lane + 1);
        row.al = -e.A1 * e.A0 * iB0;
        row.be = e.B1 - e.A1 * e.C0 * iB0 - e.C1 * A0n * iB0n;
        row.ga = -e.C1 * C0n * iB0n;
        row.de = e.D1 - e.A1 * e.D0 * iB0 - e.C1 * D0n * iB0n;
    }
    constexpr int LAST = CYCLIC ? W / 4 : W / 2;  // cyclic: the last pair is solved as a 2 x 2 system
#pragma unroll
    for (int s = 1; s <= LAST; s <<= 1) {
        const double r = 1.0 / row.be;
        Row4 lo, hi;
        lo.al = sh(row.al, lane - s); lo.ga = sh(row.ga, lane - s); lo.de = sh(row.de, lane - s);
        hi.al = sh(row.al, lane + s); hi.ga = sh(row.ga, lane + s); hi.de = sh(row.de, lane + s);
        const double lr = sh(r, lane - s), hr = sh(r, lane + s);
        if constexpr (EXACT) { lo.be = sh(row.be, lane - s); hi.be = sh(row.be, lane + s); }
        else lo.be = hi.be = 0.0;
        const bool hasl = CYCLIC || lane - s >= 0, hash = CYCLIC || lane + s <= W - 1;
        const double k1 = hasl ? cn_div<EXACT>(row.al, lo.be, lr) : 0.0;
        const double k2 = hash ? cn_div<EXACT>(row.ga, hi.be, hr) : 0.0;
        Row4 nr;
        nr.al = hasl ? -k1 * lo.al : 0.0;
        nr.ga = hash ? -k2 * hi.ga : 0.0;
        if constexpr (CYCLIC) {
            nr.be = row.be - k1 * lo.ga - k2 * hi.al;
            nr.de = row.de - k1 * lo.de - k2 * hi.de;
        } else {
            nr.be = row.be - (hasl ? k1 * lo.ga : 0.0) - (hash ? k2 * hi.al : 0.0);
            nr.de = row.de - (hasl ? k1 * lo.de : 0.0) - (hash ? k2 * hi.de : 0.0);
        }
        row = nr;
    }
    if constexpr (CYCLIC) {
        Row4 pr;
        pr.al = sh(row.al, lane ^ (W / 2)); pr.be = sh(row.be, lane ^ (W / 2));
        pr.ga = sh(row.ga, lane ^ (W / 2)); pr.de = sh(row.de, lane ^ (W / 2));
        const double ci = row.al + row.ga, cm = pr.al + pr.ga;
        u = (row.de * pr.be - ci * pr.de) / (row.be * pr.be - ci * cm);
    } else {
        u = row.de / row.be;
    }
    y0 = u;
    if constexpr (S > 1) {
        const double up = sh(u, lane - 1);
        y0 = cn_div<EXACT>(e.D0 - e.A0 * up - e.C0 * u, e.B0, iB0);  // A0 == 0 on segment 0 when not cyclic
    }
}

// back substitution of a segment
template <int S>
__device__ __forceinline__ void cn_back(double (&d)[S], const double (&ap)[S], const double (&cq)[S], double u, double y0) {
    d[0] = y0;
    if constexpr (S > 1) d[S - 1] = u;
    if constexpr (S > 2) {
#pragma unroll
        for (int k = 1; k <= S - 2; ++k) d[k] = d[k] - ap[k] * y0 - cq[k] * u;
    }
}

// z and y blocks: the interface rows of the block's TI lines change over from thread (il, seg) to one
// lane per segment through shared memory, and u and y0 back
template <int S, int W, int TI, bool CYCLIC, bool EXACT>
__device__ __forceinline__ void cn_block_reduce(const CnEnds& e, int il, int seg, double& u, double& y0) {
    constexpr int LD = W + 1;
    __shared__ double sm[8][TI * LD];
    const int p = il * LD + seg;
    sm[0][p] = e.A0; sm[1][p] = e.B0; sm[2][p] = e.C0; sm[3][p] = e.D0;
    if constexpr (S > 1) { sm[4][p] = e.A1; sm[5][p] = e.B1; sm[6][p] = e.C1; sm[7][p] = e.D1; }
    __syncthreads();
    const int line = threadIdx.x / W, lane = threadIdx.x % W, q = line * LD + lane;
    CnEnds t{sm[0][q], sm[1][q], sm[2][q], sm[3][q], 0.0, 0.0, 0.0, 0.0};
    if constexpr (S > 1) { t.A1 = sm[4][q]; t.B1 = sm[5][q]; t.C1 = sm[6][q]; t.D1 = sm[7][q]; }
    cn_reduce<S, W, CYCLIC, EXACT>(t, lane, u, y0);
    sm[0][q] = u;  // only this thread has read entry q
    sm[1][q] = y0;
    __syncthreads();
    u = sm[0][p];
    y0 = sm[1][p];
}

// Coefficients of a segment: row k couples by amu to the row before and apu to the row after,
// A = amu / D_{k-1}, B = 1 - (amu + apu) / D_k, C = apu / D_{k+1}; D[k + 1] is row k's density.
template <int S, bool EXACT>
struct CnDens {
    double D[S + 2], r[S + 2];
    __device__ __forceinline__ void invert() {
#pragma unroll
        for (int k = 0; k < S + 2; ++k) r[k] = 1.0 / D[k];
    }
    __device__ __forceinline__ double over(double a, int k) const { return cn_div<EXACT>(a, D[k], r[k]); }
};

// Threads per SM the register budgets are sized for, by the rows per segment
template <int S> __host__ __device__ constexpr int cn_minb(int nt) { return S > 12 ? 256 / nt : S > 6 ? 512 / nt : 768 / nt; }

// x lines (j, k); component blockIdx.y (0 u, 1 v, 2 w)
template <typename F> inline size_t smem_cn_x(int n) {
    const int s = n / cn_w<F>(), seg = n + n / s;
    return (size_t)cn_xlines<F>() * (size_t)(seg + 1) * (2 * sizeof(F) + sizeof(double));
}
template <int S, typename F>
__global__ void __launch_bounds__(CN_XNT, cn_minb<S>(CN_XNT)) k_io_cn_xsweep(Geo g, IoFieldsT<F> f, const DevState* __restrict__ st, int ns) {
    constexpr int W = cn_w<F>(), LPB = cn_xlines<F>();
    constexpr bool EXACT = sizeof(F) == 4;
    constexpr int L = W * S, SEG = L + W + 1;  // a line's staged row: one pad per segment
    extern __shared__ __align__(16) unsigned char smx_raw[];
    const int M = g.M, comp = blockIdx.y;
    const int warp = threadIdx.x >> 5, lane32 = threadIdx.x & 31;
    const int lane = threadIdx.x % W, lw = threadIdx.x / W;  // segment, line of the block
    double* const sm_m = reinterpret_cast<double*>(smx_raw);
    F* const sm_d = reinterpret_cast<F*>(sm_m + LPB * SEG);
    F* const sm_r = sm_d + LPB * SEG;
    const F* D = f.DST + comp * g.FS;
    F* R = f.RHS + comp * g.FI;
    // (M N lines, a multiple of LPB: every lane has a line)
    // stage the rows of this warp's 32 / W lines: density, viscosity and right-hand side
#pragma unroll
    for (int q = 0; q < 32 / W; ++q) {
        const int l = warp * (32 / W) + q;
        const long long line = (long long)blockIdx.x * LPB + l;
        const int j = 1 + (int)(line % M), k = (int)(line / M);
        const long long row = pidx(g, 0, j, k), irow = iidx(g, 0, j, k);
#pragma unroll
        for (int t = 0; t < L / 32; ++t) {
            const int i = lane32 + 32 * t, s = l * SEG + seg_pos<S>(i);
            cp_async_el(sm_d + s, D + row + i);
            cp_async_el(sm_r + s, R + irow + i);
            if (comp == 0) cp_async_el(sm_m + s, f.MU + row + i);
            else cp_async_el(reinterpret_cast<F*>(sm_m + s), f.MST + (comp == 1 ? 0 : g.FS) + row + i);
        }
    }
    cp_async_wait_all();
    __syncwarp();
    {
        const double fac = 0.50 * g.talp[ns] * st->dt * g.cvisc;
        const double coe = comp == 0 ? fac * 4.0 / 3.0 * g.dxqi : fac * g.dxqi;
        const double dpg = comp == 0 ? cn_dpgrns(g, st, ns) : 0.0;
        const int base = lw * SEG + lane * (S + 1);
        auto at = [&](int k) {  // staged position of row lane S + k, k = -1 .. S, cyclic
            if (k < 0) return lane == 0 ? lw * SEG + seg_pos<S>(L - 1) : base - 2;
            if (k >= S) return lane == W - 1 ? lw * SEG : base + S + 1;
            return base + k;
        };
        auto visc = [&](int k) { return comp == 0 ? sm_m[at(k)] : (double)*reinterpret_cast<const F*>(sm_m + at(k)); };
        CnDens<S, EXACT> dn;
        double mm[S + 1], d[S], ap[S], cq[S];
#pragma unroll
        for (int k = 0; k < S + 2; ++k) dn.D[k] = (double)sm_d[at(k - 1)];
#pragma unroll
        for (int k = 0; k < S + 1; ++k) mm[k] = visc(comp == 0 ? k - 1 : k);
#pragma unroll
        for (int k = 0; k < S; ++k) d[k] = comp == 0 ? (double)sm_r[at(k)] - dpg : (double)sm_r[at(k)];
        dn.invert();
        const CnEnds e = cn_forward<S>(d, ap, cq, [&](int k, double& a, double& b, double& c) {
            const double amu = -coe * mm[k], apu = -coe * mm[k + 1];
            a = dn.over(amu, k);
            c = dn.over(apu, k + 2);
            b = 1.0 - dn.over(amu + apu, k + 1);
        });
        double u, y0;
        cn_reduce<S, W, true, EXACT>(e, lane, u, y0);
        cn_back<S>(d, ap, cq, u, y0);
#pragma unroll
        for (int k = 0; k < S; ++k) sm_r[base + k] = (F)d[k];  // this thread's own segment
    }
    __syncwarp();
#pragma unroll
    for (int q = 0; q < 32 / W; ++q) {
        const int l = warp * (32 / W) + q;
        const long long ln = (long long)blockIdx.x * LPB + l;
        const int jl = 1 + (int)(ln % M), k = (int)(ln / M);
        if (comp == 1 && jl == 1) continue;  // MOMFA1_X_io starts at N2I = 2 for v
        const long long irow = iidx(g, 0, jl, k);
#pragma unroll
        for (int t = 0; t < L / 32; ++t) {
            const int i = lane32 + 32 * t;
            R[irow + i] = sm_r[l * SEG + seg_pos<S>(i)];
        }
    }
}

// z lines (i0 .. i0+TI-1, j); component blockIdx.z
template <int S, typename F>
__global__ void __launch_bounds__(CN_NT, cn_minb<S>(CN_NT)) k_io_cn_zsweep(Geo g, IoFieldsT<F> f, const DevState* __restrict__ st, int ns) {
    constexpr int W = cn_w<F>(), TI = cn_ti<F>();
    constexpr bool EXACT = sizeof(F) == 4;
    const int N = W * S;
    const int comp = blockIdx.z;
    const int j = 1 + blockIdx.y;
    if (comp == 1 && j == 1) return;  // uniform over the block
    const int il = threadIdx.x % TI, seg = threadIdx.x / TI;
    const int i = blockIdx.x * TI + il, k0 = seg * S;
    const double fac = 0.50 * g.talp[ns] * st->dt * g.cvisc;
    const double coe = comp == 2 ? fac * 4.0 / 3.0 * g.dzqi : fac * g.dzqi;
    const long long col = pidx(g, i, j, 0);
    const F* D = f.DST + comp * g.FS + col;
    F* R = f.RHS + comp * g.FI + iidx(g, i, j, k0);
    CnDens<S, EXACT> dn;
    double mm[S + 1], d[S], ap[S], cq[S];
#pragma unroll
    for (int k = 0; k < S; ++k) d[k] = R[g.PI_ * k];
    const long long pb = g.P * (k0 == 0 ? N - 1 : k0 - 1), pe = g.P * (k0 + S == N ? 0 : k0 + S);  // cyclic neighbours
#pragma unroll
    for (int k = 0; k < S + 2; ++k) dn.D[k] = (double)D[k == 0 ? pb : k == S + 1 ? pe : g.P * (k0 + k - 1)];
    if (comp == 2) {
        const double* m = f.MU + col;
#pragma unroll
        for (int k = 0; k < S + 1; ++k) mm[k] = m[k == 0 ? pb : g.P * (k0 + k - 1)];
    } else {
        const F* m = f.MST + (comp == 0 ? g.FS : 2 * g.FS) + col;
#pragma unroll
        for (int k = 0; k < S + 1; ++k) mm[k] = (double)m[k == S ? pe : g.P * (k0 + k)];
    }
    dn.invert();
    const CnEnds e = cn_forward<S>(d, ap, cq, [&](int k, double& a, double& b, double& c) {
        const double amu = -coe * mm[k], apu = -coe * mm[k + 1];
        a = dn.over(amu, k);
        b = 1.0 - dn.over(amu + apu, k + 1);
        c = dn.over(apu, k + 2);
    });
    double u, y0;
    cn_block_reduce<S, W, TI, true, EXACT>(e, il, seg, u, y0);
    cn_back<S>(d, ap, cq, u, y0);
#pragma unroll
    for (int k = 0; k < S; ++k) R[g.PI_ * k] = (F)d[k];
}

// y lines (i0 .. i0+TI-1, k); component blockIdx.z; then G += solution
template <int S, typename F>
__global__ void __launch_bounds__(CN_NT, cn_minb<S>(CN_NT)) k_io_cn_ysweep(Geo g, IoFieldsT<F> f, const DevState* __restrict__ st, int ns) {
    constexpr int W = cn_w<F>(), TI = cn_ti<F>();
    constexpr bool EXACT = sizeof(F) == 4;
    const int M = W * S;
    const int comp = blockIdx.z;
    const int k = blockIdx.y;
    const int il = threadIdx.x % TI, seg = threadIdx.x / TI;
    const int i = blockIdx.x * TI + il, j0 = 1 + seg * S;
    const double fac = 0.50 * g.talp[ns] * st->dt * g.cvisc;
    const double coe = comp == 1 ? fac * 4.0 / 3.0 : fac;
    const double* amv = g.amvr + comp * (M + 2) + j0;
    const double* apv = g.apvr + comp * (M + 2) + j0;
    const long long js = g.L, col = pidx(g, i, j0, k);
    const F* D = f.DST + comp * g.FS + col;
    const F* R = f.RHS + comp * g.FI + iidx(g, i, j0, k);
    F* Gc = f.G + comp * g.FS + col;
    const bool first = seg == 0, last = seg == W - 1;
    CnDens<S, EXACT> dn;
    double mm[S + 1], d[S], ap[S], cq[S];
#pragma unroll
    for (int r = 0; r < S; ++r) d[r] = (comp == 1 && r == 0 && first) ? 0.0 : (double)R[js * r];
    // The densities of rows j0 - 1 .. j0 + S.  v at j = 1: the ghost D_STG(:,0,:,2) is the y-periodic halo
    // D_STG(:,M,:,2) of a run on two or more ranks (the coupling to it is zero, so only its finiteness
    // matters); u and w do not couple to the ghost rows.
#pragma unroll
    for (int r = 0; r < S + 2; ++r) {
        long long o = js * (r - 1);
        if (r == 0 && first) o = js * (M - 1);
        if (r == S + 1 && last) o = js * (S - 1);
        dn.D[r] = (double)D[o];
    }
    double wlo = 0.0, whi = 0.0;  // half-sums of the cell and ghost viscosity in the wall rows of u and w
    if (comp == 1) {
        const double* m = f.MU + col;
#pragma unroll
        for (int r = 0; r < S + 1; ++r) mm[r] = m[js * (r - 1)];
    } else {
        const F* m = f.MST + (comp == 0 ? 0 : 2 * g.FS) + col;
#pragma unroll
        for (int r = 0; r < S + 1; ++r) mm[r] = (double)m[js * r];
        if (first) wlo = (f.MU[col] + f.MU[col - js]) * 0.5;
        if (last) whi = (f.MU[col + js * (S - 1)] + f.MU[col + js * S]) * 0.5;
    }
    dn.invert();
    const CnEnds e = cn_forward<S>(d, ap, cq, [&](int r, double& a, double& b, double& c) {
        double amu = -coe * amv[r] * mm[r], apu = -coe * apv[r] * mm[r + 1];
        if (comp != 1) {
            if (r == 0 && first) amu = -coe * g.amvr1 * wlo;
            if (r == S - 1 && last) apu = -coe * g.apvrn * whi;
            a = (r == 0 && first) ? 0.0 : dn.over(amu, r);
            c = (r == S - 1 && last) ? 0.0 : dn.over(apu, r + 2);
        } else {
            a = dn.over(amu, r);
            // the v rows divide the coupling to row j + 1 by D_STG at row j (row 2 at the wall face j = 1)
            c = (r == 0 && first) ? dn.over(apu, r + 2) : dn.over(apu, r + 1);
        }
        b = 1.0 - dn.over(amu + apu, r + 1);
    });
    double u, y0;
    cn_block_reduce<S, W, TI, false, EXACT>(e, il, seg, u, y0);
    cn_back<S>(d, ap, cq, u, y0);
    double gv[S];
#pragma unroll
    for (int r = 0; r < S; ++r) gv[r] = (double)Gc[js * r];
#pragma unroll
    for (int r = 0; r < S; ++r)
        if (!(comp == 1 && r == 0 && first)) Gc[js * r] = (F)(d[r] + gv[r]);
}
