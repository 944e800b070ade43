// Pressure Poisson solve and projection of one RK3 substep:
//   DIVG_tg (src/DIVG.f90:15-51), FFT99_POIS3D_periodicxz
//   (src/possion3d_FFT99.f90:271-505), VELOUPDT_tg
//   (src/VELO_CORRECTION.f90:14-100), PRCALC_tg
//   (src/PRESSURE_CORRECTION.f90:15-99) and the wall ghosts of
//   BC_WALL_PR_tg (src/BC_WALL.f90:293-361).
//
// Kernels:
//   k_div_fftx   divergence of u* / (alpha dt) (-> RHSLLPHI where k_correct reads it), then the real
//                x transform of every (j, k) line (two real lines packed in
//                one complex FFT), times 1/L, into the spectral array
//   k_fftz<S>    complex z transform of every (kx, j) line; forward pass
//                multiplies by 1/N (UN3M)
//   k_ysolve_warp, _seq, _2w, _scan, _reg
//                per (kx, kz) tridiagonal solve in y with diagonal
//                ACPH(j) - AK1(kx) - AK3(kz); zero mode pinned as in
//                TDMA_PHI_COEF (:225-231) and :341-344, :387-389
//                (phi_hat(0,y_1,0) = 0)
//   k_fftx_inv   inverse x transform -> DPH
//   k_correct    velocity correction, pressure update, PR wall ghosts
#pragma once
#include "common.cuh"
#include "fft.cuh"
#include "tdma.cuh"

#include <type_traits>

// Spectral element type of a step whose fields are stored as R: double2 in the
// FP64 step, float2 in the mixed-precision step (whose x and z transforms run
// in FP32; the y-solve converts to FP64 and back).
template <typename R> using SpecT = typename std::conditional<std::is_same<R, float>::value, float2, double2>::type;
template <typename C> __device__ __forceinline__ const C* twx_of(const Geo& g);
template <> __device__ __forceinline__ const double2* twx_of<double2>(const Geo& g) { return g.twx; }
template <> __device__ __forceinline__ const float2* twx_of<float2>(const Geo& g) { return g.twxf; }
template <typename C> __device__ __forceinline__ const C* twz_of(const Geo& g);
template <> __device__ __forceinline__ const double2* twz_of<double2>(const Geo& g) { return g.twz; }
template <> __device__ __forceinline__ const float2* twz_of<float2>(const Geo& g) { return g.twzf; }
__device__ __forceinline__ double2 to_d2(double2 a) { return a; }
__device__ __forceinline__ double2 to_d2(float2 a) { return make_double2((double)a.x, (double)a.y); }
template <typename C> __device__ __forceinline__ C from_d2(double2 a);
template <> __device__ __forceinline__ double2 from_d2<double2>(double2 a) { return a; }
template <> __device__ __forceinline__ float2 from_d2<float2>(double2 a) { return make_float2((float)a.x, (float)a.y); }

// x-line transforms: PX_TJ x lines per block (PX_TJ / 2 packed pairs), PX_NT
// threads, PX_MINB blocks per SM in the register budget (128 registers).  The
// block loads its lines, transforms them in shared memory and stores them,
// one phase after the other; four small blocks per SM overlap those phases
// better than two blocks of twice the size.
#define PX_TJ 16
#define PX_NT 128
#define PX_MINB 4
// FP32 transforms: eight blocks per SM within 64 registers (twice the warps to
// hide the latency of the load, transform and store phases)
template <typename C> __host__ __device__ constexpr int px_minb() { return sizeof(C) == 8 ? 8 : PX_MINB; }
#define CR_NT 256

// ---------------------------------------------------------------------------
// R is the stored type of Q, PR, RHSLLPHI and DPH (double, or float in the
// mixed-precision step, whose x and z transforms also run in FP32); the
// divergence and the correction are evaluated in FP64.  ST: RHSLLPHI is stored (see k_correct).
template <typename R, bool ST, int N1, int N2>
__global__ void __launch_bounds__(PX_NT, px_minb<SpecT<R>>()) k_div_fftx(Geo g, const R* __restrict__ Q, R* __restrict__ RHSLL,
                                                    SpecT<R>* __restrict__ SP, const DevState* __restrict__ st, int ns) {
    pdl_wait();
    using C = SpecT<R>;
    using T = typename CReal<C>::T;
    extern __shared__ __align__(16) unsigned char smp_raw[];
    C* smc = reinterpret_cast<C*>(smp_raw);
    constexpr int L = N1 * N2, LH = L / 2 + 1, LD = L + N2 + 1, NP = PX_TJ / 2;
    const int M = g.M, N = g.N;
    const int j0 = 1 + blockIdx.x * PX_TJ;
    const int k = blockIdx.y;
    const int kp = wrapp(k, N);
    const double coe0 = 1.0 / (st->dt * g.talp[ns]);
    const R* U = Q;
    const R* V = Q + g.FS;
    const R* Wf = Q + 2 * g.FS;
    const double coe1 = g.dxi / 1.0;
    // one item = VW consecutive points of both rows of a packed pair (M is a multiple of 32: every row of the
    // tile exists), read with 16-byte loads and no branch between them, so that all of two items' loads are in
    // flight together: waits for them were 0.7 of the kernel's stalls at 2.5 TB/s.  Per step 1.31 -> 1.13 ms at
    // 384 x 256 x 384 (1.42 -> 1.39 with RHSLLPHI stored), 70 -> 56 us at 128^3, FP32 at 384 x 256 x 384 0.72 -> 0.59 ms.  The pair's complex
    // values are stored to shared memory together
    constexpr int VW = V16<R>::W, LV = L / VW, NI = NP * LV;
    auto item = [&](int p) {
        const int pair = p / LV, i0 = (p - pair * LV) * VW;
        const int j = j0 + 2 * pair;
        const long long c = pidx(g, i0, j, k), cp = pidx(g, i0, j, kp);
        const int dn = i0 + VW == L ? VW - L : VW;  // u at i0 + VW (periodic)
        R u[2][VW], v[3][VW], w[2][VW], wp[2][VW], un[2];
#pragma unroll
        for (int part = 0; part < 2; ++part) {
            ld16(U + c + part * L, u[part]);
            ld16(V + c + part * L, v[part]);
            ld16(Wf + c + part * L, w[part]);
            ld16(Wf + cp + part * L, wp[part]);
            un[part] = U[c + part * L + dn];
        }
        ld16(V + c + 2 * L, v[2]);
        T val[2][VW];
#pragma unroll
        for (int part = 0; part < 2; ++part) {
            const double coe2 = g.dyfi[j + part] / 1.0;
            R out[VW];
#pragma unroll
            for (int e = 0; e < VW; ++e) {
                const double uc = u[part][e], up = e + 1 < VW ? (double)u[part][e + 1] : (double)un[part];
                const double dv = (up - uc) * coe1 + ((double)v[part + 1][e] - (double)v[part][e]) * coe2 +
                                  ((double)wp[part][e] - (double)w[part][e]) * g.dzi;
                const double x = dv * coe0;
                out[e] = (R)x;
                val[part][e] = (T)x;
            }
            if constexpr (ST) st16(RHSLL + iidx(g, i0, j + part, k), out);
        }
        C* line = smc + pair * LD + i0;
#pragma unroll
        for (int e = 0; e < VW; ++e) line[e] = mkc(val[0][e], val[1][e]);
    };
#pragma unroll 2
    for (int t = 0; t < NI / PX_NT; ++t) item(threadIdx.x + t * PX_NT);
    if (NI % PX_NT && threadIdx.x < NI % PX_NT) item(threadIdx.x + NI / PX_NT * PX_NT);
    block_fft4s<N1, N2, -1>(smc, NP, LD, twx_of<C>(g));
    // unpack: A_k = (Z_k + conj Z_{L-k}) / 2, B_k = (Z_k - conj Z_{L-k}) / (2i), both times 1/L
    const T sc = (T)(0.5 / (double)L);
    for (int p = threadIdx.x; p < NP * LH; p += PX_NT) {
        const int pair = p / LH, kx = p - pair * LH;
        const C* line = smc + pair * LD;
        const C z = line[kx];
        const C zc = line[kx == 0 ? 0 : L - kx];
        C* sp = SP + kx + (long long)LH * ((j0 + 2 * pair - 1) + (long long)M * k);
        sp[0] = mkc((z.x + zc.x) * sc, (z.y - zc.y) * sc);
        sp[LH] = mkc((z.y + zc.y) * sc, (zc.x - z.x) * sc);
    }
}

// ---------------------------------------------------------------------------
// The two passes of the four-step FFT (fft.cuh) on registers: a thread holds one length-N2 (first
// pass) or length-N1 (second pass) transform, and only the exchange between the passes goes through
// shared memory.  buf: the line's n + n2 + 1 words.
template <int N1, int N2, int SIGN, typename C>
__device__ __forceinline__ void fft_first(C (&v)[N2], C* buf, int j1, const C* __restrict__ tw) {
    SmallDft<N2, SIGN, C>::run(v);
#pragma unroll
    for (int k2 = 0; k2 < N2; ++k2) {
        C w = tw[j1 * k2];
        if (SIGN > 0) w.y = -w.y;
        buf[k2 * (N1 + 1) + j1] = (j1 == 0 || k2 == 0) ? v[k2] : cmul(v[k2], w);
    }
}
template <int N1, int SIGN, typename C>
__device__ __forceinline__ void fft_second(C (&v)[N1], const C* buf, int k2) {
#pragma unroll
    for (int j1 = 0; j1 < N1; ++j1) v[j1] = buf[k2 * (N1 + 1) + j1];
    SmallDft<N1, SIGN, C>::run(v);
}

// x-line blocks: PX_TJ y rows as PX_TJ / 2 packed pairs, N1 threads per pair
template <int N1> __host__ __device__ constexpr int px_nt() { return PX_TJ / 2 * N1; }
template <typename C, int N1> __host__ __device__ constexpr int px_rminb() { return (sizeof(C) == 8 ? 1024 : 512) / px_nt<N1>(); }
// complex z transform of TQ consecutive (kx, j) lines (index q = kx + LH*(j-1); LH M is a multiple of
// 32): thread (ql, j1) loads the N2 values of its first-pass transform straight into registers, all in
// flight together, as row pieces of TQ complex values (128 bytes), and the second pass's results go from
// registers to memory.  Staging the tile in shared memory on both sides (asynchronous copies in, a
// pass out) cost four more moves of every value and three more block barriers.  Both directions, per
// step: 0.21 -> 0.12 ms at 256 x 192 x 128, 0.18 -> 0.10 at 192 x 128 x 192, 1.29 -> 1.03 at 384 x 256 x 384 (24
// complex values in registers: the load, transform and store phases of two blocks per SM in turn), FP32 there
// 0.62 -> 0.49.  The FP32 fields are the same to the bit.
template <typename C> __host__ __device__ constexpr int fz_tq() { return 128 / (int)sizeof(C); }
template <typename C, int N1> __host__ __device__ constexpr int fz_nt() { return fz_tq<C>() * N1; }
template <typename C, int N1> __host__ __device__ constexpr int fz_minb() { return (sizeof(C) == 8 ? 1024 : 512) / fz_nt<C, N1>(); }
template <int SIGN, int N1, int N2, typename C>
__global__ void __launch_bounds__((fz_nt<C, N1>()), (fz_minb<C, N1>())) k_fftz(Geo g, C* __restrict__ SP) {
    pdl_wait();
    using T = typename CReal<C>::T;
    extern __shared__ __align__(16) unsigned char smp_raw[];
    C* smc = reinterpret_cast<C*>(smp_raw);
    constexpr int N = N1 * N2, LD = N + N2 + 1, TQ = fz_tq<C>();
    const long long Q = (long long)g.LH * g.M;
    const int ql = threadIdx.x % TQ, j1 = threadIdx.x / TQ;
    C* const sp = SP + (long long)blockIdx.x * TQ + ql;
    {
        C v[N2];
        const C* src = sp + Q * j1;
#pragma unroll
        for (int j2 = 0; j2 < N2; ++j2) v[j2] = src[Q * (N1 * j2)];
        fft_first<N1, N2, SIGN>(v, smc + ql * LD, j1, twz_of<C>(g));
    }
    __syncthreads();
    const T sc = SIGN < 0 ? (T)(1.0 / (double)N) : (T)1.0;
#pragma unroll 1
    for (int k2 = j1; k2 < N2; k2 += N1) {
        C v[N1];
        fft_second<N1, SIGN>(v, smc + ql * LD, k2);
        C* dst = sp + Q * k2;
#pragma unroll
        for (int k1 = 0; k1 < N1; ++k1) {
            C x = v[k1];
            if (SIGN < 0) { x.x = x.x * sc; x.y = x.y * sc; }
            dst[Q * (N2 * k1)] = x;
        }
    }
}

// ---------------------------------------------------------------------------
// y solve of YW_L consecutive lines q = kx + LH*kz per block, one warp per
// line, by the warp Thomas/PCR hybrid with a complex right-hand side
// (warp_tdma_c).  The coefficients (AMPH, ACPH - AK1 - AK3, APPH) are formed
// on the fly, so no per-line factor arrays are read.  For kx != 0 or kz != 0
// the systems are strictly diagonally dominant (AK1 + AK3 > 0 on top of the
// weakly dominant Neumann operator), for which the reduction is stable.  The
// singular kx = kz = 0 line keeps the reference's sequential recurrence with
// its pinned first row (TDMA_PHI_COEF :225-231, :341-344, :387-389), run by
// one lane.  Lines are staged in shared memory, line l at l*LS with row r at
// seg_pos<S>(r), LS = M + 33: conflict-free both for the coalesced tile load
// (16 lines per row) and for the per-lane segment access.  Shared memory:
// two stages of YW_L such lines in the spectrum's type, plus M FP64 complex
// values for the zero mode's forward sweep when that type is float2.
#define YW_L 16
#define YW_NT 512

struct PoisCoef {
    const double *am, *ac, *ap;
    double shift;
    __device__ __forceinline__ double A(int r) const { return am[r + 1]; }
    __device__ __forceinline__ double B(int r) const { return ac[r + 1] + shift; }
    __device__ __forceinline__ double C(int r) const { return ap[r + 1]; }
};

// Factors of the zero-mode recurrence (kx = kz = 0, phi(y_1) pinned): the
// forward sweep's pivots pp[j-1] = 1/((ACPH(j) + shift) - H(j-1) AMPH(j)) and
// multipliers hz[j-1] = H(j).  They depend on the operator only (not on dt or
// the right-hand side), so they are formed once, by the expression the
// sweep itself would evaluate, and the per-substep zero-mode solve is a chain
// of multiply-adds.  zf[0..M) = pp, zf[M..2M) = hz.
__global__ void k_ysolve_zero_factors(Geo g, double* __restrict__ zf) {
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    const int M = g.M;
    const double shift = (-g.ak1[0] / 1.0 - g.ak3[0]);
    const double b = g.acph[1] + shift;
    double hp = 0.0 / b;
    zf[0] = 1.0 / b;
    zf[M] = hp;
    for (int j = 2; j <= M; ++j) {
        const double pp = 1.0 / ((g.acph[j] + shift) - hp * g.amph[j]);
        hp = j < M ? g.apph[j] * pp : 0.0;
        zf[j - 1] = pp;
        zf[M + j - 1] = hp;
    }
}

// Persistent and double-buffered: each block owns every gridDim.x-th group of
// YW_L lines.  The copies of its next group go out (cp.async into the other
// stage) before the current group is solved and written back, so the loads
// overlap the warps' solves and the stores.  One warp per line of a group.
// The stage holds the spectrum's own type (float2 in the mixed-precision
// step); a warp widens its segment to FP64 for the solve.
template <int S, typename C>
__global__ void __launch_bounds__(YW_NT, 1) k_ysolve_warp(Geo g, C* __restrict__ SP) {
    pdl_wait();
    extern __shared__ __align__(16) unsigned char yw_raw[];
    static_assert(YW_NT == 32 * YW_L, "one warp per line of a group");
    const int M = 32 * S, LH = g.LH;
    const int LS = M + 33;
    C* const stage[2] = {reinterpret_cast<C*>(yw_raw), reinterpret_cast<C*>(yw_raw) + YW_L * LS};
    const long long nl = (long long)LH * g.N;
    const long long ngr = (nl + YW_L - 1) / YW_L;
    // the staging loops: thread t moves line t % YW_L, rows t / YW_L + (YW_NT / YW_L) * it
    const int ls = threadIdx.x % YW_L, js = threadIdx.x / YW_L;
    constexpr int RS = YW_NT / YW_L;  // rows per staging step
    auto line_ptr = [&](long long q) {
        const int kz = (int)(q / LH), kx = (int)(q - (long long)kz * LH);
        return SP + kx + (long long)LH * ((long long)M * kz);
    };
    auto issue = [&](long long gr, C* st) {
        if (gr < ngr) {
            const long long q = gr * YW_L + ls;
            if (q < nl) {
                const C* src = line_ptr(q);
                for (int j = js; j < M; j += RS) cp_async_row(st + ls * LS + seg_pos<S>(j), src + (long long)LH * j);
            }
        }
        cp_async_commit();  // an empty group past the end keeps the group count uniform
    };
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    issue(blockIdx.x, stage[0]);
    int cur = 0;
#pragma unroll 1
    for (long long gr = blockIdx.x; gr < ngr; gr += gridDim.x, cur ^= 1) {
        issue(gr + gridDim.x, stage[cur ^ 1]);
        cp_async_wait_group<1>();  // this group's copies (all but the newest group) have landed
        __syncthreads();
        C* const st = stage[cur];
        const long long q = gr * YW_L + warp;
        if (q < nl) {
            const int kz = (int)(q / LH), kx = (int)(q - (long long)kz * LH);
            C* base = st + warp * LS;
            if (q == 0) {
                // zero mode: phi(y_1) = 0 and the reference's forward/backward recurrence
                if (lane == 0) {
                    const double* pp = g.yz;
                    const double* hz = g.yz + M;
                    double2 gp = make_double2(0.0 * pp[0], 0.0 * pp[0]);
                    base[seg_pos<S>(0)] = from_d2<C>(gp);
                    // the forward intermediate g stays FP64: kept in the stage when C is
                    // double2; for a float2 stage the chain runs in a second pass below
                    if constexpr (sizeof(C) == 16) {
#pragma unroll 4
                        for (int j = 2; j <= M; ++j) {
                            const double2 rj = to_d2(base[seg_pos<S>(j - 1)]);
                            const double am = g.amph[j], p = pp[j - 1];
                            gp = make_double2((rj.x - am * gp.x) * p, (rj.y - am * gp.y) * p);
                            base[seg_pos<S>(j - 1)] = from_d2<C>(gp);
                        }
                        double2 xn = gp;
#pragma unroll 4
                        for (int j = M - 1; j >= 1; --j) {
                            const double2 gj = to_d2(base[seg_pos<S>(j - 1)]);
                            const double h = hz[j - 1];
                            xn = make_double2(gj.x - h * xn.x, gj.y - h * xn.y);
                            base[seg_pos<S>(j - 1)] = from_d2<C>(xn);
                        }
                    } else {
                        // FP32 stage: the FP64 forward values go to the FP64 scratch row of
                        // this block (after both stages), then the backward sweep
                        double2* gsc = reinterpret_cast<double2*>(reinterpret_cast<C*>(yw_raw) + 2 * YW_L * LS);
                        gsc[0] = gp;
#pragma unroll 4
                        for (int j = 2; j <= M; ++j) {
                            const double2 rj = to_d2(base[seg_pos<S>(j - 1)]);
                            const double am = g.amph[j], p = pp[j - 1];
                            gp = make_double2((rj.x - am * gp.x) * p, (rj.y - am * gp.y) * p);
                            gsc[j - 1] = gp;
                        }
                        double2 xn = gp;
                        base[seg_pos<S>(M - 1)] = from_d2<C>(xn);
#pragma unroll 4
                        for (int j = M - 1; j >= 1; --j) {
                            const double2 gj = gsc[j - 1];
                            const double h = hz[j - 1];
                            xn = make_double2(gj.x - h * xn.x, gj.y - h * xn.y);
                            base[seg_pos<S>(j - 1)] = from_d2<C>(xn);
                        }
                    }
                }
            } else {
                PoisCoef cf{g.amph, g.acph, g.apph, (-g.ak1[kx] / 1.0 - g.ak3[kz])};
                double2 d[S];
#pragma unroll
                for (int k = 0; k < S; ++k) d[k] = to_d2(base[lane * (S + 1) + k]);
                warp_tdma_c<S>(d, cf, lane);
#pragma unroll
                for (int k = 0; k < S; ++k) base[lane * (S + 1) + k] = from_d2<C>(d[k]);
            }
        }
        __syncthreads();
        {
            const long long qs = gr * YW_L + ls;
            if (qs < nl) {
                C* dst = line_ptr(qs);
                for (int j = js; j < M; j += RS) dst[(long long)LH * j] = st[ls * LS + seg_pos<S>(j)];
            }
        }
        __syncthreads();  // the stage is free for the copies issued in the next iteration but one
    }
    cp_async_wait_group<0>();
}

// ---------------------------------------------------------------------------
// Fifth y-solve variant, in mixed-precision contexts (FP64 ones have k_ysolve_reg): the sequential recurrence's
// factors (the pivots PP and multipliers H of k_ysolve_seq_factors; k_ysolve_scan_factors stores the pivots in
// the spectrum's order, F[kx + LH (t + M kz)] = PP_t, F = B_0 at t = 0, and the kernel forms each
// H_t = APPH(t+1) PP_t, H_0 = C_0 / B_0, H_{M-1} = 0, with the factor kernel's own operations) turn both
// sweeps into first-order linear recurrences,
//   forward   g_t = (r_t - A_t g_{t-1}) PP_t      (g_0 = r_0 / B_0, r_0 = 0 on the zero mode)
//   backward  x_t = g_t - H_t x_{t+1}             (H_{M-1} = 0),
// evaluated as affine scans over 32 segments of S rows per line: a segment composes its rows' maps, the 32
// maps of a line are combined by a shuffle scan (5 steps), and each segment then runs its rows' recurrence
// sequentially from its incoming value, in the reference's operation order.  Thread (il, seg) holds
// segment seg of mode line il in registers, YC_L lines (consecutive kx) per block, so the spectrum and the
// pivots move as row pieces and nothing is staged; the maps change over to one lane per segment
// through shared memory.  The maps are combined in tree order, so the result agrees with the
// sequential recurrence to rounding (1e-12 of the oracle on the Poisson problem).  Bound by latency: at
// 384x256x384 the FP32 spectrum, read and written, and the pivots are 24 B a mode, 0.07 ms of memory a solve;
// 8 lines a block (four row pieces of 64 B per warp) take 0.125 ms, the warp per line with its lines staged
// in shared memory that this replaces 0.162 (128^3: 15.6 against 18.9 us).
constexpr int YC_L = 8;

__global__ void k_ysolve_scan_factors(Geo g, double* __restrict__ F) {
    const int M = g.M, LH = g.LH;
    const long long nl = (long long)LH * g.N;
    for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < nl; q += (long long)gridDim.x * blockDim.x) {
        const int kz = (int)(q / LH), kx = (int)(q - (long long)kz * LH);
        const double shift = (-g.ak1[kx] / 1.0 - g.ak3[kz]);
        const double b = g.acph[1] + shift;
        const double c = q == 0 ? 0.0 : g.apph[1];
        double hp = c / b;
        double* f = F + kx + (long long)LH * M * kz;
        f[0] = b;
        for (int j = 2; j <= M; ++j) {
            const double pp = 1.0 / ((g.acph[j] + shift) - hp * g.amph[j]);
            hp = j < M ? g.apph[j] * pp : 0.0;
            f[(long long)LH * (j - 1)] = pp;
        }
    }
}

template <int S, typename C>
__global__ void __launch_bounds__(32 * YC_L, 2) k_ysolve_scan(Geo g, C* __restrict__ SP, const double* __restrict__ F) {
    pdl_wait();
    constexpr int M = 32 * S, TI = YC_L, LD = 33;
    __shared__ double sA[TI * LD], sBx[TI * LD], sBy[TI * LD];
    __shared__ double sam[M + 32], sap[M + 32];  // AMPH(t+1), APPH(t+1) at t + t / S: the segments' rows on different banks
    const int LH = g.LH;
    const int il = threadIdx.x % TI, seg = threadIdx.x / TI;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const unsigned q = blockIdx.x * TI + il;  // LH N is a multiple of 32
    const unsigned kz = q / (unsigned)LH, kx = q - kz * (unsigned)LH;
    const int r0 = seg * S, s0 = seg * (S + 1);  // the segment's first row and its operator-row slot
    const long long o = kx + (long long)LH * (r0 + (long long)M * kz);
    C* s = SP + o;
    const double* f = F + o;
    double2 d[S];
    double pp[S], hh[S];
#pragma unroll
    for (int k = 0; k < S; ++k) d[k] = to_d2(s[(long long)LH * k]);
#pragma unroll
    for (int k = 0; k < S; ++k) pp[k] = __ldg(f + (long long)LH * k);
    for (int t = threadIdx.x; t < M; t += 32 * TI) {
        sam[t + t / S] = g.amph[t + 1];
        sap[t + t / S] = g.apph[t + 1];
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < S; ++k) {
        const int t = r0 + k;
        if (t == 0) hh[k] = (q == 0 ? 0.0 : sap[0]) / pp[0];
        else hh[k] = t < M - 1 ? sap[s0 + k] * pp[k] : 0.0;
    }
    if (q == 0 && seg == 0) d[0] = make_double2(0.0, 0.0);  // the zero mode's pinned first row
    // forward: the segment's map g_out = A g_in + B over its rows (row 0 ignores g_in)
    double A = 1.0;
    double2 B = make_double2(0.0, 0.0);
#pragma unroll
    for (int k = 0; k < S; ++k) {
        const int t = r0 + k;
        if (t == 0) {
            A = 0.0;
            B = make_double2(d[k].x / pp[k], d[k].y / pp[k]);
        } else {
            const double al = -sam[s0 + k] * pp[k];
            B = make_double2(al * B.x + d[k].x * pp[k], al * B.y + d[k].y * pp[k]);
            A = al * A;
        }
    }
    const int p = il * LD + seg, w = warp * LD + lane;  // this thread's segment; warp: line, lane: segment
    sA[p] = A; sBx[p] = B.x; sBy[p] = B.y;
    __syncthreads();
    {   // inclusive scan over the segments (the first one's map first); each receives its predecessor's value
        A = sA[w];
        B = make_double2(sBx[w], sBy[w]);
#pragma unroll
        for (int n = 1; n < 32; n <<= 1) {
            const double Ap = __shfl_up_sync(0xffffffffu, A, n);
            const double Bx = __shfl_up_sync(0xffffffffu, B.x, n), By = __shfl_up_sync(0xffffffffu, B.y, n);
            if (lane >= n) {
                B = make_double2(A * Bx + B.x, A * By + B.y);
                A = A * Ap;
            }
        }
        double2 gp = make_double2(__shfl_up_sync(0xffffffffu, B.x, 1), __shfl_up_sync(0xffffffffu, B.y, 1));
        if (lane == 0) gp = make_double2(0.0, 0.0);
        sBx[w] = gp.x; sBy[w] = gp.y;
    }
    __syncthreads();
    {   // the segment's rows from their incoming value, in the reference's order
        double2 gp = make_double2(sBx[p], sBy[p]);
#pragma unroll
        for (int k = 0; k < S; ++k) {
            const int t = r0 + k;
            if (t == 0) {
                gp = make_double2(d[k].x / pp[k], d[k].y / pp[k]);
            } else {
                const double a = sam[s0 + k];
                gp = make_double2((d[k].x - a * gp.x) * pp[k], (d[k].y - a * gp.y) * pp[k]);
            }
            d[k] = gp;
        }
    }
    // backward: x_t = g_t - H_t x_{t+1}; the segment's map gives its first row's x from the next segment's
    // first row's (x_in): x = A x_in + B, composed from the segment's last row down
    A = 1.0;
    B = make_double2(0.0, 0.0);
#pragma unroll
    for (int k = S - 1; k >= 0; --k) {
        const double ga = -hh[k];
        B = make_double2(ga * B.x + d[k].x, ga * B.y + d[k].y);
        A = ga * A;
    }
    sA[p] = A; sBx[p] = B.x; sBy[p] = B.y;  // (this thread's own entries, read above)
    __syncthreads();
    {   // inclusive scan over the segments from the last one down
        A = sA[w];
        B = make_double2(sBx[w], sBy[w]);
#pragma unroll
        for (int n = 1; n < 32; n <<= 1) {
            const double Ap = __shfl_down_sync(0xffffffffu, A, n);
            const double Bx = __shfl_down_sync(0xffffffffu, B.x, n), By = __shfl_down_sync(0xffffffffu, B.y, n);
            if (lane + n < 32) {
                B = make_double2(A * Bx + B.x, A * By + B.y);
                A = A * Ap;
            }
        }
        double2 xn = make_double2(__shfl_down_sync(0xffffffffu, B.x, 1), __shfl_down_sync(0xffffffffu, B.y, 1));
        if (lane == 31) xn = make_double2(0.0, 0.0);  // H_{M-1} = 0: the top row is its own g
        sBx[w] = xn.x; sBy[w] = xn.y;
    }
    __syncthreads();
    double2 xn = make_double2(sBx[p], sBy[p]);
#pragma unroll
    for (int k = S - 1; k >= 0; --k) {
        xn = make_double2(d[k].x - hh[k] * xn.x, d[k].y - hh[k] * xn.y);
        s[(long long)LH * k] = from_d2<C>(xn);
    }
}

// ---------------------------------------------------------------------------
// The other y-solve variant: the reference's sequential Thomas recurrence
// (TDMAIJJ_nonCYC :95-121, zero mode pinned as above), one thread per
// (kx, kz) line.  The coefficient part of the recurrence (the pivots
// PP_j = 1/(B_j - H_{j-1} A_j) and multipliers H_j) depends on the operator
// only, not on dt or the right-hand side, so k_ysolve_seq_factors runs it
// once per line and keeps PP and H (2 M doubles per line, row-major over the
// lines: PP_j of line q at F[j*nl + q], H_j at F[(M+j)*nl + q]; row 1 keeps
// B_1 itself, which the first row divides by).  The per-substep solve is
// then two chains of multiply-adds.
//
// There are only LH * N lines (8320 at 128^3), so the solve is one thread per
// line, and what bounds it is the latency of its row loads.  Each thread
// keeps a ring of YS_G * YS_NG rows in shared memory, filled by cp.async in
// groups of YS_G rows (every row access is coalesced across the consecutive
// kx of a warp): while the chain consumes one group, the next YS_NG - 1 are
// in flight.  The forward chain leaves g_j in G (FP64; the spectral array
// itself when it is FP64, the FP64 array as scratch when the spectrum is
// FP32), which the backward chain streams back through the same ring.  No
// thread reads another's ring slots, so there is no block barrier.  The
// autotuner picks between this variant and the warp hybrid per grid.
#define YS_G 8
#define YS_NG 8
#define YS_NT 32
__host__ __device__ constexpr size_t smem_ysolve_seq() { return (size_t)YS_G * YS_NG * YS_NT * (sizeof(double2) + sizeof(double)); }
// With kg, the forward intermediate g of the block's lines stays in shared
// memory ([M][YS_NT] double2 after the ring) instead of making a round trip
// through global memory, and only the multipliers stream through the ring on
// the way back: 64 KB more at M = 128, chosen where two blocks still fit an SM.
// The M values of AMPH follow (the chain reads one per row; with the ring
// and g filling the shared memory the L1 is small, and the factor copies
// evicted them: every read went to L2).
inline size_t smem_ysolve_seq(int M, bool kg) {
    return smem_ysolve_seq() + (kg ? (size_t)M * YS_NT * sizeof(double2) : 0) + (size_t)M * sizeof(double);
}

__global__ void k_ysolve_seq_factors(Geo g, double* __restrict__ F) {
    const int M = g.M, LH = g.LH;
    const long long nl = (long long)LH * g.N;
    for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < nl; q += (long long)gridDim.x * blockDim.x) {
        const int kz = (int)(q / LH), kx = (int)(q - (long long)kz * LH);
        const double shift = (-g.ak1[kx] / 1.0 - g.ak3[kz]);
        const double b = g.acph[1] + shift;
        const double c = q == 0 ? 0.0 : g.apph[1];
        double hp = c / b;
        F[q] = b;
        F[(long long)M * nl + q] = hp;
        for (int j = 2; j <= M; ++j) {
            const double pp = 1.0 / ((g.acph[j] + shift) - hp * g.amph[j]);
            hp = j < M ? g.apph[j] * pp : 0.0;
            F[(long long)(j - 1) * nl + q] = pp;
            F[(long long)(M + j - 1) * nl + q] = hp;
        }
    }
}

template <typename C>
__device__ __forceinline__ void cp_async_row(C* dst, const C* src) {
    if constexpr (sizeof(C) == 16) cp_async16(dst, src);
    else cp_async8(reinterpret_cast<double*>(dst), reinterpret_cast<const double*>(src));
}

template <typename C, bool KG>
__global__ void __launch_bounds__(YS_NT) k_ysolve_seq(Geo g, C* SP, double2* G, const double* __restrict__ F) {
    pdl_wait();
    extern __shared__ __align__(16) unsigned char ys_raw[];
    constexpr int NR = YS_G * YS_NG;
    double2* const ringg = reinterpret_cast<double2*>(ys_raw);  // [NR][YS_NT] rows of G (backward)
    C* const ringc = reinterpret_cast<C*>(ys_raw);              // [NR][YS_NT] rows of the spectrum (forward)
    double* const ringf = reinterpret_cast<double*>(ys_raw + (size_t)NR * YS_NT * sizeof(double2));  // factors
    double2* const gsm = reinterpret_cast<double2*>(ys_raw + smem_ysolve_seq());  // [M][YS_NT] g (KG)
    const int M = g.M, LH = g.LH, th = threadIdx.x;
    double* const sam = reinterpret_cast<double*>(ys_raw + smem_ysolve_seq() +
                                                  (KG ? (size_t)M * YS_NT * sizeof(double2) : 0));  // AMPH(t+1)
    for (int t = th; t < M; t += YS_NT) sam[t] = g.amph[t + 1];
    __syncthreads();
    const long long nl = (long long)LH * g.N;
    const long long q = (long long)blockIdx.x * YS_NT + th;
    if (q >= nl) return;  // no block barrier below
    const int kz = (int)(q / LH), kx = (int)(q - (long long)kz * LH);
    const long long base = kx + (long long)LH * M * kz;
    C* const s = SP + base;
    double2* const gs = G + base;
    const double* const PP = F + q;
    const double* const HH = F + (long long)M * nl + q;
    const long long rs = LH;  // row stride of the spectrum
    // forward: g_1 = r_1 / B_1 (r_1 = 0 on the zero mode), g_t = (r_t - A_t g_{t-1}) PP_t
    const int nb = M / YS_G;
    auto issue_f = [&](int b) {
        if (b < nb) {
#pragma unroll
            for (int u = 0; u < YS_G; ++u) {
                const int row = b * YS_G + u, slot = (b % YS_NG) * YS_G + u;
                cp_async_row(ringc + slot * YS_NT + th, s + rs * row);
                cp_async8(ringf + slot * YS_NT + th, PP + (long long)row * nl);
            }
        }
        cp_async_commit();  // an empty group past the end keeps the group count uniform
    };
#pragma unroll 1
    for (int b = 0; b < YS_NG - 1; ++b) issue_f(b);
    double2 gp = make_double2(0.0, 0.0);
#pragma unroll 1
    for (int b = 0; b < nb; ++b) {
        issue_f(b + YS_NG - 1);
        cp_async_wait_group<YS_NG - 1>();  // group b has landed
#pragma unroll
        for (int u = 0; u < YS_G; ++u) {
            const int t = b * YS_G + u, slot = (b % YS_NG) * YS_G + u;
            const double2 r = to_d2(ringc[slot * YS_NT + th]);
            const double p = ringf[slot * YS_NT + th];
            if (t == 0) {
                const double2 r0 = q == 0 ? make_double2(0.0, 0.0) : r;
                gp = make_double2(r0.x / p, r0.y / p);
            } else {
                const double a = sam[t];
                gp = make_double2((r.x - a * gp.x) * p, (r.y - a * gp.y) * p);
            }
            if (t < M - 1) {
                if constexpr (KG) gsm[t * YS_NT + th] = gp;
                else gs[rs * t] = gp;
            }
        }
    }
    cp_async_wait_group<0>();
    if constexpr (!KG) __threadfence();  // the G rows written above, before the cp.async reads below
    // backward: x_M = g_M, x_t = g_t - H_t x_{t+1}, t = M-1 .. 1 (rows t-1 = M-2 .. 0)
    double2 xn = gp;
    s[rs * (M - 1)] = from_d2<C>(xn);
    const int nbb = (M - 1 + YS_G - 1) / YS_G;
    auto issue_b = [&](int b) {
        if (b < nbb) {
#pragma unroll
            for (int u = 0; u < YS_G; ++u) {
                const int t = M - 2 - b * YS_G - u, slot = (b % YS_NG) * YS_G + u;
                if (t >= 0) {
                    if constexpr (!KG) cp_async16(ringg + slot * YS_NT + th, gs + rs * t);
                    cp_async8(ringf + slot * YS_NT + th, HH + (long long)t * nl);
                }
            }
        }
        cp_async_commit();
    };
#pragma unroll 1
    for (int b = 0; b < YS_NG - 1; ++b) issue_b(b);
#pragma unroll 1
    for (int b = 0; b < nbb; ++b) {
        issue_b(b + YS_NG - 1);
        cp_async_wait_group<YS_NG - 1>();
#pragma unroll
        for (int u = 0; u < YS_G; ++u) {
            const int t = M - 2 - b * YS_G - u, slot = (b % YS_NG) * YS_G + u;
            if (t >= 0) {
                const double2 gt = KG ? gsm[t * YS_NT + th] : ringg[slot * YS_NT + th];
                const double h = ringf[slot * YS_NT + th];
                xn = make_double2(gt.x - h * xn.x, gt.y - h * xn.y);
                s[rs * t] = from_d2<C>(xn);
            }
        }
    }
    cp_async_wait_group<0>();
}

// ---------------------------------------------------------------------------
// Third y-solve variant: two-way elimination, two threads per mode line.
// The sequential recurrence is bound by one thread's chain of dependent
// instructions over all M rows.  Here the upper thread of a lane pair
// eliminates rows 0 .. m-1 downwards (Thomas: x_t = g_t - h_t x_{t+1}), the
// lower one rows M-1 .. m+1 upwards (x_t = g'_t - h'_t x_{t-1}), m = M/2;
// the middle row closes the system,
//   x_m = (r_m - A_m g_{m-1} - C_m g'_{m+1}) / (B_m - A_m h_{m-1} - C_m h'_{m+1}),
// and each thread substitutes back over its own half.  The result is the
// same tridiagonal solution with another rounding order: on the 128-row
// channel it agrees with the reference's one-way recurrence to 1e-14 on the
// kx, kz != 0 modes and to 1.2e-13 (relative) on the pinned zero mode, whose
// operator is the weakly dominant Neumann one.  The pivots are precomputed
// per line (k_ysolve_2w_factors): F[t*nl + q] holds 1/pivot of row t (upper
// rows, the middle row, lower rows), F[(M+t)*nl + q] the multiplier h_t or
// h'_t.  Rows move through the per-thread cp.async ring of k_ysolve_seq.
__global__ void k_ysolve_2w_factors(Geo g, double* __restrict__ F) {
    const int M = g.M, LH = g.LH, m = M / 2;
    const long long nl = (long long)LH * g.N;
    for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < nl; q += (long long)gridDim.x * blockDim.x) {
        const int kz = (int)(q / LH), kx = (int)(q - (long long)kz * LH);
        const double shift = (-g.ak1[kx] / 1.0 - g.ak3[kz]);
        // upper half, rows t = 0 .. m-1 (j = t + 1); the zero mode's row 1 is decoupled (phi(y_1) = 0)
        double p = 1.0 / (g.acph[1] + shift);
        double h = (q == 0 ? 0.0 : g.apph[1]) * p;
        F[q] = p;
        F[(long long)M * nl + q] = h;
        for (int t = 1; t < m; ++t) {
            const int j = t + 1;
            p = 1.0 / ((g.acph[j] + shift) - h * g.amph[j]);
            h = g.apph[j] * p;
            F[(long long)t * nl + q] = p;
            F[(long long)(M + t) * nl + q] = h;
        }
        // lower half, rows t = M-1 .. m+1
        double pb = 1.0 / (g.acph[M] + shift);
        double hb = g.amph[M] * pb;
        F[(long long)(M - 1) * nl + q] = pb;
        F[(long long)(2 * M - 1) * nl + q] = hb;
        for (int t = M - 2; t > m; --t) {
            const int j = t + 1;
            pb = 1.0 / ((g.acph[j] + shift) - hb * g.apph[j]);
            hb = g.amph[j] * pb;
            F[(long long)t * nl + q] = pb;
            F[(long long)(M + t) * nl + q] = hb;
        }
        // middle row m
        const int jm = m + 1;
        F[(long long)m * nl + q] = 1.0 / ((g.acph[jm] + shift) - g.amph[jm] * h - g.apph[jm] * hb);
        F[(long long)(M + m) * nl + q] = 0.0;
    }
}

template <typename C>
__global__ void __launch_bounds__(YS_NT) k_ysolve_2w(Geo g, C* SP, double2* G, const double* __restrict__ F) {
    pdl_wait();
    extern __shared__ __align__(16) unsigned char ys_raw[];
    constexpr int NR = YS_G * YS_NG;
    double2* const ringg = reinterpret_cast<double2*>(ys_raw);
    C* const ringc = reinterpret_cast<C*>(ys_raw);
    double* const ringf = reinterpret_cast<double*>(ys_raw + (size_t)NR * YS_NT * sizeof(double2));
    const int M = g.M, LH = g.LH, m = M / 2, th = threadIdx.x;
    const long long nl = (long long)LH * g.N;
    const long long q = ((long long)blockIdx.x * YS_NT + th) >> 1;
    if (q >= nl) return;  // both lanes of a pair leave together; no block barrier below
    const bool lower = (th & 1) != 0;
    const unsigned pair = 3u << ((th & 31) & ~1);
    const int kz = (int)(q / LH), kx = (int)(q - (long long)kz * LH);
    const long long base = kx + (long long)LH * M * kz;
    C* const s = SP + base;
    double2* const gs = G + base;
    const double* const PP = F + q;
    const double* const HH = F + (long long)M * nl + q;
    const long long rs = LH;
    // forward: upper rows 0, 1, .., m-1; lower rows M-1, M-2, .., m+1
    const int nf = lower ? m - 1 : m;
    auto frow = [&](int i) { return lower ? M - 1 - i : i; };
    const int nbf = (nf + YS_G - 1) / YS_G;
    auto issue_f = [&](int b) {
        if (b < nbf) {
#pragma unroll
            for (int u = 0; u < YS_G; ++u) {
                const int i = b * YS_G + u, slot = (b % YS_NG) * YS_G + u;
                if (i < nf) {
                    const int row = frow(i);
                    cp_async_row(ringc + slot * YS_NT + th, s + rs * row);
                    cp_async8(ringf + slot * YS_NT + th, PP + (long long)row * nl);
                }
            }
        }
        cp_async_commit();
    };
#pragma unroll 1
    for (int b = 0; b < YS_NG - 1; ++b) issue_f(b);
    double2 gp = make_double2(0.0, 0.0);
#pragma unroll 1
    for (int b = 0; b < nbf; ++b) {
        issue_f(b + YS_NG - 1);
        cp_async_wait_group<YS_NG - 1>();
#pragma unroll
        for (int u = 0; u < YS_G; ++u) {
            const int i = b * YS_G + u, slot = (b % YS_NG) * YS_G + u;
            if (i < nf) {
                const int t = frow(i);
                double2 r = to_d2(ringc[slot * YS_NT + th]);
                const double p = ringf[slot * YS_NT + th];
                if (i == 0) {
                    if (!lower && q == 0) r = make_double2(0.0, 0.0);
                    gp = make_double2(r.x * p, r.y * p);
                } else {
                    const double a = lower ? g.apph[t + 1] : g.amph[t + 1];
                    gp = make_double2((r.x - a * gp.x) * p, (r.y - a * gp.y) * p);
                }
                gs[rs * t] = gp;
            }
        }
    }
    cp_async_wait_group<0>();
    __threadfence();  // the G rows written above, before the cp.async reads below
    // middle row: the upper lane closes it with the lower lane's g'_{m+1}
    const double2 go = make_double2(__shfl_xor_sync(pair, gp.x, 1), __shfl_xor_sync(pair, gp.y, 1));
    double2 xm = make_double2(0.0, 0.0);
    if (!lower) {
        const double2 rm = to_d2(s[rs * m]);
        const double am = g.amph[m + 1], cm = g.apph[m + 1], pm = PP[(long long)m * nl];
        xm = make_double2((rm.x - am * gp.x - cm * go.x) * pm, (rm.y - am * gp.y - cm * go.y) * pm);
        s[rs * m] = from_d2<C>(xm);
    }
    double2 xn = make_double2(__shfl_sync(pair, xm.x, (th & 31) & ~1), __shfl_sync(pair, xm.y, (th & 31) & ~1));
    // backward: upper rows m-1 .. 0, lower rows m+1 .. M-1
    auto brow = [&](int i) { return lower ? m + 1 + i : m - 1 - i; };
    auto issue_b = [&](int b) {
        if (b < nbf) {
#pragma unroll
            for (int u = 0; u < YS_G; ++u) {
                const int i = b * YS_G + u, slot = (b % YS_NG) * YS_G + u;
                if (i < nf) {
                    const int t = brow(i);
                    cp_async16(ringg + slot * YS_NT + th, gs + rs * t);
                    cp_async8(ringf + slot * YS_NT + th, HH + (long long)t * nl);
                }
            }
        }
        cp_async_commit();
    };
#pragma unroll 1
    for (int b = 0; b < YS_NG - 1; ++b) issue_b(b);
#pragma unroll 1
    for (int b = 0; b < nbf; ++b) {
        issue_b(b + YS_NG - 1);
        cp_async_wait_group<YS_NG - 1>();
#pragma unroll
        for (int u = 0; u < YS_G; ++u) {
            const int i = b * YS_G + u, slot = (b % YS_NG) * YS_G + u;
            if (i < nf) {
                const double2 gt = ringg[slot * YS_NT + th];
                const double h = ringf[slot * YS_NT + th];
                xn = make_double2(gt.x - h * xn.x, gt.y - h * xn.y);
                s[rs * brow(i)] = from_d2<C>(xn);
            }
        }
    }
    cp_async_wait_group<0>();
}

// ---------------------------------------------------------------------------
// The FP64 form of the scan variant: the same two recurrences over the sequential factors, held in
// registers by the layout of the FP64 y sweep (k_ysweep_reg, momentum.cuh): thread (il, seg) owns SR
// consecutive y rows of mode line il, YR_TI lines (consecutive kx) per block, so the spectrum and the pivots
// are read and written as row pieces, with nothing staged or transposed; the segments' carries and
// multipliers change over through shared memory and are summed by Horner's rule.  Pivots in the
// spectrum's own order, F[kx + LH (t + M kz)] = PP_t; the multipliers A_t PP_t and H_t = C_t PP_t are formed
// from them.  Bound by the bytes of the spectrum and the pivots: scan kernel / this, us per launch, 39 / 22 at
// 192 x 128 x 192, 43 / 27 at 256 x 192 x 128, 264 / 133 at 384 x 256 x 384 (sequential form 213; floor of its 40
// bytes per mode row 117), 23 / 14 at 128^3.
constexpr int YR_TI = 8;
__global__ void k_ysolve_reg_factors(Geo g, double* __restrict__ F) {
    const int M = g.M, LH = g.LH;
    const long long nl = (long long)LH * g.N;
    for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < nl; q += (long long)gridDim.x * blockDim.x) {
        const int kz = (int)(q / LH), kx = (int)(q - (long long)kz * LH);
        const double shift = (-g.ak1[kx] / 1.0 - g.ak3[kz]);
        double* f = F + kx + (long long)LH * M * kz;
        double hp = 0.0;
        for (int j = 1; j <= M; ++j) {
            const double pp = 1.0 / ((g.acph[j] + shift) - (j > 1 ? hp * g.amph[j] : 0.0));
            hp = (j == M || (j == 1 && q == 0)) ? 0.0 : g.apph[j] * pp;
            f[(long long)LH * (j - 1)] = pp;
        }
    }
}

template <int NSEG, int SR>
__global__ void __launch_bounds__(YR_TI * NSEG, (SR > 12 ? 512 : SR > 8 ? 640 : 768) / (YR_TI * NSEG)) k_ysolve_reg(Geo g, double2* __restrict__ SP,
                                                                                                   const double* __restrict__ F) {
    pdl_wait();
    constexpr int M = NSEG * SR, TI = YR_TI;
    __shared__ double2 sc[NSEG][TI];            // the segments' last (first) values
    __shared__ double sm[NSEG][TI], sam[M], sap[M];  // and their products of multipliers; AMPH, APPH
    const int LH = g.LH;
    const int il = threadIdx.x % TI, seg = threadIdx.x / TI;
    const unsigned q = blockIdx.x * TI + il;    // mode line; LH N is a multiple of 32
    const unsigned kz = q / (unsigned)LH, kx = q - kz * (unsigned)LH;
    const long long o = kx + (long long)LH * (seg * SR + (long long)M * kz);
    double2* s = SP + o;
    const double* f = F + o;
    double2 d[SR];
    double pp[SR];
#pragma unroll
    for (int r = 0; r < SR; ++r) d[r] = s[(long long)LH * r];
#pragma unroll
    for (int r = 0; r < SR; ++r) pp[r] = f[(long long)LH * r];
    for (int t = threadIdx.x; t < M; t += TI * NSEG) {
        sam[t] = t == 0 ? 0.0 : -g.amph[t + 1];
        sap[t] = t == M - 1 ? 0.0 : -g.apph[t + 1];
    }
    __syncthreads();
    const double* am = sam + seg * SR;
    const double* ap = sap + seg * SR;
    // the zero mode (kx = kz = 0): phi_hat(y_1) = 0, and row 1 does not couple
    const bool zero = q == 0 && seg == 0;
    if (zero) d[0] = make_double2(0.0, 0.0);
    d[0] = c_scale(d[0], pp[0]);
    double w = am[0] * pp[0];
#pragma unroll
    for (int r = 1; r < SR; ++r) {
        const double a = am[r] * pp[r];
        d[r] = make_double2(fma(a, d[r - 1].x, d[r].x * pp[r]), fma(a, d[r - 1].y, d[r].y * pp[r]));
        w *= a;
    }
    sc[seg][il] = d[SR - 1];
    sm[seg][il] = w;
    __syncthreads();
    double2 c = make_double2(0.0, 0.0);
#pragma unroll 4
    for (int m = 0; m < NSEG - 1; ++m)
        if (m < seg) {
            const double2 v = sc[m][il];
            const double x = sm[m][il];
            c = make_double2(fma(c.x, x, v.x), fma(c.y, x, v.y));
        }
#pragma unroll
    for (int r = 0; r < SR; ++r) {
        c = c_scale(c, am[r] * pp[r]);
        d[r] = make_double2(d[r].x + c.x, d[r].y + c.y);
    }
    w = ap[SR - 1] * pp[SR - 1];
#pragma unroll
    for (int r = SR - 2; r >= 0; --r) {
        const double h = (zero && r == 0) ? 0.0 : ap[r] * pp[r];
        d[r] = make_double2(fma(h, d[r + 1].x, d[r].x), fma(h, d[r + 1].y, d[r].y));
        w *= h;
    }
    __syncthreads();  // the forward carries have been read
    sc[seg][il] = d[0];
    sm[seg][il] = w;
    __syncthreads();
    c = make_double2(0.0, 0.0);
#pragma unroll 4
    for (int m = NSEG - 1; m >= 1; --m)
        if (m > seg) {
            const double2 v = sc[m][il];
            const double x = sm[m][il];
            c = make_double2(fma(c.x, x, v.x), fma(c.y, x, v.y));
        }
#pragma unroll
    for (int r = SR - 1; r >= 0; --r) {
        c = c_scale(c, (zero && r == 0) ? 0.0 : ap[r] * pp[r]);
        s[(long long)LH * r] = make_double2(d[r].x + c.x, d[r].y + c.y);
    }
}

// ---------------------------------------------------------------------------
// Inverse x transform of PX_TJ y rows, two rows a, b packed as one complex line Z = A + iB.  Thread
// (pair, j1) forms its first-pass values Z_k, k = j1 + N1 j2, from the stored half spectra in registers
// (Z_{L-k} = conj A_k + i conj B_k; imaginary parts of the k = 0 and k = L/2 coefficients are dropped, as
// FFT99 does for ISIGN = +1): a coefficient is read for k and for L - k, the second time from L1.  Per
// step 0.108 -> 0.068 ms at 256 x 192 x 128, 0.60 -> 0.55 at 384 x 256 x 384 (FP32: 0.35 -> 0.26).  The
// forward transform keeps its staged form: it reads five field rows per line, more than the registers
// beside a first-pass transform can hold in flight (0.173 -> 0.300 ms at 192 x 128 x 192).
template <int N1, int N2, typename C>
__global__ void __launch_bounds__(px_nt<N1>(), (px_rminb<C, N1>())) k_fftx_inv(Geo g, const C* __restrict__ SP,
                                                                         typename CReal<C>::T* __restrict__ DPH) {
    pdl_wait();
    using T = typename CReal<C>::T;
    extern __shared__ __align__(16) unsigned char smp_raw[];
    C* smc = reinterpret_cast<C*>(smp_raw);
    constexpr int L = N1 * N2, LH = L / 2 + 1, LD = L + N2 + 1;
    const int M = g.M, j0 = 1 + blockIdx.x * PX_TJ, k = blockIdx.y;
    {
        const int j1 = threadIdx.x % N1, pair = threadIdx.x / N1;
        const C* ra = SP + (long long)LH * ((j0 + 2 * pair - 1) + (long long)M * k);
        const C* rb = ra + LH;
        C v[N2];
#pragma unroll
        for (int j2 = 0; j2 < N2; ++j2) {
            const int q = j1 + N1 * j2;
            const bool up = q > L / 2;
            const int ks = up ? L - q : q;
            C a = ra[ks], b = rb[ks];
            if (ks == 0 || 2 * ks == L) {
                a.y = (T)0;
                b.y = (T)0;
            }
            v[j2] = up ? mkc(a.x - (-b.y), (-a.y) + b.x) : mkc(a.x - b.y, a.y + b.x);
        }
        fft_first<N1, N2, +1>(v, smc + pair * LD, j1, twx_of<C>(g));
    }
    __syncthreads();
    for (int t = threadIdx.x; t < PX_TJ / 2 * N2; t += px_nt<N1>()) {
        const int pair = t / N2, k2 = t - pair * N2;
        C v[N1];
        fft_second<N1, +1>(v, smc + pair * LD, k2);
        T* da = DPH + pidx(g, k2, j0 + 2 * pair, k);
#pragma unroll
        for (int k1 = 0; k1 < N1; ++k1) {
            da[N2 * k1] = v[k1].x;
            da[N2 * k1 + L] = v[k1].y;  // the next row (x-periodic layout: row stride L)
        }
    }
}

// ---------------------------------------------------------------------------
// VELOUPDT_tg + PRCALC_tg + BC_WALL_PR_tg (Q walls are never written).
// Each thread updates W = 16 / sizeof(R) consecutive points of an x line with
// 16-byte loads and stores (L is a multiple of 4); the per-point arithmetic
// is FP64, in the same order for every point.
// PRCALC_tg subtracts BE times RHSLLPHI.  LAP (FP64, where lap_is_rhs of chapsim_gpu.cu finds that the caller's
// operator is the discrete Laplacian, as the reference's is): the Laplacian of the Poisson solution stands for it
// (AMPH, ACPH, APPH in y, second differences in x and z), from the DPH
// neighbours that are in cache, so the divergence kernel need not write the array nor this one read it (two
// words per point and substep).  The difference is the rounding of the Laplacian times BE = alpha dt nu / 2: relative
// to DPH 2^-53 BE (4/dx^2 + 4/dz^2 + 4/dy^2), the diffusion number's size; over three fields PR differs from the oracle's
// by 2.3e-16 rms where the array gives 2.0e-16 at REN = 2 (64 x 96 x 64, projection; 2.1e-16 with the sweeps and transforms
// in shared memory), by the same 8.7e-16 at REN = 2800.  Divergence 1.39 -> 1.13 and
// correction 1.45 -> 1.29 ms per step at 384 x 256 x 384, step 0.585 -> 0.567 ms at 128^3.  FP32 keeps the array.
template <typename R, bool LAP>
__global__ void __launch_bounds__(CR_NT) k_correct(Geo g, R* __restrict__ Q, R* __restrict__ PR,
                                                   const R* __restrict__ DPH, const R* __restrict__ RHSLL,
                                                   const DevState* __restrict__ st, int ns) {
    pdl_wait();
    constexpr int W = V16<R>::W;
    const int L = g.L, M = g.M, N = g.N;
    const unsigned LV = (unsigned)(L / W);
    const long long tot = (long long)LV * M * N;
    const long long t = (long long)blockIdx.x * CR_NT + threadIdx.x;
    if (t >= tot) return;
    const unsigned u = (unsigned)t, r = u / LV, kk = r / (unsigned)M;
    const int i0 = (int)(u - r * LV) * W, j = 1 + (int)(r - kk * (unsigned)M), k = (int)kk;
    const double dt = st->dt, ta = g.talp[ns];
    const long long c = pidx(g, i0, j, k);
    // all loads first: Q is read and written through one pointer
    R ph[W], phk[W], phj[W], uu[W], vv[W], ww[W], pr[W], ll[W], phkp[W], phjp[W];
    ld16(DPH + c, ph);
    ld16(DPH + pidx(g, i0, j, wrapm(k, N)), phk);
    if (j >= 2) ld16(DPH + c - L, phj);
    if constexpr (LAP) {
        ld16(DPH + pidx(g, i0, j, wrapp(k, N)), phkp);
        if (j < M) ld16(DPH + c + L, phjp);
    }
    ld16(Q + c, uu);
    ld16(Q + c + g.FS, vv);
    ld16(Q + c + 2 * g.FS, ww);
    ld16(PR + c, pr);
    if constexpr (!LAP) ld16(RHSLL + iidx(g, i0, j, k), ll);
    else {
        const double phip0 = DPH[pidx(g, i0 + W == L ? 0 : i0 + W, j, k)], pl = DPH[pidx(g, wrapm(i0, L), j, k)];
        const double am = j >= 2 ? g.amph[j] : 0.0, ap = j < M ? g.apph[j] : 0.0, ac = g.acph[j];
#pragma unroll
        for (int e = 0; e < W; ++e) {
            const double p = ph[e], px = e == W - 1 ? phip0 : ph[e + 1 < W ? e + 1 : e], pm = e == 0 ? pl : ph[e > 0 ? e - 1 : e];
            const double y = (j >= 2 ? am * phj[e] : 0.0) + ac * p + (j < M ? ap * phjp[e] : 0.0);
            ll[e] = ((px - p) - (p - pm)) * g.dxqi + ((phkp[e] - p) - (p - phk[e])) * g.dzqi + y;
        }
    }
    const double phim0 = DPH[pidx(g, wrapm(i0, L), j, k)];
    const double cx = dt * ta * g.dxi, cz = dt * ta * g.dzi, cy = dt * ta * g.dyci[j] / 1.0;
    const double be = 0.5 * ta * dt * g.cvisc * 1.0 / 1.0;
    R uo[W], vo[W], wo[W], pn[W];
#pragma unroll
    for (int e = 0; e < W; ++e) {
        const double p = ph[e], pim = e == 0 ? phim0 : (double)ph[e - 1];
        uo[e] = (R)(uu[e] - (p - pim) * cx);
        wo[e] = (R)(ww[e] - (p - (double)phk[e]) * cz);
        vo[e] = j >= 2 ? (R)(vv[e] - (p - (double)phj[e]) * cy) : vv[e];
        pn[e] = (R)(pr[e] + p - be * ll[e]);
    }
    st16(Q + c, uo);
    st16(Q + c + 2 * g.FS, wo);
    if (j >= 2) st16(Q + c + g.FS, vo);
    st16(PR + c, pn);
    if (j == 1) st16(PR + pidx(g, i0, 0, k), pn);
    if (j == M) st16(PR + pidx(g, i0, M + 1, k), pn);
}
