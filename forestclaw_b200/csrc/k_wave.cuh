// k_wave.cuh -- fused per-level patch update of the flux-form systems (shallow water, Euler):
// clawpack 4.6 step2 + step2_wrap with the solvers of wave_solvers.cuh, FP64 (TW = double) and
// FP32-wave (TW = float).
//
// One CTA per patch, one thread per interface of a sweep.  Phases, a barrier after each:
//   stage   q and aux by bulk asynchronous copies (cp.async.bulk, completion on an mbarrier)
//   cells   status, save_current_step, time-sync flux store, per-cell solver values (pre)
//   x1      Riemann solves of the x interfaces; waves to shared memory
//   x2      limiter, second-order correction, Godunov split -> x fluxes; transverse split
//   y1      x-transverse terms of the thread's y face (held in registers); y Riemann solves
//   y2      as x2 -> y fluxes with the held terms; transverse split
//   x3      y-transverse terms into the x fluxes
//   update  time-sync wave accumulation, q, CFL maximum
// The flux arrays fm/fp/gm/gp of clawpack46_step2.f are accumulated in the reference's order
// (x-sweeps row by row, then y-sweeps column by column) by gathering, so no atomics are needed
// and repeated runs are bitwise identical.
//
// The FP32-wave form keeps q, the flux arrays, the q update, the registers and the CFL
// reduction in FP64 and takes the Godunov split as an FP64 remainder, amdq = [f(q_i) -
// f(q_{i-1})] - apdq, so fluxes telescope to FP64 round-off and mass stays conserved to FP64
// accuracy although the waves are FP32.  It therefore stores one flux plane per direction,
// GX = fp and GY = gp: inside the Godunov range fm = (f(cell right) - f(cell left)) + fp,
// elsewhere fm = fp.  At a reflecting wall the mass flux is exactly zero, but FP32 waves
// reproduce that cancellation only to FP32 rounding (about 1e-8 of the mass per step), so the
// FP32-wave form takes the exact value, zero, for the mass component there.
//
// What bounds it: instruction issue (54 to 72 % of the slots in the shallow-water forms, 36 to 53 %
// in Euler's) and, at 11 or 12 warps per CTA and one to three CTAs per SM, latency; HBM is below 11 %.  So
// what counts is instructions per interface and CTAs per SM.  Against a kernel that solved
// each interface from the bare states and kept four flux planes per cell:
//   * square roots, sound speeds and velocities are formed once per cell for both sweeps
//     (a cell is an operand of four interfaces) and share their shared memory with the y
//     fluxes, which are first written after their last use;
//   * fluxes are stored per interface, not per cell, and nothing is zeroed;
//   * an interface keeps only what its second phase cannot form again, so two FP64 CTAs of
//     a 16x16 shallow-water patch fit an SM (80 registers; spill stores of the variant used by
//     default: Roe 8 bytes, f-wave 40);
//   * the limiter reads the upwind neighbour's wave only;
//   * LIM > 0 fixes the method at compile time (second order, second-order transverse terms,
//     that limiter on every wave); LIM = 0 reads it from the launch's parameters.
// Updates of one coarse step, one B200, against the kernels it replaced (us, ncu, warm):
//   radial dam levels 3-7, 1960 patches 16x16    FP32-wave  832 ->  620   FP64 1957 -> 1005
//   radial dam uniform, 4096 patches 16x16       FP32-wave  108 ->   87
//   radial dam uniform, 1536 patches 8x8, LIM 0                           FP64   72 ->   27
//   tsunami batch, 8180 patches 8x8              FP32-wave 1230 ->  592
//   tsunami uniform, 1024 patches 16x16                                   FP64  156 ->   71
//   shock-bubble levels 4-7, 1784 patches 16x16  FP32-wave 1139 ->  473
//   shock-bubble uniform, 512 patches 16x16                               FP64  172 ->   91
//
// Index conventions: padded 0-based cell (ic, jc), ic = i + mbc - 1 for the Fortran index i.
// Interface ic sits between cells ic-1 and ic.  x interface k: row jc = 1 + k / (NX-1),
// ic = 1 + k % (NX-1); y interface k: jc = 1 + k / (NX-2), column ic = 1 + k % (NX-2), i
// fastest, so the threads of a warp touch consecutive words.
#pragma once
#include <cuda_runtime.h>
#include <type_traits>
#include "fcb_common.h"
#include "fcb_launch.cuh"
#include "k_bulk.cuh"
#include "k_mlp.cuh"
#include "kernels.h"
#include "wave_solvers.cuh"

namespace fcb {

template <class RP, int MX, typename TW>
struct WaveGeom {
    static constexpr bool F32 = std::is_same<TW, float>::value;
    static constexpr int MY = MX, MBC = 2, NX = MX + 2 * MBC, NY = MY + 2 * MBC, NXY = NX * NY;
    static constexpr int NI = (NY - 2) * (NX - 1);               // interfaces of a sweep (square patches)
    static constexpr int MEQN = RP::MEQN, MAUX = RP::MAUX;
    static constexpr unsigned QBYTES = MEQN * NXY * 8u, ABYTES = MAUX * NXY * 8u;
    static_assert(QBYTES % 16 == 0 && ABYTES % 16 == 0, "bulk copies move multiples of 16 bytes");
    static constexpr int NF = F32 ? 1 : 2;                       // flux planes per field and direction
    static constexpr int NP = RP::NPRE + (F32 ? MEQN : 0);       // per-cell planes (FP32 form: q in TW first)
    static constexpr size_t up16(size_t n) { return (n + 15) / 16 * 16; }
    static constexpr size_t FB = up16((size_t)NF * MEQN * NI * 8), PB = up16((size_t)NP * NXY * sizeof(TW));
    static constexpr size_t OFF_A = QBYTES;
    static constexpr size_t OFF_FL = OFF_A + ABYTES;             // FP32 form: cell fluxes [NFL][NXY] double
    static constexpr size_t OFF_FX = OFF_FL + (F32 ? (size_t)RP::NFL * NXY * 8 : 0);   // [NF][MEQN][NI] double
    static constexpr size_t OFF_FY = OFF_FX + FB;                // per-cell planes, then [NF][MEQN][NI] double
    static constexpr size_t OFF_RED = OFF_FY + (FB > PB ? FB : PB);
    static constexpr size_t OFF_HIST = OFF_RED + 32 * 8;
    static constexpr size_t OFF_K = OFF_HIST + (RP::EXACT ? 32 * 4 : 0);
    static constexpr size_t OFF_BAR = OFF_K + up16(RP::NCONST * sizeof(TW));
    static constexpr size_t OFF_W = OFF_BAR + 16;                // [NW][NI] TW
    static constexpr size_t OFF_T = OFF_W + up16((size_t)RP::NW * NI * sizeof(TW));    // [4][MEQN][NI] TW
    static constexpr size_t BYTES = OFF_T + (size_t)4 * MEQN * NI * sizeof(TW);
    // conservation registers (fclaw2d_clawpatch_conservation.h:56-77), per patch
    static constexpr int R_FP0 = 0, R_FP1 = MY * MEQN, R_FM0 = 2 * MY * MEQN, R_FM1 = 3 * MY * MEQN;
    static constexpr int R_GP0 = 4 * MY * MEQN, R_GP1 = R_GP0 + MX * MEQN, R_GM0 = R_GP0 + 2 * MX * MEQN,
                         R_GM1 = R_GP0 + 3 * MX * MEQN;
    static constexpr int R_EF0 = R_GP0 + 4 * MX * MEQN, R_EF1 = R_EF0 + 2 * MY * MEQN,
                         R_EF2 = R_EF1 + 2 * MY * MEQN, R_EF3 = R_EF2 + 2 * MX * MEQN,
                         NREG = R_EF3 + 2 * MX * MEQN;
    // interface ranges (padded) of flux2 / flux2fw: Godunov and cq into the transverse split;
    // second-order correction and transverse terms (elsewhere an interface has none)
    static constexpr int GOD_LO = RP::FWAVE ? MBC : 1, GOD_HI = RP::FWAVE ? MX + MBC : NX - 2;
    static constexpr int COR_LO = RP::FWAVE ? MBC : 1, COR_HI = RP::FWAVE ? MX + MBC : NX - 1;
    __device__ static constexpr bool god(int pos) { return pos >= GOD_LO && pos <= GOD_HI; }
    __device__ static constexpr bool cor(int pos) { return pos >= COR_LO && pos <= COR_HI; }
    // interface number of face (ic, jc)
    __device__ static constexpr int kx(int ic, int jc) { return (jc - 1) * (NX - 1) + ic - 1; }
    __device__ static constexpr int ky(int ic, int jc) { return (jc - 1) * (NX - 2) + ic - 1; }
};

// Method of a launch: compile-time for LIM > 0.
template <int LIM>
struct WaveMethod {
    int order1, order2, mcapa;
    const int* lim;
    __device__ explicit WaveMethod(const StepParams* sp)
        : order1(LIM ? 2 : sp->order1), order2(LIM ? 2 : sp->order2), mcapa(LIM ? 0 : sp->mcapa), lim(sp->mthlim)
    {
    }
    __device__ __forceinline__ int limiter(int mw) const { return LIM ? LIM : lim[mw]; }
};

// Shared memory and scalars of one patch.
template <class RP, int MX, typename TW, int LIM>
struct WavePatch {
    using G = WaveGeom<RP, MX, TW>;
    static constexpr bool F32 = G::F32;
    static constexpr int NX = G::NX, NY = G::NY, NXY = G::NXY, NI = G::NI, MEQN = G::MEQN, MBC = G::MBC, MY = G::MY;
    static constexpr int MWAVES = RP::MWAVES, MAUX = G::MAUX, MA = MAUX > 0 ? MAUX : 1;
    using St = typename RP::template State<TW>;

    unsigned char* sm;
    WaveMethod<LIM> M;
    WavePar<TW> P;
    double grav, dtdx, dtdy;
    int wallf;

    __device__ __forceinline__ double* Q() const { return reinterpret_cast<double*>(sm); }
    __device__ __forceinline__ double* A() const { return reinterpret_cast<double*>(sm + G::OFF_A); }
    __device__ __forceinline__ double* FL() const { return reinterpret_cast<double*>(sm + G::OFF_FL); }
    __device__ __forceinline__ double* FX() const { return reinterpret_cast<double*>(sm + G::OFF_FX); }
    __device__ __forceinline__ double* FY() const { return reinterpret_cast<double*>(sm + G::OFF_FY); }
    __device__ __forceinline__ TW* C() const { return reinterpret_cast<TW*>(sm + G::OFF_FY); }
    __device__ __forceinline__ TW* W() const { return reinterpret_cast<TW*>(sm + G::OFF_W); }
    __device__ __forceinline__ TW* T() const { return reinterpret_cast<TW*>(sm + G::OFF_T); }
    // per-cell value j of one cell
    struct Cell {
        const TW* p;
        __device__ __forceinline__ TW operator()(int j) const { return p[j * NXY]; }
    };
    // state of cell c in TW, while the per-cell planes live
    __device__ __forceinline__ TW qc(int m, int c) const
    {
        if constexpr (F32) { return C()[m * NXY + c]; }
        else { return Q()[m * NXY + c]; }
    }
    // FP64 flux component m of cell c in direction IXY (FP32 form)
    template <int IXY> __device__ __forceinline__ double flux(int m, int c) const
    {
        const int p = RP::template flux_plane<IXY>(m);
        return p < MEQN ? Q()[p * NXY + c] : FL()[(p - MEQN) * NXY + c];
    }
    // dt/dx of a cell: with a capacity (aux field mcapa) dt / (dx kappa)
    __device__ __forceinline__ TW ratio(int ixy, int c) const
    {
        const double r = ixy == 1 ? dtdx : dtdy;
        if constexpr (MAUX > 0 && LIM == 0) { if (M.mcapa > 0) return (TW)(r / A()[(M.mcapa - 1) * NXY + c]); }
        return (TW)r;
    }

    // Riemann solve of interface k (cells cL, cR) of sweep IXY; waves to W
    template <int IXY>
    __device__ __forceinline__ int normal(int k, int cL, int cR, double seed, St& st, TW* s) const
    {
        TW qL[MEQN], qR[MEQN], dq[MEQN], aL[MA], aR[MA], da[MA], w[MWAVES][MEQN];
        for (int m = 0; m < MEQN; m++) { qL[m] = qc(m, cL); qR[m] = qc(m, cR); }
        for (int a = 0; a < MAUX; a++) { aL[a] = (TW)A()[a * NXY + cL]; aR[a] = (TW)A()[a * NXY + cR]; }
        // FP64 differences, for the solver that forms its flux difference from them (the
        // difference of two FP32 states keeps their rounding)
        for (int m = 0; m < MEQN; m++) dq[m] = (TW)(Q()[m * NXY + cR] - Q()[m * NXY + cL]);
        for (int a = 0; a < MAUX; a++) da[a] = (TW)(A()[a * NXY + cR] - A()[a * NXY + cL]);
        const TW* pc = C() + (F32 ? MEQN * NXY : 0);
        const int it = RP::template normal<IXY>(qL, qR, dq, aL, aR, da, Cell{pc + cL}, Cell{pc + cR}, P, seed, st, w, s);
#pragma unroll
        for (int mw = 0; mw < MWAVES; mw++)
#pragma unroll
            for (int m = 0; m < MEQN; m++)
                if (RP::template wp<IXY>(mw, m) >= 0) W()[RP::template wp<IXY>(mw, m) * NI + k] = w[mw][m];
        return it;
    }

    // Limiter, second-order correction, Godunov split and transverse split of interface k at
    // position pos along the sweep.  fm, fp: the interface's fluxes (FP32 form: fp only); the
    // transverse terms go to T.
    template <int IXY>
    __device__ __forceinline__ void second(int k, int cL, int cR, int pos, const St& st, double* fm, double* fp) const
    {
        constexpr int kstep = IXY == 1 ? 1 : NX - 2;
        // wall_lo: ghost on the left (low face), wall_hi: ghost on the right (high face)
        const bool wall_lo = F32 && pos == MBC && (wallf & (IXY == 1 ? 1 : 4));
        const bool wall_hi = F32 && pos == MX + MBC && (wallf & (IXY == 1 ? 2 : 8));
        TW w[MWAVES][MEQN], s[MWAVES], am[MEQN], ap[MEQN], cq[MEQN];
        RP::template expand<IXY>(st, [&](int j) { return W()[j * NI + k]; }, w, s);
        const bool god = G::god(pos), cor = G::cor(pos);
        if constexpr (RP::EXACT && F32) {
#pragma unroll
            for (int m = 0; m < MEQN; m++) {
                double a64, p64;
                RP::fluct_mixed(st, m, flux<IXY>(m, cL), flux<IXY>(m, cR), a64, p64);
                am[m] = (TW)a64; ap[m] = (TW)p64;
                fp[m] = god ? -p64 : 0.0;
            }
        } else {
            RP::template fluct<IXY>(st, w, s, am, ap);
#pragma unroll
            for (int m = 0; m < MEQN; m++) {
                if constexpr (F32) {
                    fp[m] = (double)(god ? -ap[m] : TW(0));
                    // zero mass flux through a wall: the interior cell's fluctuation cancels its own flux
                    if (m == 0 && wall_lo) fp[0] = -flux<IXY>(0, cR);
                    if (m == 0 && wall_hi) fp[0] = -((flux<IXY>(0, cR) - flux<IXY>(0, cL)) + flux<IXY>(0, cL));
                } else {
                    fm[m] = god ? am[m] : 0.0;
                    fp[m] = god ? 0.0 - ap[m] : 0.0;
                }
            }
        }
#pragma unroll
        for (int m = 0; m < MEQN; m++) cq[m] = TW(0);
        const TW dlo = ratio(IXY, cL);
        const TW dhi = RP::FWAVE ? dlo : ratio(IXY, cR);
        if (RP::FWAVE ? M.order1 != 1 : M.order1 == 2) {
            TW wlim[MWAVES];
#pragma unroll
            for (int mw = 0; mw < MWAVES; mw++) wlim[mw] = TW(1);
            if (pos >= MBC && pos <= MX + MBC) {
                // inline limiter (clawpack46_inlinelimiter.f:267-343): the projection of the
                // upwind neighbour's unlimited wave
#pragma unroll
                for (int mw = 0; mw < MWAVES; mw++) {
                    const int ml = M.limiter(mw);
                    if (ml == 0) continue;
                    const int kk = s[mw] > TW(0) ? k - kstep : k + kstep;
                    TW wnorm2 = TW(0), dot = TW(0);
#pragma unroll
                    for (int m = 0; m < MEQN; m++) {
                        if (RP::template wp<IXY>(mw, m) < 0) continue;
                        wnorm2 = wnorm2 + w[mw][m] * w[mw][m];
                        dot = dot + W()[RP::template wp<IXY>(mw, m) * NI + kk] * w[mw][m];
                    }
                    if (wnorm2 == TW(0)) continue;
                    const TW phi = limiter_phi<TW>(ml, dot / wnorm2);
                    if constexpr (F32) {
                        wlim[mw] = phi;                         // goes into the correction's factor
                    } else {
#pragma unroll
                        for (int m = 0; m < MEQN; m++) w[mw][m] = phi * w[mw][m];
                    }
                }
            }
            if (cor) {
                const TW dave = TW(0.5) * (dlo + ratio(IXY, cR));
                TW coef[MWAVES];
#pragma unroll
                for (int mw = 0; mw < MWAVES; mw++) {
                    const TW sa = fabs(s[mw]);
                    coef[mw] = mul_rn(RP::FWAVE ? sgn1(s[mw]) : sa, sub_rn(TW(1), mul_rn(sa, dave)));
                    if constexpr (F32) coef[mw] = mul_rn(coef[mw], wlim[mw]);
                }
#pragma unroll
                for (int m = 0; m < MEQN; m++) {
                    TW c = mul_rn(coef[0], w[0][m]);
#pragma unroll
                    for (int mw = 1; mw < MWAVES; mw++)
                        if (RP::template wp<IXY>(mw, m) >= 0) c = add_rn(c, mul_rn(coef[mw], w[mw][m]));
                    if (m == 0 && (wall_lo || wall_hi)) c = TW(0);
                    cq[m] = c;
                    if constexpr (F32) {
                        fp[m] = fp[m] + 0.5 * (double)c;
                    } else {
                        fm[m] = fm[m] + 0.5 * c;
                        fp[m] = fp[m] + 0.5 * c;
                    }
                }
            }
        }
        if (M.order2 > 0 && cor) {
            if (M.order1 > 1 && M.order2 == 2 && god) {
#pragma unroll
                for (int m = 0; m < MEQN; m++) { am[m] = am[m] + cq[m]; ap[m] = ap[m] - cq[m]; }
            }
            // aux of the sweep cell cL (imp 1) or cR (imp 2): below (0), here (1), above (2) the sweep line
            auto aux = [&](int row, int imp) { return (TW)A()[(imp == 1 ? cL : cR) + (row - 1) * (IXY == 1 ? NX : 1)]; };
            const auto e = RP::template split_state<IXY>(
                st, [&](int right) { return (TW)Q()[right ? cR : cL]; }, aux, P);
            TW bm[MEQN], bp[MEQN];
#pragma unroll
            for (int part = 0; part < 2; part++) {                // amdq, then apdq
                TW* as = part ? ap : am;
                const TW half = TW(0.5) * (part ? dhi : dlo);
                if constexpr (F32) {                              // the split is linear: scale what goes in
#pragma unroll
                    for (int m = 0; m < MEQN; m++) as[m] = half * as[m];
                }
                RP::template split<IXY>(e, 1 + part, aux, as, bm, bp);
#pragma unroll
                for (int m = 0; m < MEQN; m++) {
                    T()[((2 * part + 0) * MEQN + m) * NI + k] = F32 ? bm[m] : half * bm[m];
                    T()[((2 * part + 1) * MEQN + m) * NI + k] = F32 ? bp[m] : half * bp[m];
                }
            }
        }
    }

    // Transverse terms a face gets from one line of interfaces beside it: amdq of interface kr
    // (position pos + 1) and apdq of interface kl (pos), towards the lower (UP = 0) or the
    // upper (UP = 1) face.
    template <int UP>
    __device__ __forceinline__ double line(int m, int pos, int kl, int kr) const
    {
        double v = 0.0;
        if (!RP::FWAVE || G::cor(pos + 1)) v = v - (double)T()[((0 + UP) * MEQN + m) * NI + kr];
        if (!RP::FWAVE || G::cor(pos)) v = v - (double)T()[((2 + UP) * MEQN + m) * NI + kl];
        return v;
    }
    // of the y face (ic, jc) from the x sweeps of rows jc - 1 and jc
    __device__ __forceinline__ double into_y(int m, int ic, int jc) const
    {
        double g = 0.0;
        if (jc - 1 >= 1) g = line<1>(m, ic, G::kx(ic, jc - 1), G::kx(ic + 1, jc - 1));
        if (jc <= NY - 2) g = g + line<0>(m, ic, G::kx(ic, jc), G::kx(ic + 1, jc));
        return g;
    }

    // fm of the x face (ic, jc) = right face of cell c, and of the y face above it
    __device__ __forceinline__ double fm_x(int m, int ic, int jc) const
    {
        const double f = FX()[m * NI + G::kx(ic, jc)];
        if constexpr (!F32) { return f; }
        else {
            if (!G::god(ic)) return f;
            const int c = jc * NX + ic;
            if (m == 0 && !RP::EXACT && (wallf & 2) && ic == MX + MBC) return 0.0 - flux<1>(0, c - 1);
            double d = flux<1>(m, c) - flux<1>(m, c - 1);
            if constexpr (RP::SOURCE) d = d + RP::template source<1>(m, Q()[c - 1], Q()[c], A()[c - 1], A()[c], grav);
            return d + f;
        }
    }
    __device__ __forceinline__ double gm_y(int m, int ic, int jc) const
    {
        const double f = FY()[m * NI + G::ky(ic, jc)];
        if constexpr (!F32) { return f; }
        else {
            if (!G::god(jc)) return f;
            const int c = jc * NX + ic;
            if (m == 0 && !RP::EXACT && (wallf & 8) && jc == MY + MBC) return 0.0 - flux<2>(0, c - NX);
            double d = flux<2>(m, c) - flux<2>(m, c - NX);
            if constexpr (RP::SOURCE) d = d + RP::template source<2>(m, Q()[c - NX], Q()[c], A()[c - NX], A()[c], grav);
            return d + f;
        }
    }
    __device__ __forceinline__ double fp_x(int m, int ic, int jc) const
    {
        return FX()[((F32 ? 0 : MEQN) + m) * NI + G::kx(ic, jc)];
    }
    __device__ __forceinline__ double gp_y(int m, int ic, int jc) const
    {
        return FY()[((F32 ? 0 : MEQN) + m) * NI + G::ky(ic, jc)];
    }
};

// p*-seed of the exact solver for the interface between cells cL and cR (all lanes of the
// warp take part; have = false marks a lane without an interface)
template <int IXY, bool F32, int NXY>
__device__ __forceinline__ double wave_seed(const double* Q, int cL, int cR, bool have, double gamma, const void* mlp)
{
    double qL[4], qR[4];
    for (int m = 0; m < 4; m++) { qL[m] = Q[m * NXY + cL]; qR[m] = Q[m * NXY + cR]; }
    const RPEulerExact::Prim P = RPEulerExact::prim(IXY, qL, qR, gamma);
    float x[MLP_IN];
    double pbase;
    mlp_features(P.rl, P.ul, P.pl, P.rr, P.ur, P.pr, gamma, x, pbase);
    if (!have || !(x[0] == x[0] && x[1] == x[1] && x[2] == x[2] && x[3] == x[3] && x[4] == x[4] && x[5] == x[5])) {
        x[0] = 1.0f; x[1] = 0.0f; x[2] = 1.0f; x[3] = 1.0f; x[4] = 0.0f; x[5] = 1.0f;
        have = false;
    }
    const bool use = have && mlp_gate(x);
    // the network runs per warp (mma.sync over its 32 interfaces): skip warps
    // without an interface past the gate (smooth flow, weak waves)
    if (!__any_sync(0xffffffffu, use)) return 0.0;
    const MlpView W(mlp);
    MlpFrag h1, h2;
    mlp_warp_hidden<true>(W, x, h1, h2);
    const float y = mlp_warp_output(W, h2);
    if constexpr (F32) { return use ? pbase * (double)__expf(y) : 0.0; }
    else { return use ? pbase * fcb_exp((double)y) : 0.0; }
}

// The fused update of the patches from slot p0, one CTA each.  SEED: Newton starts from the
// network of the launch's parameters.
template <class RP, int MX, int NT, int MINB, typename TW, int LIM, bool SEED>
__global__ void __launch_bounds__(NT, MINB)
wave_kernel(double* __restrict__ q, double* __restrict__ qlast, const double* __restrict__ aux,
            double* __restrict__ regs, const PatchDesc* __restrict__ desc, int p0,
            const StepParams* __restrict__ spp, const LevelGroup lg, unsigned long long* __restrict__ cfl_bits)
{
    using G = WaveGeom<RP, MX, TW>;
    using WP = WavePatch<RP, MX, TW, LIM>;
    constexpr bool F32 = G::F32;
    constexpr int NX = G::NX, NY = G::NY, NXY = G::NXY, NI = G::NI, MEQN = G::MEQN, MBC = G::MBC, MY = G::MY;
    constexpr int MWAVES = RP::MWAVES;
    static_assert(NT >= NI, "one thread per interface of a sweep");
    extern __shared__ __align__(128) unsigned char sm[];
    double* red = reinterpret_cast<double*>(sm + G::OFF_RED);
    unsigned* nhist = reinterpret_cast<unsigned*>(sm + G::OFF_HIST);
    unsigned long long* bar = reinterpret_cast<unsigned long long*>(sm + G::OFF_BAR);
    const int tid = threadIdx.x, p = p0 + (int)blockIdx.x;

    // ---- stage -------------------------------------------------------------------
    if (tid == 0) {
        mbar_init(bar, 1);
        mbar_fence_init();
    }
    grid_dependency_wait();         // programmatic launch: the previous grid's writes are visible
    grid_launch_dependents();
    if (tid == 0) {
        bulk_expect(bar, G::QBYTES + G::ABYTES);
        bulk_copy(bar, sm, q + (size_t)p * MEQN * NXY, G::QBYTES);
        if constexpr (G::MAUX > 0) bulk_copy(bar, sm + G::OFF_A, aux + (size_t)p * G::MAUX * NXY, G::ABYTES);
    }
    if (RP::EXACT && tid < 32) nhist[tid] = 0u;            // Newton iterations of this patch
    const StepParams* sp = spp + group_slot(lg, (int)blockIdx.x);
    TW* konst = reinterpret_cast<TW*>(sm + G::OFF_K);
    if constexpr (RP::NCONST > 0) { if (tid == 32) RP::constants((TW)sp->gamma, konst); }
    const PatchDesc* pd = desc + p;
    const double dx = pd->dx, dy = pd->dy;
    const double dt = sp->inst_dt ? sp->dt * sp->inst_dt[pd->inst] : sp->dt;
    // reflecting walls of this patch whose ghost cells hold mirror values (FP32-wave mass rule)
    const int wallf = F32 ? (pd->phys_mask & sp->wall_faces) : 0;
    WP X{sm, WaveMethod<LIM>(sp), WavePar<TW>{(TW)sp->grav, (TW)sp->dry_tolerance, sp->gamma, sp->newton_tol, konst},
         sp->grav, dt / dx, dt / dy, wallf};
    double* Q = X.Q();
    // save_current_step: only what k_timeinterp may read (coarser levels of a subcycled step, patches
    // with fine-grid neighbours); an advance of one rank interpolates below instead
    bool save = sp->save_last && (pd->flags & PATCH_HAS_FINE_NBR);      // read while the copies travel
    __syncthreads();                                        // the barrier word is initialised
    // a thread that does not see the copies arrive writes nothing but the report of it (a decision
    // of the whole CTA before the cells phase, by thread 0 alone, took 0.8 % longer)
    const bool arrived = stage_arrived(bar);
    save = save && arrived;

    // ---- cells -------------------------------------------------------------------
    unsigned bad = 0;        // STATUS_* found in this thread's cells
    for (int c = tid; c < NXY; c += NT) {
        double qv[MEQN];
        TW qt[MEQN], cv[RP::NPRE];
#pragma unroll
        for (int m = 0; m < MEQN; m++) {
            qv[m] = Q[m * NXY + c];
            qt[m] = (TW)qv[m];
            if (!isfinite(qv[m])) bad |= STATUS_NONFINITE;
            if (save) qlast[(size_t)p * MEQN * NXY + m * NXY + c] = qv[m];
            if constexpr (F32) X.C()[m * NXY + c] = qt[m];
        }
        if (RP::DEPTH && qv[0] < 0.0) bad |= STATUS_DEPTH;
        RP::pre(qt, X.P, cv);
#pragma unroll
        for (int j = 0; j < RP::NPRE; j++) X.C()[((F32 ? MEQN : 0) + j) * NXY + c] = cv[j];
        if constexpr (F32) {
            double f[RP::NFL];
            RP::flux_planes(qv, X.P, X.grav, f);
#pragma unroll
            for (int j = 0; j < RP::NFL; j++) X.FL()[j * NXY + c] = f[j];
        }
    }
    // time-sync flux store (before the update; clawpack46_time_sync.f:37-90), FP64
    double* rg = regs + (size_t)p * G::NREG;
    if (arrived && sp->store_flux) {
        // faces 0,1: j = 1..my, k = 0,1 ; faces 2,3: i = 1..mx, k = 0,1
        for (int it = tid; it < 4 * MY + 4 * MX; it += NT) {
            int face, j, k;
            if (it < 4 * MY) { face = it / (2 * MY); int r = it % (2 * MY); j = r / 2; k = r % 2; }
            else { int r2 = it - 4 * MY; face = 2 + r2 / (2 * MX); int r = r2 % (2 * MX); j = r / 2; k = r % 2; }
            int ic, jc;
            if (face == 0) { ic = MBC - k; jc = MBC + j; }
            else if (face == 1) { ic = MX + MBC - 1 + k; jc = MBC + j; }
            else if (face == 2) { ic = MBC + j; jc = MBC - k; }
            else { ic = MBC + j; jc = MY + MBC - 1 + k; }
            double qv[MEQN], fl[MEQN];
            for (int m = 0; m < MEQN; m++) qv[m] = Q[m * NXY + jc * NX + ic];
            RP::cons_flux(face / 2, qv, X.grav, X.P.gamma, fl);
            const int n = (face < 2) ? MY : MX;
            const double el = (face < 2) ? dy : dx;
            const int base = (face == 0) ? G::R_EF0 : (face == 1) ? G::R_EF1 : (face == 2) ? G::R_EF2 : G::R_EF3;
            const bool zero = (sp->reg_reset >> ((pd->face_type >> (2 * face)) & 3)) & 1;
            for (int m = 0; m < MEQN; m++) accumulate(&rg[base + j + m * n + k * n * MEQN], zero, dt * el * fl[m]);
        }
    }
    if (bad && arrived && sp->status) atomicOr(sp->status, bad);
    if (__syncthreads_or(!arrived)) {
        // a staging copy did not arrive: report it, and wait (bounded) for it before leaving
        if (tid == 0) {
            if (sp->status) atomicOr(sp->status, (unsigned)STATUS_STAGING);
            (void)mbar_wait(bar, 0u, BULK_WAIT_LIMIT);
        }
        return;
    }

    const bool have = tid < NI;
    const int k = tid;
    const int jx = 1 + k / (NX - 1), ix = 1 + k % (NX - 1);      // x interface of this thread
    const int jy = 1 + k / (NX - 2), iy = 1 + k % (NX - 2);      // y interface
    const int cx = jx * NX + ix, cy = jy * NX + iy;              // the cells right of / above them
    typename WP::St st;
    TW cflw = TW(0);
    auto newton = [&](int r) {
        const int it = r & 0xff;
        atomicAdd(&nhist[it < 31 ? it : 31], 1u);
        if ((r & RPEulerExact::NEWTON_FAILED) && sp->status) atomicOr(sp->status, (unsigned)STATUS_NEWTON);
    };
    auto cfl = [&](const TW* s, TW d1, TW d0) {
        for (int mw = 0; mw < MWAVES; mw++) cflw = dmax1(dmax1(cflw, d1 * s[mw]), -(d0 * s[mw]));
    };

    // ---- x sweeps (clawpack46_step2.f:113-167) --------------------------------------
    {
        double seed = 0.0;
        if constexpr (SEED) seed = wave_seed<1, F32, NXY>(Q, have ? cx - 1 : 0, have ? cx : 1, have, sp->gamma, sp->mlp);
        if (have) {
            TW s[MWAVES];
            const int r = X.template normal<1>(k, cx - 1, cx, seed, st, s);
            if constexpr (RP::EXACT) newton(r);
            if (ix >= MBC && ix <= MX + MBC) cfl(s, X.ratio(1, cx), X.ratio(1, cx - 1));
        }
    }
    __syncthreads();
    if (have) {
        double fm[MEQN], fp[MEQN];
        X.template second<1>(k, cx - 1, cx, ix, st, fm, fp);
#pragma unroll
        for (int m = 0; m < MEQN; m++) {
            if constexpr (F32) X.FX()[m * NI + k] = fp[m];
            else { X.FX()[m * NI + k] = fm[m]; X.FX()[(MEQN + m) * NI + k] = fp[m]; }
        }
    }
    __syncthreads();
    // ---- y sweeps (clawpack46_step2.f:182-236) --------------------------------------
    double g[MEQN];
    {
        double seed = 0.0;
        if constexpr (SEED) seed = wave_seed<2, F32, NXY>(Q, have ? cy - NX : 0, have ? cy : 1, have, sp->gamma, sp->mlp);
        if (have) {
#pragma unroll
            for (int m = 0; m < MEQN; m++) g[m] = X.M.order2 > 0 ? X.into_y(m, iy, jy) : 0.0;
            if (F32 && ((jy == MBC && (wallf & 4)) || (jy == MY + MBC && (wallf & 8)))) g[0] = 0.0;
            TW s[MWAVES];
            const int r = X.template normal<2>(k, cy - NX, cy, seed, st, s);
            if constexpr (RP::EXACT) newton(r);
            if (jy >= MBC && jy <= MY + MBC) cfl(s, X.ratio(2, cy), X.ratio(2, cy - NX));
        }
    }
    __syncthreads();
    if (have) {
        double fm[MEQN], fp[MEQN];
        X.template second<2>(k, cy - NX, cy, jy, st, fm, fp);
#pragma unroll
        for (int m = 0; m < MEQN; m++) {
            if constexpr (F32) X.FY()[m * NI + k] = g[m] + fp[m];
            else { X.FY()[m * NI + k] = g[m] + fm[m]; X.FY()[(MEQN + m) * NI + k] = g[m] + fp[m]; }
        }
    }
    __syncthreads();
    // y-transverse terms into the x faces, column ix - 1 first
    if (have && X.M.order2 > 0) {
        const bool wall_edge = F32 && ((ix == MBC && (wallf & 1)) || (ix == MX + MBC && (wallf & 2)));
#pragma unroll
        for (int m = 0; m < MEQN; m++) {
            if (m == 0 && wall_edge) continue;
            double a = 0.0, b = 0.0;
            const bool left = ix - 1 >= 1, right = ix <= NX - 2;
            if (left) a = X.template line<1>(m, jx, G::ky(ix - 1, jx), G::ky(ix - 1, jx + 1));
            if (right) b = X.template line<0>(m, jx, G::ky(ix, jx), G::ky(ix, jx + 1));
#pragma unroll
            for (int f = 0; f < G::NF; f++) {
                double v = X.FX()[(f * MEQN + m) * NI + k];
                if (left) v = v + a;
                if (right) v = v + b;
                X.FX()[(f * MEQN + m) * NI + k] = v;
            }
        }
    }
    __syncthreads();

    // ---- time-sync wave accumulation (clawpack46_time_sync.f:163-226), FP64 ----
    if (sp->accumulate_waves) {
        const double dtdyv = dt * dy, dtdxv = dt * dx;
        const int reset = sp->reg_reset, ft = pd->face_type;
        // registers of a face reset since the last update start from zero
        auto add = [&](int face, int r, double v) {
            accumulate(&rg[r], (reset >> ((ft >> (2 * face)) & 3)) & 1, v);
        };
        for (int it = tid; it < (MY + MX) * MEQN; it += NT) {
            if (it < MY * MEQN) {
                const int j = it % MY, m = it / MY, jc = MBC + j, o = j + m * MY;
                add(0, G::R_FP0 + o, 0.0 - dtdyv * X.fp_x(m, MBC, jc));
                add(0, G::R_FM0 + o, dtdyv * X.fm_x(m, MBC, jc));
                add(1, G::R_FP1 + o, 0.0 - dtdyv * X.fp_x(m, MX + MBC, jc));
                add(1, G::R_FM1 + o, dtdyv * X.fm_x(m, MX + MBC, jc));
            } else {
                const int i2 = it - MY * MEQN, i = i2 % MX, m = i2 / MX, ic = MBC + i, o = i + m * MX;
                add(2, G::R_GP0 + o, 0.0 - dtdxv * X.gp_y(m, ic, MBC));
                add(2, G::R_GM0 + o, dtdxv * X.gm_y(m, ic, MBC));
                add(3, G::R_GP1 + o, 0.0 - dtdxv * X.gp_y(m, ic, MY + MBC));
                add(3, G::R_GM1 + o, dtdxv * X.gm_y(m, ic, MY + MBC));
            }
        }
    }
    // ---- q over i,j = 1-mbc..mx+mbc-1 (clawpack46_step2_wrap.f:107-125); faces of column or
    // row 0 are no sweep's and have no flux ----
    double* qg = q + (size_t)p * MEQN * NXY;
    double* qi = sp->qinterp && (pd->flags & PATCH_HAS_FINE_NBR) ? sp->qinterp + (size_t)p * MEQN * NXY : nullptr;
    for (int c = tid; c < NXY; c += NT) {
        const int jc = c / NX, ic = c - jc * NX;
        if (ic > NX - 2 || jc > NY - 2) continue;
        const bool band = qi && in_band(ic, jc, MX, MY, MBC);
#pragma unroll
        for (int m = 0; m < MEQN; m++) {
            const double fr = jc >= 1 ? X.fm_x(m, ic + 1, jc) : 0.0;
            const double fl = jc >= 1 && ic >= 1 ? X.fp_x(m, ic, jc) : 0.0;
            const double gt = ic >= 1 ? X.gm_y(m, ic, jc + 1) : 0.0;
            const double gb = jc >= 1 && ic >= 1 ? X.gp_y(m, ic, jc) : 0.0;
            const double old = Q[m * NXY + c];
            double v = old;
            bool capacity = false;
            if constexpr (G::MAUX > 0 && LIM == 0) capacity = X.M.mcapa > 0;
            if (capacity) v = v - (X.dtdx * (fr - fl) + X.dtdy * (gt - gb)) / X.A()[(X.M.mcapa - 1) * NXY + c];
            else v = v - X.dtdx * (fr - fl) - X.dtdy * (gt - gb);
            qg[m * NXY + c] = v;
            if (band) qi[m * NXY + c] = add_rn(old, mul_rn(sp->ti_alpha, sub_rn(v, old)));
        }
    }

    // ---- CFL maximum: warp shuffles, then one atomic per CTA -----------------
    for (int off = 16; off > 0; off >>= 1) cflw = dmax1(cflw, __shfl_xor_sync(0xffffffffu, cflw, off));
    if ((tid & 31) == 0) red[tid >> 5] = (double)cflw;
    __syncthreads();
    if (tid < 32) {
        double v = (tid < NT / 32) ? red[tid] : 0.0;
        for (int off = 16; off > 0; off >>= 1) v = dmax1(v, __shfl_xor_sync(0xffffffffu, v, off));
        if (tid == 0) {
            unsigned long long bits = (unsigned long long)__double_as_longlong(v);
            if (v != v) bits = 0x7ff8000000000000ull;   // NaN (e.g. negative depth) wins the max
            atomicMax(cfl_bits + pd->inst, bits);
        }
        if (RP::EXACT && sp->newton_hist && nhist[tid]) atomicAdd(&sp->newton_hist[tid], (unsigned long long)nhist[tid]);
    }
}

template <class RP, int MX, int NT, int MINB, typename TW, int LIM>
cudaError_t run_wave_variant(double* q, double* qlast, const double* aux, double* regs, const PatchDesc* desc, int p0,
                             int npatch, const StepParams* sp, const LevelGroup& lg, unsigned long long* cfl_bits,
                             cudaStream_t st)
{
    using G = WaveGeom<RP, MX, TW>;
    static bool attr_set = false;
    auto kern = wave_kernel<RP, MX, NT, MINB, TW, LIM, false>;
    auto seeded = kern;
    if constexpr (RP::EXACT) seeded = wave_kernel<RP, MX, NT, 1, TW, LIM, true>;   // the network takes registers
    if (!attr_set) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)G::BYTES);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(seeded, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)G::BYTES);
        if (e != cudaSuccess) return e;
        attr_set = true;
    }
    if (npatch <= 0) return cudaSuccess;
    return launch_k(lg.seeded ? seeded : kern, npatch, NT, G::BYTES, st, q, qlast, aux, regs, desc, p0, sp, lg, cfl_bits);
}

// One table entry: precision, solver id, square patch size MXV (mbc 2), threads, CTAs per SM,
// limiter fixed at compile time (0: any method).
#define FCB_WAVE_VARIANT(PREC, RPID, RPT, MXV, NT, MINB, TW, LIM)                                       \
    Step2Variant{PREC, RPID, MXV, MXV, 2, NT, MINB, 1, (int)WaveGeom<RPT, MXV, TW>::BYTES, 0,           \
                 &run_wave_variant<RPT, MXV, NT, MINB, TW, LIM>, LIM}

}  // namespace fcb
