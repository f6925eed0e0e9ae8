// k_step2.cuh -- fused per-level patch update (clawpack 4.6 step2 + step2_wrap).
//
// One CTA advances one patch.  The padded patch (mx+2mbc)(my+2mbc)meqn is staged
// in shared memory with coalesced loads; every x- and y-interface of the
// reference's sweeps gets a thread; the flux arrays fm/fp/gm/gp of
// clawpack46_step2.f are accumulated in shared memory in exactly the
// reference's order (x-sweeps row by row, then y-sweeps column by column) by
// gathering per-interface results, so no atomics are needed and repeated runs
// are bitwise identical.  The same CTA also performs, from the staged tile,
//   b4step2 (swirl edge velocities),         user_4.6/b4step2.f:25-36
//   save_current_step (q -> qlast),          fclaw2d_clawpatch.cpp (save_current_step)
//   time-sync flux store / wave accumulation clawpack46_time_sync.f:37-226
//   the conservative q update over i,j = 1-mbc..mx+mbc-1 (clawpack46_step2_wrap.f:107-125)
//   and the warp-shuffle CFL maximum.
//
// It runs application solvers (include/fc2d_b200_user.cuh); the package's own have kernels of
// their own, k_wave.cuh (shallow water, Euler) and k_adv.cuh (advection).
//
// TW is the arithmetic type of the waves, speeds, limiter, second-order correction and
// transverse splitting; built without FMA contraction, TW = double gives the bits of the FP64
// CPU path.
//
// Index conventions: padded 0-based cell (ic, jc), ic = i + mbc - 1 for the
// Fortran index i.  Interface ic sits between cells ic-1 and ic.
#pragma once
#include <cuda_runtime.h>
#include <type_traits>
#include "fcb_common.h"
#include "fcb_launch.cuh"
#include "riemann.cuh"

namespace fcb {

enum { APP_NONE = 0, APP_SWIRL = 1, APP_RADIALDAM = 2, APP_TSUNAMI = 3, APP_SHOCKBUBBLE = 4 };

// A solver struct RP declares HAS_B4STEP2 / HAS_SRC2 with the cell-wise b4step2 / src2 of
// include/fc2d_b200_user.cuh; its rpt2 receives the aux of both cells beside the interface,
// cudaclaw's layout (cudaclaw_flux2.cu:682-694): aux1/aux2/aux3[imp * maux + m], imp = 0 for
// the left cell, 1 for the right.

template <class RP, int MX, int MY, int MBC, typename TW, int NT = 0>
struct Step2Geom {
    static constexpr int NX = MX + 2 * MBC, NY = MY + 2 * MBC, NXY = NX * NY;
    static constexpr int MEQN = RP::MEQN, MWAVES = RP::MWAVES, MAUX = RP::MAUX, NEXTRA = RP::NEXTRA;
    static constexpr int NIX = (NY - 2) * (NX - 1);          // x-sweep interfaces
    // y-sweep interfaces, numbered with i fastest (k = (jc-1)(NX-2) + ic-1), so the
    // threads of a warp touch consecutive cells of a row of the shared-memory arrays
    static constexpr int NIY = (NX - 2) * (NY - 1);
    static constexpr int NI = NIX > NIY ? NIX : NIY;
    // REG: every interface of a sweep has its own thread, so the normal solve
    // (speeds, fluctuations, Roe averages) stays in registers across the
    // barrier and only the waves, which the limiter reads from the neighbours,
    // go through shared memory.
    static constexpr bool REG = NT >= NI;
    // per-interface record of the normal solve: waves, speeds, amdq, apdq, solver extra
    static constexpr int W_WAVE = 0, W_S = MWAVES * MEQN, W_AM = W_S + MWAVES, W_AP = W_AM + MEQN,
                         W_EX = W_AP + MEQN, WSZ_FULL = W_EX + NEXTRA;
    static constexpr int WSZ = REG ? MWAVES * MEQN : WSZ_FULL;
    // per-interface transverse terms: A1, A2 (from amdq), B1, B2 (from apdq)
    static constexpr int TSZ = 4 * MEQN;
    static constexpr int AUXS = MAUX > 0 ? MAUX : 0;
    static constexpr size_t DOUBLES = (size_t)MEQN * NXY * 5 + (size_t)AUXS * NXY + 64;
    static constexpr size_t TWS = (size_t)WSZ * NI + (size_t)TSZ * NI;
    static constexpr size_t SMEM_BYTES = DOUBLES * 8 + TWS * sizeof(TW) + NI;
    // conservation registers (fclaw2d_clawpatch_conservation.h:56-77), per patch
    static constexpr int R_FP0 = 0, R_FP1 = MY * MEQN, R_FM0 = 2 * MY * MEQN, R_FM1 = 3 * MY * MEQN;
    static constexpr int R_GP0 = 4 * MY * MEQN, R_GP1 = R_GP0 + MX * MEQN, R_GM0 = R_GP0 + 2 * MX * MEQN,
                         R_GM1 = R_GP0 + 3 * MX * MEQN;
    static constexpr int R_EF0 = R_GP0 + 4 * MX * MEQN, R_EF1 = R_EF0 + 2 * MY * MEQN,
                         R_EF2 = R_EF1 + 2 * MY * MEQN, R_EF3 = R_EF2 + 2 * MX * MEQN,
                         NREG = R_EF3 + 2 * MX * MEQN;
};

// The update of patch p by the whole CTA (one call per patch; the CTA may do
// several patches in turn).
template <class RP, int MX, int MY, int MBC, int NT, typename TW>
__device__ __forceinline__ void
step2_patch(double* __restrict__ q, double* __restrict__ qlast, const double* __restrict__ aux,
            double* __restrict__ regs, const PatchDesc* __restrict__ desc, const int p,
            const StepParams& sp, unsigned long long* __restrict__ cfl_bits)
{
    using G = Step2Geom<RP, MX, MY, MBC, TW, NT>;
    constexpr bool REG = G::REG;
    constexpr int NX = G::NX, NY = G::NY, NXY = G::NXY, MEQN = G::MEQN, MWAVES = G::MWAVES;
    constexpr int MAUX = G::MAUX, NEXTRA = G::NEXTRA, NI = G::NI, WSZ = G::WSZ;
    constexpr int MA = MAUX > 0 ? MAUX : 1;
    // flux2 interface ranges (padded): Godunov and amdq+=cqxx up to GOD_HI, cqxx and transverse
    // at every interface
    constexpr int GOD_HI = NX - 2, GOD_HIY = NY - 2;

    extern __shared__ double smem[];
    double* Qs = smem;                              // [MEQN][NY][NX]
    double* FMs = Qs + MEQN * NXY;
    double* FPs = FMs + MEQN * NXY;
    double* GMs = FPs + MEQN * NXY;
    double* GPs = GMs + MEQN * NXY;
    double* As = GPs + MEQN * NXY;                  // [MAUX][NY][NX]
    double* red = As + G::AUXS * NXY;               // 64 doubles for reductions
    TW* W = reinterpret_cast<TW*>(red + 64);        // [WSZ][NI]  (SoA)
    TW* Tt = W + (size_t)WSZ * NI;                  // [TSZ][NI]
    unsigned char* tflag = reinterpret_cast<unsigned char*>(Tt + (size_t)G::TSZ * NI);

    const int tid = threadIdx.x;
    const PatchDesc pd = desc[p];
    const double dx = pd.dx, dy = pd.dy;
    const double dt = sp.inst_dt ? sp.dt * sp.inst_dt[pd.inst] : sp.dt;
    const double dtdx = dt / dx, dtdy = dt / dy;
    double* qg = q + (size_t)p * MEQN * NXY;
    // save_current_step: only what k_timeinterp may read (coarser levels of a subcycled step, patches
    // with fine-grid neighbours); an advance of one rank interpolates below instead
    const bool save = sp.save_last && (pd.flags & PATCH_HAS_FINE_NBR);

    // ---- stage q (and aux) in shared memory --------------------------------
    unsigned bad = 0;        // STATUS_* found in this thread's cells
    for (int k = tid; k < MEQN * NXY; k += NT) {
        double v = qg[k];
        if (!isfinite(v)) bad |= STATUS_NONFINITE;
        Qs[k] = v;
        if (save) qlast[(size_t)p * MEQN * NXY + k] = v;
        FMs[k] = 0.0; FPs[k] = 0.0; GMs[k] = 0.0; GPs[k] = 0.0;
    }
    if (bad && sp.status) atomicOr(sp.status, bad);
    if (MAUX > 0) {
        const double* ag = aux + (size_t)p * G::AUXS * NXY;
        if (sp.app == APP_SWIRL) {
            // b4step2: aux(:,:,1) = vty*(psi(x,y+dy)-psi), aux(:,:,2) = -vtx*(psi(x+dx,y)-psi);
            // the stored aux holds the psi differences.
            const double vty = sp.vt / dy, vtx = sp.vt / dx;
            for (int k = tid; k < NXY; k += NT) {
                As[k] = vty * ag[k];
                As[NXY + k] = -(vtx * ag[NXY + k]);
            }
        } else {
            for (int k = tid; k < G::AUXS * NXY; k += NT) As[k] = ag[k];
        }
    }
    __syncthreads();
    if constexpr (RP::HAS_B4STEP2) {
        // user b4step2, cell by cell over the padded patch (cudaclaw_flux2.cu:111-150):
        // it may set the cell's aux from its q, position and time.  As the reference's
        // b4step2 it changes the patch's aux in place (the only write to the aux slab
        // during an update; each CTA writes its own patch)
        double* ag = const_cast<double*>(aux) + (size_t)p * G::AUXS * NXY;
        for (int c = tid; c < NXY; c += NT) {
            double qc[MEQN], ac[G::AUXS > 0 ? G::AUXS : 1];
            for (int m = 0; m < MEQN; m++) qc[m] = Qs[m * NXY + c];
            for (int a = 0; a < G::AUXS; a++) ac[a] = As[a * NXY + c];
            RP::b4step2(MBC, MX, MY, MEQN, qc, pd.xlower, pd.ylower, dx, dy, sp.t, dt, G::AUXS, ac,
                        c % NX - MBC + 1, c / NX - MBC + 1);
            for (int a = 0; a < G::AUXS; a++) { As[a * NXY + c] = ac[a]; ag[a * NXY + c] = ac[a]; }
        }
        __syncthreads();
    }

    const int mcapa = sp.mcapa;
    auto dtdx1d_x = [&](int ic, int jc) -> TW {
        return mcapa > 0 ? (TW)(dtdx / As[(mcapa - 1) * NXY + jc * NX + ic]) : (TW)dtdx;
    };
    auto dtdy1d_y = [&](int ic, int jc) -> TW {
        return mcapa > 0 ? (TW)(dtdy / As[(mcapa - 1) * NXY + jc * NX + ic]) : (TW)dtdy;
    };
    auto qload = [&](int m, int c) -> TW { return (TW)Qs[m * NXY + c]; };
    const TW gravw = (TW)sp.grav, drytolw = (TW)sp.dry_tolerance;

    double* rg = regs + (size_t)p * G::NREG;
    double cflmax = 0.0;

    struct State { TW wave[MWAVES][MEQN]; TW s[MWAVES]; TW am[MEQN]; TW ap[MEQN]; TW ex[NEXTRA]; };

    // Normal solve of one interface (qL = cell cL, qR = cell cR).
    auto normal_solve = [&](int ixy, int cL, int cR, int k, bool cfl_range, TW d1, TW d0, State& st) {
        TW qL[MEQN], qR[MEQN], aL[MA], aR[MA];
        for (int m = 0; m < MEQN; m++) { qL[m] = qload(m, cL); qR[m] = qload(m, cR); }
        for (int a = 0; a < MAUX; a++) { aL[a] = (TW)As[a * NXY + cL]; aR[a] = (TW)As[a * NXY + cR]; }
        RP::template rpn2<TW>(ixy, qL, qR, aL, aR, st.wave, st.s, st.am, st.ap, st.ex, gravw);
        for (int mw = 0; mw < MWAVES; mw++)
            for (int m = 0; m < MEQN; m++) W[(G::W_WAVE + mw * MEQN + m) * NI + k] = st.wave[mw][m];
        if (!REG) {
            for (int mw = 0; mw < MWAVES; mw++) W[(G::W_S + mw) * NI + k] = st.s[mw];
            for (int m = 0; m < MEQN; m++) { W[(G::W_AM + m) * NI + k] = st.am[m]; W[(G::W_AP + m) * NI + k] = st.ap[m]; }
            for (int e = 0; e < NEXTRA; e++) W[(G::W_EX + e) * NI + k] = st.ex[e];
        }
        if (cfl_range) {
            for (int mw = 0; mw < MWAVES; mw++)
                cflmax = dmax1(dmax1(cflmax, (double)(d1 * st.s[mw])), (double)(-(d0 * st.s[mw])));
        }
    };
    auto restore = [&](int k, State& st) {
        if (REG) return;
        for (int mw = 0; mw < MWAVES; mw++) {
            for (int m = 0; m < MEQN; m++) st.wave[mw][m] = W[(G::W_WAVE + mw * MEQN + m) * NI + k];
            st.s[mw] = W[(G::W_S + mw) * NI + k];
        }
        for (int m = 0; m < MEQN; m++) { st.am[m] = W[(G::W_AM + m) * NI + k]; st.ap[m] = W[(G::W_AP + m) * NI + k]; }
        for (int e = 0; e < NEXTRA; e++) st.ex[e] = W[(G::W_EX + e) * NI + k];
    };

    // Limiter, second-order correction, fadd and transverse split of one interface.
    // Returns faddm/faddp (FP64) and writes the transverse terms into Tt.
    auto interface_update = [&](int ixy, int k, int cL, int cR, int pos, int lim_lo, int lim_hi,
                                bool god, TW dlo, TW dhi, TW dave,
                                const int* a1c, const int* a2c, const int* a3c, State& st,
                                double* faddm, double* faddp) {
        TW cq[MEQN];
        for (int m = 0; m < MEQN; m++) { cq[m] = TW(0); faddm[m] = 0.0; faddp[m] = 0.0; }
        if (god) {
            for (int m = 0; m < MEQN; m++) { faddp[m] = faddp[m] - (double)st.ap[m]; faddm[m] = faddm[m] + (double)st.am[m]; }
        }
        if (sp.order1 == 2) {
            if (pos >= lim_lo && pos <= lim_hi) {
                // inline limiter (clawpack46_inlinelimiter.f:267-343) with unlimited neighbours;
                // the neighbours along the sweep are k -+ 1 (x) or k -+ (NX-2) (y)
                const int kstep = (ixy == 1) ? 1 : NX - 2;
                for (int mw = 0; mw < MWAVES; mw++) {
                    const int ml = sp.mthlim[mw];
                    if (ml == 0) continue;
                    TW wnorm2 = TW(0), dotl = TW(0), dotr = TW(0);
                    for (int m = 0; m < MEQN; m++) {
                        const TW w = st.wave[mw][m];
                        const TW wl = W[(G::W_WAVE + mw * MEQN + m) * NI + k - kstep];
                        const TW wr = W[(G::W_WAVE + mw * MEQN + m) * NI + k + kstep];
                        wnorm2 = wnorm2 + w * w;
                        dotl = dotl + wl * w;
                        dotr = dotr + w * wr;
                    }
                    if (wnorm2 == TW(0)) continue;
                    const TW r = (st.s[mw] > TW(0)) ? dotl / wnorm2 : dotr / wnorm2;
                    const TW wlim = limiter_phi<TW>(ml, r);
                    for (int m = 0; m < MEQN; m++) st.wave[mw][m] = wlim * st.wave[mw][m];
                }
            }
            for (int m = 0; m < MEQN; m++) {
                TW c = TW(0);
                for (int mw = 0; mw < MWAVES; mw++) {
                    const TW sa = fabs(st.s[mw]);
                    c = add_rn(c, mul_rn(mul_rn(sa, sub_rn(TW(1), mul_rn(sa, dave))), st.wave[mw][m]));
                }
                cq[m] = c;
                faddm[m] = faddm[m] + (double)(TW(0.5) * c);
                faddp[m] = faddp[m] + (double)(TW(0.5) * c);
            }
        }
        unsigned char fl = 0;
        if (sp.order2 > 0) {
            TW am[MEQN], ap[MEQN];
            for (int m = 0; m < MEQN; m++) { am[m] = st.am[m]; ap[m] = st.ap[m]; }
            if (sp.order1 > 1 && sp.order2 == 2 && god)
                for (int m = 0; m < MEQN; m++) { am[m] = am[m] + cq[m]; ap[m] = ap[m] - cq[m]; }
            TW qL[MEQN], qR[MEQN];
            for (int m = 0; m < MEQN; m++) { qL[m] = qload(m, cL); qR[m] = qload(m, cR); }
            TW a1[2 * MA], a2[2 * MA], a3[2 * MA], bm[MEQN], bp[MEQN];
            for (int h = 0; h < 2; h++)
                for (int a = 0; a < MAUX; a++) {
                    a1[h * MA + a] = (TW)As[a * NXY + a1c[h]];
                    a2[h * MA + a] = (TW)As[a * NXY + a2c[h]];
                    a3[h * MA + a] = (TW)As[a * NXY + a3c[h]];
                }
            RP::template rpt2<TW>(ixy, 1, qL, qR, a1, a2, a3, st.ex, am, bm, bp, gravw, drytolw);
            for (int m = 0; m < MEQN; m++) {
                Tt[(0 * MEQN + m) * NI + k] = TW(0.5) * dlo * bm[m];
                Tt[(1 * MEQN + m) * NI + k] = TW(0.5) * dlo * bp[m];
            }
            RP::template rpt2<TW>(ixy, 2, qL, qR, a1, a2, a3, st.ex, ap, bm, bp, gravw, drytolw);
            for (int m = 0; m < MEQN; m++) {
                Tt[(2 * MEQN + m) * NI + k] = TW(0.5) * dhi * bm[m];
                Tt[(3 * MEQN + m) * NI + k] = TW(0.5) * dhi * bp[m];
            }
            fl = 1;
        }
        tflag[k] = fl;
    };

    // x-sweep interface k -> row jc = 1 + k / (NX-1), interface ic = 1 + k % (NX-1)
    auto x1 = [&](int k, State& st) {
        const int jc = 1 + k / (NX - 1), ic = 1 + k % (NX - 1);
        const bool cr = (ic >= MBC && ic <= MX + MBC);
        normal_solve(1, jc * NX + ic - 1, jc * NX + ic, k, cr, cr ? dtdx1d_x(ic, jc) : TW(0),
                     cr ? dtdx1d_x(ic - 1, jc) : TW(0), st);
    };
    auto x2 = [&](int k, State& st) {
        const int jc = 1 + k / (NX - 1), ic = 1 + k % (NX - 1);
        const TW dlo = dtdx1d_x(ic - 1, jc);
        const TW dhi = dtdx1d_x(ic, jc);
        const TW dave = TW(0.5) * (dtdx1d_x(ic - 1, jc) + dtdx1d_x(ic, jc));
        // aux of cell i1 = ic-1 (amdq) / ic (apdq) on rows jc-1, jc, jc+1
        const int a1c[2] = {(jc - 1) * NX + ic - 1, (jc - 1) * NX + ic};
        const int a2c[2] = {jc * NX + ic - 1, jc * NX + ic};
        const int a3c[2] = {(jc + 1) * NX + ic - 1, (jc + 1) * NX + ic};
        double faddm[MEQN], faddp[MEQN];
        interface_update(1, k, jc * NX + ic - 1, jc * NX + ic, ic, MBC, MX + MBC,
                         ic <= GOD_HI, dlo, dhi, dave, a1c, a2c, a3c, st, faddm, faddp);
        for (int m = 0; m < MEQN; m++) {
            FMs[m * NXY + jc * NX + ic] = 0.0 + faddm[m];
            FPs[m * NXY + jc * NX + ic] = 0.0 + faddp[m];
        }
    };
    // y-sweep interface k -> row interface jc = 1 + k / (NX-2), column ic = 1 + k % (NX-2)
    auto y1 = [&](int k, State& st) {
        const int jc = 1 + k / (NX - 2), ic = 1 + k % (NX - 2);
        const bool cr = (jc >= MBC && jc <= MY + MBC);
        normal_solve(2, (jc - 1) * NX + ic, jc * NX + ic, k, cr, cr ? dtdy1d_y(ic, jc) : TW(0),
                     cr ? dtdy1d_y(ic, jc - 1) : TW(0), st);
    };
    auto y2 = [&](int k, State& st) {
        const int jc = 1 + k / (NX - 2), ic = 1 + k % (NX - 2);
        const TW dlo = dtdy1d_y(ic, jc - 1);
        const TW dhi = dtdy1d_y(ic, jc);
        const TW dave = TW(0.5) * (dtdy1d_y(ic, jc - 1) + dtdy1d_y(ic, jc));
        // aux of sweep cell i1 = jc-1 (amdq) / jc (apdq) on columns ic-1, ic, ic+1
        const int a1c[2] = {(jc - 1) * NX + ic - 1, jc * NX + ic - 1};
        const int a2c[2] = {(jc - 1) * NX + ic, jc * NX + ic};
        const int a3c[2] = {(jc - 1) * NX + ic + 1, jc * NX + ic + 1};
        double faddm[MEQN], faddp[MEQN];
        interface_update(2, k, (jc - 1) * NX + ic, jc * NX + ic, jc, MBC, MY + MBC,
                         jc <= GOD_HIY, dlo, dhi, dave, a1c, a2c, a3c, st, faddm, faddp);
        for (int m = 0; m < MEQN; m++) {
            GMs[m * NXY + jc * NX + ic] = GMs[m * NXY + jc * NX + ic] + faddm[m];
            GPs[m * NXY + jc * NX + ic] = GPs[m * NXY + jc * NX + ic] + faddp[m];
        }
    };
    // X3: gadd -> gm/gp.  gm(ic,jc) = ((0 + G2(row jc-1)) + G1(row jc)), gp identical.
    auto x3 = [&](int c) {
        const int jc = c / NX, ic = c % NX;
        if (ic < 1 || jc < 1) return;                    // accumulation range ic >= 1, rows >= 1
        for (int m = 0; m < MEQN; m++) {
            double g = 0.0;
            if (jc - 1 >= 1 && jc - 1 <= NY - 2) {       // row jc-1, its gadd(:,2)
                const int r = jc - 1;
                double v = 0.0;
                if (ic + 1 <= NX - 1) { const int kk = (r - 1) * (NX - 1) + ic; if (tflag[kk]) v = v - (double)Tt[(1 * MEQN + m) * NI + kk]; }
                { const int kk = (r - 1) * (NX - 1) + ic - 1; if (tflag[kk]) v = v - (double)Tt[(3 * MEQN + m) * NI + kk]; }
                g = g + v;
            }
            if (jc <= NY - 2) {                          // row jc, its gadd(:,1)
                const int r = jc;
                double v = 0.0;
                if (ic + 1 <= NX - 1) { const int kk = (r - 1) * (NX - 1) + ic; if (tflag[kk]) v = v - (double)Tt[(0 * MEQN + m) * NI + kk]; }
                { const int kk = (r - 1) * (NX - 1) + ic - 1; if (tflag[kk]) v = v - (double)Tt[(2 * MEQN + m) * NI + kk]; }
                g = g + v;
            }
            GMs[m * NXY + c] = g;
            GPs[m * NXY + c] = g;
        }
    };
    // Y3: gadd -> fm/fp.  fm(ic,jc) = (fm + G2(col ic-1)) + G1(col ic)
    auto y3 = [&](int c) {
        const int jc = c / NX, ic = c % NX;
        if (jc < 1) return;
        for (int m = 0; m < MEQN; m++) {
            double fm = FMs[m * NXY + c], fp = FPs[m * NXY + c];
            if (ic - 1 >= 1 && ic - 1 <= NX - 2) {
                const int col = ic - 1;
                double v = 0.0;
                if (jc + 1 <= NY - 1) { const int kk = jc * (NX - 2) + col - 1; if (tflag[kk]) v = v - (double)Tt[(1 * MEQN + m) * NI + kk]; }
                { const int kk = (jc - 1) * (NX - 2) + col - 1; if (tflag[kk]) v = v - (double)Tt[(3 * MEQN + m) * NI + kk]; }
                fm = fm + v; fp = fp + v;
            }
            if (ic >= 1 && ic <= NX - 2) {
                const int col = ic;
                double v = 0.0;
                if (jc + 1 <= NY - 1) { const int kk = jc * (NX - 2) + col - 1; if (tflag[kk]) v = v - (double)Tt[(0 * MEQN + m) * NI + kk]; }
                { const int kk = (jc - 1) * (NX - 2) + col - 1; if (tflag[kk]) v = v - (double)Tt[(2 * MEQN + m) * NI + kk]; }
                fm = fm + v; fp = fp + v;
            }
            FMs[m * NXY + c] = fm;
            FPs[m * NXY + c] = fp;
        }
    };

    // =================== x-sweeps (clawpack46_step2.f:113-167) ===================
    State st;
    if (REG) { if (tid < G::NIX) x1(tid, st); }
    else for (int k = tid; k < G::NIX; k += NT) x1(k, st);
    __syncthreads();
    if (REG) { if (tid < G::NIX) x2(tid, st); }
    else for (int k = tid; k < G::NIX; k += NT) { restore(k, st); x2(k, st); }
    __syncthreads();
    // X3 and the y-sweep normal solves touch disjoint data: one phase
    for (int c = tid; c < NXY; c += NT) x3(c);
    // =================== y-sweeps (clawpack46_step2.f:182-236) ===================
    if (REG) { if (tid < G::NIY) y1(tid, st); }
    else for (int k = tid; k < G::NIY; k += NT) y1(k, st);
    __syncthreads();
    if (REG) { if (tid < G::NIY) y2(tid, st); }
    else for (int k = tid; k < G::NIY; k += NT) { restore(k, st); y2(k, st); }
    __syncthreads();
    for (int c = tid; c < NXY; c += NT) y3(c);
    __syncthreads();

    // ---- time-sync wave accumulation (clawpack46_time_sync.f:163-226), FP64 ----
    if (sp.accumulate_waves) {
        const double dtdyv = dt * dy, dtdxv = dt * dx;
        // registers of a face reset since the last update start from zero
        auto z = [&](int face) { return ((sp.reg_reset >> ((pd.face_type >> (2 * face)) & 3)) & 1) != 0; };
        const bool z0 = z(0), z1 = z(1), z2 = z(2), z3 = z(3);
        for (int it = tid; it < (MY + MX) * MEQN; it += NT) {
            if (it < MY * MEQN) {
                const int j = it % MY, m = it / MY;
                const int jc = MBC + j;
                const int cl = m * NXY + jc * NX + MBC, cr = m * NXY + jc * NX + MX + MBC;
                double* r;
                r = &rg[G::R_FP0 + j + m * MY]; *r = (z0 ? 0.0 : *r) - dtdyv * FPs[cl];
                r = &rg[G::R_FM0 + j + m * MY]; *r = (z0 ? 0.0 : *r) + dtdyv * FMs[cl];
                r = &rg[G::R_FP1 + j + m * MY]; *r = (z1 ? 0.0 : *r) - dtdyv * FPs[cr];
                r = &rg[G::R_FM1 + j + m * MY]; *r = (z1 ? 0.0 : *r) + dtdyv * FMs[cr];
            } else {
                const int i2 = it - MY * MEQN;
                const int i = i2 % MX, m = i2 / MX;
                const int ic = MBC + i;
                const int cb = m * NXY + MBC * NX + ic, ct = m * NXY + (MY + MBC) * NX + ic;
                double* r;
                r = &rg[G::R_GP0 + i + m * MX]; *r = (z2 ? 0.0 : *r) - dtdxv * GPs[cb];
                r = &rg[G::R_GM0 + i + m * MX]; *r = (z2 ? 0.0 : *r) + dtdxv * GMs[cb];
                r = &rg[G::R_GP1 + i + m * MX]; *r = (z3 ? 0.0 : *r) - dtdxv * GPs[ct];
                r = &rg[G::R_GM1 + i + m * MX]; *r = (z3 ? 0.0 : *r) + dtdxv * GMs[ct];
            }
        }
    }

    // ---- q update over i,j = 1-mbc..mx+mbc-1 (clawpack46_step2_wrap.f:107-125) ----
    double* qi = sp.qinterp && (pd.flags & PATCH_HAS_FINE_NBR) ? sp.qinterp + (size_t)p * MEQN * NXY : nullptr;
    auto interpolate = [&](int m, int c, int ic, int jc, double v) {
        if (qi && in_band(ic, jc, MX, MY, MBC)) {
            const double old = Qs[m * NXY + c];
            qi[m * NXY + c] = add_rn(old, mul_rn(sp.ti_alpha, sub_rn(v, old)));
        }
    };
    if constexpr (RP::HAS_SRC2) {
        // with a user src2 (clawpack46_update, fc2d_clawpack46.cpp:436-441: src2 after
        // step2), every padded cell gets its updated q (cells the update skips keep
        // theirs) passed through the cell-wise source term before it is stored
        for (int c = tid; c < NXY; c += NT) {
            const int jc = c / NX, ic = c % NX;
            double qc[MEQN], ac[G::AUXS > 0 ? G::AUXS : 1];
            for (int m = 0; m < MEQN; m++) {
                const int b = m * NXY;
                double v = Qs[b + c];
                if (ic <= NX - 2 && jc <= NY - 2) {
                    if (mcapa == 0)
                        v = v - dtdx * (FMs[b + c + 1] - FPs[b + c]) - dtdy * (GMs[b + c + NX] - GPs[b + c]);
                    else
                        v = v - (dtdx * (FMs[b + c + 1] - FPs[b + c]) + dtdy * (GMs[b + c + NX] - GPs[b + c])) /
                                    As[(mcapa - 1) * NXY + c];
                }
                qc[m] = v;
            }
            for (int a = 0; a < G::AUXS; a++) ac[a] = As[a * NXY + c];
            RP::src2(MBC, MX, MY, MEQN, qc, pd.xlower, pd.ylower, dx, dy, sp.t, dt, G::AUXS, ac, ic - MBC + 1,
                     jc - MBC + 1);
            for (int m = 0; m < MEQN; m++) {
                qg[m * NXY + c] = qc[m];
                interpolate(m, c, ic, jc, qc[m]);
            }
        }
    } else
    for (int k = tid; k < MEQN * NXY; k += NT) {
        const int m = k / NXY, c = k % NXY;
        const int jc = c / NX, ic = c % NX;
        if (ic <= NX - 2 && jc <= NY - 2) {
            const int b = m * NXY;
            double v = Qs[k];
            if (mcapa == 0)
                v = v - dtdx * (FMs[b + c + 1] - FPs[b + c]) - dtdy * (GMs[b + c + NX] - GPs[b + c]);
            else
                v = v - (dtdx * (FMs[b + c + 1] - FPs[b + c]) + dtdy * (GMs[b + c + NX] - GPs[b + c])) /
                            As[(mcapa - 1) * NXY + c];
            qg[k] = v;
            interpolate(m, c, ic, jc, v);
        }
    }

    // ---- CFL maximum: warp shuffles, then one atomic per CTA -----------------
    for (int off = 16; off > 0; off >>= 1) cflmax = dmax1(cflmax, __shfl_xor_sync(0xffffffffu, cflmax, off));
    if ((tid & 31) == 0) red[tid >> 5] = cflmax;
    __syncthreads();
    if (tid < 32) {
        double v = (tid < NT / 32) ? red[tid] : 0.0;
        for (int off = 16; off > 0; off >>= 1) v = dmax1(v, __shfl_xor_sync(0xffffffffu, v, off));
        if (tid == 0) {
            unsigned long long bits = (unsigned long long)__double_as_longlong(v);
            if (v != v) bits = 0x7ff8000000000000ull;   // NaN (e.g. negative depth) wins the max
            atomicMax(cfl_bits + pd.inst, bits);
        }
    }
}

// The fused update of npatch patches starting at slot p0.  One CTA per patch, or
// (PERSIST) a grid of a few CTAs per SM, each taking patches p0 + blockIdx.x,
// + gridDim.x, ... in turn, its shared memory reused patch after patch.
template <class RP, int MX, int MY, int MBC, int NT, typename TW, int MINB = 2, bool PERSIST = false>
__global__ void __launch_bounds__(NT, MINB)
step2_kernel(double* __restrict__ q, double* __restrict__ qlast, const double* __restrict__ aux,
             double* __restrict__ regs, const PatchDesc* __restrict__ desc, int p0, int npatch,
             const StepParams* __restrict__ spp, const LevelGroup lg, unsigned long long* __restrict__ cfl_bits)
{
    grid_dependency_wait();         // programmatic launch: the previous grid's writes are visible
    grid_launch_dependents();
    // per-launch parameters live in device memory (graph replay); a launch over
    // several levels holds one block per level, highest level first
    if constexpr (!PERSIST) {
        (void)npatch;
        const int p = p0 + (int)blockIdx.x;
        const StepParams sp = spp[group_slot(lg, (int)blockIdx.x)];
        step2_patch<RP, MX, MY, MBC, NT, TW>(q, qlast, aux, regs, desc, p, sp, cfl_bits);
    } else {
        for (int b = blockIdx.x; b < npatch; b += gridDim.x) {
            const int p = p0 + b;
            const StepParams sp = spp[group_slot(lg, b)];
            step2_patch<RP, MX, MY, MBC, NT, TW>(q, qlast, aux, regs, desc, p, sp, cfl_bits);
            __syncthreads();   // the next patch restages the shared memory
        }
    }
}

}  // namespace fcb
