// riemann.cuh -- parts the update kernels share: limiters, the pressure function, fluxes and
// star pressure of the exact Euler solver, and uncontracted arithmetic.  The solvers themselves
// are in wave_solvers.cuh (shallow water, Euler) and k_adv.cuh (advection); application solvers
// run in k_step2.cuh.
#pragma once
#include <cuda_runtime.h>
#include "fcb_math.cuh"

namespace fcb {

template <typename T> __device__ __forceinline__ T dmin1(T a, T b) { return a < b ? a : b; }
template <typename T> __device__ __forceinline__ T dmax1(T a, T b) { return a > b ? a : b; }
template <typename T> __device__ __forceinline__ T sgn1(T x) { return copysign(T(1), x); }

// Whether padded cell (ic, jc) lies in the band of width mbc inside an mx x my patch that time
// interpolation fills (fclaw2d_clawpatch46_timeinterp.f:33-70).
__device__ __forceinline__ bool in_band(int ic, int jc, int mx, int my, int mbc)
{
    return ic >= mbc && ic < mx + mbc && jc >= mbc && jc < my + mbc &&
           (ic < 2 * mbc || ic >= mx || jc < 2 * mbc || jc >= my);
}

// Correctly rounded, uncontracted multiply / add.  The FP32-wave units are built with
// FMA contraction; the second-order correction must not be contracted, or the
// exactly opposite terms of the waves at a reflecting wall leave the rounding
// error of one product as a flux through the wall.
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float add_rn(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float sub_rn(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double add_rn(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double sub_rn(double a, double b) { return __dsub_rn(a, b); }

// min and max in one instruction that return NaN where an operand is NaN, as the comparisons of
// dmin1 and dmax1 do below (fminf and fmaxf return the other operand).
__device__ __forceinline__ float min_nan(float a, float b)
{
    float d;
    asm("min.NaN.f32 %0, %1, %2;" : "=f"(d) : "f"(a), "f"(b));
    return d;
}
__device__ __forceinline__ float max_nan(float a, float b)
{
    float d;
    asm("max.NaN.f32 %0, %1, %2;" : "=f"(d) : "f"(a), "f"(b));
    return d;
}

// ---------------------------------------------------------------------------
// 2D Euler, exact Riemann solver (no counterpart in the reference): the pressure function,
// fluxes and star pressure.  Newton iteration on p* (Toro, Riemann Solvers and Numerical
// Methods for Fluid Dynamics, ch. 4: pressure functions 4.6-4.7, PVRS start 4.47, sampling
// 4.5).  The interface solve is WaveEulerExact (wave_solvers.cuh).
// ---------------------------------------------------------------------------
struct RPEulerExact {
    __device__ static void prefun(double g1, double g4, double g5, double g6, double p, double rk, double pk,
                                  double ak, double& f, double& fd)
    {
        if (p <= pk) {
            const double prat = p / pk;
            const double z = fcb_exp(g1 * fcb_log(prat));
            f = g4 * ak * (z - 1.0);
            fd = (z / prat) / (rk * ak);
        } else {
            const double bk = g6 * pk;
            const double qrt = sqrt((g5 / rk) / (bk + p));
            f = (p - pk) * qrt;
            fd = (1.0 - 0.5 * (p - pk) / (bk + p)) * qrt;
        }
    }
    // FP32 pressure function for the FP32-wave form.  On the rarefaction side
    // z - 1 = (p/pk)^g1 - 1 comes from full-precision log1pf / expm1f (not the
    // fast-math exp/log), so weak waves, where p/pk is close to 1, keep their
    // relative accuracy.
    static constexpr float NEWTON_TOL32 = 4.0e-7f;
    __device__ static void prefun32(float g1, float g4, float g5, float g6, float p, float rk, float pk, float ak,
                                    float& f, float& fd)
    {
        if (p <= pk) {
            const float prat = p / pk;
            const float zm1 = expm1f(g1 * log1pf(prat - 1.0f));
            f = g4 * ak * zm1;
            fd = ((zm1 + 1.0f) / prat) / (rk * ak);
        } else {
            const float bk = g6 * pk;
            const float qrt = sqrtf((g5 / rk) / (bk + p));
            f = (p - pk) * qrt;
            fd = (1.0f - 0.5f * (p - pk) / (bk + p)) * qrt;
        }
    }
    __device__ static void eflux(double r, double u, double v, double p, double en, double* f)
    {
        f[0] = r * u;
        f[1] = r * u * u + p;
        f[2] = r * u * v;
        f[3] = u * (en + p);
    }
    // Euler flux of one cell in direction idir (0: x, 1: y), the time-sync rpn2_cons
    __device__ static void cons_flux(int idir, const double* q, double gam, double* flux)
    {
        const int mu = (idir == 0) ? 1 : 2, mv = (idir == 0) ? 2 : 1;
        const double r = q[0], un = q[mu] / r;
        const double p = (gam - 1.0) * (q[3] - 0.5 * (q[1] * q[1] + q[2] * q[2]) / r);
        flux[0] = q[mu];
        flux[mu] = q[mu] * un + p;
        flux[mv] = q[mv] * un;
        flux[3] = un * (q[3] + p);
    }
    // Primitive states of one interface (normal/tangential by ixy) and the PVRS start.
    struct Prim { double rl, ul, vl, pl, al, rr, ur, vr, pr, ar; };
    __device__ static Prim prim(int ixy, const double* qL, const double* qR, double gam)
    {
        const int mu = (ixy == 1) ? 1 : 2, mv = (ixy == 1) ? 2 : 1;
        const double gm1 = gam - 1.0;
        Prim w;
        w.rl = qL[0]; w.ul = qL[mu] / w.rl; w.vl = qL[mv] / w.rl;
        w.pl = gm1 * (qL[3] - 0.5 * (qL[mu] * qL[mu] + qL[mv] * qL[mv]) / w.rl);
        w.rr = qR[0]; w.ur = qR[mu] / w.rr; w.vr = qR[mv] / w.rr;
        w.pr = gm1 * (qR[3] - 0.5 * (qR[mu] * qR[mu] + qR[mv] * qR[mv]) / w.rr);
        w.al = sqrt(gam * w.pl / w.rl);
        w.ar = sqrt(gam * w.pr / w.rr);
        return w;
    }
    // Star pressure of primitive states (Newton from seed, or PVRS if seed <= 0).
    __device__ static double pstar(double rl, double ul, double pl, double rr, double ur, double pr, double gam,
                                   double tol, double seed, int& iters)
    {
        const double g1 = (gam - 1.0) / (2.0 * gam), g4 = 2.0 / (gam - 1.0), g5 = 2.0 / (gam + 1.0);
        const double g6 = (gam - 1.0) / (gam + 1.0);
        const double al = sqrt(gam * pl / rl), ar = sqrt(gam * pr / rr);
        const double du = ur - ul, tolpre = 1.0e-6;
        double p;
        if (seed > 0.0 && isfinite(seed)) p = seed;
        else {
            const double ppv = 0.5 * (pl + pr) - 0.125 * du * (rl + rr) * (al + ar);
            p = ppv > tolpre ? ppv : tolpre;
        }
        if (pl == pr && ul == ur) { iters = 0; return pl; }
        const bool seeded = seed > 0.0 && isfinite(seed);
        int it = 0;
        bool ok = false;
        for (int pass = 0; pass < (seeded ? 2 : 1) && !ok; pass++) {
            if (pass == 1) {        // the seed failed: start again from PVRS
                const double ppv = 0.5 * (pl + pr) - 0.125 * du * (rl + rr) * (al + ar);
                p = ppv > tolpre ? ppv : tolpre;
            }
            for (int k = 1; k <= 64; k++) {
                double fl, fdl, fr, fdr;
                prefun(g1, g4, g5, g6, p, rl, pl, al, fl, fdl);
                prefun(g1, g4, g5, g6, p, rr, pr, ar, fr, fdr);
                double pn = p - (fl + fr + du) / (fdl + fdr);
                if (pn < 0.0) pn = tolpre;
                const double change = 2.0 * fabs(pn - p) / (pn + p);
                p = pn;
                it++;
                if (change <= tol) { ok = true; break; }
            }
            ok = ok && isfinite(p);
        }
        iters = (it > 64 ? 64 : it) | (ok ? 0 : NEWTON_FAILED);
        return p;
    }
    // Returned with the iteration count when Newton converged neither from the seed nor from PVRS.
    static constexpr int NEWTON_FAILED = 0x100;
};

// clawpack46_inlinelimiter.f:59-104
template <typename T>
__device__ __forceinline__ T limiter_phi(int mthlim, T r)
{
    switch (mthlim) {
    case 1: return dmax1(T(0), dmin1(T(1), r));
    case 2: return dmax1(dmax1(T(0), dmin1(T(1), T(2) * r)), dmin1(T(2), r));
    case 3: return (r + fabs(r)) / (T(1) + fabs(r));
    case 4:
        if constexpr (sizeof(T) == 4) {
            // one instruction each.  A ratio of squared waves that overflow FP32 is inf/inf: its NaN
            // reaches q and the status word, where fminf and fmaxf gave the limiter 2 unnoticed.
            return max_nan(0.0f, min_nan(min_nan(fmaf(0.5f, r, 0.5f), 2.0f), 2.0f * r));
        } else {
            T c = (T(1) + r) / T(2);
            return dmax1(T(0), dmin1(dmin1(c, T(2)), T(2) * r));
        }
    case 5: return r;
    case 6: { T th = T((double)1.3f); return dmax1(T(0), dmin1(dmin1(th * r, (T(1) + r) / T(2)), th)); }
    default: return T(1);
    }
}

}  // namespace fcb
