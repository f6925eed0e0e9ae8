// wave_solvers.cuh -- Riemann solvers of the fused update of the flux-form systems
// (k_wave.cuh): shallow water (Roe, f-waves) and the exact Euler solver.
//
// A solver is split so that nothing is computed twice that a patch can share:
//   pre      per cell, once for both sweeps: square roots, sound speeds and velocities
//            (every cell is an operand of four interfaces);
//   normal   the Riemann solve of one interface from its two cells' states and pre values;
//            returns the Newton iterations of the exact solver.  The waves go to shared
//            memory for the limiters of the neighbours; State holds the little an interface
//            needs again after the barrier;
//   expand   waves and speeds after the barrier: the products of `normal` formed again from
//            State, or (Euler) read back through ow, cheaper than registers held meanwhile;
//   fluct    amdq and apdq;
//   split    the transverse solve of one fluctuation.
// Every expression has the operands and the order of the cited Fortran, so that the FP64
// instantiation (built without FMA contraction) gives the bits of the FP64 CPU path; what is
// dropped are additions of products with structurally zero wave components, which can only
// change the sign of a zero.
//
// wp<IXY>(mw, m): shared-memory plane of component m of wave mw, or -1 where it is zero.
// T = double, or float for the FP32-wave form, whose Godunov split takes amdq as the FP64
// remainder of the flux difference: amdq = (f(qR) - f(qL)) - apdq, with the cell fluxes of
// flux_planes / flux.
#pragma once
#include <cuda_runtime.h>
#include "riemann.cuh"

namespace fcb {

// Scalars of a launch every solver function may need; k: constants of the solver in shared
// memory (RP::NCONST of them, RP::constants), formed once per CTA.
template <typename T>
struct WavePar { T grav, drytol; double gamma, tol; const T* k; };

// normal (mu) and transverse (mv) momentum component of a sweep
template <int IXY> struct Dir { static constexpr int mu = IXY == 1 ? 1 : 2, mv = IXY == 1 ? 2 : 1; };

// ---------------------------------------------------------------------------
// Shallow water, Roe solver with Harten-Hyman entropy fix.
// applications/clawpack/shallow/2d/rp/clawpack46_rpn2.f:1-247, clawpack46_rpt2.f:248-321
// ---------------------------------------------------------------------------
struct WaveShallowRoe {
    static constexpr int MEQN = 3, MWAVES = 3, MAUX = 0, NPRE = 3, NW = 7, NFL = 3, NCONST = 0;
    static constexpr bool FWAVE = false, DEPTH = true, EXACT = false;
    enum { P_RS = 0, P_N1 = 1, P_N2 = 2 };   // sqrt h, (hu, hv)/sqrt h
    template <int IXY> __host__ __device__ static constexpr int wp(int mw, int m)
    {
        return mw == 0 ? m : mw == 2 ? 4 + m : m == Dir<IXY>::mv ? 3 : -1;
    }
    template <typename T> __device__ static void pre(const T* q, const WavePar<T>& P, T* c)
    {
        const T rs = sqrt(q[0]);
        c[P_RS] = rs; c[P_N1] = q[1] / rs; c[P_N2] = q[2] / rs;
    }
    // Whether |hu|/h can reach sqrt(g h): false only where hu^2 is clearly below g h^3 (one per
    // cent, far beyond rounding), so the caller's exact test of hu/h -+ sqrt(g h) would fail too.
    template <typename T> __device__ __forceinline__ static bool fast(T h, T hu, T grav)
    {
        return !(hu * hu < T(0.99) * (grav * (h * (h * h))));
    }
    // FP64 cell fluxes of the FP32-wave form: f_x = (hu, F0, F2), f_y = (hv, F2, F1)
    __device__ static void flux_planes(const double* q, const WavePar<float>&, double grav, double* f)
    {
        const double inv = 1.0 / q[0];
        f[0] = q[1] * q[1] * inv + 0.5 * grav * q[0] * q[0];
        f[1] = q[2] * q[2] * inv + 0.5 * grav * q[0] * q[0];
        f[2] = q[1] * q[2] * inv;
    }
    // plane of component m of the flux in direction IXY: a q plane (< MEQN) or MEQN + flux plane
    template <int IXY> __host__ __device__ static constexpr int flux_plane(int m)
    {
        return m == 0 ? Dir<IXY>::mu : m == Dir<IXY>::mu ? 3 + (IXY - 1) : 3 + 2;
    }
    template <typename T> struct State { T a1, a2, a3, u, v, a, am[3]; };
    template <int IXY, typename T, class C>
    __device__ static int normal(const T* qL, const T* qR, const T* dq, const T* aL, const T* aR, const T* da, C cL, C cR,
                                 const WavePar<T>& P, double, State<T>& st, T w[3][3], T* s)
    {
        (void)dq; (void)aL; (void)aR; (void)da;
        constexpr int mu = Dir<IXY>::mu, mv = Dir<IXY>::mv;
        constexpr int NN = IXY == 1 ? P_N1 : P_N2, NT = IXY == 1 ? P_N2 : P_N1;
        // :91-99
        const T h = (qL[0] + qR[0]) / T(2);
        const T hsq2 = cL(P_RS) + cR(P_RS);
        const T u = (cL(NN) + cR(NN)) / hsq2;
        const T v = (cL(NT) + cR(NT)) / hsq2;
        const T a = sqrt(P.grav * h);
        // :105-129
        const T d1 = qR[0] - qL[0], d2 = qR[mu] - qL[mu], d3 = qR[mv] - qL[mv];
        const T a1 = ((u + a) * d1 - d2) / (T(2) * a);
        const T a2 = -(v * d1) + d3;
        T a3;
        if constexpr (sizeof(T) == 4) { a3 = d1 - a1; }           // the two acoustic strengths sum to d1
        else { a3 = (-((u - a) * d1) + d2) / (T(2) * a); }
        st.a1 = a1; st.a2 = a2; st.a3 = a3; st.u = u; st.v = v; st.a = a;
        const T sl = u - a, sr = u + a;
        const T w0n = a1 * sl, w0t = a1 * v, w2n = a3 * sr, w2t = a3 * v;
        // entropy fix :170-229.  The characteristic speeds of the cells and the middle states (a
        // quotient and a square root each) decide only supersonic and transonic interfaces, and
        // are formed only where one is possible.
        T am[3] = {T(0), T(0), T(0)};
        auto speed = [&](T h_, T hu_, T sign) { return hu_ / h_ + sign * sqrt(P.grav * h_); };
        if (!(sl > T(0) && speed(qL[0], qL[mu], T(-1)) > T(0))) {
            const T h1 = qL[0] + a1, hu1 = qL[mu] + w0n;
            T sf = sl < T(0) ? sl : T(0);
            if (hu1 > T(0) && fast(h1, hu1, P.grav)) {
                const T s1 = speed(h1, hu1, T(-1)), s0 = speed(qL[0], qL[mu], T(-1));
                if (s0 < T(0) && s1 > T(0)) sf = s0 * ((s1 - sl) / (s1 - s0));
            }
            am[0] = sf * a1; am[mu] = sf * w0n; am[mv] = sf * w0t;
            if (!(u > T(0))) {
                am[mv] = am[mv] + u * a2;
                const T h3 = qR[0] - a3, hu3 = qR[mu] - w2n;
                sf = sr;
                bool third = sr < T(0);
                if (hu3 < T(0) && fast(h3, hu3, P.grav)) {
                    const T s3 = speed(h3, hu3, T(1)), s03 = speed(qR[0], qR[mu], T(1));
                    if (s3 < T(0) && s03 > T(0)) { sf = s3 * ((s03 - sr) / (s03 - s3)); third = true; }
                }
                if (third) {
                    am[0] = am[0] + sf * a3; am[mu] = am[mu] + sf * w2n; am[mv] = am[mv] + sf * w2t;
                }
            }
        }
        for (int m = 0; m < 3; m++) st.am[m] = am[m];
        expand<IXY>(st, 0, w, s);
        return 0;
    }
    // waves and speeds of the interface
    template <int IXY, typename T, class OW>
    __device__ static void expand(const State<T>& st, OW, T w[3][3], T* s)
    {
        constexpr int mu = Dir<IXY>::mu, mv = Dir<IXY>::mv;
        s[0] = st.u - st.a; s[1] = st.u; s[2] = st.u + st.a;
        w[0][0] = st.a1; w[0][mu] = st.a1 * s[0]; w[0][mv] = st.a1 * st.v;
        w[1][0] = T(0); w[1][mu] = T(0); w[1][mv] = st.a2;
        w[2][0] = st.a3; w[2][mu] = st.a3 * s[2]; w[2][mv] = st.a3 * st.v;
    }
    // :234-242
    template <int IXY, typename T>
    __device__ static void fluct(const State<T>& st, const T w[3][3], const T* s, T* am, T* ap)
    {
        for (int m = 0; m < 3; m++) {
            T df = s[0] * w[0][m];
            if (wp<IXY>(1, m) >= 0) df = df + s[1] * w[1][m];
            df = df + s[2] * w[2][m];
            am[m] = st.am[m];
            ap[m] = df - st.am[m];
        }
    }
    // shared part of the two transverse solves of an interface
    template <typename T> struct Split { T u, v, a; };
    template <int IXY, typename T, class QC, class AC>
    __device__ static Split<T> split_state(const State<T>& st, QC, AC, const WavePar<T>&) { return {st.u, st.v, st.a}; }
    template <int IXY, typename T, class AC>
    __device__ static void split(const Split<T>& e, int imp, AC, const T* asdq, T* bm, T* bp)
    {
        (void)imp;
        constexpr int mu = Dir<IXY>::mu, mv = Dir<IXY>::mv;
        const T u = e.u, v = e.v, a = e.a;
        const T a1 = ((v + a) * asdq[0] - asdq[mv]) / (T(2) * a);
        const T a2 = asdq[mu] - u * asdq[0];
        const T a3 = (-((v - a) * asdq[0]) + asdq[mv]) / (T(2) * a);
        const T sb0 = v - a, sb1 = v, sb2 = v + a;
        if (sb0 < T(0) && sb2 > T(0)) {
            // subcritical, the rule: the outer waves go one way each (the products left out are
            // zeros)
            const T m1 = dmin1(sb1, T(0)) * a2, p1 = dmax1(sb1, T(0)) * a2;
            bm[0] = sb0 * a1; bp[0] = sb2 * a3;
            bm[mu] = sb0 * (a1 * u) + m1; bp[mu] = p1 + sb2 * (a3 * u);
            bm[mv] = sb0 * (a1 * sb0); bp[mv] = sb2 * (a3 * sb2);
            return;
        }
        const T m0 = dmin1(sb0, T(0)), m1 = dmin1(sb1, T(0)), m2 = dmin1(sb2, T(0));
        const T p0 = dmax1(sb0, T(0)), p1 = dmax1(sb1, T(0)), p2 = dmax1(sb2, T(0));
        const T w0u = a1 * u, w0v = a1 * sb0, w2u = a3 * u, w2v = a3 * sb2;
        bm[0] = m0 * a1 + m2 * a3;
        bp[0] = p0 * a1 + p2 * a3;
        bm[mu] = (m0 * w0u + m1 * a2) + m2 * w2u;
        bp[mu] = (p0 * w0u + p1 * a2) + p2 * w2u;
        bm[mv] = m0 * w0v + m2 * w2v;
        bp[mv] = p0 * w0v + p2 * w2v;
    }
    // flux of the time-sync store (applications/clawpack/shallow/2d/radialdam/rpn2cons_update.f)
    __device__ static void cons_flux(int idir, const double* q, double grav, double, double* f)
    {
        const int mu = (idir == 0) ? 1 : 2, mv = (idir == 0) ? 2 : 1;
        const double hun = q[mu], hut = q[mv], h = q[0];
        const double un = hun / h;
        f[0] = hun;
        f[mu] = (hun * hun) / h + 0.5 * grav * (h * h);
        f[mv] = un * hut;
    }
    // source part of the flux difference in the FP32-wave form: none
    template <int IXY> __device__ static double source(int, double, double, double, double, double) { return 0.0; }
    static constexpr bool SOURCE = false;
};

// ---------------------------------------------------------------------------
// Shallow water f-waves with bathymetry b = aux(:,:,1).
// applications/clawpack/shallow/2d/rp/rpn2_tsunami.f90:3-222, rpt2_tsunami.f90:3-170
// ---------------------------------------------------------------------------
struct WaveShallowFWave {
    static constexpr int MEQN = 3, MWAVES = 3, MAUX = 1, NPRE = 6, NW = 7, NFL = 3, NCONST = 0;
    static constexpr bool FWAVE = true, DEPTH = true, EXACT = false;
    enum { P_RS = 0, P_C = 1, P_U1 = 2, P_U2 = 3, P_E1 = 4, P_E2 = 5 };   // sqrt h, sqrt gh, (hu, hv)/h, (hu^2, hv^2)/h
    template <int IXY> __host__ __device__ static constexpr int wp(int mw, int m)
    {
        return mw == 0 ? m : mw == 2 ? 4 + m : m == Dir<IXY>::mv ? 3 : -1;
    }
    template <typename T> __device__ static void pre(const T* q, const WavePar<T>& P, T* c)
    {
        c[P_RS] = sqrt(q[0]);
        c[P_C] = sqrt(P.grav * q[0]);
        c[P_U1] = q[1] / q[0]; c[P_U2] = q[2] / q[0];
        c[P_E1] = (q[1] * q[1]) / q[0]; c[P_E2] = (q[2] * q[2]) / q[0];
    }
    __device__ static void flux_planes(const double* q, const WavePar<float>& P, double grav, double* f)
    {
        WaveShallowRoe::flux_planes(q, P, grav, f);
    }
    template <int IXY> __host__ __device__ static constexpr int flux_plane(int m)
    {
        return WaveShallowRoe::flux_plane<IXY>(m);
    }
    // t1, t2, t3: speeds of the transverse solve; dry: both cells below the tolerance
    template <typename T> struct State { T b1, b2, b3, s1, s3, vL, vR, t1, t2, t3; bool dry; };
    template <int IXY, typename T, class C>
    __device__ static int normal(const T* qL, const T* qR, const T* dq, const T* aL, const T* aR, const T* da, C cL, C cR,
                                 const WavePar<T>& P, double, State<T>& st, T w[3][3], T* s)
    {
        constexpr int UN = IXY == 1 ? P_U1 : P_U2, UT = IXY == 1 ? P_U2 : P_U1, EN = IXY == 1 ? P_E1 : P_E2;
        const T grav = P.grav;
        const T hL = qL[0], hR = qR[0];
        const T uR = cR(UN), vR = cR(UT), uL = cL(UN), vL = cL(UT);
        const T gL = cL(P_C), gR = cR(P_C);
        const T uhat = (gL * uL + gR * uR) / (gR + gL);
        const T chat = sqrt(grav * T(0.5) * (hR + hL));
        const T hbar = T(0.5) * (hR + hL);
        T fd1, fd2;
        if constexpr (sizeof(T) == 4) {
            // FP32: from the FP64 differences; g/2 (hR^2 - hL^2) is g hbar (hR - hL), so still
            // water over any bottom balances to the rounding of h + b
            fd1 = dq[IXY];
            fd2 = grav * hbar * (dq[0] + da[0]) + (cR(EN) - cL(EN));
        } else {
            const T phiR = T(0.5) * grav * (hR * hR) + cR(EN);
            const T phiL = T(0.5) * grav * (hL * hL) + cL(EN);
            fd1 = (hR * uR) - (hL * uL);
            fd2 = phiR - phiL + grav * hbar * (aR[0] - aL[0]);
        }
        const T fd3 = hR * uR * vR - hL * uL * vL;
        const T s1 = fmin(uL - gL, uhat - chat);
        const T s3 = fmax(uR + gR, uhat + chat);
        st.b1 = -(fd2 - s3 * fd1) / (s3 - s1);
        if constexpr (sizeof(T) == 4) { st.b3 = fd1 - st.b1; }    // the two strengths sum to fd1
        else { st.b3 = (fd2 - s1 * fd1) / (s3 - s1); }
        st.b2 = fd3 - st.b1 * vL - st.b3 * vR;
        st.s1 = s1; st.s3 = s3; st.vL = vL; st.vR = vR;
        // speeds of the transverse solve (rpt2_tsunami.f90:60-118), the same for both
        // fluctuations; between wet cells its celerity is chat, and in FP32 its velocities are
        // averaged with the weights at hand (sqrt(g h) in place of sqrt h)
        const bool dl = hL < P.drytol, dr = hR < P.drytol;
        const T hl = dl ? T(0) : hL, hr = dr ? T(0) : hR;
        st.dry = hl <= P.drytol && hr <= P.drytol;
        const bool wet = !dl && !dr;
        T vhat, ct = chat;
        if (sizeof(T) == 4 && wet) {
            vhat = (gL * vL + gR * vR) / (gR + gL);
            st.t2 = uhat;
        } else {
            const T ul = dl ? T(0) : uL, vl = dl ? T(0) : vL, ur = dr ? T(0) : uR, vr = dr ? T(0) : vR;
            const T rl = dl ? T(0) : cL(P_RS), rr = dr ? T(0) : cR(P_RS);
            const T rs = rr + rl;
            vhat = (vr * rr) / rs + (vl * rl) / rs;
            st.t2 = (ur * rr) / rs + (ul * rl) / rs;
            if (!wet) ct = sqrt(grav * ((hr + hl) / T(2)));
        }
        st.t1 = fmin(vhat - ct, (dl ? T(0) : vL) - (dl ? T(0) : gL));
        st.t3 = fmax(vhat + ct, (dr ? T(0) : vR) + (dr ? T(0) : gR));
        expand<IXY>(st, 0, w, s);
        return 0;
    }
    template <int IXY, typename T, class OW>
    __device__ static void expand(const State<T>& st, OW, T w[3][3], T* s)
    {
        constexpr int mu = Dir<IXY>::mu, mv = Dir<IXY>::mv;
        s[0] = st.s1; s[1] = T(0.5) * (st.s1 + st.s3); s[2] = st.s3;
        w[0][0] = st.b1; w[0][mu] = st.b1 * st.s1; w[0][mv] = st.b1 * st.vL;
        w[1][0] = T(0); w[1][mu] = T(0); w[1][mv] = st.b2;
        w[2][0] = st.b3; w[2][mu] = st.b3 * st.s3; w[2][mv] = st.b3 * st.vR;
    }
    // a wave goes left or right by the sign bit of its speed: (1 -+ sgn s)/2 is 0 or 1
    template <int IXY, typename T>
    __device__ static void fluct(const State<T>&, const T w[3][3], const T* s, T* am, T* ap)
    {
        const bool n0 = signbit(s[0]), n1 = signbit(s[1]), n2 = signbit(s[2]);
        for (int m = 0; m < 3; m++) {
            T l = n0 ? w[0][m] : T(0), r = n0 ? T(0) : w[0][m];
            if (wp<IXY>(1, m) >= 0) { l = l + (n1 ? w[1][m] : T(0)); r = r + (n1 ? T(0) : w[1][m]); }
            am[m] = l + (n2 ? w[2][m] : T(0));
            ap[m] = r + (n2 ? T(0) : w[2][m]);
        }
    }
    template <typename T> struct Split { T t1, t2, t3, hL, hR; bool dry; };
    template <int IXY, typename T, class QC, class AC>
    __device__ static Split<T> split_state(const State<T>& st, QC depth, AC, const WavePar<T>&)
    {
        return {st.t1, st.t2, st.t3, depth(0), depth(1), st.dry};
    }
    // aux(k, imp): bathymetry of the fluctuation's cell (k = 1) and of the cells below (0) and above (2)
    template <int IXY, typename T, class AC>
    __device__ static void split(const Split<T>& e, int imp, AC aux, const T* asdq, T* bm, T* bp)
    {
        constexpr int mu = Dir<IXY>::mu, mv = Dir<IXY>::mv;
        bool skip = e.dry;
        if (!skip) {
            const T eta = (imp == 1 ? e.hL : e.hR) + aux(1, imp);
            skip = eta < fmax(aux(0, imp), aux(2, imp));
        }
        if (skip) {
            for (int m = 0; m < 3; m++) { bm[m] = T(0); bp[m] = T(0); }
            return;
        }
        const T s1 = e.t1, s2 = e.t2, s3 = e.t3;
        const T d1 = asdq[0], d2 = asdq[mu], d3 = asdq[mv];
        T b0, b2;
        if constexpr (sizeof(T) == 4) {
            b0 = (s3 * d1 - d3) / (s3 - s1);
            b2 = d1 - b0;
        } else {
            b0 = (s3 * d1 / (s3 - s1)) - (d3 / (s3 - s1));
            b2 = (d3 / (s3 - s1)) - (s1 * d1 / (s3 - s1));
        }
        const T b1 = -(s2 * d1) + d2;
        const T g0 = s1 * b0, g1 = s2 * b1, g2 = s3 * b2;
        const bool n0 = signbit(s1), n1 = signbit(s2), n2 = signbit(s3);
        const T m0 = n0 ? g0 : T(0), m1 = n1 ? g1 : T(0), m2 = n2 ? g2 : T(0);
        const T p0 = n0 ? T(0) : g0, p1 = n1 ? T(0) : g1, p2 = n2 ? T(0) : g2;
        bm[0] = m0 + m2; bp[0] = p0 + p2;
        bm[mu] = (m0 * s2 + m1) + m2 * s2; bp[mu] = (p0 * s2 + p1) + p2 * s2;
        bm[mv] = m0 * s1 + m2 * s3; bp[mv] = p0 * s1 + p2 * s3;
    }
    __device__ static void cons_flux(int idir, const double* q, double grav, double gamma, double* f)
    {
        WaveShallowRoe::cons_flux(idir, q, grav, gamma, f);
    }
    // f-waves sum to the flux difference plus the source g hbar (bR - bL) of the normal momentum
    static constexpr bool SOURCE = true;
    template <int IXY> __device__ static double source(int m, double hL, double hR, double bL, double bR, double grav)
    {
        return m == Dir<IXY>::mu ? grav * (0.5 * (hR + hL)) * (bR - bL) : 0.0;
    }
};

// ---------------------------------------------------------------------------
// 2D Euler, exact Riemann solver (RPEulerExact in riemann.cuh has the pressure function and
// the sources): Newton on p*,
//   amdq = F(q0) - F(qL), apdq = F(qR) - F(q0), q0 the Godunov state at x/t = 0,
//   waves w1 = q*L - qL, w2 = q*R - q*L, w3 = qR - q*R,
//   speeds s1 = left shock speed or rarefaction head, s2 = u*, s3 the right one.
// The Roe averages (clawpack46_rpn2_euler4.f:83-100) serve the transverse solver
// clawpack46_rpt2_euler4.f:56-94.  The waves stay in shared memory between the phases.
// ---------------------------------------------------------------------------
struct WaveEulerExact {
    static constexpr int MEQN = 4, MWAVES = 3, MAUX = 0, NPRE = 8, NW = 12, NFL = 5, NCONST = 7;
    static constexpr bool FWAVE = false, DEPTH = false, EXACT = true, SOURCE = false;
    static constexpr int NEWTON_FAILED = RPEulerExact::NEWTON_FAILED;
    // velocities, pressure, sound speed, sqrt rho, (rho u, rho v, E + p)/sqrt rho
    enum { P_U1 = 0, P_U2 = 1, P_P = 2, P_A = 3, P_RS = 4, P_N1 = 5, P_N2 = 6, P_H = 7 };
    template <int IXY> __host__ __device__ static constexpr int wp(int mw, int m) { return 4 * mw + m; }
    // functions of gamma (Toro's G1..G7)
    template <typename T> __device__ static void constants(T gam, T* k)
    {
        k[0] = (gam - T(1)) / (T(2) * gam); k[1] = (gam + T(1)) / (T(2) * gam);
        k[2] = T(2) * gam / (gam - T(1)); k[3] = T(2) / (gam - T(1)); k[4] = T(2) / (gam + T(1));
        k[5] = (gam - T(1)) / (gam + T(1)); k[6] = (gam - T(1)) / T(2);
    }
    __device__ static void pre(const double* q, const WavePar<double>& P, double* c)
    {
        const double gamma1 = P.gamma - 1.0, r = q[0];
        const double p = gamma1 * (q[3] - 0.5 * (q[1] * q[1] + q[2] * q[2]) / r);
        const double rs = sqrt(r);
        c[P_U1] = q[1] / r; c[P_U2] = q[2] / r; c[P_P] = p; c[P_A] = sqrt(P.gamma * p / r);
        c[P_RS] = rs; c[P_N1] = q[1] / rs; c[P_N2] = q[2] / rs; c[P_H] = (q[3] + p) / rs;
    }
    // FP32: the primitive state with correctly rounded, uncontracted operations
    __device__ static void pre(const float* q, const WavePar<float>& P, float* c)
    {
        const float gam = (float)P.gamma, gamma1 = gam - 1.0f, r = q[0];
        const float ke = __fdiv_rn(__fmul_rn(0.5f, __fadd_rn(__fmul_rn(q[1], q[1]), __fmul_rn(q[2], q[2]))), r);
        const float p = __fmul_rn(gamma1, __fsub_rn(q[3], ke));
        const float rs = sqrtf(r);
        c[P_U1] = __fdiv_rn(q[1], r); c[P_U2] = __fdiv_rn(q[2], r); c[P_P] = p; c[P_A] = sqrtf(gam * p / r);
        c[P_RS] = rs; c[P_N1] = q[1] / rs; c[P_N2] = q[2] / rs; c[P_H] = (q[3] + p) / rs;
    }
    // FP64 cell fluxes of the FP32-wave form: f_x = (m1, F0, F2, F3), f_y = (m2, F2, F1, F4)
    __device__ static void flux_planes(const double* q, const WavePar<float>& P, double, double* f)
    {
        const double u = q[1] / q[0], v = q[2] / q[0];
        const double p = (P.gamma - 1.0) * (q[3] - 0.5 * (q[1] * q[1] + q[2] * q[2]) / q[0]);
        f[0] = q[1] * u + p; f[1] = q[2] * v + p; f[2] = q[2] * u;
        f[3] = u * (q[3] + p); f[4] = v * (q[3] + p);
    }
    template <int IXY> __host__ __device__ static constexpr int flux_plane(int m)
    {
        return m == 0 ? Dir<IXY>::mu : m == Dir<IXY>::mu ? 4 + (IXY - 1) : m == Dir<IXY>::mv ? 4 + 2 : 4 + 3 + (IXY - 1);
    }
    // FP64: am, ap.  FP32: the Godunov flux f0 (src 0), or the flux of the left (1) or right
    // (2) cell where the states do not jump in p and u.
    template <typename T> struct State { T s[3], ex[5], f[8]; int src; };
    template <int IXY, typename T, class OW>
    __device__ static void expand(const State<T>& st, OW ow, T w[3][4], T* s)
    {
        for (int mw = 0; mw < 3; mw++) {
            s[mw] = st.s[mw];
            for (int m = 0; m < 4; m++) w[mw][m] = ow(4 * mw + m);
        }
    }
    template <int IXY>
    __device__ static void fluct(const State<double>& st, const double[3][4], const double*, double* am, double* ap)
    {
        for (int m = 0; m < 4; m++) { am[m] = st.f[m]; ap[m] = st.f[4 + m]; }
    }
    // FP32: amdq and apdq in FP64 from the cell fluxes
    __device__ static void fluct_mixed(const State<float>& st, int m, double fL, double fR, double& am, double& ap)
    {
        const double f = st.src == 0 ? (double)st.f[m] : st.src == 1 ? fL : fR;
        am = f - fL;
        ap = fR - f;
    }
    template <int IXY, typename T, class C>
    __device__ static void roe(const T* qL, const T* qR, C cL, C cR, T gamma1, T* ex)
    {
        constexpr int NN = IXY == 1 ? P_N1 : P_N2, NT = IXY == 1 ? P_N2 : P_N1;
        const T rhsq2 = cL(P_RS) + cR(P_RS);
        const T u = (cL(NN) + cR(NN)) / rhsq2;
        const T v = (cL(NT) + cR(NT)) / rhsq2;
        const T enth = (cL(P_H) + cR(P_H)) / rhsq2;
        const T a2 = gamma1 * (enth - T(0.5) * (u * u + v * v));
        ex[0] = u; ex[1] = v; ex[2] = enth; ex[3] = sqrt(a2); ex[4] = gamma1 / a2;
    }
    template <int IXY, class C>
    __device__ static int normal(const double* qL, const double* qR, const double*, const double*, const double*, const double*, C cL, C cR,
                                 const WavePar<double>& P, double seed, State<double>& st, double w[3][4], double* s)
    {
        constexpr int mu = Dir<IXY>::mu, mv = Dir<IXY>::mv;
        constexpr int UN = IXY == 1 ? P_U1 : P_U2, UT = IXY == 1 ? P_U2 : P_U1;
        const double gam = P.gamma, gamma1 = gam - 1.0;
        roe<IXY>(qL, qR, cL, cR, gamma1, st.ex);
        const double g1 = P.k[0], g2 = P.k[1], g3 = P.k[2], g4 = P.k[3], g5 = P.k[4], g6 = P.k[5], g7 = P.k[6];
        const double rl = qL[0], ul = cL(UN), vl = cL(UT), pl = cL(P_P), al = cL(P_A);
        const double rr = qR[0], ur = cR(UN), vr = cR(UT), pr = cR(P_P), ar = cR(P_A);
        const double du = ur - ul;
        const double tolpre = 1.0e-6;
        const bool seeded = seed > 0.0 && isfinite(seed);
        const double ppv = 0.5 * (pl + pr) - 0.125 * du * (rl + rr) * (al + ar);
        double p = seeded ? seed : ppv > tolpre ? ppv : tolpre;
        double fl = 0.0, fr = 0.0, fdl, fdr;
        int it = 0;
        bool ok = true;
        if (pl == pr && ul == ur) {
            // no pressure or normal-velocity jump: p* = p, u* = u exactly (the first
            // Newton step's values, bit for bit), no iteration
            p = pl;
        } else {
            // Newton from the seed; where it does not converge, again from PVRS
            ok = false;
            for (int pass = 0; pass < (seeded ? 2 : 1) && !ok; pass++) {
                if (pass == 1) p = ppv > tolpre ? ppv : tolpre;
                for (int k = 1; k <= 64; k++) {
                    RPEulerExact::prefun(g1, g4, g5, g6, p, rl, pl, al, fl, fdl);
                    RPEulerExact::prefun(g1, g4, g5, g6, p, rr, pr, ar, fr, fdr);
                    double pn = p - (fl + fr + du) / (fdl + fdr);
                    if (pn < 0.0) pn = tolpre;
                    const double change = 2.0 * fabs(pn - p) / (pn + p);
                    p = pn;
                    it++;
                    if (change <= P.tol) { ok = true; break; }
                }
                ok = ok && isfinite(p);
            }
            if (it > 64) it = 64;
        }
        const double ps = p;
        const double us = 0.5 * (ul + ur) + 0.5 * (fr - fl);
        // star densities and sound speeds (p* = pK: rhoK, aK exactly, as log 1 = 0, exp 0 = 1)
        double rsl, rsr, asl, asr;
        if (ps > pl) { const double q = ps / pl; rsl = rl * ((q + g6) / (g6 * q + 1.0)); asl = sqrt(gam * ps / rsl); }
        else if (ps == pl) { rsl = rl; asl = al; }
        else { const double lq = fcb_log(ps / pl); rsl = rl * fcb_exp(lq / gam); asl = al * fcb_exp(g1 * lq); }
        if (ps > pr) { const double q = ps / pr; rsr = rr * ((q + g6) / (g6 * q + 1.0)); asr = sqrt(gam * ps / rsr); }
        else if (ps == pr) { rsr = rr; asr = ar; }
        else { const double lq = fcb_log(ps / pr); rsr = rr * fcb_exp(lq / gam); asr = ar * fcb_exp(g1 * lq); }
        const double shl = ul - al, shr = ur + ar;
        const double sl = ps > pl ? ul - al * sqrt(g2 * (ps / pl) + g1) : shl;
        const double sr = ps > pr ? ur + ar * sqrt(g2 * (ps / pr) + g1) : shr;
        s[0] = sl; s[1] = us; s[2] = sr;
        for (int mw = 0; mw < 3; mw++) st.s[mw] = s[mw];
        const double esl = ps / gamma1 + 0.5 * rsl * (us * us + vl * vl);
        const double esr = ps / gamma1 + 0.5 * rsr * (us * us + vr * vr);
        // waves in (rho, m_n, m_t, E) order, stored at the natural components
        const double qln[4] = {qL[0], qL[mu], qL[mv], qL[3]}, qrn[4] = {qR[0], qR[mu], qR[mv], qR[3]};
        const double qsl[4] = {rsl, rsl * us, rsl * vl, esl};
        const double qsr[4] = {rsr, rsr * us, rsr * vr, esr};
        constexpr int comp[4] = {0, mu, mv, 3};
        for (int k = 0; k < 4; k++) {
            w[0][comp[k]] = qsl[k] - qln[k];
            w[1][comp[k]] = qsr[k] - qsl[k];
            w[2][comp[k]] = qrn[k] - qsr[k];
        }
        // Godunov state at x/t = 0
        double r0, u0, v0, p0, e0;
        int which;
        if (0.0 <= us) {
            v0 = vl;
            if (ps > pl) which = (0.0 <= sl) ? 0 : 1;
            else if (0.0 <= shl) which = 0;
            else which = (0.0 > us - asl) ? 1 : 2;
        } else {
            v0 = vr;
            if (ps > pr) which = (0.0 >= sr) ? 4 : 3;
            else if (0.0 >= shr) which = 4;
            else which = (0.0 < us + asr) ? 3 : 5;
        }
        if (which == 0) { r0 = rl; u0 = ul; p0 = pl; e0 = qL[3]; }
        else if (which == 4) { r0 = rr; u0 = ur; p0 = pr; e0 = qR[3]; }
        else if (which == 1) { r0 = rsl; u0 = us; p0 = ps; e0 = esl; }
        else if (which == 3) { r0 = rsr; u0 = us; p0 = ps; e0 = esr; }
        else if (which == 2) {
            const double c = g5 + (g6 / al) * ul;
            const double lc = fcb_log(c);
            r0 = rl * fcb_exp(g4 * lc);
            u0 = g5 * (al + g7 * ul);
            p0 = pl * fcb_exp(g3 * lc);
            e0 = p0 / gamma1 + 0.5 * r0 * (u0 * u0 + v0 * v0);
        } else {
            const double c = g5 - (g6 / ar) * ur;
            const double lc = fcb_log(c);
            r0 = rr * fcb_exp(g4 * lc);
            u0 = g5 * (-ar + g7 * ur);
            p0 = pr * fcb_exp(g3 * lc);
            e0 = p0 / gamma1 + 0.5 * r0 * (u0 * u0 + v0 * v0);
        }
        double f0[4], flv[4], frv[4];
        RPEulerExact::eflux(r0, u0, v0, p0, e0, f0);
        RPEulerExact::eflux(rl, ul, vl, pl, qL[3], flv);
        RPEulerExact::eflux(rr, ur, vr, pr, qR[3], frv);
        for (int k = 0; k < 4; k++) { st.f[comp[k]] = f0[k] - flv[k]; st.f[4 + comp[k]] = frv[k] - f0[k]; }
        return it | (ok ? 0 : NEWTON_FAILED);
    }
    // FP32-wave form: primitive states, Roe averages, the Newton iteration on p* (only where p
    // or u jumps), star states, the Godunov state and the waves in FP32.  FP32 resolves p* to a
    // few ulp, so the iteration stops at a relative change of max(tol, NEWTON_TOL32).
    template <int IXY, class C>
    __device__ static int normal(const float* qL, const float* qR, const float*, const float*, const float*, const float*, C cL, C cR,
                                 const WavePar<float>& P, double seed, State<float>& st, float w[3][4], float* s)
    {
        constexpr int mu = Dir<IXY>::mu, mv = Dir<IXY>::mv;
        constexpr int UN = IXY == 1 ? P_U1 : P_U2, UT = IXY == 1 ? P_U2 : P_U1;
        const float gam = (float)P.gamma, gamma1 = gam - 1.0f;
        roe<IXY>(qL, qR, cL, cR, gamma1, st.ex);
        const float g1 = P.k[0], g2 = P.k[1], g3 = P.k[2], g4 = P.k[3], g5 = P.k[4], g6 = P.k[5], g7 = P.k[6];
        const float rl = qL[0], ul = cL(UN), vl = cL(UT), pl = cL(P_P), al = cL(P_A);
        const float rr = qR[0], ur = cR(UN), vr = cR(UT), pr = cR(P_P), ar = cR(P_A);
        int it = 0;
        bool ok = true;
        float ps, us;
        const bool nojump = (pl == pr && ul == ur);
        if (nojump) {
            ps = pl; us = ul;
        } else {
            const float du = ur - ul, tolpre = 1.0e-6f;
            const bool seeded = seed > 0.0 && isfinite(seed);
            const float ppv = 0.5f * (pl + pr) - 0.125f * du * (rl + rr) * (al + ar);
            float p = seeded ? (float)seed : ppv > tolpre ? ppv : tolpre;
            const float tol = fmaxf((float)P.tol, RPEulerExact::NEWTON_TOL32);
            float fl = 0.0f, fr = 0.0f, fdl, fdr;
            bool conv = false;
            for (int pass = 0; pass < (seeded ? 2 : 1) && !conv; pass++) {
                if (pass == 1) p = ppv > tolpre ? ppv : tolpre;
                for (int k = 1; k <= 64; k++) {
                    RPEulerExact::prefun32(g1, g4, g5, g6, p, rl, pl, al, fl, fdl);
                    RPEulerExact::prefun32(g1, g4, g5, g6, p, rr, pr, ar, fr, fdr);
                    float pn = p - (fl + fr + du) / (fdl + fdr);
                    if (pn < 0.0f) pn = tolpre;
                    const float change = 2.0f * fabsf(pn - p) / (pn + p);
                    p = pn;
                    it++;
                    if (change <= tol) { conv = true; break; }
                }
                conv = conv && isfinite(p);
            }
            ok = conv;
            if (it > 64) it = 64;
            ps = p;
            us = 0.5f * (ul + ur) + 0.5f * (fr - fl);
        }
        float rsl, rsr, asl, asr;
        if (ps > pl) { const float q = ps / pl; rsl = rl * ((q + g6) / (g6 * q + 1.0f)); asl = sqrtf(gam * ps / rsl); }
        else if (ps == pl) { rsl = rl; asl = al; }
        else { const float lq = __logf(ps / pl); rsl = rl * __expf(lq / gam); asl = al * __expf(g1 * lq); }
        if (ps > pr) { const float q = ps / pr; rsr = rr * ((q + g6) / (g6 * q + 1.0f)); asr = sqrtf(gam * ps / rsr); }
        else if (ps == pr) { rsr = rr; asr = ar; }
        else { const float lq = __logf(ps / pr); rsr = rr * __expf(lq / gam); asr = ar * __expf(g1 * lq); }
        const float shl = ul - al, shr = ur + ar;
        const float sl = (ps > pl) ? ul - al * sqrtf(g2 * (ps / pl) + g1) : shl;
        const float sr = (ps > pr) ? ur + ar * sqrtf(g2 * (ps / pr) + g1) : shr;
        s[0] = sl; s[1] = us; s[2] = sr;
        for (int mw = 0; mw < 3; mw++) st.s[mw] = s[mw];
        const float esl = ps / gamma1 + 0.5f * rsl * (us * us + vl * vl);
        const float esr = ps / gamma1 + 0.5f * rsr * (us * us + vr * vr);
        const float qln[4] = {qL[0], qL[mu], qL[mv], qL[3]}, qrn[4] = {qR[0], qR[mu], qR[mv], qR[3]};
        const float qsl[4] = {rsl, rsl * us, rsl * vl, esl};
        const float qsr[4] = {rsr, rsr * us, rsr * vr, esr};
        constexpr int comp[4] = {0, mu, mv, 3};
        for (int k = 0; k < 4; k++) {
            // without a jump the star states are the outer states: only the contact/shear wave
            w[0][comp[k]] = nojump ? 0.0f : qsl[k] - qln[k];
            w[1][comp[k]] = nojump ? qrn[k] - qln[k] : qsr[k] - qsl[k];
            w[2][comp[k]] = nojump ? 0.0f : qrn[k] - qsr[k];
        }
        float r0, u0, v0, p0, e0;
        int which;
        if (0.0f <= us) {
            v0 = vl;
            if (ps > pl) which = (0.0f <= sl) ? 0 : 1;
            else if (0.0f <= shl) which = 0;
            else which = (0.0f > us - asl) ? 1 : 2;
        } else {
            v0 = vr;
            if (ps > pr) which = (0.0f >= sr) ? 4 : 3;
            else if (0.0f >= shr) which = 4;
            else which = (0.0f < us + asr) ? 3 : 5;
        }
        if (which == 0) { r0 = rl; u0 = ul; p0 = pl; e0 = qL[3]; }
        else if (which == 4) { r0 = rr; u0 = ur; p0 = pr; e0 = qR[3]; }
        else if (which == 1) { r0 = rsl; u0 = us; p0 = ps; e0 = esl; }
        else if (which == 3) { r0 = rsr; u0 = us; p0 = ps; e0 = esr; }
        else if (which == 2) {
            const float c = g5 + (g6 / al) * ul, lc = __logf(c);
            r0 = rl * __expf(g4 * lc); u0 = g5 * (al + g7 * ul); p0 = pl * __expf(g3 * lc);
            e0 = p0 / gamma1 + 0.5f * r0 * (u0 * u0 + v0 * v0);
        } else {
            const float c = g5 - (g6 / ar) * ur, lc = __logf(c);
            r0 = rr * __expf(g4 * lc); u0 = g5 * (-ar + g7 * ur); p0 = pr * __expf(g3 * lc);
            e0 = p0 / gamma1 + 0.5f * r0 * (u0 * u0 + v0 * v0);
        }
        // without a jump the Godunov state on the sampled side of the contact is that side's
        // own state: its FP64 flux
        st.src = nojump ? (which <= 2 ? 1 : 2) : 0;
        st.f[0] = r0 * u0; st.f[mu] = r0 * u0 * u0 + p0; st.f[mv] = r0 * u0 * v0; st.f[3] = u0 * (e0 + p0);
        return it | (ok ? 0 : NEWTON_FAILED);
    }
    // clawpack46_rpt2_euler4.f:56-94 with the Roe averages of the interface
    template <typename T> struct Split { T u, v, enth, a, g1a2; };
    template <int IXY, typename T, class QC, class AC>
    __device__ static Split<T> split_state(const State<T>& st, QC, AC, const WavePar<T>&)
    {
        return {st.ex[0], st.ex[1], st.ex[2], st.ex[3], st.ex[4]};
    }
    template <int IXY, typename T, class AC>
    __device__ static void split(const Split<T>& e, int, AC, const T* asdq, T* bm, T* bp)
    {
        constexpr int mu = Dir<IXY>::mu, mv = Dir<IXY>::mv;
        const T u = e.u, v = e.v, enth = e.enth, a = e.a;
        const T u2v2 = u * u + v * v;
        const T euv = enth - u2v2;
        const T a3 = e.g1a2 * (euv * asdq[0] + u * asdq[mu] + v * asdq[mv] - asdq[3]);
        const T a2 = asdq[mu] - u * asdq[0];
        const T a4 = (asdq[mv] + (a - v) * asdq[0] - a * a3) / (T(2) * a);
        const T a1 = asdq[0] - a3 - a4;
        T wb[4][3], sb[3];
        wb[0][0] = a1; wb[mu][0] = a1 * u; wb[mv][0] = a1 * (v - a); wb[3][0] = a1 * (enth - v * a); sb[0] = v - a;
        wb[0][1] = a3; wb[mu][1] = a3 * u + a2; wb[mv][1] = a3 * v; wb[3][1] = a3 * T(0.5) * u2v2 + a2 * u; sb[1] = v;
        wb[0][2] = a4; wb[mu][2] = a4 * u; wb[mv][2] = a4 * (v + a); wb[3][2] = a4 * (enth + v * a); sb[2] = v + a;
        for (int m = 0; m < 4; m++) {
            T b1 = dmin1(sb[0], T(0)) * wb[m][0], b2 = dmax1(sb[0], T(0)) * wb[m][0];
            for (int mw = 1; mw < 3; mw++) {
                b1 = b1 + dmin1(sb[mw], T(0)) * wb[m][mw];
                b2 = b2 + dmax1(sb[mw], T(0)) * wb[m][mw];
            }
            bm[m] = b1; bp[m] = b2;
        }
    }
    __device__ static void cons_flux(int idir, const double* q, double, double gamma, double* f)
    {
        RPEulerExact::cons_flux(idir, q, gamma, f);
    }
    template <int IXY> __device__ static double source(int, double, double, double, double, double) { return 0.0; }
};

}  // namespace fcb
