// k_adv.cuh -- fused per-level patch update of scalar advection with edge velocities in aux:
// clawpack 4.6 step2 + step2_wrap, FP64 (TW = double) and FP32-wave (TW = float: waves, limiter,
// second-order correction and transverse split in FP32; the Godunov split, the flux sums and
// the q update in FP64).
//   plane     applications/clawpack/advection/2d/all/clawpack46_rpn2adv.f, clawpack46_rpt2adv.f
//   manifold  clawpack46_rpn2adv_manifold.f, clawpack46_rpt2adv_manifold.f: aux = (capacity kappa,
//             edge velocities scaled by the edge lengths, i.e. psi differences)
//
// One wave per interface, wave = q_R - q_L with the face velocity as its speed, so an interface
// needs no record of its Riemann solve: its neighbours' waves are differences of q.  What the
// update needs from an interface is a = s (q_R - q_L) (amdq where s < 0, apdq where s > 0, the
// other being zero) and the second-order correction cq, and of the two transverse splits that
// meet at a face only the one from upwind is not zero (min(v,0) and max(v,0) of one face
// velocity).  Phases, a barrier after each:
//   stage   q and aux by bulk asynchronous copies
//   cells   status, save_current_step, velocity scaling (b4step2), dt/dx/kappa
//   faces   a and cq of every x and y interface, from q alone (the y sweep does not read the x
//           sweep's results), indexed by the cell right of or above it
//   cross   the transverse terms of every face, from the records of the crossing sweep
//   update  per cell the four face fluxes, formed from the records; q; CFL maximum; time-sync
//           wave accumulation
// Sums keep the order of clawpack46_step2.f, so FP64 results are the CPU path's bits; what is
// dropped are additions of zeros.  At a corner of the cubed sphere (three blocks meet) the
// faces phase runs sweep by sweep with that sweep's corner cells.
//
// What bounds it: issue and shared-memory latency (HBM below 15 %); a general kernel that keeps
// waves, four transverse terms per interface and four flux planes ran at one CTA per SM with
// six barriers.  Updates of one coarse step, one B200 (us, ncu, warm): 256 patches of 32x32 FP64
// 29.3 -> 10.9, cubed sphere levels 3-6, 804 patches of 32x32 FP32-wave 325 -> 131.
#pragma once
#include <cuda_runtime.h>
#include <type_traits>
#include "fcb_common.h"
#include "fcb_launch.cuh"
#include "k_bulk.cuh"
#include "kernels.h"
#include "riemann.cuh"

namespace fcb {

// aux fields of the x- and y-face velocities and (1-based, 0: none) of the capacity
struct AdvPlane { static constexpr int MAUX = 2, U = 0, V = 1, CAPA = 0; };
struct AdvManifold { static constexpr int MAUX = 3, U = 1, V = 2, CAPA = 1; };

template <class RP, int MX, typename TW>
struct AdvGeom {
    static constexpr bool F32 = std::is_same<TW, float>::value;
    static constexpr int MY = MX, MBC = 2, NX = MX + 2 * MBC, NY = MY + 2 * MBC, NXY = NX * NY, MAUX = RP::MAUX;
    static constexpr unsigned QBYTES = NXY * 8u, ABYTES = MAUX * NXY * 8u;
    static_assert(QBYTES % 16 == 0, "bulk copies move multiples of 16 bytes");
    static constexpr size_t OFF_A = QBYTES;                                  // aux [MAUX][NXY] double
    static constexpr size_t OFF_F = OFF_A + ABYTES;                          // a of x, y faces [2][NXY] double
    static constexpr size_t OFF_V = OFF_F + 2 * QBYTES;                      // transverse terms of x, y faces [2][NXY] double
    static constexpr size_t OFF_C = OFF_V + 2 * QBYTES;                      // cq of x, y faces [2][NXY] TW
    static constexpr size_t OFF_R = OFF_C + 2 * (size_t)NXY * sizeof(TW);    // dt/(dx kappa), capacity only [NXY] TW
    static constexpr size_t OFF_Q = OFF_R + (MAUX == 3 ? (size_t)NXY * sizeof(TW) : 0);   // FP32 form: q in TW [NXY]
    static constexpr size_t OFF_RED = OFF_Q + (F32 ? (size_t)NXY * sizeof(TW) : 0);
    static constexpr size_t OFF_BAR = OFF_RED + 32 * 8;
    static constexpr size_t BYTES = OFF_BAR + 16;
    // registers (fclaw2d_clawpatch_conservation.h:56-77), one field
    static constexpr int R_FP0 = 0, R_FP1 = MY, R_FM0 = 2 * MY, R_FM1 = 3 * MY, R_GP0 = 4 * MY, R_GP1 = R_GP0 + MX,
                         R_GM0 = R_GP0 + 2 * MX, R_GM1 = R_GP0 + 3 * MX, NREG = R_GP0 + 4 * MX + 4 * MY + 4 * MX;
};

// Method of a launch: LIM > 0 fixes it at compile time (second order, second-order transverse
// terms, that limiter, and the capacity in aux field 1 of a manifold, none on the plane).
template <int LIM, int CAPA>
struct AdvMethod {
    int o1, o2, l, m;
    __device__ explicit AdvMethod(const StepParams* sp)
        : o1(LIM ? 2 : sp->order1), o2(LIM ? 2 : sp->order2), l(LIM ? LIM : sp->mthlim[0]), m(LIM ? CAPA : sp->mcapa)
    {
    }
    __device__ __forceinline__ int order1() const { return LIM ? 2 : o1; }
    __device__ __forceinline__ int order2() const { return LIM ? 2 : o2; }
    __device__ __forceinline__ int limiter() const { return LIM ? LIM : l; }
    __device__ __forceinline__ int mcapa() const { return LIM ? CAPA : m; }
};

template <class RP, int MX, typename TW, int LIM>
struct AdvPatch {
    using G = AdvGeom<RP, MX, TW>;
    static constexpr int NX = G::NX, NY = G::NY, NXY = G::NXY, MBC = G::MBC, MY = G::MY;
    unsigned char* sm;
    AdvMethod<LIM, RP::CAPA> M;
    double dtdx, dtdy;
    bool plane;                  // the ratio plane serves both directions

    __device__ __forceinline__ double* Q() const { return reinterpret_cast<double*>(sm); }
    __device__ __forceinline__ double* A(int f) const { return reinterpret_cast<double*>(sm + G::OFF_A) + f * NXY; }
    template <int IXY> __device__ __forceinline__ double* F() const
    {
        return reinterpret_cast<double*>(sm + G::OFF_F) + (IXY - 1) * NXY;
    }
    template <int IXY> __device__ __forceinline__ double* V() const
    {
        return reinterpret_cast<double*>(sm + G::OFF_V) + (IXY - 1) * NXY;
    }
    template <int IXY> __device__ __forceinline__ TW* C() const
    {
        return reinterpret_cast<TW*>(sm + G::OFF_C) + (IXY - 1) * NXY;
    }
    __device__ __forceinline__ TW* R() const { return reinterpret_cast<TW*>(sm + G::OFF_R); }
    __device__ __forceinline__ TW* Qt() const
    {
        if constexpr (G::F32) { return reinterpret_cast<TW*>(sm + G::OFF_Q); }
        else { return Q(); }
    }
    // velocity of the x (y) face left of (below) cell c
    template <int IXY> __device__ __forceinline__ double vel(int c) const { return A(IXY == 1 ? RP::U : RP::V)[c]; }
    // dt/dx of cell c in direction IXY, with a capacity dt / (dx kappa)
    template <int IXY> __device__ __forceinline__ TW ratio(int c) const
    {
        if (M.mcapa() > 0) {
            if (G::MAUX == 3 && (IXY == 1 || plane)) return R()[c];
            return (TW)((IXY == 1 ? dtdx : dtdy) / A(M.mcapa() - 1)[c]);
        }
        return (TW)(IXY == 1 ? dtdx : dtdy);
    }

    // Riemann solve, limiter and second-order correction of the face between cells c - step
    // and c at position pos along the sweep; the CFL number goes into cfl.
    template <int IXY>
    __device__ __forceinline__ void face(int c, int pos, TW& cfl) const
    {
        constexpr int step = IXY == 1 ? 1 : NX;
        const double sd = vel<IXY>(c);
        const TW s = (TW)sd;
        const TW* q = Qt();
        TW d = q[c] - q[c - step];
        F<IXY>()[c] = G::F32 ? sd * (Q()[c] - Q()[c - step]) : (double)(s * d);
        const bool inner = pos >= MBC && pos <= MX + MBC;
        const TW rl = ratio<IXY>(c - step), rr = ratio<IXY>(c);
        if (inner) cfl = dmax1(dmax1(cfl, rr * s), -(rl * s));
        TW cq = TW(0);
        if (M.order1() == 2) {
            if (inner && M.limiter() != 0) {
                // inline limiter (clawpack46_inlinelimiter.f:267-343), upwind difference
                const int cu = s > TW(0) ? c - step : c + step;
                const TW du = q[cu] - q[cu - step];
                const TW wnorm2 = d * d;
                if (wnorm2 != TW(0)) d = limiter_phi<TW>(M.limiter(), (du * d) / wnorm2) * d;
            }
            const TW sa = fabs(s), dave = TW(0.5) * (rl + rr);
            cq = mul_rn(mul_rn(sa, sub_rn(TW(1), mul_rn(sa, dave))), d);
        }
        C<IXY>()[c] = cq;
    }
    // amdq and apdq of face c as the transverse split takes them
    template <int IXY> __device__ __forceinline__ TW minus(int c, int pos) const
    {
        const TW a = vel<IXY>(c) < 0.0 ? (TW)F<IXY>()[c] : TW(0);
        return M.order1() > 1 && M.order2() == 2 && pos <= MX + 2 * MBC - 2 ? a + C<IXY>()[c] : a;
    }
    template <int IXY> __device__ __forceinline__ TW plus(int c) const
    {
        const TW a = vel<IXY>(c) > 0.0 ? (TW)F<IXY>()[c] : TW(0);
        return M.order1() > 1 && M.order2() == 2 ? a - C<IXY>()[c] : a;
    }
    // Transverse terms of the face left of (IXY 1) or below (IXY 2) cell c: those of the crossing
    // sweep from the upwind line, whose cell there is cu.  pos, npos: the face's position along
    // its sweep, and across it.
    template <int IXY>
    __device__ __forceinline__ void cross(int c, int pos, int npos) const
    {
        constexpr int step = IXY == 1 ? 1 : NX, side = IXY == 1 ? NX : 1, N = IXY == 1 ? NX : NY;
        const double s = vel<IXY>(c);
        double v = 0.0;
        if (M.order2() > 0 && (s > 0.0 ? pos - 1 >= 1 : s < 0.0 && pos <= N - 2)) {
            const int cu = s > 0.0 ? c - step : c;
            const TW sv = (TW)s, r = TW(0.5) * ratio<3 - IXY>(cu);
            v = 0.0 - (double)(r * (sv * minus<3 - IXY>(cu + side, npos + 1)));
            v = v - (double)(r * (sv * plus<3 - IXY>(cu)));
        }
        V<IXY>()[c] = v;
    }
    // Fluxes fm, fp of that face.
    template <int IXY>
    __device__ __forceinline__ void flux(int c, int pos, double& fm, double& fp) const
    {
        constexpr int N = IXY == 1 ? NX : NY;
        const double s = vel<IXY>(c), a = F<IXY>()[c], v = V<IXY>()[c];
        const double h = G::F32 ? 0.5 * (double)C<IXY>()[c] : (double)(TW(0.5) * C<IXY>()[c]);
        const bool god = pos <= N - 2;
        fm = ((god && s < 0.0 ? a : 0.0) + h) + v;
        fp = ((god && s > 0.0 ? 0.0 - a : 0.0) + h) + v;
    }
};

template <class RP, int MX, int NT, int MINB, typename TW, int LIM>
__global__ void __launch_bounds__(NT, MINB)
adv_kernel(double* __restrict__ q, double* __restrict__ qlast, const double* __restrict__ aux,
           double* __restrict__ regs, const PatchDesc* __restrict__ desc, int p0,
           const StepParams* __restrict__ spp, const LevelGroup lg, unsigned long long* __restrict__ cfl_bits)
{
    using G = AdvGeom<RP, MX, TW>;
    constexpr int NX = G::NX, NY = G::NY, NXY = G::NXY, MBC = G::MBC, MY = G::MY;
    extern __shared__ __align__(128) unsigned char sm[];
    double* red = reinterpret_cast<double*>(sm + G::OFF_RED);
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
        bulk_copy(bar, sm, q + (size_t)p * NXY, G::QBYTES);
        bulk_copy(bar, sm + G::OFF_A, aux + (size_t)p * G::MAUX * NXY, G::ABYTES);
    }
    const StepParams* sp = spp + group_slot(lg, (int)blockIdx.x);
    const PatchDesc* pd = desc + p;
    const double dx = pd->dx, dy = pd->dy;
    const double dt = sp->inst_dt ? sp->dt * sp->inst_dt[pd->inst] : sp->dt;
    const int bcc = (pd->flags / PATCH_BCC3) & 15;
    const AdvPatch<RP, MX, TW, LIM> X{sm, AdvMethod<LIM, RP::CAPA>(sp), dt / dx, dt / dy, dx == dy};
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
    // b4step2: aux(:,:,1) = vty*(psi(x,y+dy)-psi), aux(:,:,2) = -vtx*(psi(x+dx,y)-psi); the
    // stored aux holds the psi differences
    const bool swirl = sp->app == FC2D_B200_APP_SWIRL;
    const double vty = sp->vt / dy, vtx = sp->vt / dx;
    for (int c = tid; c < NXY; c += NT) {
        const double v = Q[c];
        if (!isfinite(v)) bad |= STATUS_NONFINITE;
        if (save) qlast[(size_t)p * NXY + c] = v;
        if constexpr (G::F32) X.Qt()[c] = (TW)v;
        if (swirl) {
            X.A(0)[c] = vty * X.A(0)[c];
            X.A(1)[c] = -(vtx * X.A(1)[c]);
        }
        if (G::MAUX == 3 && X.M.mcapa() > 0) X.R()[c] = (TW)(X.dtdx / X.A(X.M.mcapa() - 1)[c]);
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

    // ---- faces (clawpack46_step2.f:113-236) ------------------------------------------
    TW cflw = TW(0);
    auto faces = [&](bool xs, bool ys) {
        for (int c = tid; c < NXY; c += NT) {
            const int jc = c / NX, ic = c - jc * NX;
            if (xs && ic >= 1 && jc >= 1 && jc <= NY - 2) X.template face<1>(c, ic, cflw);
            if (ys && jc >= 1 && ic >= 1 && ic <= NX - 2) X.template face<2>(c, jc, cflw);
        }
    };
    // clawpack46_fix_corners (clawpack46_step2.f:242-310): at a corner of the cubed sphere
    // (three blocks meet, no corner neighbour) the mbc x mbc corner ghost cells take rotated
    // copies of face ghost cells before each sweep (sweep 0: x, 1: y).  Sources are face
    // ghost cells, never corner cells, so the copies are independent.
    auto fix_corners = [&](int sweep) {
        for (int t = tid; t < 4 * MBC * MBC; t += NT) {
            const int k = t / (MBC * MBC), r = t % (MBC * MBC), ibc = 1 + r / MBC, jbc = 1 + r % MBC;
            if (!((bcc >> k) & 1)) continue;
            const int i1 = (k & 1) ? MX + ibc : 1 - ibc, j1 = (k & 2) ? MY + jbc : 1 - jbc;
            // int(ihat - jhat), int(ihat + jhat) with ihat = 0.5 or mx + 0.5, jhat = 0.5 or my + 0.5
            const int ih = (k & 1) ? MX : 0, jh = (k & 2) ? MY : 0;
            const int dmi = ih - jh, dpl = ih + jh + 1;
            const bool use_b = (sweep == 0 && (k == 0 || k == 3)) || (sweep == 1 && (k == 1 || k == 2));
            const int id = use_b ? j1 + dmi : -j1 + dpl, jd = use_b ? -i1 + dpl : i1 - dmi;
            const int dst = (j1 + MBC - 1) * NX + (i1 + MBC - 1), src = (jd + MBC - 1) * NX + (id + MBC - 1);
            Q[dst] = Q[src];
            if constexpr (G::F32) X.Qt()[dst] = X.Qt()[src];
        }
        __syncthreads();
    };
    if (bcc) {
        fix_corners(0);
        faces(true, false);
        __syncthreads();
        fix_corners(1);
        faces(false, true);
    } else {
        faces(true, true);
    }
    __syncthreads();
    // ---- transverse terms, once per face (two cells read each) --------------------------
    for (int c = tid; c < NXY; c += NT) {
        const int jc = c / NX, ic = c - jc * NX;
        if (ic >= 1 && jc >= 1 && jc <= NY - 2) X.template cross<1>(c, ic, jc);
        if (jc >= 1 && ic >= 1 && ic <= NX - 2) X.template cross<2>(c, jc, ic);
    }
    __syncthreads();

    // ---- time-sync wave accumulation (clawpack46_time_sync.f:163-226), FP64 ----
    if (sp->accumulate_waves) {
        double* rg = regs + (size_t)p * G::NREG;
        const double dtdyv = dt * dy, dtdxv = dt * dx;
        // registers of a face reset since the last update start from zero
        auto add = [&](int face, int r, double v) {
            accumulate(&rg[r], (sp->reg_reset >> ((pd->face_type >> (2 * face)) & 3)) & 1, v);
        };
        for (int it = tid; it < MY + MX; it += NT) {
            double fm, fp;
            if (it < MY) {
                const int jc = MBC + it, c = jc * NX + MBC;
                X.template flux<1>(c, MBC, fm, fp);
                add(0, G::R_FP0 + it, 0.0 - dtdyv * fp);
                add(0, G::R_FM0 + it, dtdyv * fm);
                X.template flux<1>(c + MX, MX + MBC, fm, fp);
                add(1, G::R_FP1 + it, 0.0 - dtdyv * fp);
                add(1, G::R_FM1 + it, dtdyv * fm);
            } else {
                const int i = it - MY, ic = MBC + i, c = MBC * NX + ic;
                X.template flux<2>(c, MBC, fm, fp);
                add(2, G::R_GP0 + i, 0.0 - dtdxv * fp);
                add(2, G::R_GM0 + i, dtdxv * fm);
                X.template flux<2>(c + MY * NX, MY + MBC, fm, fp);
                add(3, G::R_GP1 + i, 0.0 - dtdxv * fp);
                add(3, G::R_GM1 + i, dtdxv * fm);
            }
        }
    }
    // ---- q over i,j = 1-mbc..mx+mbc-1 (clawpack46_step2_wrap.f:107-125); faces of column or
    // row 0 are no sweep's and have no flux ----
    double* qg = q + (size_t)p * NXY;
    double* qi = sp->qinterp && (pd->flags & PATCH_HAS_FINE_NBR) ? sp->qinterp + (size_t)p * NXY : nullptr;
    for (int c = tid; c < NXY; c += NT) {
        const int jc = c / NX, ic = c - jc * NX;
        if (ic <= NX - 2 && jc <= NY - 2) {
            double fr = 0.0, fl = 0.0, gt = 0.0, gb = 0.0, none;
            if (jc >= 1) {
                X.template flux<1>(c + 1, ic + 1, fr, none);
                if (ic >= 1) X.template flux<1>(c, ic, none, fl);
            }
            if (ic >= 1) {
                X.template flux<2>(c + NX, jc + 1, gt, none);
                if (jc >= 1) X.template flux<2>(c, jc, none, gb);
            }
            const double old = Q[c];
            double v = old;
            if (X.M.mcapa() == 0) v = v - X.dtdx * (fr - fl) - X.dtdy * (gt - gb);
            else v = v - (X.dtdx * (fr - fl) + X.dtdy * (gt - gb)) / X.A(X.M.mcapa() - 1)[c];
            qg[c] = v;
            if (qi && in_band(ic, jc, MX, MY, MBC)) qi[c] = add_rn(old, mul_rn(sp->ti_alpha, sub_rn(v, old)));
        } else if (bcc) {
            // cells the update skips keep the step's (corner-fixed) values, as the
            // reference fixes the corners of q in place
            const int kx = ic >= MX + MBC ? 1 : (ic < MBC ? 0 : -1);
            const int ky = jc >= MY + MBC ? 1 : (jc < MBC ? 0 : -1);
            if (kx >= 0 && ky >= 0 && ((bcc >> (kx + 2 * ky)) & 1)) qg[c] = Q[c];
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
            if (v != v) bits = 0x7ff8000000000000ull;   // NaN wins the max
            atomicMax(cfl_bits + pd->inst, bits);
        }
    }
}

template <class RP, int MX, int NT, int MINB, typename TW, int LIM>
cudaError_t run_adv_variant(double* q, double* qlast, const double* aux, double* regs, const PatchDesc* desc, int p0,
                            int npatch, const StepParams* sp, const LevelGroup& lg, unsigned long long* cfl_bits,
                            cudaStream_t st)
{
    using G = AdvGeom<RP, MX, TW>;
    static bool attr_set = false;
    auto kern = adv_kernel<RP, MX, NT, MINB, TW, LIM>;
    if (!attr_set) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)G::BYTES);
        if (e != cudaSuccess) return e;
        attr_set = true;
    }
    if (npatch <= 0) return cudaSuccess;
    return launch_k(kern, npatch, NT, G::BYTES, st, q, qlast, aux, regs, desc, p0, sp, lg, cfl_bits);
}

// One table entry: precision, solver id, square patch size MXV (mbc 2), threads, CTAs per SM,
// limiter fixed at compile time (0: any method).
#define FCB_ADV_VARIANT(PREC, RPID, RPT, MXV, NT, MINB, TW, LIM)                                             \
    Step2Variant{PREC, RPID, MXV, MXV, 2, NT, MINB, 0, (int)AdvGeom<RPT, MXV, TW>::BYTES, 0,            \
                 &run_adv_variant<RPT, MXV, NT, MINB, TW, LIM>, LIM}

}  // namespace fcb
