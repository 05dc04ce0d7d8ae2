// Kernels of one GAMERA MHD time step on sm_100a.
//
// This header is compiled twice (gam_step_strict.cu without FMA contraction,
// gam_step_fast.cu with it) inside the namespace named by GAM_NS, and each
// kernel is templated on the real type R of the bulk data (double for the
// drop-in form, float for the precision form; scalars, the dt reduction and
// the totals stay double).
//
// Step = stepGamera (gamapp.F90:73-91):
//   k_step_begin     AdvanceMHD time trap, AB2 spacing      (mhdgroup.F90:25-31, 457)
//   k_predict        Predictor/PredictCell/ExtrapAB2 + bFlux2Fld of the
//                    half state; per-cell primitives of both states and
//                    per-face B = flux/area, computed once for all stencils
//                                                           (mhdgroup.F90:444-615)
//   k_mom2face(eD)   Mom2Face                               (fields.F90:235-285)
//   k_vxb(eD)        GetCornerV/D/B, EdgeLRs, edge EMF      (fields.F90:184-228, 288-517)
//   k_stress(d)      Fluxes: recon + PDM, MagKinFlux, GasKinFlux, HOGS
//                                                           (stress.F90:204-599, recon.F90)
//   k_update_faces   E2Flux on the new buffer               (fields.F90:18-51)
//   k_update_cells   Flux2Deltas, CellReynolds, bFlux2Fld, CellMaxwell, and the
//                    per-cell CFL dt with a block min       (stress.F90:148-194,
//                    mhdgroup.F90:79-329, gridutils.F90:49-106)
//   finalize_dt      time bookkeeping + CalcDT checks, in the last block of the
//                    update where nothing comes between     (gamapp.F90:110-111, step.F90:58-168)
//   k_bc             EnforceBCs (the kinds that copy values) fused with bFlux2Fld
//                    of the cells whose faces changed       (bcs.F90:279-450, gamapp.F90:86-88)
//
// Every expression keeps the reference's evaluation order (Fortran a+b+c is
// (a+b)+c, x**2.0 is x*x, dot_product is a sequential sum from 0), so the
// strict build reproduces an IEEE-strict CPU step bit for bit.
#pragma once

#include <algorithm>
#include <cuda_runtime.h>
#include <nvtx3/nvToolsExt.h>
#include <stdint.h>
#include <type_traits>
#include "gam_layout.cuh"
#include "gam_math.cuh"
#include "gam_quot.cuh"
#include "gam_types.cuh"

#ifndef GAM_NS
#error "GAM_NS must name the namespace of this build"
#endif
#ifndef GAM_STRICT_KERNELS
#define GAM_STRICT_KERNELS 0  // 1: the strict build (launch bounds measured for it)
#endif

namespace GAM_NS {

static constexpr double TINY = 1.0e-12;
static constexpr double HUGE_DT = 1.0e12;
static constexpr double PI_D = 3.141592653589793;
static constexpr double SQRT_PI_D = 1.7724538509055159;  // sqrt(pi) rounded to double

// interpolation weights (recon.F90:22-23, 28-29)
__device__ __forceinline__ double w8(int n) {
    switch (n) {
        case 0: return -3.0 / 840.0;
        case 1: return 29.0 / 840.0;
        case 2: return -139.0 / 840.0;
        case 3: return 533.0 / 840.0;
        case 4: return 533.0 / 840.0;
        case 5: return -139.0 / 840.0;
        case 6: return 29.0 / 840.0;
        default: return -3.0 / 840.0;
    }
}
__device__ __forceinline__ double up7c(int n) {
    switch (n) {
        case 0: return -3.0 / 420.0;
        case 1: return 25.0 / 420.0;
        case 2: return -101.0 / 420.0;
        case 3: return 319.0 / 420.0;
        case 4: return 214.0 / 420.0;
        case 5: return -38.0 / 420.0;
        default: return 4.0 / 420.0;
    }
}

template <class R> __device__ __forceinline__ R Rc(double x) { return (R)x; }

template <class R> struct Mth;
template <> struct Mth<double> {
#ifdef GAM_CUDA_MATH
    // product build: CUDA's erfc/exp (a few ulp, like libm's, and cheaper)
    static __device__ __forceinline__ double erfc_(double x) { return erfc(x); }
    static __device__ __forceinline__ double exp_(double x) { return exp(x); }
#else
    // strict build: the self-written erfc/exp shared with the CPU restatement
    static __device__ __forceinline__ double erfc_(double x) { return gam::gam_erfc(x); }
    static __device__ __forceinline__ double exp_(double x) { return gam::gam_exp(x); }
#endif
    static __device__ __forceinline__ double sqrt_(double x) { return sqrt(x); }
    static __device__ __forceinline__ double rsqrt_(double x) { return rsqrt(x); }
};
template <> struct Mth<float> {
    static __device__ __forceinline__ float erfc_(float x) { return erfcf(x); }
    static __device__ __forceinline__ float exp_(float x) { return expf(x); }
    static __device__ __forceinline__ float sqrt_(float x) { return sqrtf(x); }
    static __device__ __forceinline__ float rsqrt_(float x) { return rsqrtf(x); }
};

// Quotients a/d that share the divisor d. The FMA form (GAM_FAST_RECIP)
// takes one reciprocal and multiplies (at most one ulp more than the division,
// and a fraction of its instructions). Every other build returns the IEEE
// quotient bit for bit: FP64 through gam::QuotExact (one division per divisor,
// three fmas and a multiply per numerator), FP32 by plain division.
// Quot1 is the same for a divisor with a single numerator, where QuotExact
// would cost more than the division it replaces.
// many<N> takes N numerators at once (one range check for all of them). The
// two-argument form takes the divisor's rounded reciprocal from a table. close is
// rounded like a division in every form: where only the reciprocal is kept, the
// product gets the correction by its exact remainder (gam_quot.cuh).
template <class R> struct Quot {
#ifdef GAM_FAST_RECIP
    R r;
    __device__ __forceinline__ explicit Quot(R d) : r((R)1 / d) {}
    __device__ __forceinline__ Quot(R, R rd) : r(rd) {}
    __device__ __forceinline__ R operator()(R a) const { return a * r; }
    __device__ __forceinline__ R close(R a, R d) const {
        const R q = a * r, e = fma(-d, q, a);
        return e - e == (R)0 ? fma(e, r, q) : q;  // an infinite quotient stays infinite
    }
    // the same for a finite quotient; NaN for another
    __device__ __forceinline__ R close_finite(R a, R d) const {
        const R q = a * r;
        return fma(fma(-d, q, a), r, q);
    }
#else
    R d;
    __device__ __forceinline__ explicit Quot(R dd) : d(dd) {}
    __device__ __forceinline__ Quot(R dd, R) : d(dd) {}
    __device__ __forceinline__ R operator()(R a) const { return a / d; }
    __device__ __forceinline__ R close(R a, R) const { return a / d; }
    __device__ __forceinline__ R close_finite(R a, R) const { return a / d; }
#endif
    template <int N> __device__ __forceinline__ void many(const R* a, R* o) const {
#pragma unroll
        for (int n = 0; n < N; n++) o[n] = (*this)(a[n]);
    }
};
#ifndef GAM_FAST_RECIP
template <> struct Quot<double> {
    gam::QuotExact q;
    __device__ __forceinline__ explicit Quot(double d) : q(d) {}
    __device__ __forceinline__ Quot(double d, double rd) : q(d, rd) {}
    __device__ __forceinline__ double operator()(double a) const { return q(a); }
    __device__ __forceinline__ double close(double a, double) const { return q(a); }
    __device__ __forceinline__ double close_finite(double a, double) const { return q(a); }
    template <int N> __device__ __forceinline__ void many(const double* a, double* o) const { q.many<N>(a, o); }
};
#endif
// The quotient of code that runs twice at most (strict FP64): first with the
// branch-free quotients, which note in ok an operand that they do not cover,
// then, if there was one, with EXACT divisions. The other forms have one kind.
template <class R, bool EXACT> struct QuotTry : Quot<R> {
    using Quot<R>::Quot;
    __device__ __forceinline__ R operator()(R a, bool&) const { return Quot<R>::operator()(a); }
};
#ifndef GAM_FAST_RECIP
template <> struct QuotTry<double, false> : Quot<double> {
    using Quot<double>::Quot;
    __device__ __forceinline__ double operator()(double a, bool& ok) const { return this->q.quick(a, ok); }
};
template <> struct QuotTry<double, true> {
    double d;
    __device__ __forceinline__ explicit QuotTry(double dd) : d(dd) {}
    __device__ __forceinline__ QuotTry(double dd, double) : d(dd) {}
    __device__ __forceinline__ double operator()(double a, bool&) const { return a / d; }
};
#endif
// whether a form has the two kinds
template <class R> struct TwoTries { static constexpr bool v = std::is_same<R, double>::value
#ifdef GAM_FAST_RECIP
    && false
#endif
    ; };
// a/d for a finite nonzero divisor d, equal to the IEEE quotient. A zero
// numerator returns a*d (the signed zero of a/d) without entering the
// division, whose IEEE routine leaves its fast path for a zero numerator;
// zero numerators are common in the step (velocities and field components
// that are exactly zero over much of a grid).
template <class R> __device__ __forceinline__ R qdiv(R a, R d) { return a == (R)0 ? a * d : a / d; }
template <class R> struct Quot1 {
#ifdef GAM_FAST_RECIP
    R r;
    __device__ __forceinline__ explicit Quot1(R d) : r((R)1 / d) {}
    __device__ __forceinline__ R operator()(R a) const { return a * r; }
#else
    R d;
    __device__ __forceinline__ explicit Quot1(R dd) : d(dd) {}
    __device__ __forceinline__ R operator()(R a) const { return qdiv(a, d); }
#endif
};

// a/(gamma - 1) with the reciprocal from the parameters, rounded like a division
// in every form: pressure and internal energy go through gamma - 1 and back every
// step, and a rounded reciprocal would pull the energy the same way each time
// (FP32: 5e-7 instead of 2e-7 off after 20 steps).
template <class R> __device__ __forceinline__ R over_gm1(const DevParams<R>& P, R a) {
    return Quot<R>(P.gm1, P.rgm1).close(a, P.gm1);
}
template <class R, bool EXACT> __device__ __forceinline__ R over_gm1(const DevParams<R>& P, R a, bool& ok) {
#ifdef GAM_FAST_RECIP
    return over_gm1(P, a);
#else
    return QuotTry<R, EXACT>(P.gm1, P.rgm1)(a, ok);
#endif
}

// std::max / std::min semantics: max(a,b) = (a < b) ? b : a, min(a,b) = (b < a) ? b : a
template <class R> __device__ __forceinline__ R rmax(R a, R b) { return (a < b) ? b : a; }
template <class R> __device__ __forceinline__ R rmin(R a, R b) { return (b < a) ? b : a; }
template <class R> __device__ __forceinline__ R sgn1(R b) { return copysign((R)1, b); }

__device__ __forceinline__ bool thread_ijk(const Range& r, int& ii, int& jj, int& kk) {
    ii = r.i0 + blockIdx.x * blockDim.x + threadIdx.x;
    jj = r.j0 + blockIdx.y * blockDim.y + threadIdx.y;
    kk = r.k0 + blockIdx.z * blockDim.z + threadIdx.z;
    return ii <= r.i1 && jj <= r.j1 && kk <= r.k1;
}

__device__ __forceinline__ long lidx(const GamBox& b, int ii, int jj, int kk) {
    return (long)ii + (long)b.sx * jj + b.sk * kk;
}
__device__ __forceinline__ long dstride(const GamBox& b, int d) { return d == 0 ? 1L : (d == 1 ? (long)b.sx : b.sk); }

// ----------------------------------------------------------------- recon
// pdmLR (recon.F90:231-272) on a 4-point limiter stencil nq[0..3] = cells -2..1
template <class R>
__device__ __forceinline__ void pdm_lr(R pdmb, const R* v, R Qi, R& Ql, R& Qr) {
    R v0 = v[0], v1 = v[1], v2 = v[2], v3 = v[3];
    R maxV = rmax(v1, v2), minV = rmin(v1, v2);
    R vN = rmax(minV, rmin(Qi, maxV));
    R dv0 = pdmb * (v1 - v0), dv1 = pdmb * (v2 - v1), dv2 = pdmb * (v3 - v2);
    R s0 = sgn1(dv0), s1 = sgn1(dv1), s2 = sgn1(dv2);
    R q0 = fabs(s0 + s1), q1 = fabs(s1 + s2);
    R dvL = vN - v1, dvR = v2 - vN;
    Ql = vN - s1 * rmax((R)0, fabs(dvL) - q0 * fabs(dv0));
    Qr = vN + s1 * rmax((R)0, fabs(dvR) - q1 * fabs(dv2));
}
// PDM (recon.F90:275-301)
template <class R>
__device__ __forceinline__ R pdm1(R pdmb, R q0, R q1, R q2, R qI) {
    R maxQ = rmax(q1, q2), minQ = rmin(q1, q2);
    R qN = rmax(minQ, rmin(qI, maxQ));
    R dq0 = pdmb * (q1 - q0), dq1 = pdmb * (q2 - q1);
    R s0 = sgn1(dq0), s1 = sgn1(dq1);
    R s01 = fabs(s0 + s1);
    R dqL = qN - q1;
    return qN - s1 * rmax((R)0, fabs(dqL) - s01 * fabs(dq0));
}
// PDM on both sides of a face between the cells v1 and v2, for the interpolants QL
// and QR: pdmLR's states with QL in 8CENT, in Up7LRs pdm1's and its from the other
// side. The right state is the left one with the stencil mirrored; where mirroring a
// zero difference changes its sign, the term it selects is zero. The two differ
// beside a cell that is not a number: pdmLR's bounds are then v1, mirrored ones v2.
// FP64: the signs of the differences are taken from their bits and twice the
// limiter difference enters by one fma (exact, since 2|x| is): 15 FP64
// instructions instead of 22.
__device__ __forceinline__ double pdm_cut(double pd, double v, double qN, double vd) {
    // qN - s max(0, |qN - v| - |s + s'| |pd|), s = sign of vd, s' = sign of pd
    const int sp = __double2hiint(pd), sv = __double2hiint(vd);
    const double k = __hiloint2double((sp ^ sv) < 0 ? 0 : (int)0xC0000000, 0);  // -2 or 0
    const double t = fma(k, fabs(pd), fabs(qN - v));
    const double m = (0.0 < t) ? t : 0.0;
    return qN - __hiloint2double(__double2hiint(m) ^ (sv & (int)0x80000000), __double2loint(m));
}
__device__ __forceinline__ void pdm_both(double pdmb, double v0, double v1, double v2, double v3, double QL, double QR,
                                         bool up7, double& L, double& U) {
    const double d1 = v2 - v1, pd0 = pdmb * (v1 - v0), pd2 = pdmb * (v2 - v3);
    const bool dn = ((unsigned)__double2hiint(d1) ^ 0x80000000u) < 0x7ff00001u;  // negative, and a number
    const double hi = dn ? v1 : v2, lo = dn ? v2 : v1;
    const double qL = rmax(lo, rmin(QL, hi)), q7 = rmin(hi, rmax(lo, QR)), qR = up7 ? q7 : qL;
    const double vd = pdmb * d1;
    L = pdm_cut(pd0, v1, qL, vd);
    U = pdm_cut(pd2, v2, qR, -vd);
}
__device__ __forceinline__ void pdm_both(float pdmb, float v0, float v1, float v2, float v3, float QL, float QR,
                                         bool up7, float& L, float& U) {
    const float hi = rmax(v1, v2), lo = rmin(v1, v2);
    const float qL = rmax(lo, rmin(QL, hi)), q7 = rmax(rmin(v2, v1), rmin(QR, rmax(v2, v1))), qR = up7 ? q7 : qL;
    const float d0 = pdmb * (v1 - v0), d1 = pdmb * (v2 - v1), d2 = pdmb * (v3 - v2);
    const float s0 = sgn1(d0), s1 = sgn1(d1), s2 = sgn1(d2);
    L = qL - s1 * rmax(0.0f, fabs(qL - v1) - fabs(s0 + s1) * fabs(d0));
    U = qR + s1 * rmax(0.0f, fabs(v2 - qR) - fabs(s1 + s2) * fabs(d2));
}
template <class R> __device__ __forceinline__ R central8(const R* q) {
    R s = (R)0;
#pragma unroll
    for (int n = 0; n < 8; n++) s += Rc<R>(w8(n)) * q[n];
    return s;
}
// GetLRs = Cen8LRs (recon.F90:125-158) or Up7LRs (:162-198) on the volume
// weighted stencil QdV[0..7] = dV*Q at cells -4..3 (precomputed per cell),
// limiter nq[0..3] at cells -2..1, and the volume interpolant Vi.
template <class R, class Q>
__device__ __forceinline__ void lrs_from_qdv(const DevParams<R>& P, const R* QdV, const R* nq, const Q& Vi, R& Ql,
                                             R& Qr) {
    if (!P.up7) {
        R s = (R)0;
#pragma unroll
        for (int n = 0; n < 8; n++) s += Rc<R>(w8(n)) * QdV[n];
        R Qi = Vi(s);
        pdm_lr(P.pdmb, nq, Qi, Ql, Qr);
    } else {
        R a = QdV[0] * Rc<R>(up7c(0));
#pragma unroll
        for (int n = 1; n < 7; n++) a = a + QdV[n] * Rc<R>(up7c(n));
        R b = QdV[7] * Rc<R>(up7c(0));
#pragma unroll
        for (int n = 1; n < 7; n++) b = b + QdV[7 - n] * Rc<R>(up7c(n));
        Ql = Vi(a);
        Qr = Vi(b);
        Ql = pdm1(P.pdmb, nq[0], nq[1], nq[2], Ql);
        Qr = pdm1(P.pdmb, nq[3], nq[2], nq[1], Qr);
    }
}

// ----------------------------------------------------------------- EOS
// CellC2P (gamutils.F90:301-321)
template <class R>
__device__ __forceinline__ void cell_c2p(const DevParams<R>& P, const R* U, R* W) {
    R rho = U[0];
    const Quot<R> qr(rho);
    R V[3];
    qr.template many<3>(U + 1, V);
    R Vx = V[0], Vy = V[1], Vz = V[2];
    R E = U[4];
    R KinE = (R)0.5 * rho * (Vx * Vx + Vy * Vy + Vz * Vz);
    W[0] = rmax(rho, P.dFloor);
    W[1] = Vx;
    W[2] = Vy;
    W[3] = Vz;
    W[4] = rmax(P.gm1 * (E - KinE), P.pFloor);
}
// CellP2C (gamutils.F90:362-383)
template <class R>
__device__ __forceinline__ void cell_p2c(const DevParams<R>& P, const R* W, R* U) {
    R rho = rmax(W[0], P.dFloor);
    R Vx = W[1], Vy = W[2], Vz = W[3];
    R IntE = over_gm1(P, rmax(W[4], P.pFloor));
    R KinE = (R)0.5 * rho * (Vx * Vx + Vy * Vy + Vz * Vz);
    U[0] = rho;
    U[1] = rho * Vx;
    U[2] = rho * Vy;
    U[3] = rho * Vz;
    U[4] = IntE + KinE;
}

// norm2 as gfortran evaluates it (scaled sum of squares)
__device__ __forceinline__ double norm2s3(const double* a) {
    double scale = 1.0, res = 0.0;
#pragma unroll
    for (int q = 0; q < 3; q++) {
        if (a[q] != 0.0) {
            double ax = fabs(a[q]);
            if (scale < ax) {
                double val = scale / ax;
                res = 1.0 + res * val * val;
                scale = ax;
            } else {
                double val = ax / scale;
                res += val * val;
            }
        }
    }
    return scale * sqrt(res);
}
// sqrt(2.0) of the nuclear option's interface speed (stress.F90:405): a
// default-real constant in the reference, which gfortran folds to this float
#define GAM_SQRT2_R4 ((double)1.41421354f)

// PredictCell (mhdgroup.F90:528-562, AB2, single fluid): the half-step
// conserved state from the primitives of State n (W) and n-1 (oW)
template <class R>
__device__ __forceinline__ void predict_prim(const DevParams<R>& P, const R* W, const R* oW, R pdt, const Quot<R>& odt,
                                             R* pQ) {
    R dif[5], dQ[5], pW[5];
#pragma unroll
    for (int v = 0; v < 5; v++) dif[v] = W[v] - oW[v];
    odt.template many<5>(dif, dQ);
#pragma unroll
    for (int v = 0; v < 5; v++) pW[v] = W[v] + pdt * dQ[v];
    pW[0] = rmax(pW[0], P.dFloor);
    pW[4] = rmax(pW[4], P.pFloor);
    cell_p2c(P, pW, pQ);
}
template <class R>
__device__ __forceinline__ void predict_cell(const DevParams<R>& P, const R* Q, const R* oQ, R pdt, const Quot<R>& odt,
                                             R* pQ) {
    R W[5], oW[5];
    cell_c2p(P, oQ, oW);
    cell_c2p(P, Q, W);
    predict_prim(P, W, oW, pdt, odt, pQ);
}

// ExtrapAB3 (mhdgroup.F90:721-731)
template <class R> __device__ __forceinline__ R extrap_ab3(R dt, R Q, R oQ, R ooQ, R odt, R oodt) {
    R dQ = qdiv(Q - oQ, odt);
    R odQ = qdiv(oQ - ooQ, oodt);
    R tScl = (dt + odt) / (odt + oodt);
    return Q + dt * dQ + dt * tScl * (dQ - odQ);
}
// PredictCell with doAB3: the third level of the gas is oState's
// (ooQ = oState%Gas, mhdgroup.F90:500-502), as in the reference
template <class R>
__device__ __forceinline__ void predict_prim_ab3(const DevParams<R>& P, const R* W, const R* oW, R pdt, R odt, R oodt,
                                                 R* pQ) {
    R pW[5];
#pragma unroll
    for (int v = 0; v < 5; v++) pW[v] = extrap_ab3(pdt, W[v], oW[v], oW[v], odt, oodt);
    pW[0] = rmax(pW[0], P.dFloor);
    pW[4] = rmax(pW[4], P.pFloor);
    cell_p2c(P, pW, pQ);
}
template <class R>
__device__ __forceinline__ void predict_cell_ab3(const DevParams<R>& P, const R* Q, const R* oQ, R pdt, R odt, R oodt,
                                                 R* pQ) {
    R W[5], oW[5];
    cell_c2p(P, oQ, oW);
    cell_c2p(P, Q, W);
    predict_prim_ab3(P, W, oW, pdt, odt, oodt, pQ);
}

// Boris-limited speed Ca v / sqrt(Ca^2 + v^2) (fields.F90:211-213,
// gridutils.F90:91-93, gamutils.F90:356-358)
template <class T> __device__ __forceinline__ T boris_speed(T Ca, T v) { return Ca * v / sqrt(Ca * Ca + v * v); }

// gamCellBxyz (gridutils.F90:648-680) from the six face fluxes of cell c, with
// the quotient by the cell volume qV. The metric is read through the read-only
// path: the compiler may then move these loads above stores to the state and
// work arrays.
template <class R, class Q>
__device__ __forceinline__ void cell_bxyz_q(const GamBox& b, const Geo<R>& g, long c, R fI, R fIp, R fJ, R fJp, R fK,
                                            R fKp, const Q& qV, R* B) {
    const long fs = b.fs;
    if constexpr (std::is_same<R, float>::value) {
        // sum of flux x (face centroid - cell centroid): the same value as the
        // form below, without the cancellation of absolute coordinates
#pragma unroll
        for (int x = 0; x < 3; x++) {
            const R* d = g.dxf + (long)x * fs + c;
            R t = fIp * __ldg(d + 3 * fs) + fJp * __ldg(d + 9 * fs) + fKp * __ldg(d + 15 * fs) - fI * __ldg(d) -
                  fJ * __ldg(d + 6 * fs) - fK * __ldg(d + 12 * fs);
            B[x] = qV(t);
        }
        return;
    }
    R Div = fIp - fI + fJp - fJ + fKp - fK;
#pragma unroll
    for (int x = 0; x < 3; x++) {
        R xfI = __ldg(g.xfc + (x + 0) * fs + c);
        R xfJ = __ldg(g.xfc + (x + 3) * fs + c);
        R xfK = __ldg(g.xfc + (x + 6) * fs + c);
        R xfIp = __ldg(g.xfc + (x + 0) * fs + c + 1);
        R xfJp = __ldg(g.xfc + (x + 3) * fs + c + b.sx);
        R xfKp = __ldg(g.xfc + (x + 6) * fs + c + b.sk);
        R t = qV(fIp * xfIp + fJp * xfJp + fKp * xfKp - fI * xfI - fJ * xfJ - fK * xfK);
        B[x] = t - qV(Div * __ldg(g.xyzcc + x * fs + c));
    }
}
template <class R>
__device__ __forceinline__ void cell_bxyz(const GamBox& b, const Geo<R>& g, long c, R fI, R fIp, R fJ, R fJp, R fK,
                                          R fKp, R* B) {
    cell_bxyz_q(b, g, c, fI, fIp, fJ, fJp, fK, fKp, Quot<R>(g.vol[c]), B);
}

// ----------------------------------------------------------------- bounds checks
// Built with -DGAM_BOUNDS_CHECK (libgamgpu_check.so): every kernel checks the
// lowest and highest linear box index its stencils will touch before loading
// anything; a failed check records the kernel and the index in the scalars
// and the thread returns without touching memory (no trap). The host reads
// the record after the call. Without the macro the checks compile to nothing.
#ifdef GAM_BOUNDS_CHECK
__device__ __forceinline__ bool box_ok(const GamBox& b, long lo, long hi, const GamScalars* csc, int kid) {
    GamScalars* sc = const_cast<GamScalars*>(csc);
    const long lim = sc->oobLimit > 0 ? (long)sc->oobLimit : b.nbox;
    if (lo >= 0 && hi < lim) return true;
    if (atomicExch(&sc->oob, 1) == 0) {
        sc->oobKernel = kid;
        sc->oobIndex = lo < 0 ? lo : hi;
    }
    return false;
}
#define GAM_BOX_CHECK(lo, hi, kid) \
    if (!box_ok(b, (long)(lo), (long)(hi), sc, (kid))) return
// for kernels whose threads must reach a later barrier: a value, not a return
#define GAM_BOX_OK(lo, hi, kid) box_ok(b, (long)(lo), (long)(hi), sc, (kid))
#else
#define GAM_BOX_OK(lo, hi, kid) true
#define GAM_BOX_CHECK(lo, hi, kid) \
    do {                           \
    } while (0)
#endif

// ----------------------------------------------------------------- LFM pole
// Index maps across the LFM axis (ringutils.F90:482-659, box indices): the
// pole at js (doS) / je+1 (doE), k shifted by half a ring (WrapK).
__device__ __forceinline__ int ring_wrapk(const GamBox& b, int kk) {
    int kp = kk + b.Nkp / 2;
    if (kp > GAM_NG + b.Nkp - 1) kp -= b.Nkp;
    return kp;
}
// lfmIJKcc for a ghost row across the pole: its conjugate cell (true) or
// nothing (false)
__device__ __forceinline__ bool ring_conj_cc(const GamBox& b, const RingData& Rg, int& jj, int& kk) {
    const int G = GAM_NG;
    if (Rg.doS && jj < G) {
        jj = 2 * G - 1 - jj;
        kk = ring_wrapk(b, kk);
        return true;
    }
    if (Rg.doE && jj > G + b.Njp - 1 && jj <= G + b.Njp + 3) {
        jj = 2 * G + 2 * b.Njp - 1 - jj;
        kk = ring_wrapk(b, kk);
        return true;
    }
    return false;
}
// The pole boundary lfmIn / lfmOut (bcs.F90:1019-1106) as a map of value
// comp (-1 cell, 0..2 face normal) at (jj, kk): the source and its sign
// (J and K faces reversed); the J faces' pole face itself is not mirrored
__device__ __forceinline__ int ring_bc_jmap(const GamBox& b, const RingData& Rg, int comp, int& jj, int& kk) {
    const int G = GAM_NG, N = b.Njp;
    if (comp == 1) {
        if (Rg.doS && jj < G) {
            jj = 2 * G - jj;
            kk = ring_wrapk(b, kk);
            return -1;
        }
        if (Rg.doE && jj >= G + N + 1 && jj <= G + N + 4) {
            jj = 2 * G + 2 * N - jj;
            kk = ring_wrapk(b, kk);
            return -1;
        }
        return 1;
    }
    if (ring_conj_cc(b, Rg, jj, kk)) return comp == 2 ? -1 : 1;
    return 1;
}

// ----------------------------------------------------------------- kernels
// AdvanceMHD entry: time trap and AB2 spacing (mhdgroup.F90:25-31, 457)
__global__ void k_step_begin(GamScalars* sc) {
    if (sc->halted) return;
    if (fabs(sc->otime - sc->time) < TINY) sc->otime = sc->time - sc->dt;
    sc->odt = sc->time - sc->otime;
    sc->oodt = sc->otime - sc->ootime;  // Predictor (mhdgroup.F90:459-463), used with doAB3
    sc->pdt = 0.5 * sc->dt;
    sc->rodt = 1.0 / sc->odt;
    sc->rdt = 1.0 / sc->dt;
}

// The predictor's work at box position c (see k_predict): faces, then the cell.
// Quotients by one density share its reciprocal; no branch between them in the
// first try (192^3, strict: 862 -> 661 us; FMA form 713 -> 608).
template <class R, bool AB3, bool EXACT>
__device__ __forceinline__ void predict_at(const GamBox& b, const DevParams<R>& P, const Geo<R>& g,
                                           const StateBuf<R>& cur, const StateBuf<R>& old, const Work<R>& w,
                                           const R* __restrict__ oomf, int ii, int jj, int kk, long c, bool isCell, R pdt,
                                           R odt, R rodt, R oodt, bool& ok) {
    const long fs = b.fs;
    // The state and work pointers may alias as far as the compiler knows, so
    // every state load is issued before the first store.
    R fQ[3], foQ[3], fA[3], Q[5], oQ[5], uQ[3], uoQ[3];
    R fooQ[3], uooQ[3];  // AB3: ooState fluxes of the lower / upper faces
    if (P.doMHD) {
#pragma unroll
        for (int d = 0; d < 3; d++) {
            fQ[d] = cur.mf[d * fs + c];
            foQ[d] = old.mf[d * fs + c];
            fA[d] = g.face[d * fs + c];
            if constexpr (AB3) fooQ[d] = oomf[d * fs + c];
        }
    }
    if (isCell) {
#pragma unroll
        for (int v = 0; v < 5; v++) {
            Q[v] = cur.Gas[v * fs + c];
            oQ[v] = old.Gas[v * fs + c];
        }
        if (P.doMHD) {
            const long off[3] = {1, (long)b.sx, b.sk};
#pragma unroll
            for (int d = 0; d < 3; d++) {
                uQ[d] = cur.mf[d * fs + c + off[d]];
                uoQ[d] = old.mf[d * fs + c + off[d]];
                if constexpr (AB3) uooQ[d] = oomf[d * fs + c + off[d]];
            }
        }
    }
    R hm[3];
    const QuotTry<R, EXACT> qodt(odt, rodt);
    if (P.doMHD) {
        if constexpr (AB3) {
#pragma unroll
            for (int d = 0; d < 3; d++) hm[d] = extrap_ab3(pdt, fQ[d], foQ[d], fooQ[d], odt, oodt);
        } else {
#pragma unroll
            for (int d = 0; d < 3; d++) hm[d] = fQ[d] + pdt * qodt(fQ[d] - foQ[d], ok);  // ExtrapAB2
        }
#pragma unroll
        for (int d = 0; d < 3; d++) {
            R A = fA[d];
            R Am = rmax(A, (R)TINY);
            const QuotTry<R, EXACT> qAm(Am);
            const R bh = qAm(hm[d], ok);
            w.abh[d * fs + c] = A * bh;
            // the area itself divides Bnf: the same quotient, but for areas below TINY
#ifdef GAM_FAST_RECIP
            w.Bnf[d * fs + c] = Am == A ? qAm.close(hm[d], A) : qdiv(hm[d], A);
#else
            w.Bnf[d * fs + c] = Am == A ? bh : qdiv(hm[d], A);
#endif
            w.bn[d * fs + c] = P.doLFMLim ? qAm(fQ[d], ok) : bh;
        }
    }
    if (!isCell) return;
    R pQ[5], Wn[5];
    {
        // CellC2P of State n and BlockCon2Prim's primitives of it divide by the
        // same density unless the floor acts on it
        R W[5], oW[5];
        const R rho = Q[0], D = rmax(rho, P.dFloor);
        const QuotTry<R, EXACT> qD(D), qo(oQ[0]);
        Wn[0] = W[0] = D;
#pragma unroll
        for (int x = 0; x < 3; x++) Wn[1 + x] = W[1 + x] = qD(Q[1 + x], ok);
        Wn[4] = rmax(P.gm1 * (Q[4] - qD((R)0.5 * (Q[1] * Q[1] + Q[2] * Q[2] + Q[3] * Q[3]), ok)), P.pFloor);
        if (D != rho) {
#pragma unroll
            for (int x = 0; x < 3; x++) W[1 + x] = Q[1 + x] / rho;
        }
        W[4] = rmax(P.gm1 * (Q[4] - (R)0.5 * rho * (W[1] * W[1] + W[2] * W[2] + W[3] * W[3])), P.pFloor);
#pragma unroll
        for (int x = 0; x < 3; x++) oW[1 + x] = qo(oQ[1 + x], ok);
        oW[0] = rmax(oQ[0], P.dFloor);
        oW[4] = rmax(P.gm1 * (oQ[4] - (R)0.5 * oQ[0] * (oW[1] * oW[1] + oW[2] * oW[2] + oW[3] * oW[3])), P.pFloor);
        if constexpr (AB3) {
            predict_prim_ab3(P, W, oW, pdt, odt, oodt, pQ);
        } else {
            R pW[5];
#pragma unroll
            for (int v = 0; v < 5; v++) pW[v] = W[v] + pdt * qodt(W[v] - oW[v], ok);
            pW[0] = rmax(pW[0], P.dFloor);
            pW[4] = rmax(pW[4], P.pFloor);
            const R KinE = (R)0.5 * pW[0] * (pW[1] * pW[1] + pW[2] * pW[2] + pW[3] * pW[3]);  // CellP2C
            pQ[0] = pW[0];
#pragma unroll
            for (int x = 0; x < 3; x++) pQ[1 + x] = pW[0] * pW[1 + x];
            pQ[4] = over_gm1<R, EXACT>(P, pW[4], ok) + KinE;
        }
    }
    const R vol = __ldg(g.vol + c);
    {
        // BlockCon2Prim of the half state, and volume * momentum / density by the same density
        R Wh[5];
        Wh[0] = rmax(pQ[0], P.dFloor);
        const QuotTry<R, EXACT> qh(Wh[0]);
#pragma unroll
        for (int x = 0; x < 3; x++) Wh[1 + x] = qh(pQ[1 + x], ok);
        Wh[4] = rmax(P.gm1 * (pQ[4] - qh((R)0.5 * (pQ[1] * pQ[1] + pQ[2] * pQ[2] + pQ[3] * pQ[3]), ok)), P.pFloor);
#pragma unroll
        for (int v = 0; v < 5; v++) {
            w.QW[v * fs + c] = vol * Wh[v];
            w.Wn[v * fs + c] = P.doLFMLim ? Wn[v] : Wh[v];
        }
        w.Dh[c] = Wh[0];
#pragma unroll
        for (int x = 0; x < 3; x++) w.VdV[x * fs + c] = qh(vol * pQ[1 + x], ok);
    }
    if (P.doMHD) {
        // upper faces of this cell, recomputed with the same ExtrapAB2
        R up[3];
        if constexpr (AB3) {
#pragma unroll
            for (int d = 0; d < 3; d++) up[d] = extrap_ab3(pdt, uQ[d], uoQ[d], uooQ[d], odt, oodt);
        } else {
#pragma unroll
            for (int d = 0; d < 3; d++) up[d] = uQ[d] + pdt * qodt(uQ[d] - uoQ[d], ok);
        }
        R B[3];
        int jc = jj, kc = kk;
        if (P.ring.on && ring_conj_cc(b, P.ring, jc, kc)) {
            // RingFlux2FieldFix in the predictor's bFlux2Fld: the conjugate
            // cell's field from its own extrapolated fluxes
            const long cc = lidx(b, ii, jc, kc);
            const long off[3] = {1, (long)b.sx, b.sk};
            R lo[3], hi[3];
#pragma unroll
            for (int d = 0; d < 3; d++) {
                const long f0 = d * fs + cc, f1 = f0 + off[d];
                if constexpr (AB3) {
                    lo[d] = extrap_ab3(pdt, cur.mf[f0], old.mf[f0], oomf[f0], odt, oodt);
                    hi[d] = extrap_ab3(pdt, cur.mf[f1], old.mf[f1], oomf[f1], odt, oodt);
                } else {
                    lo[d] = cur.mf[f0] + pdt * qodt(cur.mf[f0] - old.mf[f0], ok);
                    hi[d] = cur.mf[f1] + pdt * qodt(cur.mf[f1] - old.mf[f1], ok);
                }
            }
            const QuotTry<R, EXACT> qv(__ldg(g.vol + cc));
            cell_bxyz_q(b, g, cc, lo[0], hi[0], lo[1], hi[1], lo[2], hi[2], [&](R a) { return qv(a, ok); }, B);
        } else {
            const QuotTry<R, EXACT> qv(vol);
            cell_bxyz_q(b, g, c, hm[0], up[0], hm[1], up[1], hm[2], up[2], [&](R a) { return qv(a, ok); }, B);
        }
#pragma unroll
        for (int x = 0; x < 3; x++) {
            w.QB[x * fs + c] = vol * B[x];
            if (!P.doLFMLim) w.Bl[x * fs + c] = B[x];
        }
    }
}

// Predictor over every face and cell of the ghosted box. Besides the half
// state it stores the operands every later stencil uses, each computed once:
// volume * primitive (the recon operand QdV of Cen8LRs/Up7LRs), the limiter
// primitives, volume * momentum / density (Mom2Face), and per face
// area * flux/max(area,TINY) and flux/max(area,TINY) (EdgeLRs), flux/area (Fluxes).
template <class R, int MINB, bool AB3 = false>
__global__ void __launch_bounds__(256, MINB) k_predict(GamBox b, DevParams<R> P, Geo<R> g, StateBuf<R> cur,
                                                 StateBuf<R> old, Work<R> w, GamScalars* sc,
                                                 const R* __restrict__ oomf) {
    if (sc->halted) {  // the steps after a failed one leave its ghosts alone
        if (blockIdx.x + blockIdx.y + blockIdx.z + threadIdx.x + threadIdx.y == 0) sc->fixGhosts = 0;
        return;
    }
    int ii, jj, kk;
    Range r{0, b.Ni, 0, b.Nj, 0, b.Nk};
    if (!thread_ijk(r, ii, jj, kk)) return;
    const long c = lidx(b, ii, jj, kk);
    const R pdt = (R)sc->pdt, odt = (R)sc->odt;
    const bool isCell = ii < b.Ni && jj < b.Nj && kk < b.Nk;
    GAM_BOX_CHECK(c, isCell ? c + b.sk : c, 1);
    [[maybe_unused]] R oodt = (R)0;
    if constexpr (AB3) oodt = (R)sc->oodt;
#ifdef GAM_GEO_TABLES
    const R rodt = (R)sc->rodt;
#else
    const R rodt = (R)1 / odt;
#endif
    bool ok = true;
    predict_at<R, AB3, false>(b, P, g, cur, old, w, oomf, ii, jj, kk, c, isCell, pdt, odt, rodt, oodt, ok);
    if constexpr (TwoTries<R>::v) {  // an operand out of the quick quotients' range: once more
        if (!ok)
            predict_at<R, AB3, true>(b, P, g, cur, old, w, oomf, ii, jj, kk, c, isCell, pdt, odt, rodt, oodt, ok);
    }
}

// Quotient by the volume interpolated to the face c of direction D: from the
// tables made with the geometry, else from the volumes (differentiation form)
template <class R> __device__ __forceinline__ Quot<R> face_quot(const GamBox& b, const Geo<R>& g, long c, int D) {
#ifdef GAM_GEO_TABLES
#ifdef GAM_FAST_RECIP
    return Quot<R>((R)0, g.rvif[D * b.fs + c]);
#else
    return Quot<R>(g.vif[D * b.fs + c], g.rvif[D * b.fs + c]);
#endif
#else
    const long s = dstride(b, D);
    R vol[8];
#pragma unroll
    for (int n = 0; n < 8; n++) vol[n] = g.vol[c + (n - 4) * s];
    return Quot<R>(central8(vol));
#endif
}
// the same with the volume floored at TINY (Mom2Face)
template <class R> __device__ __forceinline__ Quot<R> face_quot_floor(const GamBox& b, const Geo<R>& g, long c, int D) {
#ifdef GAM_GEO_TABLES
    R v = (R)0, rv = g.rvif[D * b.fs + c];
#ifndef GAM_FAST_RECIP
    v = g.vif[D * b.fs + c];
#endif
    if (!(rv > (R)0 && rv < (R)(1.0 / TINY))) {
        v = (R)TINY;
        rv = (R)(1.0 / TINY);
    }
    return Quot<R>(v, rv);
#else
    const long s = dstride(b, D);
    R vol[8];
#pragma unroll
    for (int n = 0; n < 8; n++) vol[n] = g.vol[c + (n - 4) * s];
    return Quot<R>(rmax(central8(vol), (R)TINY));
#endif
}

// Edge geometry of the EMF in direction eD (fields.F90:84-170): face
// direction dT1 (Mom2Face sweep), dT2 (corner sweep)
__device__ __forceinline__ void edge_dirs(int eD, int& dT1, int& dT2) {
    dT1 = (eD + 1) % 3;
    dT2 = (eD + 2) % 3;
}

// Mom2Face for edge direction eD over the reference's loop range (192^3, the
// three directions with the interpolated volume from its table: strict 503 ->
// 375 us, FMA form 470 -> 325, FP32 276 -> 234); stores
// area(dT1) * Vf, the operand of GetCornerV's weighted interpolation.
template <class R>
__global__ void __launch_bounds__(256) k_mom2face(GamBox b, DevParams<R> P, Geo<R> g, Work<R> w, int eD, Range r,
                                                  const GamScalars* sc) {
    if (sc->halted) return;
    int ii, jj, kk;
    if (!thread_ijk(r, ii, jj, kk)) return;
    int dT1, dT2;
    edge_dirs(eD, dT1, dT2);
    const long fs = b.fs;
    const long c = lidx(b, ii, jj, kk);
    const long s = dstride(b, dT1);
    GAM_BOX_CHECK(c - 4 * s, c + 3 * s, 2 + 2 * eD);
    const Quot<R> qdV = face_quot_floor<R>(b, g, c, dT1);
    const R A = g.face[dT1 * fs + c];
    R num[3], quo[3];
#pragma unroll
    for (int x = 0; x < 3; x++) {
        R q[8];
#pragma unroll
        for (int n = 0; n < 8; n++) q[n] = w.VdV[x * fs + c + (n - 4) * s];
        num[x] = central8(q);
    }
    qdV.template many<3>(num, quo);
#pragma unroll
    for (int x = 0; x < 3; x++) w.AVf[(x + 3 * eD) * fs + c] = A * quo[x];
}

// EdgeLRs (fields.F90:288-362), the weighted sums of its reconstruction from
// the operand p (the edge's own face) with stride s: one sum in 8CENT, in sR too
template <class R> __device__ __forceinline__ void edge_sums(bool up7, const R* p, int s, R& sL, R& sR) {
    R q[8];
#pragma unroll
    for (int n = 0; n < 8; n++) q[n] = p[(n - 4) * s];
    if (!up7) {
        sL = sR = central8(q);
    } else {
        sL = q[0] * Rc<R>(up7c(0));
        sR = q[7] * Rc<R>(up7c(0));
#pragma unroll
        for (int n = 1; n < 7; n++) {
            sL = sL + q[n] * Rc<R>(up7c(n));
            sR = sR + q[7 - n] * Rc<R>(up7c(n));
        }
    }
}

// The metric of an edge that edge_emf takes
template <class R> struct EdgeMetric {
    R t1[3], t2[3];              // tangents
    R xni, yni, xnj, ynj, detT;  // B map
    R fA1, fA2, rA1;             // interpolated areas (not in the forms that multiply by 1/area), 1/fA1
    R edge;
};
// The EMF of edge c (VxB edge loop, fields.F90:184-228) from its block's boxes in
// shared memory (EdgeTile) and its metric. SAVE: also the corner values into
// w.esv, where that is not null (see flux_face).
template <class R, int E, bool SAVE>
__device__ __forceinline__ void edge_emf(const GamBox& b, const DevParams<R>& P, const Geo<R>& g, const Work<R>& w,
                                         long c, const R* sm, int tx, int ty, int tz, const EdgeMetric<R>& m,
                                         const Quot<R>& qA1, const Quot<R>& qA2, const Quot<R>& qdt, R dt) {
    using T_ = EdgeTile<E>;
    constexpr int eD = E, dT1 = T_::d1, dT2 = T_::d2;
    const long fs = b.fs;
    const R* pD = sm + T_::at(5, tx, ty, tz);
    // GetCornerD (fields.F90:427-454): normal-plane unit offsets e1 < e2
    constexpr int e1 = E == 0 ? 1 : 0, e2 = E == 2 ? 1 : 2;
    constexpr int h1 = T_::str(5, e1), h2 = T_::str(5, e2);
    R Dc = (R)0.25 * (pD[0] + pD[-h1] + pD[-h2] + pD[-h1 - h2]);
    // GetCornerB: EdgeLRs for dT1 faces along dT2 and dT2 faces along dT1, and
    // GetCornerV (fields.F90:457-517), whose area stencil is the first one's:
    // all sums, then their quotients by the two interpolated areas
    R num[5], quo[5], n2[2], q2[2];
    edge_sums(P.up7, sm + T_::at(0, tx, ty, tz), T_::str(0, dT2), num[0], num[1]);
    edge_sums(P.up7, sm + T_::at(1, tx, ty, tz), T_::str(1, dT1), n2[0], n2[1]);
#pragma unroll
    for (int x = 0; x < 3; x++) {
        const R* p = sm + T_::at(2, tx, ty, tz) + x * T_::size(2);
        R q[8];
#pragma unroll
        for (int n = 0; n < 8; n++) q[n] = p[(n - 4) * T_::str(2, dT2)];
        num[2 + x] = central8(q);
    }
    qA1.template many<5>(num, quo);
    qA2.template many<2>(n2, q2);
    R VC[3] = {quo[2], quo[3], quo[4]};
#ifdef GAM_FAST_RECIP
    const bool small = !(m.rA1 > (R)0 && m.rA1 <= (R)(1.0 / TINY));
#else
    const bool small = m.fA1 < (R)TINY;
#endif
    if (small) {  // GetCornerV divides by an area of TINY at least
#pragma unroll
        for (int x = 0; x < 3; x++) VC[x] = num[2 + x] / (R)TINY;
    }
    R bT1L, bT1R, bT2L, bT2R;
    auto limit = [&](bool up7) {
        const R *p1 = sm + T_::at(3, tx, ty, tz), *p2 = sm + T_::at(4, tx, ty, tz);
        constexpr int r1 = T_::str(3, dT2), r2 = T_::str(4, dT1);
        pdm_both(P.pdmb, p1[-2 * r1], p1[-r1], p1[0], p1[r1], quo[0], quo[1], up7, bT1L, bT1R);
        pdm_both(P.pdmb, p2[-2 * r2], p2[-r2], p2[0], p2[r2], q2[0], q2[1], up7, bT2L, bT2R);
    };
    // each with its own code: a choice inside costs the FMA form's edges 6 us of 250 (192^3)
    if (P.up7)
        limit(true);
    else
        limit(false);
    R v1 = VC[0] * m.t1[0] + VC[1] * m.t1[1] + VC[2] * m.t1[2];
    R v2 = VC[0] * m.t2[0] + VC[1] * m.t2[1] + VC[2] * m.t2[2];
    R vDiff = Mth<R>::sqrt_(v1 * v1 + v2 * v2);
#ifdef GAM_FAST_RECIP
    // the reference multiplies by the area and divides by it again
    R bT1 = (R)0.5 * (bT1L + bT1R), bT2 = (R)0.5 * (bT2L + bT2R);
    R db1 = bT1R - bT1L, db2 = bT2R - bT2L;
#else
    bT1L = bT1L * m.fA1;
    bT1R = bT1R * m.fA1;
    bT2L = bT2L * m.fA2;
    bT2R = bT2R * m.fA2;
    const R m1[2] = {(R)0.5 * (bT1L + bT1R), bT1R - bT1L}, m2[2] = {(R)0.5 * (bT2L + bT2R), bT2R - bT2L};
    R o1[2], o2[2];
    qA1.template many<2>(m1, o1);
    qA2.template many<2>(m2, o2);
    R bT1 = o1[0], bT2 = o2[0];
    R db1 = o1[1], db2 = o2[1];
#endif
    R Jd = db2 - db1;
    R b1 = m.detT * (m.ynj * bT1 - m.yni * bT2);
    R b2 = m.detT * (-(m.xnj * bT1) + m.xni * bT2);
    if (P.doBackground) {
        b1 = b1 + (R)g.edgB0[(0 + 2 * eD) * fs + c];
        b2 = b2 + (R)g.edgB0[(1 + 2 * eD) * fs + c];
    }
    R vA = qdiv(Mth<R>::sqrt_(b1 * b1 + b2 * b2), Mth<R>::sqrt_(Dc));
    if (P.doBoris) vA = boris_speed((R)P.Ca, vA);
    vDiff = vDiff + vA;
    // FP32 divides: 192^3, the I edges 150 us, 156 with the corrected product. (A bound
    // that is infinite, or not a number, bounds nothing.)
    const R vMax = sizeof(R) == 4 ? P.CFL * m.edge / dt : qdt.close_finite(P.CFL * m.edge, dt);
    vDiff = rmin(vDiff, vMax);
    R e = -(v1 * b2 - v2 * b1) + P.Vd0 * vDiff * Jd;
    w.E[eD * fs + c] = e * m.edge;
    if (SAVE && w.esv) {
        R* o = w.esv + (long)(GAM_ESV_NC * eD) * fs + c;
        o[0] = Dc;
        o[fs] = bT1L;
        o[2 * fs] = bT1R;
        o[3 * fs] = m.fA1;
        o[4 * fs] = bT2L;
        o[5 * fs] = bT2R;
        o[6 * fs] = m.fA2;
#pragma unroll
        for (int x = 0; x < 3; x++) o[(7 + x) * fs] = VC[x];
    }
}

#ifdef GAM_GEO_TABLES
// ----------------------------------------------------------------- TMA
// Box copies of a (i, j, k, component) field into shared memory and the
// mbarrier that counts their bytes.
__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void tma_bar_init(uint64_t* bar) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(bar)) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void tma_expect(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void tma_load(void* dst, const CUtensorMap* map, int i, int j, int k, int comp,
                                         uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], "
        "[%6];" ::"r"(smem_u32(dst)), "l"(map), "r"(i), "r"(j), "r"(k), "r"(comp), "r"(smem_u32(bar))
        : "memory");
}
__device__ __forceinline__ uint64_t device_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}
// Wait for the first phase; false when it does not complete in half a second (each
// try waits in hardware for a while, the first ones without a look at the clock)
__device__ __forceinline__ bool tma_wait(uint64_t* bar) {
    uint64_t t0 = 0;
    for (int n = 0;; n = n < 64 ? n + 1 : n) {
        uint32_t done;
        asm volatile(
            "{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], 0; selp.b32 %0, 1, 0, p; }"
            : "=r"(done)
            : "r"(smem_u32(bar))
            : "memory");
        if (done) return true;
        if (n < 64) continue;
        const uint64_t t = device_ns();
        if (t0 == 0) t0 = t;
        if (t - t0 > 500000000u) return false;
    }
}
// ... in the step's kernels: a wait that ran out is noted for the end of the step
// (finalize_dt), which stops there. It does not set halted, which other blocks look
// at. The copies may still be under way into this block's memory, so it waits
// once more before it gives the memory up.
__device__ __forceinline__ bool tma_wait(uint64_t* bar, GamScalars* sc) {
    if (tma_wait(bar)) return true;
    sc->copyFailed = 1;
    tma_wait(bar);
    return false;
}
#ifdef GAM_BOUNDS_CHECK
#define GAM_COPY_BYTES(n) ((n) + sc->copyStall)  // test hook: bytes that never come
#else
#define GAM_COPY_BYTES(n) (n)
#endif

// VxB edge loop for direction E (fields.F90:184-228), one edge per thread. The
// stencils (the two EdgeLRs with their limiters, GetCornerV's, GetCornerD's)
// are read from shared memory, where one thread has the block's boxes copied
// by TMA; the metric's loads are issued meanwhile, and what the geometry alone
// gives (interpolated areas, the B map's determinant) comes from tables (see
// k_stress). 192^3, the three directions: strict 366/404/416 -> 289/299/299 us,
// FMA form 328/372/376 -> 246/248/242, FP32 211/224/225 -> 148/137/140.
template <class R, int E, int MINB>
__global__ void __launch_bounds__(EdgeTile<E>::NT, MINB)
    k_vxb(GamBox b, DevParams<R> P, Geo<R> g, Work<R> w, Range r, GamScalars* sc,
          const __grid_constant__ GamEdgeMaps maps) {
    using T_ = EdgeTile<E>;
    constexpr int eD = E, dT1 = T_::d1, dT2 = T_::d2;
    extern __shared__ __align__(128) unsigned char flux_smem[];
    __shared__ __align__(8) uint64_t bar;
    if (sc->halted) return;
    R* sm = (R*)flux_smem;
    const int tx = threadIdx.x % T_::T0, ty = threadIdx.x / T_::T0 % T_::T1, tz = threadIdx.x / (T_::T0 * T_::T1);
    const int i0 = r.i0 + blockIdx.x * T_::T0, j0 = r.j0 + blockIdx.y * T_::T1, k0 = r.k0 + blockIdx.z * T_::T2;
    if (threadIdx.x == 0) {
        tma_bar_init(&bar);
        tma_expect(&bar, GAM_COPY_BYTES(T_::all() * sizeof(R)));
#pragma unroll
        for (int q = 0; q < 6; q++)
            tma_load(sm + T_::off(q), &maps.m[q], i0 - T_::org(q, 0), j0 - T_::org(q, 1), k0 - T_::org(q, 2),
                     q == 2 ? 3 * E : (q == 0 || q == 3) ? dT1 : (q == 1 || q == 4) ? dT2 : 0, &bar);
    }
    const int ii = i0 + tx, jj = j0 + ty, kk = k0 + tz;
    const bool in = ii <= r.i1 && jj <= r.j1 && kk <= r.k1;
    const long fs = b.fs;
    const long c = lidx(b, min(ii, r.i1), min(jj, r.j1), min(kk, r.k1));
    const R* Te = g.Te + c;
    EdgeMetric<R> m;
#pragma unroll
    for (int x = 0; x < 3; x++) {
        m.t1[x] = Te[(3 + x + 9 * eD) * fs];
        m.t2[x] = Te[(6 + x + 9 * eD) * fs];
    }
    m.xni = g.Teb[(0 + 4 * eD) * fs + c];
    m.yni = g.Teb[(1 + 4 * eD) * fs + c];
    m.xnj = g.Teb[(2 + 4 * eD) * fs + c];
    m.ynj = g.Teb[(3 + 4 * eD) * fs + c];
    m.rA1 = g.rfae[(2 * eD) * fs + c];
#ifdef GAM_FAST_RECIP
    m.fA1 = m.fA2 = (R)0;  // not used
#else
    m.fA1 = g.fae[(2 * eD) * fs + c];
    m.fA2 = g.fae[(2 * eD + 1) * fs + c];
#endif
    const R dt = (R)sc->dt;
    const Quot<R> qA1(m.fA1, m.rA1), qA2(m.fA2, g.rfae[(2 * eD + 1) * fs + c]), qdt(dt, (R)sc->rdt);
    m.detT = g.rdet[eD * fs + c];
    m.edge = g.edge[eD * fs + c];
    __syncthreads();  // the barrier's initialisation
    if (!tma_wait(&bar, sc)) return;
    if (!in) return;
    {
        [[maybe_unused]] const long sA = dstride(b, dT1), sB = dstride(b, dT2), sM = sA > sB ? sA : sB;
        [[maybe_unused]] const long lo = c - sA - sB < c - 4 * sM ? c - sA - sB : c - 4 * sM;
        GAM_BOX_CHECK(lo, c + 3 * sM, 3 + 2 * eD);
    }
    edge_emf<R, E, false>(b, P, g, w, c, sm, tx, ty, tz, m, qA1, qA2, qdt, dt);
}

#endif  // GAM_GEO_TABLES

// One-sided Gaussian-moment fluxes for one side q (sgn = -1 LEFT, +1 RIGHT).
// MagKinFlux (stress.F90:513-599).
template <class R, bool BORIS = false>
__device__ __forceinline__ void mag_kin_flux(const DevParams<R>& P, R sgn, const R* W, const R* Bm, R Bn,
                                             const R* T, const double* B0, double B0n, R* mF, R& bbD, R& VaD) {
    R D = W[0], Pr = W[4];
    const Quot<R> qD(D);
    R Bx = Bm[0], By = Bm[1], Bz = Bm[2];
    R dPb = (R)0.5 * (Bx * Bx + By * By + Bz * Bz);
    R Va2;
    R B0x = (R)0, B0y = (R)0, B0z = (R)0;
    if (P.doBackground) {
        B0x = (R)B0[0]; B0y = (R)B0[1]; B0z = (R)B0[2];
        R sx = Bx + B0x, sy = By + B0y, sz = Bz + B0z;
        Va2 = qD(sx * sx + sy * sy + sz * sz);
        bbD = bbD + (R)0.5 * (sx * sx + sy * sy + sz * sz);
    } else {
        Va2 = qD((R)2 * dPb);
        bbD = bbD + (R)0.5 * (Bx * Bx + By * By + Bz * Bz);
    }
    R Vac2 = Va2;
    if constexpr (BORIS) {  // Boris-corrected Va^2
        const R Ca = (R)P.Ca;
        Vac2 = Va2 / ((R)1 + (Va2 / (Ca * Ca)));
    }
    R Nx = T[0], Ny = T[1], Nz = T[2];
    R Vn = Nx * W[1] + Ny * W[2] + Nz * W[3];
#ifdef GAM_FAST_RECIP
    // sqrt(1/x) as one reciprocal square root (about one ulp)
    const R sqlam = Mth<R>::rsqrt_(qD((R)2 * Pr) + Vac2);
#else
    R lambda = (R)1 / (qD((R)2 * Pr) + Vac2);
    const R sqlam = Mth<R>::sqrt_(lambda);
#endif
    R Vn0 = (R)0.5 * Mth<R>::erfc_(sgn * sqlam * Vn);
    VaD = VaD + (R)0.5 * Mth<R>::sqrt_(Vac2);
    mF[0] = mF[0] + Vn0 * (dPb * Nx - Bx * Bn);
    mF[1] = mF[1] + Vn0 * (dPb * Ny - By * Bn);
    mF[2] = mF[2] + Vn0 * (dPb * Nz - Bz * Bn);
    if (P.doBackground) {
        R B0nR = (R)B0n;
        R BdB0 = B0x * Bx + B0y * By + B0z * Bz;
        mF[0] = mF[0] + Vn0 * (-(B0x * Bn) - Bx * B0nR + BdB0 * Nx);
        mF[1] = mF[1] + Vn0 * (-(B0y * Bn) - By * B0nR + BdB0 * Ny);
        mF[2] = mF[2] + Vn0 * (-(B0z * Bn) - Bz * B0nR + BdB0 * Nz);
    }
}
// GasKinFlux (stress.F90:432-511)
template <class R>
__device__ __forceinline__ void gas_kin_flux(const DevParams<R>& P, R sgn, const R* W, const R* T, R* gF, R* dW) {
    R D = W[0], Pr = W[4], Vx = W[1], Vy = W[2], Vz = W[3];
    R E = (R)0.5 * D * (Vx * Vx + Vy * Vy + Vz * Vz) + over_gm1(P, Pr);
    R lambda = D / ((R)2 * Pr);
    R Vn = T[0] * Vx + T[1] * Vy + T[2] * Vz;
    R Vt1 = T[3] * Vx + T[4] * Vy + T[5] * Vz;
    R Vt2 = T[6] * Vx + T[7] * Vy + T[8] * Vz;
    const R sqlam = Mth<R>::sqrt_(lambda);
    R Vn0 = (R)0.5 * Mth<R>::erfc_(sgn * sqlam * Vn);
#ifdef GAM_FAST_RECIP
    // sqrt(pi lambda) = sqrt(pi) sqrt(lambda): one square root instead of two
    R Vn1 = Vn * Vn0 - qdiv((R)0.5 * sgn * Mth<R>::exp_(-(lambda * Vn * Vn)), (R)SQRT_PI_D * sqlam);
#else
    R Vn1 = Vn * Vn0 - qdiv((R)0.5 * sgn * Mth<R>::exp_(-(lambda * Vn * Vn)), Mth<R>::sqrt_((R)PI_D * lambda));
#endif
    gF[0] = gF[0] + D * Vn1;
    gF[4] = gF[4] + (E + (R)0.5 * Pr) * Vn1 + (R)0.5 * Pr * Vn0 * Vn;
    R fMn = D * Vn * Vn1 + Pr * Vn0;
    R fMt1 = D * Vt1 * Vn1;
    R fMt2 = D * Vt2 * Vn1;
    R fMx = T[0] * fMn + T[3] * fMt1 + T[6] * fMt2;
    R fMy = T[1] * fMn + T[4] * fMt1 + T[7] * fMt2;
    R fMz = T[2] * fMn + T[5] * fMt1 + T[8] * fMt2;
    gF[1] = gF[1] + fMx;
    gF[2] = gF[2] + fMy;
    gF[3] = gF[3] + fMz;
    dW[0] = dW[0] + sgn * D;
    dW[1] = dW[1] + sgn * D * Vx;
    dW[2] = dW[2] + sgn * D * Vy;
    dW[3] = dW[3] + sgn * D * Vz;
    dW[4] = dW[4] + sgn * E;
}

// The fluxes of face c (Fluxes, stress.F90:204-429) from its block's stencil
// boxes in shared memory (FluxTile) and its metric. SAVE (the differentiation
// form): also the face states into w.fsv, where that is not null (a run-time
// choice, so that both ways are one code with one rounding).
template <class R, int D, bool BORIS, bool SAVE>
__device__ __forceinline__ void flux_face(const GamBox& b, const DevParams<R>& P, const Work<R>& w, const GamScalars* sc,
                                          const R* __restrict__ gasN, const R* __restrict__ gasO, long c, const R* sQ,
                                          const R* sL, int tx, int tn, const Quot<R>& Vi, const R* T, R fa, R Bn,
                                          const double* B0, double B0n) {
    using T_ = FluxTile<R, D>;
    const long fs = b.fs;
    [[maybe_unused]] const long s = D == 0 ? 1L : (D == 1 ? (long)b.sx : b.sk);
    R MagL[3] = {(R)0, (R)0, (R)0}, MagR[3] = {(R)0, (R)0, (R)0};
    R WL[5], WR[5];
    // reconstruction, GRP variables at a time: their interpolants, one range
    // check for the quotients, the limiter
    constexpr int GRP = 4;
    const R* pQ = sQ + tn * T_::QX + tx;
    const R* pL = sL + tn * T_::QX + tx + (D == 0 ? 2 : 0);
    constexpr int st = D == 0 ? 1 : T_::TX;
    const int nvar = P.doMHD ? 8 : 5;
#pragma unroll
    for (int n0 = 0; n0 < 8; n0 += GRP) {
        if (n0 >= nvar) break;
        R a[2 * GRP], Qi[2 * GRP];
#pragma unroll
        for (int n = 0; n < GRP; n++) {
            const R* p = pQ + (n0 + n) * T_::QN * T_::QX;
            if (!P.up7) {
                R q[8];
#pragma unroll
                for (int m = 0; m < 8; m++) q[m] = p[m * st];
                a[n] = central8(q);
            } else {
                a[n] = p[0] * Rc<R>(up7c(0));
                a[GRP + n] = p[7 * st] * Rc<R>(up7c(0));
#pragma unroll
                for (int m = 1; m < 7; m++) {
                    a[n] = a[n] + p[m * st] * Rc<R>(up7c(m));
                    a[GRP + n] = a[GRP + n] + p[(7 - m) * st] * Rc<R>(up7c(m));
                }
            }
        }
        Vi.template many<GRP>(a, Qi);
        if (P.up7) {
            Vi.template many<GRP>(a + GRP, Qi + GRP);
        } else {
#pragma unroll
            for (int n = 0; n < GRP; n++) Qi[GRP + n] = Qi[n];
        }
#pragma unroll
        for (int n = 0; n < GRP; n++) {
            const int v = n0 + n;
            const R* p = pL + v * T_::LN * T_::QX;
            R l, u;
            pdm_both(P.pdmb, p[0], p[st], p[2 * st], p[3 * st], Qi[n], Qi[GRP + n], P.up7, l, u);
            if (v < 5) {
                WL[v] = l;
                WR[v] = u;
            } else {
                MagL[v - 5] = l;
                MagR[v - 5] = u;
            }
        }
    }
    R VaD = (R)0, bbD = (R)0;
    if (P.doMHD) {
        R mF[3] = {(R)0, (R)0, (R)0};
        mag_kin_flux<R, BORIS>(P, (R)-1, WL, MagL, Bn, T, B0, B0n, mF, bbD, VaD);
        mag_kin_flux<R, BORIS>(P, (R)1, WR, MagR, Bn, T, B0, B0n, mF, bbD, VaD);
        if constexpr (BORIS) {  // Boris hogs on the magnetic fluxes (stress.F90:335-349)
            const R Ca = (R)P.Ca;
#pragma unroll
            for (int x = 0; x < 3; x++) {
                R deeV = WR[1 + x] - WL[1 + x];
                R deeP = qdiv(bbD * deeV, Ca * Ca);
                mF[x] = mF[x] - P.cHogM * VaD * deeP;
            }
        }
#pragma unroll
        for (int x = 0; x < 3; x++) w.mF[(x + 3 * D) * fs + c] = fa * mF[x];
    }
    R gF[5] = {(R)0, (R)0, (R)0, (R)0, (R)0}, dW[5] = {(R)0, (R)0, (R)0, (R)0, (R)0};
    gas_kin_flux(P, (R)-1, WL, T, gF, dW);
    gas_kin_flux(P, (R)1, WR, T, gF, dW);
    R gv[5];
#pragma unroll
    for (int v = 0; v < 5; v++) gv[v] = gF[v] - (R)1 * P.cHogH * VaD * dW[v];
    if constexpr (BORIS) {
        // the nuclear option (stress.F90:399-417, cLim = 1.5): where the mean
        // interface speed reaches cLim Ca, diffuse with speed Ca on the jump of
        // the half-step conserved state between the face's two cells, which is
        // recomputed here (the predictor keeps primitives only)
        double vl[3] = {(double)WL[1], (double)WL[2], (double)WL[3]}, vr[3] = {(double)WR[1], (double)WR[2], (double)WR[3]};
        const R vL = (R)norm2s3(vl), vR = (R)norm2s3(vr);
        const R Vn = Mth<R>::sqrt_(vL * vL + vR * vR) / (R)GAM_SQRT2_R4;
        const R Ca = (R)P.Ca;
        if (Vn >= (R)1.5 * Ca) {
            R Ql[5], oQl[5], Qr[5], oQr[5], pQl[5], pQr[5];
#pragma unroll
            for (int v = 0; v < 5; v++) {
                Ql[v] = gasN[v * fs + c - s];
                oQl[v] = gasO[v * fs + c - s];
                Qr[v] = gasN[v * fs + c];
                oQr[v] = gasO[v * fs + c];
            }
            const R pdt = (R)sc->pdt, odt = (R)sc->odt;
            if (P.doAB3) {
                const R oodt = (R)sc->oodt;
                predict_cell_ab3(P, Ql, oQl, pdt, odt, oodt, pQl);
                predict_cell_ab3(P, Qr, oQr, pdt, odt, oodt, pQr);
            } else {
                const Quot<R> qodt(odt);
                predict_cell(P, Ql, oQl, pdt, qodt, pQl);
                predict_cell(P, Qr, oQr, pdt, qodt, pQr);
            }
#pragma unroll
            for (int v = 0; v < 5; v++) gv[v] = gv[v] - Ca * (pQr[v] - pQl[v]);
        }
    }
#pragma unroll
    for (int v = 0; v < 5; v++) w.gF[(v + 5 * D) * fs + c] = fa * gv[v];
    if (SAVE && w.fsv) {
        R* o = w.fsv + (long)(GAM_FSV_NC * D) * fs + c;
#pragma unroll
        for (int v = 0; v < 5; v++) {
            o[v * fs] = WL[v];
            o[(5 + v) * fs] = WR[v];
            o[(17 + v) * fs] = dW[v];
        }
#pragma unroll
        for (int x = 0; x < 3; x++) {
            o[(10 + x) * fs] = MagL[x];
            o[(13 + x) * fs] = MagR[x];
        }
        o[16 * fs] = VaD;
    }
}

#ifdef GAM_GEO_TABLES
// Face fluxes of direction D (Fluxes, stress.F90:204-429), one face per
// thread. The stencil operands are the per-cell products volume*primitive and
// volume*B of the half state (QdV of Cen8LRs) and the limiter values of 16
// fields. One thread has the block's tile of all of them copied to shared
// memory by TMA (four box copies, one mbarrier); the metric's loads are issued
// meanwhile. What bounds the kernel is the FP64 pipe's issue and the latency of
// the formulas' chains: with plain loads through L1 (about half of them
// missing) every variable exposed a memory latency, a third of all stalls.
// MINB bounds the registers for occupancy.
template <class R, int D, int MINB, bool BORIS = false>
__global__ void __launch_bounds__(FluxTile<R, D>::NT, MINB)
    k_stress(GamBox b, DevParams<R> P, Geo<R> g, Work<R> w, Range r, GamScalars* sc, const R* __restrict__ gasN,
             const R* __restrict__ gasO, const __grid_constant__ GamFluxMaps maps) {
    using T_ = FluxTile<R, D>;
    extern __shared__ __align__(128) unsigned char flux_smem[];
    __shared__ __align__(8) uint64_t bar;
    if (sc->halted) return;
    R* sQ = (R*)flux_smem;                // [8][QN][QX]: QW (5), QB (3)
    R* sL = (R*)(flux_smem + T_::LOFF);   // [8][LN][QX]: Wn (5), limiter B (3)
    const int tx = threadIdx.x % T_::TX, tn = threadIdx.x / T_::TX;
    const int i0 = r.i0 + blockIdx.x * T_::TX;
    const int j0 = r.j0 + blockIdx.y * (D == 2 ? 1 : T_::TN);
    const int k0 = r.k0 + blockIdx.z * (D == 2 ? T_::TN : 1);
    if (threadIdx.x == 0) {
        tma_bar_init(&bar);
        tma_expect(&bar, GAM_COPY_BYTES(P.doMHD ? T_::BYTES : T_::BYTES_GAS));
        const int qi = D == 0 ? i0 - 4 : i0, qj = D == 1 ? j0 - 4 : j0, qk = D == 2 ? k0 - 4 : k0;
        const int lj = D == 1 ? j0 - 2 : j0, lk = D == 2 ? k0 - 2 : k0;
        tma_load(sQ, &maps.QW, qi, qj, qk, 0, &bar);
        tma_load(sL, &maps.Wn, qi, lj, lk, 0, &bar);
        if (P.doMHD) {
            tma_load(sQ + 5 * T_::QN * T_::QX, &maps.QB, qi, qj, qk, 0, &bar);
            tma_load(sL + 5 * T_::LN * T_::QX, &maps.Bl, qi, lj, lk, 0, &bar);
        }
    }
    const int ii = i0 + tx, jj = D == 2 ? j0 : j0 + tn, kk = D == 2 ? k0 + tn : k0;
    const long fs = b.fs;
    [[maybe_unused]] const long s = D == 0 ? 1L : (D == 1 ? (long)b.sx : b.sk);
    // threads past the range take the range's last face (and store nothing)
    const bool in = ii <= r.i1 && jj <= r.j1 && kk <= r.k1;
    const long c = lidx(b, min(ii, r.i1), min(jj, r.j1), min(kk, r.k1));
    R T[9];
#pragma unroll
    for (int n = 0; n < 9; n++) T[n] = g.Tf[(n + 9 * D) * fs + c];
    const R fa = g.face[D * fs + c];
    const Quot<R> Vi = face_quot<R>(b, g, c, D);
    R Bn = (R)0;
    double B0[3] = {0.0, 0.0, 0.0}, B0n = 0.0;
    if (P.doMHD) {
        Bn = w.Bnf[D * fs + c];
        if (P.doBackground) {
#pragma unroll
            for (int x = 0; x < 3; x++) B0[x] = g.fcB0[(x + 3 * D) * fs + c];
            B0n = qdiv(g.bFlux0[D * fs + c], (double)fa);
        }
    }
    __syncthreads();  // the barrier's initialisation
    if (!tma_wait(&bar, sc)) return;
    if (!in) return;
    GAM_BOX_CHECK(c - 4 * s, c + 3 * s, 8 + D);
    flux_face<R, D, BORIS, false>(b, P, w, sc, gasN, gasO, c, sQ, sL, tx, tn, Vi, T, fa, Bn, B0, B0n);
}
#endif  // GAM_GEO_TABLES

// E2Flux into the new buffer; faces outside its range are copied. With
// doAB3 the buffer's old content (oState, n-1) first moves to ooState
// (CopyState(oState, ooState), mhdgroup.F90:100-102).
// Where r ends before the box, its last index stands for the box's last layer: the
// slots there of the other directions' components belong to no face, no boundary
// fills them, and they keep State's values.
template <class R>
__global__ void __launch_bounds__(256) k_update_faces(GamBox b, DevParams<R> P, StateBuf<R> cur, StateBuf<R> nxt,
                                                      Work<R> w, Range r, const GamScalars* sc, R* __restrict__ oomf) {
    if (sc->halted) return;
    int ii, jj, kk;
    if (!thread_ijk(r, ii, jj, kk)) return;
    if (ii == r.i1) ii = b.Ni;
    if (jj == r.j1) jj = b.Nj;
    if (kk == r.k1) kk = b.Nk;
    const long fs = b.fs;
    const long c = lidx(b, ii, jj, kk);
    const int G = GAM_NG;
    {
        const bool inr0 = P.doMHD && ii >= G && ii <= G + b.Nip && jj >= G && jj <= G + b.Njp && kk >= G &&
                          kk <= G + b.Nkp;
        GAM_BOX_CHECK(c, inr0 ? c + b.sk : c, 11);
    }
    if (oomf) {
#pragma unroll
        for (int x = 0; x < 3; x++) oomf[x * fs + c] = nxt.mf[x * fs + c];
    }
    const bool inr = P.doMHD && ii >= G && ii <= G + b.Nip && jj >= G && jj <= G + b.Njp && kk >= G && kk <= G + b.Nkp;
    if (!inr) {
#pragma unroll
        for (int x = 0; x < 3; x++) nxt.mf[x * fs + c] = cur.mf[x * fs + c];
        return;
    }
    const R* E = w.E;
    const long sj = b.sx, sk = b.sk;
    const R dt = (R)sc->dt;
    R dfi = E[2 * fs + c + sj] - E[2 * fs + c] - E[1 * fs + c + sk] + E[1 * fs + c];
    R dfj = E[0 * fs + c + sk] - E[0 * fs + c] - E[2 * fs + c + 1] + E[2 * fs + c];
    R dfk = E[1 * fs + c + 1] - E[1 * fs + c] - E[0 * fs + c + sj] + E[0 * fs + c];
    nxt.mf[0 * fs + c] = cur.mf[0 * fs + c] - dt * dfi;
    nxt.mf[1 * fs + c] = cur.mf[1 * fs + c] - dt * dfj;
    nxt.mf[2 * fs + c] = cur.mf[2 * fs + c] - dt * dfk;
}

__device__ __forceinline__ unsigned long long dbits(double x) { return (unsigned long long)__double_as_longlong(x); }
// Scalars of the coming step from the current ones: AdvanceMHD's time trap and
// the AB2 spacing (mhdgroup.F90:25-31, 457), Predictor (:459-463)
__device__ __forceinline__ void step_scalars(GamScalars* sc) {
    const double ot = fabs(sc->otime - sc->time) < TINY ? sc->time - sc->dt : sc->otime;
    sc->odt = sc->time - ot;
    sc->oodt = ot - sc->ootime;  // used with doAB3
    sc->pdt = 0.5 * sc->dt;
    sc->rodt = 1.0 / sc->odt;
    sc->rdt = 1.0 / sc->dt;
}
// The end of a step: time bookkeeping and CalcDT's checks (gamapp.F90:110-111,
// step.F90:58-168), by one thread; then the scalars of the next step
__device__ __forceinline__ void finalize_dt(GamScalars* sc) {
    if (fabs(sc->otime - sc->time) < TINY) sc->otime = sc->time - sc->dt;  // the time trap of this step
    sc->ootime = sc->otime;        // CopyState(oState, ooState) (mhdgroup.F90:100-102)
    sc->otime = sc->time;          // CopyState (mhdgroup.F90:255)
    sc->time = sc->time + sc->dt;  // mhdgroup.F90:106
    sc->ts = sc->ts + 1;
    sc->t = sc->t + sc->dt;
    if (sc->copyFailed) {  // its fluxes or EMFs are not those of the state
        sc->status = 6;
        sc->halted = sc->fixGhosts = 1;
        return;
    }
    if (sc->fixedTimestep) {
        step_scalars(sc);
        return;
    }
    const double dtOld = sc->dt;
    double dtMin = __longlong_as_double((long long)sc->dtmin_bits);
    sc->dtmin_bits = dbits(HUGE_DT);
    bool isDisaster = (dtMin == HUGE_DT) || sc->nbad > 0;
    bool isBad = false;
    if (sc->ts > 0) {
        if (dtOld / dtMin >= 10.0) isBad = true;
        if (sc->dt0 > TINY && dtMin / sc->dt0 <= sc->limDT0) isBad = true;
        if (dtMin <= TINY) isDisaster = true;
    }
    double dt = dtMin;
    if (sc->t + dt > sc->tFin) dt = fmax(sc->tFin - sc->t, TINY);
    if (sc->dt0 > TINY && dt > 10.0 * sc->dt0) dt = 10.0 * sc->dt0;
    sc->dt = dt;
    if (isDisaster) { sc->status = 5; sc->halted = 1; }
    else if (isBad) { sc->status = 4; sc->halted = 1; }
    else step_scalars(sc);
    sc->fixGhosts = sc->halted;
}
// The block's smallest dt candidate into the step's minimum, and whether one of
// its cells has none. The minimum only falls, so a block that is not below the
// value it reads leaves the atomic out: tens of thousands of them on one address
// (69 us of a 96 x 96 x 128 CalcDT pass, one per warp) queue up behind each other.
// last > 0: the last of that many blocks ends the step (finalize_dt).
__device__ __forceinline__ void block_min_dt(double mydt, bool bad, double* smin, GamScalars* sc, unsigned last = 0) {
    for (int o = 16; o > 0; o >>= 1) mydt = fmin(mydt, __shfl_xor_sync(0xffffffffu, mydt, o));
    const int t = threadIdx.x + blockDim.x * (threadIdx.y + blockDim.y * threadIdx.z);
    const int lane = t & 31, wid = t >> 5, nw = (blockDim.x * blockDim.y * blockDim.z + 31) >> 5;
    if (lane == 0) smin[wid] = mydt;
    const int anybad = __syncthreads_or(bad ? 1 : 0);
    if (wid == 0) {
        double v = lane < nw ? smin[lane] : HUGE_DT;
        for (int o = 16; o > 0; o >>= 1) v = fmin(v, __shfl_xor_sync(0xffffffffu, v, o));
        if (lane == 0) {
            if (v < HUGE_DT && dbits(v) < *(volatile unsigned long long*)&sc->dtmin_bits)
                atomicMin(&sc->dtmin_bits, dbits(v));
            if (anybad) atomicAdd(&sc->nbad, 1);
            if (last) {
                __threadfence();
                if (atomicAdd(&sc->done, 1u) == last - 1) {
                    sc->done = 0;
                    __threadfence();
                    finalize_dt(sc);
                }
            }
        }
    }
}

// CellDT (gridutils.F90:49-106), evaluated in FP64
template <class R, bool BORIS>
__device__ __forceinline__ double cell_dt(const DevParams<R>& P, const double* U, const double* Bt, double dl,
                                          double gamma, double gm1, double CFL) {
    double rho = U[0];
    const Quot<double> qr(rho);
    double Vel[3];
    qr.many<3>(U + 1, Vel);
    double Vx = Vel[0], Vy = Vel[1], Vz = Vel[2];
    double MagV = sqrt(Vx * Vx + Vy * Vy + Vz * Vz);
    double ke = 0.5 * rho * (MagV * MagV);
    double e = U[4] - ke;
    double Pr = gm1 * e;
    double Cs = sqrt(qr.close(gamma * Pr, rho));
    double Valf = 0.0;
    if (P.doMHD) {
        double MagB = sqrt(Bt[0] * Bt[0] + Bt[1] * Bt[1] + Bt[2] * Bt[2]);
        Valf = qdiv(MagB, sqrt(rho));
        if constexpr (BORIS) Valf = boris_speed(P.Ca, Valf);
    }
    double vCFL = MagV + sqrt(Cs * Cs + Valf * Valf) + 0.0;
    return CFL * dl / vCFL;
}

// CellBoris (mhdgroup.F90:334-382, single fluid): U2 the hydro-updated state
// (in place), U0 State n, B2 and B0 the total fields at n+1 and n
template <class R>
__device__ __forceinline__ void cell_boris(const DevParams<R>& P, R* U2, const R* U0, const R* B2, const R* B0,
                                           const R* dGasH, const R* dGasM, R Ca, R dt) {
    R W2[5];
    cell_c2p(P, U2, W2);
    const R D2 = rmax(W2[0], P.dFloor);
    const R P2 = rmax(W2[4], P.pFloor);
    const R D0 = rmax(U0[0], P.dFloor);
    R V0[3], B1[3], dPGas[3], dPMag[3], bhat1[3], dMom[3];
#pragma unroll
    for (int x = 0; x < 3; x++) {
        V0[x] = qdiv(U0[1 + x], D0);
        B1[x] = (R)0.5 * (B2[x] + B0[x]);
    }
    const R alpha = (B1[0] * B1[0] + B1[1] * B1[1] + B1[2] * B1[2]) / (D2 * Ca * Ca);
    const R dRho = dt * dGasH[0];
#pragma unroll
    for (int x = 0; x < 3; x++) {
        dPGas[x] = dt * dGasH[1 + x];
        dPMag[x] = dt * dGasM[x];
    }
    const R pCon = (R)1 / ((R)1 + alpha);
    // normVec (math.F90:332-343)
    const R nA = Mth<R>::sqrt_(B1[0] * B1[0] + B1[1] * B1[1] + B1[2] * B1[2]);
#pragma unroll
    for (int x = 0; x < 3; x++) bhat1[x] = nA <= (R)TINY ? (R)0 : B1[x] / nA;
    if (alpha > (R)TINY) {
        R sum[3];
#pragma unroll
        for (int x = 0; x < 3; x++) sum[x] = dPGas[x] + dPMag[x];
        const R pg = dPGas[0] * bhat1[0] + dPGas[1] * bhat1[1] + dPGas[2] * bhat1[2];
        const R ps = sum[0] * bhat1[0] + sum[1] * bhat1[1] + sum[2] * bhat1[2];
        const R pv = V0[0] * bhat1[0] + V0[1] * bhat1[1] + V0[2] * bhat1[2];
#pragma unroll
        for (int x = 0; x < 3; x++)
            dMom[x] = pg * bhat1[x] + pCon * (sum[x] - ps * bhat1[x]) + alpha * pCon * dRho * (V0[x] - pv * bhat1[x]);
    } else {
#pragma unroll
        for (int x = 0; x < 3; x++) dMom[x] = dPGas[x] + dPMag[x];
    }
    W2[0] = D2;
#pragma unroll
    for (int x = 0; x < 3; x++) W2[1 + x] = (D0 * V0[x] + dMom[x]) / D2;
    W2[4] = P2;
    cell_p2c(P, W2, U2);
}

// Flux2Deltas + CellReynolds + bFlux2Fld + CellMaxwell of an active cell, copy +
// bFlux2Fld of a ghost cell: the new conserved state U and field Bc
template <class R, bool BORIS, bool EXACT>
__device__ __forceinline__ void update_cell(const GamBox& b, const DevParams<R>& P, const Geo<R>& g,
                                            const StateBuf<R>& cur, const StateBuf<R>& nxt, const Work<R>& w, int ii,
                                            int jj, int kk, long c, bool active, R dt, R* U, R* Bc, bool& ok) {
    const long fs = b.fs;
    // bFlux2Fld and Flux2Deltas divide by the same cell volume
    const QuotTry<R, EXACT> qv(__ldg(g.vol + c));
    auto qdV = [&](R a) { return qv(a, ok); };
#pragma unroll
    for (int x = 0; x < 3; x++) Bc[x] = (R)0;
    if (P.doMHD) {
        const long sj = b.sx, sk = b.sk;
        int jc = jj, kc = kk;
        // RingFlux2FieldFix: a cell across the pole takes its conjugate's
        // field (the same volume, so the same quotient)
        const long cb = (P.ring.on && ring_conj_cc(b, P.ring, jc, kc)) ? lidx(b, ii, jc, kc) : c;
        cell_bxyz_q(b, g, cb, nxt.mf[cb], nxt.mf[cb + 1], nxt.mf[fs + cb], nxt.mf[fs + cb + sj], nxt.mf[2 * fs + cb],
                  nxt.mf[2 * fs + cb + sk], qdV, Bc);
    }
    if (active) {
        const long sj = b.sx, sk = b.sk;
        R dGasH[5];
#pragma unroll
        for (int v = 0; v < 5; v++) {
            const R* gI = w.gF + (v + 0) * fs;
            const R* gJ = w.gF + (v + 5) * fs;
            const R* gK = w.gF + (v + 10) * fs;
            dGasH[v] = qdV(gI[c] - gI[c + 1] + gJ[c] - gJ[c + sj] + gK[c] - gK[c + sk]);
            U[v] = cur.Gas[v * fs + c] + dt * dGasH[v];
        }
        if (P.doMHD) {
            R dGasM[3];
#pragma unroll
            for (int x = 0; x < 3; x++) {
                const R* mI = w.mF + (x + 0) * fs;
                const R* mJ = w.mF + (x + 3) * fs;
                const R* mK = w.mF + (x + 6) * fs;
                dGasM[x] = qdV(mI[c] - mI[c + 1] + mJ[c] - mJ[c + sj] + mK[c] - mK[c + sk]);
                if (P.doBackground) dGasM[x] = dGasM[x] + (R)g.dpB0[x * fs + c];
            }
            if constexpr (BORIS) {
                R U0[5], B2[3], B0[3];
#pragma unroll
                for (int v = 0; v < 5; v++) U0[v] = cur.Gas[v * fs + c];
#pragma unroll
                for (int x = 0; x < 3; x++) {
                    B2[x] = Bc[x];
                    B0[x] = cur.B[x * fs + c];
                    if (P.doBackground) {
                        const R b0 = (R)g.B0[x * fs + c];
                        B2[x] = B2[x] + b0;
                        B0[x] = B0[x] + b0;
                    }
                }
                cell_boris(P, U, U0, B2, B0, dGasH, dGasM, (R)P.Ca, dt);
            } else {
            // CellMaxwell (mhdgroup.F90:299-329)
            R D = rmax(U[0], P.dFloor);
            const QuotTry<R, EXACT> qd(D);
            auto qD = [&](R a) { return qd(a, ok); };
            R Mx = U[1], My = U[2], Mz = U[3], TotE = U[4];
            R KinE = qD((R)0.5 * (Mx * Mx + My * My + Mz * Mz));
            R Pr = rmax(P.gm1 * (TotE - KinE), P.pFloor);
            Mx = Mx + dt * dGasM[0];
            My = My + dt * dGasM[1];
            Mz = Mz + dt * dGasM[2];
            KinE = qD((R)0.5 * (Mx * Mx + My * My + Mz * Mz));
            U[0] = D;
            U[1] = Mx;
            U[2] = My;
            U[3] = Mz;
            U[4] = KinE + over_gm1<R, EXACT>(P, Pr, ok);
            }
        }
    } else {
#pragma unroll
        for (int v = 0; v < 5; v++) U[v] = cur.Gas[v * fs + c];
    }
}

// Whether the ring average or a hook may change cell (ii, jj, .) after the
// update: its CFL dt is then taken by k_dt_only (grids with rings)
template <class R> __device__ __forceinline__ bool dt_after_rings(const GamBox& b, const DevParams<R>& P, int ii, int jj) {
    const int G = GAM_NG;
    return P.doBoris || (P.ring.doS && jj < G + P.ring.NumR) || (P.ring.doE && jj >= G + b.Njp - P.ring.NumR) ||
           (P.ion.push && ii < G + P.ion.nIonP) || (P.ion.wind && ii >= G + b.Nip - 1);
}

// update_cell for every cell, then the CFL dt of cells in the dt range. Bound by
// the latency of its ~85 loads per cell: the strict form's branch at each
// quotient kept the next loads waiting (192^3: 932 -> 792 us with quick
// quotients and one check at the end; the FMA form, which has none, 640). Slower:
// the face values in shared memory by TMA (924 us, FMA 903, FP32 389 against 380),
// E2Flux in the same kernel (FMA 800 against 641 + 104, FP32 539 against 380 + 75).
template <class R, int MINB, bool BORIS = false>
__global__ void __launch_bounds__(128, MINB) k_update_cells(GamBox b, DevParams<R> P, Geo<R> g, StateBuf<R> cur,
                                                      StateBuf<R> nxt, Work<R> w, GamScalars* sc, double gamma_d,
                                                      double gm1_d, Range r, int fin) {
    __shared__ double smin[32];
    if (sc->halted) return;
    int ii, jj, kk;
    bool ok = thread_ijk(r, ii, jj, kk);
    ok = ok && GAM_BOX_OK(lidx(b, ii, jj, kk), lidx(b, ii, jj, kk) + b.sk, 12);
    double mydt = HUGE_DT;
    bool bad = false;
    if (ok) {
        const long fs = b.fs;
        const long c = lidx(b, ii, jj, kk);
        const int G = GAM_NG;
        const bool active = ii >= G && ii < G + b.Nip && jj >= G && jj < G + b.Njp && kk >= G && kk < G + b.Nkp;
        const R dt = (R)sc->dt;
        R U[5], Bc[3];
        bool tok = true;
        update_cell<R, BORIS, false>(b, P, g, cur, nxt, w, ii, jj, kk, c, active, dt, U, Bc, tok);
        if constexpr (TwoTries<R>::v) {
            if (!tok) update_cell<R, BORIS, true>(b, P, g, cur, nxt, w, ii, jj, kk, c, active, dt, U, Bc, tok);
        }
        // dt range isDT..ieDT = is-1..ie+1 (init.F90:511-530, single domain);
        // evaluated before the stores so that none of its loads waits on them
        // (PushIon and NudgeSW change the first shells and the last one after
        // the update: their dt is taken after them, by k_ion_push / k_nudge_sw)
        const bool indt = ii >= G - P.dtIlo && ii <= G + b.Nip - 1 + P.dtIhi && jj >= G - P.dtJlo &&
                          jj <= G + b.Njp - 1 + P.dtJhi && kk >= G - P.dtKlo &&
                          kk <= G + b.Nkp - 1 + P.dtKhi && !(P.ion.push && active && ii < G + P.ion.nIonP) &&
                          !(P.ion.wind && active && ii == G + b.Nip - 1);
        if (indt && !sc->fixedTimestep && !(P.ring.on && dt_after_rings(b, P, ii, jj))) {
            double Ud[5], Bt[3];
#pragma unroll
            for (int v = 0; v < 5; v++) Ud[v] = (double)U[v];
#pragma unroll
            for (int x = 0; x < 3; x++) {
                Bt[x] = (double)Bc[x];
                if (P.doBackground) Bt[x] = Bt[x] + g.B0[x * fs + c];
            }
            double dtc = cell_dt<R, BORIS>(P, Ud, Bt, (double)g.dl[c], gamma_d, gm1_d, sc->CFL);
            if (dtc > 0.0 && dtc < 1.0e300) mydt = dtc;  // finite positive
            else bad = true;
        }
#pragma unroll
        for (int v = 0; v < 5; v++) nxt.Gas[v * fs + c] = U[v];
        if (P.doMHD) {
#pragma unroll
            for (int x = 0; x < 3; x++) nxt.B[x * fs + c] = Bc[x];
        }
    }
    block_min_dt(mydt, bad, smin, sc, fin ? gridDim.x * gridDim.y * gridDim.z : 0u);
}

// ---- model hooks of the ionospheric boundary (bc[0] = 7; earthcmi.F90)
// HackE, first part: IonEFix (msphutils.F90:214-240), the J and K EMFs of
// the first shell i = is over jsg..jeg, ksg..keg from the coupling field
// (edge length x inEijk(5), formed on the host)
template <class R>
__global__ void __launch_bounds__(256) k_ion_efix(GamBox b, DevParams<R> P, Work<R> w, const GamScalars* sc) {
    if (sc->halted) return;
    const long q = blockIdx.x * (long)blockDim.x + threadIdx.x;
    if (q >= (long)b.Nj * b.Nk) return;
    const int jj = (int)(q % b.Nj), kk = (int)(q / b.Nj);
    const long c = lidx(b, GAM_NG, jj, kk);
    GAM_BOX_CHECK(c, c, 15);
    w.E[b.fs + c] = (R)P.ion.Ee[2 * q];
    w.E[2 * b.fs + c] = (R)P.ion.Ee[2 * q + 1];
}
// HackE, last part: FixEFieldLFM (gamdebug.F90:149-175), the I and J EMFs
// of k = ks and ke+1 set to their mean, i = is..ie+1, j = j0..j1 (js..je+1)
template <class R>
__global__ void __launch_bounds__(256) k_fix_e_lfm(GamBox b, R* __restrict__ E, int j0, int j1, const GamScalars* sc) {
    if (sc->halted) return;
    const int G = GAM_NG;
    const long q = blockIdx.x * (long)blockDim.x + threadIdx.x;
    const int ni = b.Nip + 1;
    if (q >= (long)ni * (j1 - j0 + 1)) return;
    const int ii = G + (int)(q % ni), jj = j0 + (int)(q / ni);
    const long c0 = lidx(b, ii, jj, G), c1 = lidx(b, ii, jj, G + b.Nkp);
    GAM_BOX_CHECK(c0, c1, 15);
    const long fs = b.fs;
    const R Ei = (R)0.5 * (E[c0] + E[c1]);
    const R Ej = (R)0.5 * (E[fs + c0] + E[fs + c1]);
    E[c0] = Ei;
    E[c1] = Ei;
    E[fs + c0] = Ej;
    E[fs + c1] = Ej;
}
// HackStep: PushIon (earthcmi.F90:586-663) on the first nIonP active
// shells after the update, then CalcDT's CellDT of those cells (k_update_cells
// leaves them out) into the step's dt minimum
template <class R, bool BORIS>
__global__ void __launch_bounds__(128) k_ion_push(GamBox b, DevParams<R> P, Geo<R> g, StateBuf<R> nxt,
                                                  GamScalars* sc, double gamma_d, double gm1_d) {
    __shared__ double smin[32];
    if (sc->halted) return;
    const int G = GAM_NG;
    const long q = blockIdx.x * (long)blockDim.x + threadIdx.x;
    const int np = P.ion.nIonP;
    double mydt = HUGE_DT;
    bool bad = false;
    if (q < (long)np * b.Njp * b.Nkp) {
        const int ii = G + (int)(q % np);
        const long r = q / np;
        const int jj = G + (int)(r % b.Njp), kk = G + (int)(r / b.Njp);
        const long fs = b.fs, c = lidx(b, ii, jj, kk);
        GAM_BOX_CHECK(c, c, 15);
        R U[5], W[5];
#pragma unroll
        for (int v = 0; v < 5; v++) U[v] = nxt.Gas[v * fs + c];
        if (!(U[0] < (R)0)) {  // RhoMin(BLK) = 0
            cell_c2p(P, U, W);
            const int dN = ii - G + 1;
            double f = sc->dt / ((double)dN * P.ion.dtCpl);
            f = (1.0 < f) ? 1.0 : f;  // min(dt, 1.0)
            const R fr = (R)f;
            const double* Vp = P.ion.Vp + 3 * q;
#pragma unroll
            for (int x = 0; x < 3; x++) {
                const R dV = (R)Vp[x] - W[1 + x];
                W[1 + x] = W[1 + x] + fr * dV;
            }
            cell_p2c(P, W, U);
#pragma unroll
            for (int v = 0; v < 5; v++) nxt.Gas[v * fs + c] = U[v];
        }
        if (!sc->fixedTimestep && !P.ring.on) {  // with rings, CalcDT runs after the ring average
            double Ud[5], Bt[3];
#pragma unroll
            for (int v = 0; v < 5; v++) Ud[v] = (double)U[v];
#pragma unroll
            for (int x = 0; x < 3; x++) {
                Bt[x] = (double)nxt.B[x * fs + c];
                if (P.doBackground) Bt[x] = Bt[x] + g.B0[x * fs + c];
            }
            const double dtc = cell_dt<R, BORIS>(P, Ud, Bt, (double)g.dl[c], gamma_d, gm1_d, sc->CFL);
            if (dtc > 0.0 && dtc < 1.0e300) mydt = dtc;
            else bad = true;
        }
    }
    block_min_dt(mydt, bad, smin, sc);
}

// HackE, wind part: WindEFix (apps/wind.F90:489-566), the EMFs of shells
// ie-2..ie+1 blended with the wind's (weights and wind EMFs formed on the
// host), then DiffuseOuter (:570-616) on the outermost, from State n's fluxes
template <class R>
__global__ void __launch_bounds__(256) k_wind_efix(GamBox b, DevParams<R> P, Geo<R> g, StateBuf<R> S, Work<R> w,
                                                   const GamScalars* sc) {
    if (sc->halted) return;
    const int G = GAM_NG;
    const long q = blockIdx.x * (long)blockDim.x + threadIdx.x;
    if (q >= 4L * (b.Njp + 1) * (b.Nkp + 1)) return;
    const int sh = (int)(q & 3);
    const long r = q >> 2;
    const int jj = G + (int)(r % (b.Njp + 1)), kk = G + (int)(r / (b.Njp + 1));
    const int ii = G + b.Nip - 3 + sh;
    const long fs = b.fs, c = lidx(b, ii, jj, kk);
    GAM_BOX_CHECK(c - b.sk, c, 15);
    const double* t = P.ion.We + 7 * q;
    // CalcElecField starts every step from E = 0 (fields.F90:88): the edges it
    // does not compute (I edges at ie+1, J edges at je+1, K edges at ke+1) hold
    // zero when the wind blends into them; here they hold last step's blend
    const bool computed[3] = {ii < G + b.Nip, jj < G + b.Njp, kk < G + b.Nkp};
#pragma unroll
    for (int n = 0; n < 3; n++) {
        const R mhdE = computed[n] ? w.E[n * fs + c] : (R)0;
        if (t[n] >= 0.0) {
            const R wSW = (R)t[n];
            w.E[n * fs + c] = ((R)1 - wSW) * mhdE + wSW * (R)t[3 + n];
        } else {
            w.E[n * fs + c] = mhdE;
        }
    }
    if (sh != 3) return;
    const long sj = b.sx, sk = b.sk;
    const R* mf = S.mf;
    const R* fa = g.face;
    R bP = mf[fs + c] / rmax(fa[fs + c], (R)TINY);
    R bM = mf[fs + c - 1] / rmax(fa[fs + c - 1], (R)TINY);
    R db2 = bP - bM;
    bP = mf[c] / fa[c];
    bM = mf[c - sj] / fa[c - sj];
    R db1 = bP - bM;
    const R JdK = db2 - db1;
    bP = mf[c] / fa[c];
    bM = mf[c - sk] / fa[c - sk];
    db2 = bP - bM;
    bP = mf[2 * fs + c] / fa[2 * fs + c];
    bM = mf[2 * fs + c - 1] / fa[2 * fs + c - 1];
    db1 = bP - bM;
    const R JdJ = db2 - db1;
    const R dl = Mth<R>::sqrt_(g.edge[fs + c] * g.edge[2 * fs + c]);
    const R Vd = rmin((R)P.ion.vSW, P.CFL * dl / (R)sc->dt);
    const R Ed[3] = {(R)0, Vd * JdJ * dl, Vd * JdK * dl};
    const R wK = (R)t[6];
#pragma unroll
    for (int x = 0; x < 3; x++) w.E[x * fs + c] = w.E[x * fs + c] + wK * Ed[x];
}
// HackStep, wind part: NudgeSW (apps/wind.F90:394-486), the last active cell
// nudged towards the wind, then its CellDT into the step's dt minimum
template <class R, bool BORIS>
__global__ void __launch_bounds__(128) k_nudge_sw(GamBox b, DevParams<R> P, Geo<R> g, StateBuf<R> nxt,
                                                  GamScalars* sc, double gamma_d, double gm1_d) {
    __shared__ double smin[32];
    if (sc->halted) return;
    const int G = GAM_NG;
    const long q = blockIdx.x * (long)blockDim.x + threadIdx.x;
    double mydt = HUGE_DT;
    bool bad = false;
    if (q < (long)b.Njp * b.Nkp) {
        const int jj = G + (int)(q % b.Njp), kk = G + (int)(q / b.Njp), ii = G + b.Nip - 1;
        const long fs = b.fs, c = lidx(b, ii, jj, kk);
        GAM_BOX_CHECK(c, c, 15);
        R U[5];
#pragma unroll
        for (int v = 0; v < 5; v++) U[v] = nxt.Gas[v * fs + c];
        const double wSW = P.ion.Wn[q];
        if (wSW > TINY) {
            const double a = P.ion.dtSW0 / wSW, dt = sc->dt;
            const double dtSW = (a < dt) ? dt : a;  // max(dtSW0 / wSW, dt)
            const R f = (R)(dt / dtSW);
            const double* ws = P.wind.state;
            const R gWs[5] = {(R)ws[0], (R)ws[2], (R)ws[3], (R)ws[4], (R)ws[1]};
            R gWm[5], gW[5];
            cell_c2p(P, U, gWm);
#pragma unroll
            for (int v = 0; v < 5; v++) gW[v] = gWm[v] + f * (gWs[v] - gWm[v]);
            cell_p2c(P, gW, U);
#pragma unroll
            for (int v = 0; v < 5; v++) nxt.Gas[v * fs + c] = U[v];
        }
        if (!sc->fixedTimestep && !P.ring.on) {  // with rings, CalcDT runs after the ring average
            double Ud[5], Bt[3];
#pragma unroll
            for (int v = 0; v < 5; v++) Ud[v] = (double)U[v];
#pragma unroll
            for (int x = 0; x < 3; x++) {
                Bt[x] = (double)nxt.B[x * fs + c];
                if (P.doBackground) Bt[x] = Bt[x] + g.B0[x * fs + c];
            }
            const double dtc = cell_dt<R, BORIS>(P, Ud, Bt, (double)g.dl[c], gamma_d, gm1_d, sc->CFL);
            if (dtc > 0.0 && dtc < 1.0e300) mydt = dtc;
            else bad = true;
        }
    }
    block_min_dt(mydt, bad, smin, sc);
}


// ----------------------------------------------------------------- ring averaging
// Ring averaging about the LFM axis (ringav.F90, ringrecon.F90,
// ringutils.F90; gid "lfm" with the reference's defaults: no shift, no
// velocity cleaning, ring variables rho, momentum, internal energy). One
// thread per ring (pole, slice i, ring nR): the ring is the k circle of row
// js+nR-1 (S) or je-nR+1 (E); its work is sequential along k in the
// reference's order, so the bits match the CPU restatement.

// PoleE (ringav.F90:394-430) over slices i0..i1, or the same touch-up of
// WindEFix (apps/wind.F90:549-564): on each pole row the K EMFs zero and the
// I EMFs their mean over ks..ke, over the whole ghosted k range
// One warp per (pole, slice): the row is staged in shared memory by the
// lanes and summed by lane 0 in k order (the CPU code's sum).
template <class R> __device__ __forceinline__ R ring_row_mean(const R* __restrict__ f, long c0, long sk, int Np, R* row) {
    const int lane = threadIdx.x;
    for (int n = lane; n < Np; n += 32) row[n] = f[c0 + n * sk];
    __syncwarp();
    R sum = (R)0;
    if (lane == 0)
        for (int n = 0; n < Np; n++) sum = sum + row[n];
    sum = __shfl_sync(0xffffffffu, sum, 0);
    return sum / (R)Np;
}
template <class R>
__global__ void __launch_bounds__(32) k_ring_pole_e(GamBox b, RingData Rg, R* __restrict__ E, int i0, int i1,
                                                    const GamScalars* sc) {
    if (sc->halted) return;
    const int G = GAM_NG, ni = i1 - i0 + 1;
    const int pole = blockIdx.x / ni, ii = i0 + (int)(blockIdx.x % ni);
    if (!(pole == 0 ? Rg.doS : Rg.doE)) return;
    const int jp = pole == 0 ? G : G + b.Njp;
    const long fs = b.fs;
    if (!GAM_BOX_OK(lidx(b, ii, jp, 0), lidx(b, ii, jp, b.Nk - 1), 15)) return;
    extern __shared__ __align__(16) unsigned char ring_smem[];
    const R avg = ring_row_mean(E, lidx(b, ii, jp, G), b.sk, Rg.Np, (R*)ring_smem);
    for (int kk = threadIdx.x; kk < b.Nk; kk += 32) {
        const long c = lidx(b, ii, jp, kk);
        E[2 * fs + c] = (R)0;
        E[c] = avg;
    }
}

// RingFlux (ringutils.F90:662-678): no flux through the pole faces (every i,
// k), then FixGasFluxLFM (gamdebug.F90:91-124): the K fluxes of k = ks and
// ke+1 set to their mean, i = is..ie, j = js..je
template <class R>
__global__ void __launch_bounds__(256) k_ring_flux(GamBox b, DevParams<R> P, Work<R> w, const GamScalars* sc) {
    if (sc->halted) return;
    const int G = GAM_NG;
    const long q = blockIdx.x * (long)blockDim.x + threadIdx.x;
    const long fs = b.fs;
    const long nz = (long)b.Ni * b.Nk;
    if (q < 2 * nz) {
        const int pole = (int)(q / nz);
        if (!(pole == 0 ? P.ring.doS : P.ring.doE)) return;
        const long r = q % nz;
        const int ii = (int)(r % b.Ni), kk = (int)(r / b.Ni);
        const long c = lidx(b, ii, pole == 0 ? G : G + b.Njp, kk);
        GAM_BOX_CHECK(c, c, 15);
#pragma unroll
        for (int v = 0; v < 5; v++) w.gF[(v + 5) * fs + c] = (R)0;
        if (P.doMHD) {
#pragma unroll
            for (int x = 0; x < 3; x++) w.mF[(x + 3) * fs + c] = (R)0;
        }
        return;
    }
    if (!P.doMHD) return;
    const long r = q - 2 * nz;
    if (r >= (long)b.Nip * b.Njp) return;
    const int ii = G + (int)(r % b.Nip), jj = G + (int)(r / b.Nip);
    const long c0 = lidx(b, ii, jj, G), c1 = lidx(b, ii, jj, G + b.Nkp);
    GAM_BOX_CHECK(c0, c1, 15);
#pragma unroll
    for (int v = 0; v < 5; v++) {
        R* gK = w.gF + (v + 10) * fs;
        const R gFa = (R)0.5 * (gK[c0] + gK[c1]);
        gK[c0] = gFa;
        gK[c1] = gFa;
    }
#pragma unroll
    for (int x = 0; x < 3; x++) {
        R* mK = w.mF + (x + 6) * fs;
        const R mFa = (R)0.5 * (mK[c0] + mK[c1]);
        mK[c0] = mFa;
        mK[c1] = mFa;
    }
}

// HackFlux = IonFlux (earthcmi.F90:357-404) on the inner tile with rings: the
// I fluxes of the first face ring at each pole (i = is, j = je then js) set
// to their ring mean, one thread per pole and component
template <class R> __global__ void __launch_bounds__(32) k_ion_flux(GamBox b, DevParams<R> P, Work<R> w,
                                                                      const GamScalars* sc) {
    if (sc->halted) return;
    const int G = GAM_NG;
    const int pole = blockIdx.x / 8, comp = blockIdx.x % 8;  // pole 0: E (je), 1: S (js); comp 0-4 gas, 5-7 magnetic
    if (!(pole == 0 ? P.ring.doE : P.ring.doS)) return;
    if (comp >= 5 && !P.doMHD) return;
    const int jr = pole == 0 ? G + b.Njp - 1 : G;
    R* f = comp < 5 ? w.gF + (long)comp * b.fs : w.mF + (long)(comp - 5) * b.fs;  // the I direction's components
    if (!GAM_BOX_OK(lidx(b, G, jr, G), lidx(b, G, jr, G + b.Nkp - 1), 15)) return;
    extern __shared__ __align__(16) unsigned char ring_smem[];
    const R avg = ring_row_mean(f, lidx(b, G, jr, G), b.sk, P.ring.Np, (R*)ring_smem);
    for (int kk = G + threadIdx.x; kk < G + b.Nkp; kk += 32) f[lidx(b, G, jr, kk)] = avg;
}

// the smoothing EMF rows each step starts from zero (InitRAVec): S rows
// js..js+NumR+1, E rows je-NumR..je+1, every i and k
template <class R> __global__ void __launch_bounds__(256) k_ring_zero_e(GamBox b, RingData Rg, const GamScalars* sc) {
    if (sc->halted) return;
    const int G = GAM_NG, nr = Rg.NumR + 2;
    const long q = blockIdx.x * (long)blockDim.x + threadIdx.x;
    const long nrow = (long)b.Ni * b.Nk;
    if (q >= 2L * nr * nrow) return;
    const int pole = (int)(q / (nr * nrow));
    if (!(pole == 0 ? Rg.doS : Rg.doE)) return;
    const long r = q % (nr * nrow);
    const int row = (int)(r / nrow), ii = (int)(r % nrow % b.Ni), kk = (int)(r % nrow / b.Ni);
    const int jj = pole == 0 ? G + row : G + b.Njp - Rg.NumR - 1 + row;
    R* E = (R*)Rg.smoothE;
    const long c = lidx(b, ii, jj, kk), fs = b.fs;
#pragma unroll
    for (int x = 0; x < 3; x++) E[x * fs + c] = (R)0;
}

// minmod (math.F90:192-197): sign() as copysign, min() as a < b
template <class R> __device__ __forceinline__ R ring_min(R a, R b2) { return b2 < a ? b2 : a; }
template <class R> __device__ __forceinline__ R ring_minmod(R x, R y) {
    return (R)0.5 * (copysign((R)1, x) + copysign((R)1, y)) * ring_min(fabs(x), fabs(y));
}
// the interval L/R of a chunk (ringrecon.F90:224-285: PPM, PLM, PCM)
template <class R>
__device__ __forceinline__ void ring_lr(int recon, R fm2, R fm1, R f, R fp1, R fp2, R& vm, R& vp) {
    if (recon == 2) {
        vm = f;
        vp = f;
        return;
    }
    if (recon == 1) {
        const R dwL = f - fm1, dwR = fp1 - f, dwC = (fp1 - fm1) / (R)2;
        const R min1 = ring_min((R)2 * fabs(dwL), (R)2 * fabs(dwR));
        const R min2 = ring_min(min1, fabs(dwC));
        const R dwM = copysign(min2, dwC);
        vp = f + (R)0.5 * dwM;
        vm = f - (R)0.5 * dwM;
        return;
    }
    const R dvm2 = fm1 - fm2, dvm1 = f - fm1, dvp1 = fp1 - f, dvp2 = fp2 - fp1;
    R dvc = (R)0.5 * (dvm2 + dvm1), SM = (R)2 * ring_minmod(dvm2, dvm1);
    const R Sm1 = ring_minmod(dvc, SM);
    dvc = (R)0.5 * (dvm1 + dvp1);
    SM = (R)2 * ring_minmod(dvm1, dvp1);
    const R Sp1 = ring_minmod(dvc, SM);
    dvc = (R)0.5 * (dvp2 + dvp1);
    SM = (R)2 * ring_minmod(dvp2, dvp1);
    const R Sp2 = ring_minmod(dvc, SM);
    vp = (R)0.5 * (f + fp1) - (Sp2 - Sp1) / (R)6;
    vm = (R)0.5 * (f + fm1) - (Sp1 - Sm1) / (R)6;
    R ap = vp - f, am = vm - f;
    if (ap * am >= (R)0) {
        ap = (R)0;
        am = (R)0;
    } else {
        if (fabs(ap) >= (R)2 * fabs(am)) ap = (R)(-2) * am;
        if (fabs(am) >= (R)2 * fabs(ap)) am = (R)(-2) * ap;
    }
    vp = f + ap;
    vm = f + am;
}
// the parabola of chunk c (1-based) from the chunk values chv(1-2 .. Nc+2)
// (ReconstructRing, ringrecon.F90:34-91): coefficients a, b, c
template <class R>
__device__ __forceinline__ void ring_parabola(int recon, const R* chW, int c, R& a, R& bq, R& cq) {
    R fL, fR;
    const R* p = chW + c + 1;  // chv(c) = chW[c + 1]
    ring_lr(recon, p[-2], p[-1], p[0], p[1], p[2], fL, fR);
    const R f = p[0];
    a = (R)3 * (fL + fR - (R)2 * f);
    bq = (R)2 * ((R)3 * f - fR - (R)2 * fL);
    cq = fL;
}
template <class R> __device__ __forceinline__ R ring_interp(R a, R bq, R cq, int m, int dJ) {
    return (a / (R)3) * (R)(3 * m * m - 3 * m + 1) / (R)(dJ * dJ) + (R)0.5 * bq * (R)(2 * m - 1) / (R)dJ + cq;
}
// periodic ghosts of the chunk values chv(1..Nc)
template <class R> __device__ __forceinline__ void ring_chunk_ghosts(R* chW, int Nc) {
    for (int n = 1; n <= 2; n++) {
        chW[1 - n + 1] = chW[Nc - n + 1 + 1];
        chW[Nc + n + 1] = chW[n + 1];
    }
}

// CalcSmoothE (ringav.F90:212-344) for one ring, one block per ring: the J
// fluxes through the ring (then the I fluxes) cleaned of Fourier modes
// 0..nft, chunk-averaged, reconstructed, dirtied again; the change of each
// face's flux accumulated along its chunk into the I (J) EMFs of the
// smoothing field. Every sum keeps the sequential order of the CPU code
// (one lane per sum); the lanes split the independent cells and chunks. A ring's
// chain of dependent steps bounds both smoothing kernels, so a block of RING_NT
// threads takes a ring's cells at once (one warp per ring took four rounds of
// loads and divisions on a ring of 128).
constexpr int RING_NT = 128;
template <class R>
__global__ void __launch_bounds__(RING_NT) k_ring_smooth_e(GamBox b, RingData Rg, StateBuf<R> S, const GamScalars* sc) {
    if (sc->halted) return;
    const int G = GAM_NG, Np = Rg.Np, nsl = b.Nip + 1, lane = threadIdx.x;
    const long t = blockIdx.x;
    const long nper = (long)nsl * Rg.NumR;
    if (t >= 2 * nper) return;
    const int pole = (int)(t / nper);
    if (!(pole == 0 ? Rg.doS : Rg.doE)) return;
    const int nS = G + (int)(t % nper % nsl), nR = 1 + (int)(t % nper / nsl);
    const int NumCh = Rg.Nch[nR - 1], dC = Np / NumCh;
    extern __shared__ __align__(16) unsigned char ring_smem[];
    R* bF = (R*)ring_smem;  // the ring's fluxes
    R* cl = bF + Np;        // cleaned fluxes, then the flux changes
    R* chW = cl + Np;       // chunk values with 2 periodic ghosts each side
    __shared__ R cf[6];     // CleanRing's coefficients (m, cos / sin)
    R* E = (R*)Rg.smoothE;
    const long fs = b.fs;
    const double* cs = Rg.ftab;
    for (int dd = 0; dd < 2; dd++) {
        const int fD = dd == 0 ? 1 : 0, eD = dd == 0 ? 0 : 1;
        const R eScl = dd == 0 ? (R)1 : (R)(-1);
        const int jf = pole == 1 ? G + b.Njp - nR : (fD == 1 ? G + nR : G + nR - 1);
        const int je = pole == 1 ? G + b.Njp - nR : (eD == 0 ? G + nR : G + nR - 1);
        const R* mf = S.mf + fD * fs;
        if (!GAM_BOX_OK(lidx(b, nS, jf, G), lidx(b, nS, jf, G + Np - 1), 15)) return;
        for (int n = lane; n < Np; n += RING_NT) bF[n] = mf[lidx(b, nS, jf, G + n)];
        __syncthreads();
        // CleanRing's coefficients: one lane per sum, sequential over the ring
        if (lane < 2 * (Rg.nft + 1)) {
            const int m = lane >> 1;
            const double* tab = cs + (long)lane * Np;  // (2 m + c) Np
            R acc = (R)0;
            for (int n = 0; n < Np; n++) acc = acc + bF[n] * (R)tab[n];
            cf[lane] = (m == 0 ? (R)0.5 * (R)Rg.aScl : (R)1 * (R)Rg.aScl) * acc;
        }
        __syncthreads();
        for (int n = lane; n < Np; n += RING_NT) {
            R Q = bF[n];
            for (int m = 0; m <= Rg.nft; m++)
                Q = Q - cf[2 * m] * (R)cs[(2 * m) * Np + n] - cf[2 * m + 1] * (R)cs[(2 * m + 1) * Np + n];
            cl[n] = Q;
        }
        __syncthreads();
        for (int c = lane; c < NumCh; c += RING_NT) {
            R sum = (R)0;
            for (int l = c * dC; l < (c + 1) * dC; l++) sum = sum + cl[l];
            chW[c + 2] = sum / (R)dC;
        }
        __syncthreads();
        if (lane == 0) ring_chunk_ghosts(chW, NumCh);
        __syncthreads();
        // reconstruct and dirty each cell, then its flux change
        for (int n = lane; n < Np; n += RING_NT) {
            const int c = n / dC, m = n - c * dC + 1;
            R a, bq, cq;
            ring_parabola(Rg.recon, chW, c + 1, a, bq, cq);
            R ra = ring_interp(a, bq, cq, m, dC);
            for (int mm = 0; mm <= Rg.nft; mm++)
                ra = ra + cf[2 * mm] * (R)cs[(2 * mm) * Np + n] + cf[2 * mm + 1] * (R)cs[(2 * mm + 1) * Np + n];
            cl[n] = ra - bF[n];
        }
        __syncthreads();
        // the changes accumulated along each chunk into the EMFs
        for (int c = lane; c < NumCh; c += RING_NT) {
            R cum = (R)0;
            for (int m = 0; m < dC; m++) {
                const int n = c * dC + m;
                const long ce = eD * fs + lidx(b, nS, je, G + n);
                if (m == 0) {
                    E[ce] = (R)0;
                    cum = -cl[n];
                } else {
                    E[ce] = eScl * cum;
                    cum = cum - cl[n];
                }
            }
        }
        __syncthreads();
        // replicate k = ks at ke+1 (chunk 0 is lane 0's)
        if (lane == 0) E[eD * fs + lidx(b, nS, je, G + Np)] = E[eD * fs + lidx(b, nS, je, G)];
        __syncthreads();
    }
}

// E2Flux with the smoothing field and dt = 1 (fields.F90:18-51) over the
// faces it changes: rows js..js+NumR and je-NumR..je, i = is..ie+1, k = ks..ke+1
template <class R> __global__ void __launch_bounds__(256) k_ring_e2flux(GamBox b, RingData Rg, StateBuf<R> S,
                                                                          const GamScalars* sc) {
    if (sc->halted) return;
    const int G = GAM_NG, nr = Rg.NumR + 1;
    const long q = blockIdx.x * (long)blockDim.x + threadIdx.x;
    const int ni = b.Nip + 1, nk = b.Nkp + 1;
    const long nrow = (long)ni * nk;
    if (q >= 2L * nr * nrow) return;
    const int pole = (int)(q / (nr * nrow));
    if (!(pole == 0 ? Rg.doS : Rg.doE)) return;
    const long r = q % (nr * nrow);
    const int row = (int)(r / nrow), ii = G + (int)(r % nrow % ni), kk = G + (int)(r % nrow / ni);
    const int jj = pole == 0 ? G + row : G + b.Njp - 1 - Rg.NumR + row;
    const R* E = (const R*)Rg.smoothE;
    const long fs = b.fs, c = lidx(b, ii, jj, kk), sj = b.sx, sk = b.sk;
    GAM_BOX_CHECK(c, c + sj + sk + 1, 15);
    const R* Ei = E;
    const R* Ej = E + fs;
    const R* Ek = E + 2 * fs;
    const R dfi = Ek[c + sj] - Ek[c] - Ej[c + sk] + Ej[c];
    const R dfj = Ei[c + sk] - Ei[c] - Ek[c + 1] + Ek[c];
    const R dfk = Ej[c + 1] - Ej[c] - Ei[c + sj] + Ei[c];
    S.mf[c] = S.mf[c] - (R)1 * dfi;
    S.mf[fs + c] = S.mf[fs + c] - (R)1 * dfj;
    S.mf[2 * fs + c] = S.mf[2 * fs + c] - (R)1 * dfk;
}

// CleanLoops (ringav.F90:347-391): the K fluxes of the pole's first ring
// lose their mean, slices is..ie+1
template <class R> __global__ void __launch_bounds__(32) k_ring_clean_loops(GamBox b, RingData Rg, StateBuf<R> S,
                                                                              const GamScalars* sc) {
    if (sc->halted) return;
    const int G = GAM_NG, ni = b.Nip + 1;
    const int pole = blockIdx.x / ni, ii = G + (int)(blockIdx.x % ni);
    if (!(pole == 0 ? Rg.doS : Rg.doE)) return;
    const int jr = pole == 0 ? G : G + b.Njp - 1;
    R* mK = S.mf + 2 * b.fs;
    if (!GAM_BOX_OK(lidx(b, ii, jr, G), lidx(b, ii, jr, G + b.Nkp), 15)) return;
    extern __shared__ __align__(16) unsigned char ring_smem[];
    const R avg = ring_row_mean(mK, lidx(b, ii, jr, G), b.sk, Rg.Np, (R*)ring_smem);
    const R tScl = (R)Rg.tScl;
    for (int kk = G + threadIdx.x; kk <= G + b.Nkp; kk += 32) {
        const long c = lidx(b, ii, jr, kk);
        mK[c] = mK[c] - tScl * avg;
    }
}

// bFlux2Fld with RingFlux2FieldFix over the cells whose faces the ring
// average changed: j rows 0..js+NumR(+1) and je-NumR-1..Nj-1, every i and k
template <class R> __global__ void __launch_bounds__(128) k_ring_bfield(GamBox b, Geo<R> g, RingData Rg,
                                                                          StateBuf<R> S, const GamScalars* sc) {
    if (sc->halted) return;
    const int G = GAM_NG, nr = G + Rg.NumR + 2;
    const long q = blockIdx.x * (long)blockDim.x + threadIdx.x;
    const long nrow = (long)b.Ni * b.Nk;
    if (q >= 2L * nr * nrow) return;
    const int pole = (int)(q / (nr * nrow));
    if (!(pole == 0 ? Rg.doS : Rg.doE)) return;
    const long r = q % (nr * nrow);
    const int row = (int)(r / nrow), ii = (int)(r % nrow % b.Ni), kk = (int)(r % nrow / b.Ni);
    const int jj = pole == 0 ? row : b.Nj - nr + row;
    const long fs = b.fs, c = lidx(b, ii, jj, kk);
    int jc = jj, kc = kk;
    const long cb = ring_conj_cc(b, Rg, jc, kc) ? lidx(b, ii, jc, kc) : c;
    GAM_BOX_CHECK(cb, cb + b.sk, 15);
    R B[3];
    cell_bxyz(b, g, cb, S.mf[cb], S.mf[cb + 1], S.mf[fs + cb], S.mf[fs + cb + b.sx], S.mf[2 * fs + cb],
              S.mf[2 * fs + cb + b.sk], B);
#pragma unroll
    for (int x = 0; x < 3; x++) S.B[x * fs + c] = B[x];
}

// SmoothGas (ringav.F90:78-210) for one ring, one block per ring: the ring
// variables (rho, momentum, internal energy; Gas2Ring, ringutils.F90:
// 804-830) chunk-averaged, reconstructed per chunk and written back as gas
// (Ring2Gas :832-856); each chunk sum sequential on one lane
template <class R>
__global__ void __launch_bounds__(RING_NT) k_ring_smooth_gas(GamBox b, DevParams<R> P, StateBuf<R> S, const GamScalars* sc) {
    if (sc->halted) return;
    const RingData& Rg = P.ring;
    const int G = GAM_NG, Np = Rg.Np, nsl = b.Nip, lane = threadIdx.x;
    const long t = blockIdx.x;
    const long nper = (long)nsl * Rg.NumR;
    if (t >= 2 * nper) return;
    const int pole = (int)(t / nper);
    if (!(pole == 0 ? Rg.doS : Rg.doE)) return;
    const int nS = G + (int)(t % nper % nsl), nR = 1 + (int)(t % nper / nsl);
    const int NumCh = Rg.Nch[nR - 1], dC = Np / NumCh;
    const int jr = pole == 0 ? G + nR - 1 : G + b.Njp - nR;
    const int cst = NumCh + 4;
    extern __shared__ __align__(16) unsigned char ring_smem[];
    R* rW = (R*)ring_smem;  // 5 x Np ring variables
    R* chW = rW + 5 * Np;   // 5 x (NumCh + 4) chunk values
    const long fs = b.fs;
    if (!GAM_BOX_OK(lidx(b, nS, jr, G), lidx(b, nS, jr, G + Np - 1), 15)) return;
    for (int n = lane; n < Np; n += RING_NT) {
        const long c = lidx(b, nS, jr, G + n);
        R W[5];
#pragma unroll
        for (int v = 0; v < 5; v++) W[v] = S.Gas[v * fs + c];
        const R D = rmax(W[0], P.dFloor);
        const R KinE = (R)0.5 * (W[1] * W[1] + W[2] * W[2] + W[3] * W[3]) / D;
        const R Pr = rmax(P.gm1 * (W[4] - KinE), P.pFloor);
        W[0] = D;
        W[4] = Pr / P.gm1;
#pragma unroll
        for (int v = 0; v < 5; v++) rW[v * Np + n] = W[v];
    }
    __syncthreads();
    for (int q = lane; q < 5 * NumCh; q += RING_NT) {
        const int v = q / NumCh, c = q % NumCh;
        R sum = (R)0;
        for (int l = c * dC; l < (c + 1) * dC; l++) sum = sum + rW[v * Np + l];
        chW[v * cst + c + 2] = sum / (R)dC;
    }
    __syncthreads();
    if (lane < 5) ring_chunk_ghosts(chW + lane * cst, NumCh);
    __syncthreads();
    for (int n = lane; n < Np; n += RING_NT) {
        const int c = n / dC, m = n - c * dC + 1;
        R W[5];
#pragma unroll
        for (int v = 0; v < 5; v++) {
            R a, bq, cq;
            ring_parabola(Rg.recon, chW + v * cst, c + 1, a, bq, cq);
            W[v] = ring_interp(a, bq, cq, m, dC);
        }
        const R D = rmax(W[0], P.dFloor);
        R Pr = P.gm1 * W[4];
        Pr = rmax(Pr, P.pFloor);
        const R KinE = (R)0.5 * (W[1] * W[1] + W[2] * W[2] + W[3] * W[3]) / D;
        const long c2 = lidx(b, nS, jr, G + n);
        S.Gas[c2] = D;
        S.Gas[fs + c2] = W[1];
        S.Gas[2 * fs + c2] = W[2];
        S.Gas[3 * fs + c2] = W[3];
        S.Gas[4 * fs + c2] = KinE + Pr / P.gm1;
    }
}

// Con2Fast (gamutils.F90:255-269 with CellPress2Cs :238-253, Boris :356-358)
template <class R> __device__ __forceinline__ R con2fast(const DevParams<R>& P, const R* gCon, const R* Bin) {
    R rho = rmax(gCon[0], P.dFloor);
    R Vx = gCon[1] / rho, Vy = gCon[2] / rho, Vz = gCon[3] / rho;
    R KinE = (R)0.5 * rho * (Vx * Vx + Vy * Vy + Vz * Vz);
    R Pr = rmax(P.gm1 * (gCon[4] - KinE), P.pFloor);
    R Cs = Mth<R>::sqrt_(P.gamma * Pr / rho);
    double Bd[3] = {(double)Bin[0], (double)Bin[1], (double)Bin[2]};
    R MagB = (R)norm2s3(Bd);
    R Va = MagB / Mth<R>::sqrt_(gCon[0]);
    if (P.doBoris) Va = boris_speed((R)P.Ca, Va);
    return Mth<R>::sqrt_(Cs * Cs + Va * Va);
}
// NudgeSW's ring branch (apps/wind.F90:458-484): the last active cell and the
// one across the E pole flow out at the fast speed when they flow in
template <class R>
__global__ void __launch_bounds__(128) k_ring_nudge_axis(GamBox b, DevParams<R> P, StateBuf<R> S, const GamScalars* sc) {
    if (sc->halted) return;
    const int G = GAM_NG;
    const long q = blockIdx.x * (long)blockDim.x + threadIdx.x;
    if (q >= 2L * b.Nkp) return;
    const int kk = G + (int)(q % b.Nkp), jj = G + b.Njp - 1 + (int)(q / b.Nkp), ii = G + b.Nip - 1;
    const long fs = b.fs, c = lidx(b, ii, jj, kk);
    GAM_BOX_CHECK(c, c, 15);
    if (!(S.Gas[fs + c] > (R)0)) return;
    R U[5], W[5], B[3];
#pragma unroll
    for (int v = 0; v < 5; v++) U[v] = S.Gas[v * fs + c];
#pragma unroll
    for (int x = 0; x < 3; x++) B[x] = S.B[x * fs + c];
    const R Cx = con2fast(P, U, B);
    cell_c2p(P, U, W);
    W[1] = -Cx;
    cell_p2c(P, W, U);
#pragma unroll
    for (int v = 0; v < 5; v++) S.Gas[v * fs + c] = U[v];
}

// UpdateStateData time bookkeeping + CalcDT decisions (gamapp.F90:110-111,
// mhdgroup.F90:106, step.F90:58-168). A failure halts the remaining kernels.
__global__ void k_dt_finalize(GamScalars* sc) {
    if (sc->halted) return;
    finalize_dt(sc);
}

// Boundary kinds: 0 periodic, 1 none, 2 zero-gradient, 3 inner sphere,
// 4 solar wind, 6 uniform inflow (include/gamgpu.h).
enum { BCK_PERIODIC = 0, BCK_NONE = 1, BCK_ZEROGRAD = 2, BCK_SPHIN = 3, BCK_WIND = 4, BCK_HALO = 5, BCK_INFLOW = 6,
       BCK_ION = 7, BCK_LFM = 8 };

// Gather maps of the boundary conditions that copy values (bcs.F90:279-450
// periodic, :799-892 zero-gradient, :934-957 SphIn). x is the box index along
// the BC's direction, n the active count, normal = the value sits on a face
// normal to that direction. Returns the source index (x when untouched).
__device__ __forceinline__ int bmap_lo(int kind, int x, int n) {
    const int G = GAM_NG;
    if (x >= G) return x;
    if (kind == BCK_PERIODIC) return x + n;
    if (kind == BCK_ZEROGRAD || kind == BCK_SPHIN) return G;
    return x;
}
__device__ __forceinline__ int bmap_hi(int kind, int x, int n, bool normal) {
    const int G = GAM_NG;
    if (normal) {
        if (x < G + n + 1 || x > G + n + 4) return x;
        if (kind == BCK_PERIODIC) return x - n;
        if (kind == BCK_ZEROGRAD) return G + n;  // magFlux(je+n+1,JDIR) = magFlux(je+1,JDIR)
        return x;
    }
    if (x < G + n || x > G + n + 3) return x;
    if (kind == BCK_PERIODIC) return x - n;
    if (kind == BCK_ZEROGRAD) return G + n - 1;
    return x;
}
// do25D periodic k: every ghost slab copies ks (bcs.F90:387-394, 423-429)
__device__ __forceinline__ int bmap_25d(int x) {
    const int G = GAM_NG;
    if ((x >= G - 4 && x < G) || (x > G && x <= G + 4)) return G;
    return x;
}

// Source of value (ii,jj,kk) of component comp (-1 cell, 0..2 face normal)
// after the K, then J, then I boundary conditions that are gathers (the
// reference applies INI, OUTI, INJ, OUTJ, INK, OUTK in that order, so a value
// ends up copied from the I-map of the J-map of the K-map of its index). Each
// map applies only over its loop ranges: periodic over the whole box,
// zero-gradient and SphIn over cell ranges of the other two indices. The
// non-periodic I sides (SphIn, wind) were applied before, in place. withB:
// follow only the BCs that also copy Bxyz (periodic and the LFM pole;
// zero-gradient does not). The LFM pole (lfmIn / lfmOut, over the whole
// box) maps a ghost row to its conjugate across the axis and reverses J and
// K fluxes: the return value is the sign of the source.
template <class R>
__device__ __forceinline__ int bc_source(const GamBox& b, const DevParams<R>& P, int comp, bool withB, int& ii,
                                         int& jj, int& kk) {
    int sgn = 1;
    if (P.do25D)
        kk = bmap_25d(kk);
    else if (P.bc[4] == BCK_PERIODIC) {
        kk = bmap_lo(BCK_PERIODIC, kk, b.Nkp);
        kk = bmap_hi(BCK_PERIODIC, kk, b.Nkp, comp == 2);
    }
    if (P.ring.on) {
        sgn = ring_bc_jmap(b, P.ring, comp, jj, kk);
    } else if (P.bc[2] == BCK_PERIODIC || (!withB && ii < b.Ni && kk < b.Nk)) {
        jj = bmap_lo(P.bc[2], jj, b.Njp);
        jj = bmap_hi(P.bc[3], jj, b.Njp, comp == 1);
    }
    if (P.bc[0] == BCK_PERIODIC) {
        ii = bmap_lo(BCK_PERIODIC, ii, b.Nip);
        ii = bmap_hi(BCK_PERIODIC, ii, b.Nip, comp == 0);
    }
    return sgn;
}


// face * (n . B) on face d of box cell c (zeroGrad_obcI, bcs.F90:842-844)
template <class R>
__device__ __forceinline__ R face_proj(const GamBox& b, const Geo<R>& g, int d, long c, const R* B) {
    const long fs = b.fs;
    const R* n = g.Tf + (long)(9 * d) * fs + c;
    return g.face[d * fs + c] * (B[0] * n[0] + B[1] * n[fs] + B[2] * n[2 * fs]);
}

// ---- the solar-wind time series (apps/wind.F90), in FP64 in both forms.
// InterpWgts (:825-868) with doWindInterp = F: the row at or below t (0-based)
__device__ __forceinline__ int wind_row(const WindData& W, double t) {
    if (t >= W.tMax) return W.n - 1;
    if (t <= W.tMin) return 0;
    const int i0 = (int)floor((t - W.tMin) / W.dtW) + 1;  // 1-based, as the reference
    return i0 + 1 <= W.n ? i0 - 1 : W.n - 2;
}
// InterpWind (:766-809) without the spin-up sequence
__device__ __forceinline__ void wind_interp(const WindData& W, double t, double& D, double& P, double* V, double* B) {
    const double* r = W.ts + 12 * wind_row(W, t);
    D = r[1];
    V[0] = r[2]; V[1] = r[3]; V[2] = r[4];
    P = r[5];
    B[1] = r[7];
    B[2] = r[8];
    B[0] = W.Bx0 + W.ByC * B[1] + W.BzC * B[2];
    if (t <= W.tMin) B[0] = B[1] = B[2] = 0.0;
}
// PlaceWind (:812-822) and RefreshWind (:116-157) at time t
__device__ __forceinline__ void wind_refresh(const WindData& W, double t, double* xyzW, double* vFr) {
    const double* r = W.ts + 12 * wind_row(W, t);
    xyzW[0] = r[9]; xyzW[1] = r[10]; xyzW[2] = r[11];
    double D, P, V0[3], B[3];
    wind_interp(W, t, D, P, V0, B);
    const double vSpd = -norm2s3(V0);
    const double bcc = sqrt(W.ByC * W.ByC + W.BzC * W.BzC);
    const double btt = sqrt(1.0 + bcc * bcc);
    if (bcc > TINY) {
        const double CosBp = W.ByC / bcc, SinBp = W.BzC / bcc, CosF = 1.0 / btt, SinF = bcc / btt;
        vFr[0] = vSpd * (CosF * CosF);
        vFr[1] = -(vSpd * CosF * SinF * CosBp);
        vFr[2] = -(vSpd * CosF * SinF * SinBp);
    } else {
        vFr[0] = vSpd; vFr[1] = 0.0; vFr[2] = 0.0;
    }
}
// GetWindAt (:160-176): the wind rewound by the lag time to xyz
__device__ __forceinline__ void wind_at(const WindData& W, const double* xyzW, const double* vFr, const double* xyz,
                                        double t, double& D, double& P, double* V, double* B) {
    const double vMag = norm2s3(vFr);
    const double DelT = ((xyz[0] - xyzW[0]) * vFr[0] + (xyz[1] - xyzW[1]) * vFr[1] + (xyz[2] - xyzW[2]) * vFr[2]) /
                        (vMag * vMag);
    wind_interp(W, t - DelT, D, P, V, B);
}
// wgtWind (:180-203) with RampDown (math.F90:97-111); CUDA's acos and exp
__device__ __forceinline__ double wind_weight(const WindData& W, const double* xyzW, const double* vFr,
                                              const double* xyz, double t) {
    double D, P, V[3], B[3];
    wind_at(W, xyzW, vFr, xyz, t, D, P, V, B);
    const double nA = sqrt(xyz[0] * xyz[0] + xyz[1] * xyz[1] + xyz[2] * xyz[2]);
    const double vA = sqrt(V[0] * V[0] + V[1] * V[1] + V[2] * V[2]);
    double c = 0.0;
#pragma unroll
    for (int x = 0; x < 3; x++) {
        const double nh = nA <= TINY ? 0.0 : xyz[x] / nA;
        const double vh = vA <= TINY ? 0.0 : V[x] / vA;
        c = x == 0 ? (-vh) * nh : c + (-vh) * nh;
    }
    const double dTh = acos(c) * 180.0 / PI_D;
    if (dTh <= 90.0) return 1.0;
    if (dTh >= 180.0) return 0.0;
    const double rScl = (dTh - 90.0) / 90.0;
    return exp(-1.0 / (1.0 - rScl * rScl) + 1.0);
}

// The non-periodic I boundaries, in place: the SphIn copy or the uniform
// inflow on the inner side (bcs.F90:934-957), the solar-wind blend
// (apps/wind.F90:206-300) or zeroGrad_obcI (bcs.F90:820-850) on the outer
// side, for ghost layer n = 1..4 of every (j, k). Writes touch ghost cells and
// ghost faces only; the reads are of the first / last active cell.
template <class R>
__global__ void __launch_bounds__(256) k_bc_iside(GamBox b, DevParams<R> P, Geo<R> g, StateBuf<R> s,
                                                  const GamScalars* sc) {
    if (sc->halted) return;
    const long t = blockIdx.x * (long)blockDim.x + threadIdx.x;
    const int n = 1 + (int)(t & 3);
    const long q = t >> 2;
    const int jj = (int)(q % (b.Nj + 1)), kk = (int)(q / (b.Nj + 1));
    if (kk > b.Nk) return;
    const long fs = b.fs;
    const int G = GAM_NG;
    const bool cellJK = jj < b.Nj && kk < b.Nk;
    GAM_BOX_CHECK(lidx(b, 0, jj, kk), lidx(b, b.Ni, jj, kk), 14);  // the row this thread writes in
    if (P.bc[0] == BCK_SPHIN && cellJK) {
        const long dst = lidx(b, G - n, jj, kk), src = lidx(b, G, jj, kk);
#pragma unroll
        for (int v = 0; v < 5; v++) s.Gas[v * fs + dst] = s.Gas[v * fs + src];
#pragma unroll
        for (int x = 0; x < 3; x++) s.mf[x * fs + dst] = s.mf[x * fs + src];
#pragma unroll
        for (int x = 0; x < 3; x++) s.B[x * fs + dst] = s.B[x * fs + src];
    }
    if (P.bc[0] == BCK_ION) {
        // IonInner (earthcmi.F90:441-583) with CellPlasmaBC (msphingest.F90:
        // 268-372, single fluid, no ingestion): density and pressure of the
        // mirror cell is+n-1 (k wrapped, lfmIJKcc ringutils.F90:482-518), the
        // velocity of the table; zero flux through the ghost layer's faces
        // (isGoodFaceIJK ranges, gridutils.F90:985-1015)
        const long cg = lidx(b, G - n, jj, kk);
        if (cellJK) {
            int kp = kk, jp = jj;
            if (kk < G) kp = kk + b.Nkp;
            else if (kk >= G + b.Nkp) kp = kk - b.Nkp;
            if (P.ring.on) {  // across the LFM pole: the conjugate's mirror cell
                int kr = kk;
                if (ring_conj_cc(b, P.ring, jp, kr)) kp = kr;
            }
            const long src = lidx(b, G + n - 1, jp, kp);
            GAM_BOX_CHECK(src, src, 14);
            R pU[5], pW[5], gC[5];
#pragma unroll
            for (int v = 0; v < 5; v++) pU[v] = s.Gas[v * fs + src];
            cell_c2p(P, pU, pW);
            const double* V = P.ion.Vg + 3 * ((n - 1) + 4 * ((long)jj + (long)b.Nj * kk));
            const R gW[5] = {pW[0], (R)V[0], (R)V[1], (R)V[2], pW[4]};
            cell_p2c(P, gW, gC);
#pragma unroll
            for (int v = 0; v < 5; v++) s.Gas[v * fs + cg] = gC[v];
        }
        if (jj < b.Nj && kk < b.Nk) s.mf[cg] = (R)0;
        if (jj <= b.Nj && kk < b.Nk) s.mf[fs + cg] = (R)0;
        if (jj < b.Nj && kk <= b.Nk) s.mf[2 * fs + cg] = (R)0;
    }
    if (P.bc[0] == BCK_INFLOW && cellJK) {
        const double* w = P.inflow;
        R gW[5] = {(R)w[0], (R)w[2], (R)w[3], (R)w[4], (R)w[1]}, gC[5];
        cell_p2c(P, gW, gC);
        const R Bin[3] = {(R)w[5], (R)w[6], (R)w[7]};
        const long c = lidx(b, G - n, jj, kk);
#pragma unroll
        for (int v = 0; v < 5; v++) s.Gas[v * fs + c] = gC[v];
#pragma unroll
        for (int d = 0; d < 3; d++) s.mf[d * fs + c] = face_proj(b, g, d, c, Bin);
    }
    if (P.bc[1] == BCK_ZEROGRAD && cellJK) {
        const int ie = G + b.Nip - 1;
        const long cp = lidx(b, ie, jj, kk), cg = lidx(b, ie + n, jj, kk);
        GAM_BOX_CHECK(cp, cp + b.sk, 14);
#pragma unroll
        for (int v = 0; v < 5; v++) s.Gas[v * fs + cg] = s.Gas[v * fs + cp];
        R B[3];
        cell_bxyz(b, g, cp, s.mf[cp], s.mf[cp + 1], s.mf[fs + cp], s.mf[fs + cp + b.sx], s.mf[2 * fs + cp],
                  s.mf[2 * fs + cp + b.sk], B);
        s.mf[cg + 1] = face_proj(b, g, 0, cg + 1, B);
        s.mf[fs + cg] = face_proj(b, g, 1, cg, B);
        s.mf[2 * fs + cg] = face_proj(b, g, 2, cg, B);
    }
    if (P.bc[1] != BCK_WIND) return;
    const WindData& W = P.wind;
    const long wi = (n - 1) + 4 * (jj + (long)(b.Nj + 1) * kk);
    const int ig = G + b.Nip - 1 + n, ip = G + b.Nip - 1;
    // a time series: RefreshWind at Model%t (the time after this step's
    // update), then the wind at each point's lag time (apps/wind.F90:218-223)
    const bool series = W.n > 0;
    const double tnow = sc->t;
    double xyzW[3] = {0.0, 0.0, 0.0}, vFr[3] = {-1.0, 0.0, 0.0};
    if (series) wind_refresh(W, tnow, xyzW, vFr);
    if (cellJK) {
        const double MinMach = 1.0;
        double wSW, Dsw = W.state[0], Psw = W.state[1], Vsw[3] = {W.state[2], W.state[3], W.state[4]};
        if (series) {
            const long cg = lidx(b, ig, jj, kk);
            const double xc[3] = {(double)g.xyzcc[cg], (double)g.xyzcc[fs + cg], (double)g.xyzcc[2 * fs + cg]};
            wSW = wind_weight(W, xyzW, vFr, xc, tnow);
            if (wSW > TINY) {
                double Bsw[3];
                wind_at(W, xyzW, vFr, xc, tnow, Dsw, Psw, Vsw, Bsw);
            }
        } else {
            wSW = W.wC[wi];
        }
        const double wMHD = 1.0 - wSW;
        R gW_sw[5] = {(R)0, (R)0, (R)0, (R)0, (R)0}, gW_in[5] = {(R)0, (R)0, (R)0, (R)0, (R)0};
        if (wSW > TINY) {
            gW_sw[0] = (R)Dsw;
            gW_sw[4] = (R)Psw;
            gW_sw[1] = (R)Vsw[0];
            gW_sw[2] = (R)Vsw[1];
            gW_sw[3] = (R)Vsw[2];
        }
        if (wMHD > TINY) {
            const long cp = lidx(b, ip, jj, kk);
            R gCon[5], Bin[3];
#pragma unroll
            for (int v = 0; v < 5; v++) gCon[v] = s.Gas[v * fs + cp];
#pragma unroll
            for (int x = 0; x < 3; x++) Bin[x] = s.B[x * fs + cp];
            cell_c2p(P, gCon, gW_in);
            // Con2Fast (gamutils.F90:255-269) with CellPress2Cs (:238-253)
            R rho = rmax(gCon[0], P.dFloor);
            R Vx = gCon[1] / rho, Vy = gCon[2] / rho, Vz = gCon[3] / rho;
            R KinE = (R)0.5 * rho * (Vx * Vx + Vy * Vy + Vz * Vz);
            R Pr = rmax(P.gm1 * (gCon[4] - KinE), P.pFloor);
            R Cs = Mth<R>::sqrt_(P.gamma * Pr / rho);
            double Bd[3] = {(double)Bin[0], (double)Bin[1], (double)Bin[2]};
            R MagB = (R)norm2s3(Bd);
            R Va = MagB / Mth<R>::sqrt_(gCon[0]);
            if (P.doBoris) Va = boris_speed((R)P.Ca, Va);
            R Cx = Mth<R>::sqrt_(Cs * Cs + Va * Va);
            const long cf = lidx(b, ip + 1, jj, kk);
            R nH[3] = {g.Tf[0 * fs + cf], g.Tf[1 * fs + cf], g.Tf[2 * fs + cf]};
            R V[3] = {gW_in[1], gW_in[2], gW_in[3]};
            R dn = V[0] * nH[0] + V[1] * nH[1] + V[2] * nH[2];
            if (dn < (R)MinMach * Cx) {
#pragma unroll
                for (int x = 0; x < 3; x++) V[x] = V[x] - dn * nH[x] + (R)MinMach * Cx * nH[x];
            }
            gW_in[1] = V[0];
            gW_in[2] = V[1];
            gW_in[3] = V[2];
        }
        R gW[5], gC[5];
#pragma unroll
        for (int v = 0; v < 5; v++) gW[v] = (R)wSW * gW_sw[v] + (R)wMHD * gW_in[v];
        cell_p2c(P, gW, gC);
        const long cg = lidx(b, ig, jj, kk);
#pragma unroll
        for (int v = 0; v < 5; v++) s.Gas[v * fs + cg] = gC[v];
    }
    // face fluxes: I face ig+1, J and K faces of cell ig
#pragma unroll
    for (int d = 0; d < 3; d++) {
        const long cf = lidx(b, d == 0 ? ig + 1 : ig, jj, kk), cin = lidx(b, d == 0 ? ip + 1 : ip, jj, kk);
        double w, sw;
        if (series) {
            // WindMagFlux (apps/wind.F90:378-391) with Project2Face (bcs.F90:250-263)
            const double xf[3] = {(double)g.xfc[(3 * d) * fs + cf], (double)g.xfc[(3 * d + 1) * fs + cf],
                                  (double)g.xfc[(3 * d + 2) * fs + cf]};
            w = wind_weight(W, xyzW, vFr, xf, tnow);
            double D, Pw, V[3], Bf[3];
            wind_at(W, xyzW, vFr, xf, tnow, D, Pw, V, Bf);
            const R* nh = g.Tf + (long)(9 * d) * fs + cf;
            sw = (double)g.face[d * fs + cf] * ((double)nh[0] * Bf[0] + (double)nh[fs] * Bf[1] + (double)nh[2 * fs] * Bf[2]);
        } else {
            w = W.wF[d * W.nw + wi];
            sw = W.sF[d * W.nw + wi];
        }
        s.mf[d * fs + cf] = (R)w * (R)sw + ((R)1 - (R)w) * s.mf[d * fs + cin];
    }
}
// Bxyz of the wind (apps/wind.F90:341-351) or inflow ghost cells from their
// new fluxes: ig = ie + n (outer) or is - n (inner)
template <class R>
__global__ void __launch_bounds__(256) k_bc_iside_b(GamBox b, Geo<R> g, StateBuf<R> s, const GamScalars* sc,
                                                    int outer, int wrapk = 0) {
    if (sc->halted) return;
    const long t = blockIdx.x * (long)blockDim.x + threadIdx.x;
    const int n = 1 + (int)(t & 3);
    const long q = t >> 2;
    const int jj = (int)(q % b.Nj), kk = (int)(q / b.Nj);
    if (kk >= b.Nk) return;
    const long fs = b.fs;
    const int ii = outer ? GAM_NG + b.Nip - 1 + n : GAM_NG - n;
    const long c = lidx(b, ii, jj, kk);
    // the ionospheric boundary takes the field of the k-wrapped cell
    // (IonInner's CellBxyz of lfmIJKcc's cell, earthcmi.F90:530-543)
    int kp = kk;
    if (wrapk && kk < GAM_NG) kp = kk + b.Nkp;
    else if (wrapk && kk >= GAM_NG + b.Nkp) kp = kk - b.Nkp;
    const long cs = lidx(b, ii, jj, kp);
    GAM_BOX_CHECK(cs, cs + b.sk, 14);
    R B[3];
    cell_bxyz(b, g, cs, s.mf[cs], s.mf[cs + 1], s.mf[fs + cs], s.mf[fs + cs + b.sx], s.mf[2 * fs + cs],
              s.mf[2 * fs + cs + b.sk], B);
#pragma unroll
    for (int x = 0; x < 3; x++) s.B[x * fs + c] = B[x];
}

// The gather boundary conditions (periodic, zero-gradient J) as one pass over
// the ghost shell, then the final bFlux2Fld of every ghost cell and of every
// cell whose faces changed. copyB: the initial EnforceBCs of CalcGridInfo
// (init.F90:226-238), which copies Bxyz with the BCs instead of recomputing it.
// The launch enumerates the shell outside the deep interior [G+1, G+N-2]^3;
// per dimension the "outer" indices are [0, G] and [G+N-1, Nmax].
struct Shell {
    int nx, ny, nz;         // face-box extents (Ni+1, Nj+1, Nk+1)
    int a[3], bnd[3];       // deep interior [a, bnd] per dimension (empty if bnd < a)
    long nA, nB, nC;        // counts of the three parts
};
static inline Shell make_shell(const GamBox& b) {
    Shell sh;
    sh.nx = b.Ni + 1; sh.ny = b.Nj + 1; sh.nz = b.Nk + 1;
    const int N[3] = {b.Nip, b.Njp, b.Nkp}, M[3] = {sh.nx, sh.ny, sh.nz};
    int nout[3], nin[3];
    for (int d = 0; d < 3; d++) {
        sh.a[d] = GAM_NG + 1;
        sh.bnd[d] = GAM_NG + N[d] - 2;
        nin[d] = sh.bnd[d] >= sh.a[d] ? sh.bnd[d] - sh.a[d] + 1 : 0;
        nout[d] = M[d] - nin[d];
    }
    sh.nA = (long)nout[2] * sh.ny * sh.nx;
    sh.nB = (long)nin[2] * nout[1] * sh.nx;
    sh.nC = (long)nin[2] * nin[1] * nout[0];
    return sh;
}
__device__ __forceinline__ int outer_coord(int o, int a, int bnd) { return (bnd >= a && o >= a) ? o - a + bnd + 1 : o; }
// 32-bit index arithmetic: a box whose fields fit the device holds far fewer
// than 2^32 positions, and the 64-bit divisions were most of the work of a
// thread with nothing to copy
__device__ __forceinline__ bool shell_ijk(const Shell& sh, unsigned t, int& ii, int& jj, int& kk) {
    const unsigned nx = sh.nx, ny = sh.ny;
    if (t < (unsigned)sh.nA) {
        const unsigned q = t / nx;
        ii = t - q * nx;
        const unsigned z = q / ny;
        jj = q - z * ny;
        kk = outer_coord((int)z, sh.a[2], sh.bnd[2]);
        return true;
    }
    t -= (unsigned)sh.nA;
    const int nin1 = sh.bnd[1] >= sh.a[1] ? sh.bnd[1] - sh.a[1] + 1 : 0;
    if (t < (unsigned)sh.nB) {
        const unsigned q = t / nx, nout1 = ny - nin1;
        ii = t - q * nx;
        const unsigned z = q / nout1;
        jj = outer_coord((int)(q - z * nout1), sh.a[1], sh.bnd[1]);
        kk = sh.a[2] + (int)z;
        return true;
    }
    t -= (unsigned)sh.nB;
    if (t < (unsigned)sh.nC) {
        const unsigned nout0 = nx - (sh.bnd[0] >= sh.a[0] ? sh.bnd[0] - sh.a[0] + 1 : 0);
        const unsigned q = t / nout0;
        ii = outer_coord((int)(t - q * nout0), sh.a[0], sh.bnd[0]);
        const unsigned z = q / (unsigned)nin1;
        jj = sh.a[1] + (int)(q - z * nin1);
        kk = sh.a[2] + (int)z;
        return true;
    }
    return false;
}

__device__ __forceinline__ bool in_range(const Range& r, int ii, int jj, int kk) {
    return ii >= r.i0 && ii <= r.i1 && jj >= r.j0 && jj <= r.j1 && kk >= r.k0 && kk <= r.k1;
}
// A step that failed CalcDT stops before its boundary conditions with the ghosts
// of its start (the update's copies, mhdgroup.F90:202-256) and their field. The
// update's ranges uc, uf leave out the layers that the boundaries fill, so those
// are copied here; the others may hold more than a copy (NudgeSW across the pole).
template <class R>
__device__ void failed_ghosts(const GamBox& b, const DevParams<R>& P, const Geo<R>& g, const StateBuf<R>& s,
                              const StateBuf<R>& cur, const Range& uc, const Range& uf, int ii, int jj, int kk,
                              bool isCell) {
    const long fs = b.fs, c = lidx(b, ii, jj, kk);
    auto face = [&](int d, int x, int y, int z) {
        const long q = d * fs + lidx(b, x, y, z);
        return in_range(uf, x, y, z) ? s.mf[q] : cur.mf[q];
    };
    if (!in_range(uf, ii, jj, kk)) {
#pragma unroll
        for (int d = 0; d < 3; d++) s.mf[d * fs + c] = cur.mf[d * fs + c];
    }
    if (!isCell || in_range(uc, ii, jj, kk)) return;
#pragma unroll
    for (int v = 0; v < 5; v++) s.Gas[v * fs + c] = cur.Gas[v * fs + c];
    if (!P.doMHD) return;
    int jb = jj, kb = kk;
    if (P.ring.on) ring_conj_cc(b, P.ring, jb, kb);  // RingFlux2FieldFix
    R B[3];
    cell_bxyz(b, g, lidx(b, ii, jb, kb), face(0, ii, jb, kb), face(0, ii + 1, jb, kb), face(1, ii, jb, kb),
              face(1, ii, jb + 1, kb), face(2, ii, jb, kb), face(2, ii, jb, kb + 1), B);
#pragma unroll
    for (int x = 0; x < 3; x++) s.B[x * fs + c] = B[x];
}

// Every load of a position comes before its first store: a source position is
// an active one that no thread writes, but the compiler cannot know that, and a
// load, store, load chain over 11 values took 25 us on a grid of 128 x 128 x 4,
// now 17; 192^3 strict 136 -> 121 us, FP32 88 -> 82. Blocks of 128 at 6 (FP64) or 8
// per SM: without the bound the loads held at once take 83 registers and FP64
// 192^3 takes 170 us.
template <class R>
__global__ void __launch_bounds__(128, sizeof(R) == 8 ? 6 : 8)
    k_bc(GamBox b, DevParams<R> P, Geo<R> g, StateBuf<R> s, StateBuf<R> cur, const GamScalars* sc, int copyB, Shell sh,
         Range uc, Range uf) {
    if (sc->halted && !(sc->fixGhosts && !copyB)) return;
    int ii, jj, kk;
    if (!shell_ijk(sh, blockIdx.x * blockDim.x + threadIdx.x, ii, jj, kk)) return;
    const long fs = b.fs;
    const long c = lidx(b, ii, jj, kk);
    GAM_BOX_CHECK(c, c, 14);
    const bool isCell = ii < b.Ni && jj < b.Nj && kk < b.Nk;
    if (sc->halted) {
        failed_ghosts(b, P, g, s, cur, uc, uf, ii, jj, kk, isCell);
        return;
    }
    R fv[3], gv[5], bv[3], B[3];
    bool fm[3], gm = false, bm = false, bnew = false;
    // faces
#pragma unroll
    for (int d = 0; d < 3; d++) {
        int x = ii, y = jj, z = kk;
        const int sg = bc_source(b, P, d, false, x, y, z);
        GAM_BOX_CHECK(lidx(b, x, y, z), lidx(b, x, y, z), 14);
        fm[d] = x != ii || y != jj || z != kk;
        if (fm[d]) {
            fv[d] = s.mf[d * fs + lidx(b, x, y, z)];
            if (sg < 0) fv[d] = -fv[d];
        }
    }
    if (isCell) {
        int x = ii, y = jj, z = kk;
        bc_source(b, P, -1, false, x, y, z);
        GAM_BOX_CHECK(lidx(b, x, y, z), lidx(b, x, y, z), 14);
        gm = x != ii || y != jj || z != kk;
        if (gm) {
            const long src = lidx(b, x, y, z);
#pragma unroll
            for (int v = 0; v < 5; v++) gv[v] = s.Gas[v * fs + src];
        }
        if (copyB) {
            int xb = ii, yb = jj, zb = kk;
            bc_source(b, P, -1, true, xb, yb, zb);
            GAM_BOX_CHECK(lidx(b, xb, yb, zb), lidx(b, xb, yb, zb), 14);
            bm = xb != ii || yb != jj || zb != kk;
            if (bm) {
                const long src = lidx(b, xb, yb, zb);
#pragma unroll
                for (int q = 0; q < 3; q++) bv[q] = s.B[q * fs + src];
            }
        } else if (P.doMHD) {
            // the six faces of this cell after the boundary fill
            auto srcf = [&](int d, int a0, int a1, int a2) -> long {
                int x = a0, y = a1, z = a2;
                bc_source(b, P, d, false, x, y, z);
                return lidx(b, x, y, z);
            };
            // RingFlux2FieldFix: a cell across the LFM pole takes its conjugate's field
            int jb = jj, kb = kk;
            const bool conj = P.ring.on && ring_conj_cc(b, P.ring, jb, kb);
            const long fI = srcf(0, ii, jb, kb), fIp = srcf(0, ii + 1, jb, kb);
            const long fJ = srcf(1, ii, jb, kb), fJp = srcf(1, ii, jb + 1, kb);
            const long fK = srcf(2, ii, jb, kb), fKp = srcf(2, ii, jb, kb + 1);
            {
                long lo = fI, hi = fI;
                for (long v : {fIp, fJ, fJp, fK, fKp}) {
                    lo = v < lo ? v : lo;
                    hi = v > hi ? v : hi;
                }
                GAM_BOX_CHECK(lo, hi, 14);
            }
            const bool facesMapped = fI != c || fIp != c + 1 || fJ != c || fJp != c + b.sx || fK != c || fKp != c + b.sk;
            const int G = GAM_NG;
            const bool ghost =
                ii < G || ii >= G + b.Nip || jj < G || jj >= G + b.Njp || kk < G || kk >= G + b.Nkp;
            bnew = ghost || facesMapped;
            if (bnew)
                cell_bxyz(b, g, conj ? lidx(b, ii, jb, kb) : c, s.mf[fI], s.mf[fIp], s.mf[fs + fJ], s.mf[fs + fJp],
                          s.mf[2 * fs + fK], s.mf[2 * fs + fKp], B);
        }
    }
#pragma unroll
    for (int d = 0; d < 3; d++)
        if (fm[d]) s.mf[d * fs + c] = fv[d];
    if (gm) {
#pragma unroll
        for (int v = 0; v < 5; v++) s.Gas[v * fs + c] = gv[v];
    }
    if (bm || bnew) {
#pragma unroll
        for (int x = 0; x < 3; x++) s.B[x * fs + c] = bm ? bv[x] : B[x];
    }
}

// All boundary conditions of one EnforceBCs (+ final bFlux2Fld unless copyB).
// S: the state to fill; cur: the step's start, uc and uf: the cells and faces that
// the update wrote (a failed step's ghosts)
template <class R>
void launch_bcs(const Ctx<R>& C, const StateBuf<R>& S, const StateBuf<R>& cur, const Range& uc, const Range& uf,
                cudaStream_t s, int copyB) {
    const GamBox& b = C.b;
    const bool iside = C.P.bc[0] == BCK_SPHIN || C.P.bc[0] == BCK_INFLOW || C.P.bc[0] == BCK_ION ||
                       C.P.bc[1] == BCK_WIND || C.P.bc[1] == BCK_ZEROGRAD;
    if (iside) {
        const long n = 4L * (b.Nj + 1) * (b.Nk + 1);
        k_bc_iside<R><<<(unsigned)((n + 255) / 256), 256, 0, s>>>(b, C.P, C.g, S, C.sc);
        // the wind's and the inflow's own Bxyz of their ghost cells matter
        // only where no final bFlux2Fld follows (the initial fill); a step
        // recomputes every ghost
        const long m = 4L * b.Nj * b.Nk;
        if (C.P.bc[1] == BCK_WIND && copyB)
            k_bc_iside_b<R><<<(unsigned)((m + 255) / 256), 256, 0, s>>>(b, C.g, S, C.sc, 1);
        if (C.P.bc[0] == BCK_INFLOW && copyB)
            k_bc_iside_b<R><<<(unsigned)((m + 255) / 256), 256, 0, s>>>(b, C.g, S, C.sc, 0);
        if (C.P.bc[0] == BCK_ION && copyB)
            k_bc_iside_b<R><<<(unsigned)((m + 255) / 256), 256, 0, s>>>(b, C.g, S, C.sc, 0, 1);
    }
    const Shell sh = make_shell(b);
    const long nsh = sh.nA + sh.nB + sh.nC;
    k_bc<R><<<(unsigned)((nsh + 127) / 128), 128, 0, s>>>(b, C.P, C.g, S, cur, C.sc, copyB, sh, uc, uf);
}

// CalcDT on a state without changing it (gam_calc_dt): min of CellDT over
// the dt range into sc->dtmin_bits. As a part of a step (countBad): of the cells
// that the update left to it.
template <class R>
__global__ void __launch_bounds__(128) k_dt_only(GamBox b, DevParams<R> P, Geo<R> g, StateBuf<R> s,
                                                 GamScalars* sc, double gamma_d, double gm1_d, int countBad) {
    __shared__ double smin[32];
    int ii, jj, kk;
    const int G = GAM_NG;
    Range r{G - P.dtIlo, G + b.Nip - 1 + P.dtIhi, G - P.dtJlo, G + b.Njp - 1 + P.dtJhi, G - P.dtKlo,
            G + b.Nkp - 1 + P.dtKhi};
    double mydt = HUGE_DT;
    bool bad = false;
    if (thread_ijk(r, ii, jj, kk) && !(countBad && !dt_after_rings(b, P, ii, jj)) &&
        GAM_BOX_OK(lidx(b, ii, jj, kk), lidx(b, ii, jj, kk), 13)) {
        const long fs = b.fs;
        const long c = lidx(b, ii, jj, kk);
        double Ud[5], Bt[3] = {0.0, 0.0, 0.0};
#pragma unroll
        for (int v = 0; v < 5; v++) Ud[v] = (double)s.Gas[v * fs + c];
        if (P.doMHD) {
#pragma unroll
            for (int x = 0; x < 3; x++) {
                Bt[x] = (double)s.B[x * fs + c];
                if (P.doBackground) Bt[x] = Bt[x] + g.B0[x * fs + c];
            }
        }
        double dtc = P.doBoris ? cell_dt<R, true>(P, Ud, Bt, (double)g.dl[c], gamma_d, gm1_d, sc->CFL)
                                : cell_dt<R, false>(P, Ud, Bt, (double)g.dl[c], gamma_d, gm1_d, sc->CFL);
        if (dtc > 0.0 && dtc < 1.0e300) mydt = dtc;
        else bad = countBad != 0;
    }
    if (sc->fixedTimestep && countBad) return;
    block_min_dt(mydt, bad, smin, sc);
}


// bFlux2Fld over every cell of a state (gridutils.F90:281-301)
template <class R>
__global__ void __launch_bounds__(128) k_bfield_all(GamBox b, Geo<R> g, StateBuf<R> s, const GamScalars* sc,
                                                    RingData ring) {
    int ii, jj, kk;
    Range r{0, b.Ni - 1, 0, b.Nj - 1, 0, b.Nk - 1};
    if (!thread_ijk(r, ii, jj, kk)) return;
    const long fs = b.fs;
    const long c = lidx(b, ii, jj, kk);
    int jc = jj, kc = kk;
    const long cb = (ring.on && ring_conj_cc(b, ring, jc, kc)) ? lidx(b, ii, jc, kc) : c;
    GAM_BOX_CHECK(cb, cb + b.sk, 16);
    R B[3];
    cell_bxyz(b, g, cb, s.mf[cb], s.mf[cb + 1], s.mf[fs + cb], s.mf[fs + cb + b.sx], s.mf[2 * fs + cb],
              s.mf[2 * fs + cb + b.sk], B);
#pragma unroll
    for (int x = 0; x < 3; x++) s.B[x * fs + c] = B[x];
}

// ----------------------------------------------------------------- launches
// The grids of FluxTile's blocks over the faces r of direction D, and of EdgeTile's
// over the edges r of direction E
template <class R, int D> dim3 flux_grid(const Range& r) {
    using T_ = FluxTile<R, D>;
    return dim3((unsigned)((r.i1 - r.i0 + T_::TX) / T_::TX),
                (unsigned)(D == 2 ? r.j1 - r.j0 + 1 : (r.j1 - r.j0 + T_::TN) / T_::TN),
                (unsigned)(D == 2 ? (r.k1 - r.k0 + T_::TN) / T_::TN : r.k1 - r.k0 + 1));
}
template <int E> dim3 edge_grid(const Range& r) {
    using T_ = EdgeTile<E>;
    return dim3((unsigned)((r.i1 - r.i0 + T_::T0) / T_::T0), (unsigned)((r.j1 - r.j0 + T_::T1) / T_::T1),
                (unsigned)((r.k1 - r.k0 + T_::T2) / T_::T2));
}
#ifdef GAM_GEO_TABLES  // the builds that hold the step
static inline dim3 grid_for(const Range& r, dim3 blk) {
    return dim3((unsigned)((r.i1 - r.i0 + 1 + blk.x - 1) / blk.x), (unsigned)((r.j1 - r.j0 + 1 + blk.y - 1) / blk.y),
                (unsigned)((r.k1 - r.k0 + 1 + blk.z - 1) / blk.z));
}

template <class R, int E> void launch_vxb(const Ctx<R>& C, const Range& r, cudaStream_t s) {
    using T_ = EdgeTile<E>;
    const dim3 gr = edge_grid<E>(r);
    const unsigned sm = T_::all() * sizeof(R);
    // blocks of 256 per SM: 3 in FP64 (strict 289/299/299 us for the three
    // directions at 192^3; 2: 372/376/377, 4: 305/313/325), 5 in FP32
    // (148/137/140; 4: 156/152/154)
    k_vxb<R, E, sizeof(R) == 4 ? 5 : 3><<<gr, T_::NT, sm, s>>>(C.b, C.P, C.g, C.w, r, C.sc, C.fmaps->e[E]);
}

// RingAverage (ringav.F90:26-75), its magnetic part on the new fluxes: smoothing
// EMFs of both poles, PoleE and FixEFieldLFM on them, E2Flux with dt = 1, CleanLoops
template <class R> void launch_ring_flux_average(const Ctx<R>& C, const StateBuf<R>& O, cudaStream_t s) {
    const GamBox& b = C.b;
    const RingData& Rg = C.P.ring;
    const int G = GAM_NG;
    const long nz = 2L * (Rg.NumR + 2) * b.Ni * b.Nk;
    k_ring_zero_e<R><<<(unsigned)((nz + 255) / 256), 256, 0, s>>>(b, Rg, C.sc);
    const long ne = 2L * (b.Nip + 1) * Rg.NumR;
    const size_t smE = (size_t)(2 * Rg.Np + Rg.chunkStride / 5) * sizeof(R);
    k_ring_smooth_e<R><<<(unsigned)ne, RING_NT, smE, s>>>(b, Rg, O, C.sc);
    R* E = (R*)Rg.smoothE;
    const int ni = b.Nip + 1;
    k_ring_pole_e<R><<<(unsigned)(2 * ni), 32, Rg.Np * sizeof(R), s>>>(b, Rg, E, G, G + b.Nip, C.sc);
    // FixEFieldLFM over the rows that can be nonzero (the others hold zeros)
    const int sj1 = std::min(G + Rg.NumR + 1, G + b.Njp), ej0 = std::max(G + b.Njp - 1 - Rg.NumR, G);
    if (Rg.doS)
        k_fix_e_lfm<R><<<(unsigned)(((long)ni * (sj1 - G + 1) + 255) / 256), 256, 0, s>>>(b, E, G, sj1, C.sc);
    if (Rg.doE)
        k_fix_e_lfm<R><<<(unsigned)(((long)ni * (G + b.Njp - ej0 + 1) + 255) / 256), 256, 0, s>>>(
            b, E, ej0, G + b.Njp, C.sc);
    const long nf = 2L * (Rg.NumR + 1) * (b.Nip + 1) * (b.Nkp + 1);
    k_ring_e2flux<R><<<(unsigned)((nf + 255) / 256), 256, 0, s>>>(b, Rg, O, C.sc);
    if (Rg.clean) k_ring_clean_loops<R><<<(unsigned)(2 * ni), 32, Rg.Np * sizeof(R), s>>>(b, Rg, O, C.sc);
}
// ... bFlux2Fld of the cells around the rings
template <class R> void launch_ring_field(const Ctx<R>& C, const StateBuf<R>& O, cudaStream_t s) {
    const long nb = 2L * (GAM_NG + C.P.ring.NumR + 2) * C.b.Ni * C.b.Nk;
    k_ring_bfield<R><<<(unsigned)((nb + 127) / 128), 128, 0, s>>>(C.b, C.g, C.P.ring, O, C.sc);
}
// ... and SmoothGas of both poles on the updated state
template <class R> void launch_ring_gas_average(const Ctx<R>& C, const StateBuf<R>& O, cudaStream_t s) {
    const RingData& Rg = C.P.ring;
    const long ng = 2L * C.b.Nip * Rg.NumR;
    const size_t smG = (size_t)(5 * Rg.Np + Rg.chunkStride) * sizeof(R);
    k_ring_smooth_gas<R><<<(unsigned)ng, RING_NT, smG, s>>>(C.b, C.P, O, C.sc);
}

// The kernels of one stepGamera in order, each handed to f(id, launch) with
// id: 0 begin, 1 predict, 2/3 mom2face/vxb I, 4/5 J, 6/7 K, 8/9/10 stress
// I/J/K, 11 update_faces, 12 update_cells, 13 dt_finalize, 14 bc.
// st[cur] is State (n); st[1-cur] holds oState (n-1) on entry and State
// (n+1) on exit.
template <class R, class F> void for_each_kernel(const Ctx<R>& C, int cur, cudaStream_t& s, F&& f, int fold = 0) {
    const GamBox& b = C.b;
    const int G = GAM_NG;
    const StateBuf<R> S = C.st[cur], O = C.st[1 - cur];
    const dim3 blk(32, 4, 1);
    const Range all{0, b.Ni, 0, b.Nj, 0, b.Nk};
    // The update copies State n into the ghosts. Those of a periodic direction are
    // all filled by the step's boundaries, so there only the one layer that CalcDT
    // looks at is needed (at 128 x 128 x 4 less than half of the box, at 192^3 91 %;
    // a step of that small grid 0.161 -> 0.149 ms with this and k_bc's loads).
    Range cells{0, b.Ni - 1, 0, b.Nj - 1, 0, b.Nk - 1}, faces = all;
    const int N[3] = {b.Nip, b.Njp, b.Nkp};
    int* lim[3][4] = {{&cells.i0, &cells.i1, &faces.i0, &faces.i1}, {&cells.j0, &cells.j1, &faces.j0, &faces.j1},
                      {&cells.k0, &cells.k1, &faces.k0, &faces.k1}};
    for (int d = 0; d < 3; d++) {
        if (C.P.bc[2 * d] != BCK_PERIODIC || C.P.bc[2 * d + 1] != BCK_PERIODIC || (d == 2 && C.P.do25D)) continue;
        // rows start where the box's do: a warp's values lie in whole lines then
        *lim[d][0] = d == 0 ? 0 : G - 1;
        *lim[d][1] = G + N[d];
        if (!C.oomf) {  // ooState takes the fluxes of every face
            *lim[d][2] = *lim[d][0];
            *lim[d][3] = G + N[d] + 1;
        }
    }
    const int kke = C.P.do25D ? G : G + b.Nkp - 1;  // last active k of the stress sweep
    f(0, [&] { k_step_begin<<<1, 1, 0, s>>>(C.sc); });
    const dim3 pblk(32, 8, 1);
    f(1, [&] {
        if (C.P.doAB3)
            k_predict<R, sizeof(R) == 8 ? 3 : 4, true><<<grid_for(all, pblk), pblk, 0, s>>>(b, C.P, C.g, S, O, C.w, C.sc,
                                                                                          C.oomf);
        else  // 3 blocks/SM in FP64 (192^3, strict: 661 us; 4: 745, 2: 754), 4 in FP32
            k_predict<R, sizeof(R) == 8 ? 3 : 4><<<grid_for(all, pblk), pblk, 0, s>>>(b, C.P, C.g, S, O, C.w, C.sc, nullptr);
    });
    if (C.P.doMHD) {
        // the faces whose velocities the edges' stencils (along dT2) take (the
        // ghosts left out: 192^3 strict 375 -> 353 us for the three)
        const Range mf[3] = {{G, G + b.Nip - 1, G, G + b.Njp, 0, b.Nk - 1},
                             {0, b.Ni - 1, G, G + b.Njp - 1, G, G + b.Nkp},
                             {G, G + b.Nip, 0, b.Nj - 1, G, G + b.Nkp - 1}};
        const Range ed[3] = {{G, G + b.Nip - 1, G, G + b.Njp, G, G + b.Nkp},
                             {G, G + b.Nip, G, G + b.Njp - 1, G, G + b.Nkp},
                             {G, G + b.Nip, G, G + b.Njp, G, G + b.Nkp - 1}};
        for (int eD = 0; eD < 3; eD++) {
            f(2 + 2 * eD, [&] { k_mom2face<R><<<grid_for(mf[eD], blk), blk, 0, s>>>(b, C.P, C.g, C.w, eD, mf[eD], C.sc); });
            f(3 + 2 * eD, [&] {
                if (eD == 0) launch_vxb<R, 0>(C, ed[0], s);
                else if (eD == 1) launch_vxb<R, 1>(C, ed[1], s);
                else launch_vxb<R, 2>(C, ed[2], s);
            });
        }
    }
    const Range fr[3] = {{G, G + b.Nip, G, G + b.Njp - 1, G, kke},
                         {G, G + b.Nip - 1, G, G + b.Njp, G, kke},
                         {G, G + b.Nip - 1, G, G + b.Njp - 1, G, G + b.Nkp}};
    auto stress = [&](auto Dc) {
        constexpr int D = decltype(Dc)::value;
        const Range& r = fr[D];
        using T_ = FluxTile<R, D>;
        const dim3 sg = flux_grid<R, D>(r);
        const GamFluxMaps& M = C.fmaps->m[cur][D];
        // blocks per SM (registers against warps; 192^3, I/J/K sweeps): the strict
        // form 5 (782/739/808 us; 4: 852/770/775, 7: 895/854/859), the FMA form 5
        // (598/560/563; 4: 627/576/586, 6: 648/611/636), FP32 5 of 256 threads on
        // the J and K sweeps (263/264; 4: 269/275) and 7 of 128 on the I sweep
        constexpr int MB = sizeof(R) == 8 ? 5 : (D == 0 ? 7 : 5);
        if (C.P.doBoris)
            k_stress<R, D, sizeof(R) == 8 ? 5 : 3, true><<<sg, T_::NT, T_::SMEM, s>>>(b, C.P, C.g, C.w, r, C.sc, S.Gas, O.Gas, M);
        else
            k_stress<R, D, MB><<<sg, T_::NT, T_::SMEM, s>>>(b, C.P, C.g, C.w, r, C.sc, S.Gas, O.Gas, M);
    };
    f(8, [&] { stress(std::integral_constant<int, 0>()); });
    f(9, [&] { stress(std::integral_constant<int, 1>()); });
    if (!C.P.do25D) f(10, [&] { stress(std::integral_constant<int, 2>()); });
    f(11, [&] {
        if (C.P.ion.on && C.P.doMHD) {  // HackE (EFix, earthcmi.F90:321-354)
            const long ne = (long)b.Nj * b.Nk, nf = (long)(b.Nip + 1) * (b.Njp + 1);
            if (C.P.bc[0] == BCK_ION)  // the inner tile (hasLowerBC(IDIR))
                k_ion_efix<R><<<(unsigned)((ne + 255) / 256), 256, 0, s>>>(b, C.P, C.w, C.sc);
            if (C.P.ion.wind) {
                const long nw = 4L * (b.Njp + 1) * (b.Nkp + 1);
                k_wind_efix<R><<<(unsigned)((nw + 255) / 256), 256, 0, s>>>(b, C.P, C.g, S, C.w, C.sc);
                if (C.P.ring.on)  // WindEFix's touch-up of the pole rows of its shells
                    k_ring_pole_e<R><<<8, 32, C.P.ring.Np * sizeof(R), s>>>(b, C.P.ring, C.w.E, GAM_NG + b.Nip - 3,
                                                                          GAM_NG + b.Nip, C.sc);
            }
            if (C.P.bc[4] != BCK_HALO)
                k_fix_e_lfm<R><<<(unsigned)((nf + 255) / 256), 256, 0, s>>>(b, C.w.E, GAM_NG, GAM_NG + b.Njp, C.sc);
        }
        if (C.P.ring.on && C.P.doMHD) {  // PoleE before E2Flux (mhdgroup.F90:140-142)
            const int ni = b.Nip + 1;
            k_ring_pole_e<R><<<(unsigned)(2 * ni), 32, C.P.ring.Np * sizeof(R), s>>>(b, C.P.ring, C.w.E, GAM_NG,
                                                                                    GAM_NG + b.Nip, C.sc);
            const long nf = (long)ni * (b.Njp + 1);
            k_fix_e_lfm<R><<<(unsigned)((nf + 255) / 256), 256, 0, s>>>(b, C.w.E, GAM_NG, GAM_NG + b.Njp, C.sc);
        }
        Range fl = faces;  // with the last layers
        fl.i1 += fl.i1 < b.Ni;
        fl.j1 += fl.j1 < b.Nj;
        fl.k1 += fl.k1 < b.Nk;
        k_update_faces<R><<<grid_for(fl, blk), blk, 0, s>>>(b, C.P, S, O, C.w, fl, C.sc, C.oomf);
        // RingAverage's magnetic part takes the new fluxes alone, and only CellBoris
        // looks at the field before it: here it runs beside the flux sweeps, and the
        // update finds the averaged fluxes (96 x 96 x 128 cells: 65 us of small launches
        // beside the sweeps, and the field around the rings formed once, 20 us)
        if (C.P.ring.on && C.P.doMHD && !C.P.doBoris) launch_ring_flux_average(C, O, s);
    });
    f(12, [&] {
        if (C.P.ring.on) {  // RingFlux (stress.F90:137-139), before the fluxes become deltas
            const long n = 2L * b.Ni * b.Nk + (long)b.Nip * b.Njp;
            k_ring_flux<R><<<(unsigned)((n + 255) / 256), 256, 0, s>>>(b, C.P, C.w, C.sc);
            if (C.P.bc[0] == BCK_ION && C.P.ion.on)
                k_ion_flux<R><<<16, 32, C.P.ring.Np * sizeof(R), s>>>(b, C.P, C.w, C.sc);
        }
        if (C.P.doBoris)
            k_update_cells<R, sizeof(R) == 8 ? 6 : 8, true><<<grid_for(cells, blk), blk, 0, s>>>(b, C.P, C.g, S, O, C.w, C.sc, C.gamma, C.gm1, cells, fold);
        else  // strict: 5 blocks/SM (792 us at 192^3; 6: 836; dipole of 1.2e6 cells 158, 6: 171); the other forms 8 (FMA: 643 us; 7: 650, 6: 710)
            k_update_cells<R, GAM_STRICT_KERNELS ? 5 : 8><<<grid_for(cells, blk), blk, 0, s>>>(b, C.P, C.g, S, O, C.w, C.sc, C.gamma, C.gm1, cells, fold);
        if (C.P.ring.on) {  // RingAverage (mhdgroup.F90:69-74)
            if (C.P.doMHD && C.P.doBoris) {
                launch_ring_flux_average(C, O, s);
                launch_ring_field(C, O, s);
            }
            launch_ring_gas_average(C, O, s);
        }
        if (C.P.ion.push) {  // HackStep (PerStep, earthcmi.F90:224-263): PushIon, before CalcDT
            const long np = (long)C.P.ion.nIonP * b.Njp * b.Nkp;
            if (C.P.doBoris)
                k_ion_push<R, true><<<(unsigned)((np + 127) / 128), 128, 0, s>>>(b, C.P, C.g, O, C.sc, C.gamma, C.gm1);
            else
                k_ion_push<R, false><<<(unsigned)((np + 127) / 128), 128, 0, s>>>(b, C.P, C.g, O, C.sc, C.gamma, C.gm1);
        }
        if (C.P.ion.wind) {  // HackStep, wind part: NudgeSW
            const long nn = (long)b.Njp * b.Nkp;
            if (C.P.doBoris)
                k_nudge_sw<R, true><<<(unsigned)((nn + 127) / 128), 128, 0, s>>>(b, C.P, C.g, O, C.sc, C.gamma, C.gm1);
            else
                k_nudge_sw<R, false><<<(unsigned)((nn + 127) / 128), 128, 0, s>>>(b, C.P, C.g, O, C.sc, C.gamma, C.gm1);
            if (C.P.ring.on && C.P.ring.doE)
                k_ring_nudge_axis<R><<<(unsigned)((2 * b.Nkp + 127) / 128), 128, 0, s>>>(b, C.P, O, C.sc);
        }
        if (C.P.ring.on) {  // CalcDT after the ring average and the hooks (gamapp.F90:78-80)
            const dim3 blk2(32, 4, 1);
            const Range r{GAM_NG - C.P.dtIlo, GAM_NG + b.Nip - 1 + C.P.dtIhi, GAM_NG - C.P.dtJlo,
                          GAM_NG + b.Njp - 1 + C.P.dtJhi, GAM_NG - C.P.dtKlo, GAM_NG + b.Nkp - 1 + C.P.dtKhi};
            k_dt_only<R><<<grid_for(r, blk2), blk2, 0, s>>>(b, C.P, C.g, O, C.sc, C.gamma, C.gm1, 1);
        }
    });
    if (!fold) f(13, [&] { k_dt_finalize<<<1, 1, 0, s>>>(C.sc); });
    f(14, [&] { launch_bcs(C, O, S, cells, faces, s, 0); });
}

// One step. With side streams (C.aux, C.ev) the independent kernels run as
// parallel branches of the captured graph: the three Mom2Face -> EMF chains
// (then the face update) beside the three flux directions; the cell update
// joins them. Every branch writes its own arrays, so the result is the same
// bits as the sequential order.
//
// A grid of a few cells is bound by the chain of its launches: the step's
// scalars are ready from the step before (finalize_dt; launch_begin before the
// first), and the last block of the cell update ends the step where no later
// kernel adds to CalcDT (rings, the ionospheric hooks).
template <class R> void launch_step(const Ctx<R>& C, int cur, cudaStream_t s) {
    cudaStream_t cs = s;
    const int fold = !C.P.ring.on && !C.P.ion.push && !C.P.ion.wind;
    if (!C.aux[0]) {
        for_each_kernel(C, cur, cs, [](int id, auto&& L) { if (id) L(); }, fold);
        return;
    }
    for_each_kernel(C, cur, cs, [&](int id, auto&& L) {
        switch (id) {
            case 0: return;
            case 1:
                cs = s;
                L();
                cudaEventRecord(C.ev[0], s);
                for (int q = 0; q < 5; q++) cudaStreamWaitEvent(C.aux[q], C.ev[0], 0);
                return;
            case 2: case 3: cs = C.aux[0]; break;
            case 4: case 5: cs = C.aux[1]; break;
            case 6: case 7: cs = C.aux[2]; break;
            case 8: cs = s; break;
            case 9: cs = C.aux[3]; break;
            case 10: cs = C.aux[4]; break;
            case 11:
                cudaEventRecord(C.ev[1], C.aux[1]);
                cudaEventRecord(C.ev[2], C.aux[2]);
                cudaStreamWaitEvent(C.aux[0], C.ev[1], 0);
                cudaStreamWaitEvent(C.aux[0], C.ev[2], 0);
                cs = C.aux[0];
                break;
            case 12:
                cudaEventRecord(C.ev[3], C.aux[0]);
                cudaEventRecord(C.ev[4], C.aux[3]);
                cudaEventRecord(C.ev[5], C.aux[4]);
                cudaStreamWaitEvent(s, C.ev[3], 0);
                cudaStreamWaitEvent(s, C.ev[4], 0);
                cudaStreamWaitEvent(s, C.ev[5], 0);
                cs = s;
                break;
            default: cs = s; break;
        }
        L();
    }, fold);
}
// the scalars of the first step after the host may have set some
template <class R> void launch_begin(const Ctx<R>& C, cudaStream_t s) { k_step_begin<<<1, 1, 0, s>>>(C.sc); }

// Device time of each kernel of a step (ms, average of reps back-to-back
// launches; ms[15]). The kernels after k_step_begin read their inputs and
// write other arrays, so repeating one changes nothing; the time bookkeeping
// kernels are not run.
// The reference's clock label of each kernel id of for_each_kernel
// (gamapp.F90:96-99, mhdgroup.F90, fields.F90, stress.F90, step.F90 Tic/Toc)
inline const char* kernel_label(int id) {
    static const char* L[15] = {"Gamera", "Predictor", "Mom2Face", "VxB", "Mom2Face", "VxB", "Mom2Face", "VxB",
                                "Fluxes", "Fluxes", "Fluxes", "CT-Update", "Maxwell", "DT", "BCs"};
    return (id >= 0 && id < 15) ? L[id] : "Gamera";
}

template <class R> void profile_step(const Ctx<R>& C, int cur, cudaStream_t s, int reps, double* ms) {
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    for (int q = 0; q < 15; q++) ms[q] = 0.0;
    cudaStream_t cs = s;
    for_each_kernel(C, cur, cs, [&](int id, auto&& L) {
        if (id == 0 || id == 13) return;
        L();  // warm
        nvtxRangePushA(kernel_label(id));
        cudaEventRecord(e0, s);
        for (int r = 0; r < reps; r++) L();
        cudaEventRecord(e1, s);
        nvtxRangePop();
        cudaEventSynchronize(e1);
        float t = 0.f;
        cudaEventElapsedTime(&t, e0, e1);
        ms[id] = t / reps;
    });
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
}

// Kernel attributes that must be set before a launch is captured in a graph.
template <class R> void prepare() {}

// CalcDT on st[cur] into sc->dtmin_bits (the caller resets it first).
template <class R> void launch_dt_only(const Ctx<R>& C, int cur, cudaStream_t s) {
    const GamBox& b = C.b;
    const int G = GAM_NG;
    const dim3 blk(32, 4, 1);
    const Range r{G - C.P.dtIlo, G + b.Nip - 1 + C.P.dtIhi, G - C.P.dtJlo, G + b.Njp - 1 + C.P.dtJhi,
                  G - C.P.dtKlo, G + b.Nkp - 1 + C.P.dtKhi};
    k_dt_only<R><<<grid_for(r, blk), blk, 0, s>>>(b, C.P, C.g, C.st[cur], C.sc, C.gamma, C.gm1, 0);
}

// CalcGridInfo after the initial condition (init.F90:217-238): Bxyz from the
// fluxes, first EnforceBCs, oState = State.
// bFlux2Fld of State (st[cur]) over every cell (gridutils.F90:281-301)
template <class R> void launch_bfield(const Ctx<R>& C, int cur, cudaStream_t s) {
    const GamBox& b = C.b;
    const dim3 blk(32, 4, 1);
    const Range cells{0, b.Ni - 1, 0, b.Nj - 1, 0, b.Nk - 1};
    k_bfield_all<R><<<grid_for(cells, blk), blk, 0, s>>>(b, C.g, C.st[cur], C.sc, C.P.ring);
}

template <class R> void launch_init(const Ctx<R>& C, int cur, cudaStream_t s) {
    const GamBox& b = C.b;
    const dim3 blk(32, 4, 1);
    const Range all{0, b.Ni, 0, b.Nj, 0, b.Nk};
    const Range cells{0, b.Ni - 1, 0, b.Nj - 1, 0, b.Nk - 1};
    const StateBuf<R> S = C.st[cur], O = C.st[1 - cur];
    if (C.P.doMHD) k_bfield_all<R><<<grid_for(cells, blk), blk, 0, s>>>(b, C.g, S, C.sc, C.P.ring);
    launch_bcs(C, S, S, cells, all, s, 1);
    cudaMemcpyAsync(O.Gas, S.Gas, 5 * b.fs * sizeof(R), cudaMemcpyDeviceToDevice, s);
    cudaMemcpyAsync(O.mf, S.mf, 3 * b.fs * sizeof(R), cudaMemcpyDeviceToDevice, s);
    cudaMemcpyAsync(O.B, S.B, 3 * b.fs * sizeof(R), cudaMemcpyDeviceToDevice, s);
    if (C.oomf) cudaMemcpyAsync(C.oomf, S.mf, 3 * b.fs * sizeof(R), cudaMemcpyDeviceToDevice, s);  // ooState = State
}

// ----------------------------------------------------------------- k-slab tiling
// One step in two phases for a caller that reduces dt over several domains:
// phase 0 = begin .. cell update (the dt candidates in sc->dtmin_bits and
// sc->nbad), phase 1 = dt decision and boundary fill. The caller writes the
// global min / count into sc between them (gamapp_mpi.F90:495-512).
template <class R> void launch_step_phase(const Ctx<R>& C, int cur, cudaStream_t s, int phase) {
    cudaStream_t cs = s;
    for_each_kernel(C, cur, cs, [&](int id, auto&& L) {
        if ((id <= 12) == (phase == 0)) L();
    });
}

// Halo of a tile (the depth-4 exchange of updateMpiBCs/haloUpdate,
// gamapp_mpi.F90:573-782) along direction d (0 I, 1 J, 2 K): 11 components
// (Gas 0-4, magFlux 5-7, Bxyz 8-10) x 4 layers along d x the full ghosted
// face-box extents (u, v) of the other two directions (u the lower of the
// two), element (q, l, v, u) at ((q * 4 + l) * nv + v) * nu + u. Pack side 0
// = what this tile sends down (cells and the other faces at G..G+3 along d,
// d-faces at G+1..G+4: the neighbour's upper ghosts); side 1 = what it sends
// up (everything at Nd..Nd+3: the neighbour's lower ghosts). Unpack side 0
// fills this tile's lower ghosts (0..3), side 1 its upper ghosts (cells and
// the other faces at G+Nd.., d-faces at G+Nd+1..), the indices the periodic
// rules of bcs.F90:279-450 use. Exchanging I, then J, then K with the full
// extents carries the edge and corner ghosts through the earlier exchanges.
// The k-slab API's sides are d = 2.
__device__ __forceinline__ int halo_pos(const GamBox& b, int d, int side, bool unpack, int q, int l) {
    const int G = GAM_NG;
    const int Nd = d == 0 ? b.Nip : (d == 1 ? b.Njp : b.Nkp);
    const bool dface = q == 5 + d;
    if (!unpack) return side == 0 ? G + l + (dface ? 1 : 0) : Nd + l;
    return side == 0 ? l : G + Nd + l + (dface ? 1 : 0);
}
template <class R> __device__ __forceinline__ R* halo_ptr(const StateBuf<R>& S, long fs, int q) {
    return q < 5 ? S.Gas + (long)q * fs : (q < 8 ? S.mf + (long)(q - 5) * fs : S.B + (long)(q - 8) * fs);
}
// face-box extents across direction d: nu (the lower other direction), nv
__host__ __device__ __forceinline__ void halo_extents(const GamBox& b, int d, long& nu, long& nv) {
    nu = d == 0 ? b.Nj + 1 : b.Ni + 1;
    nv = d == 2 ? b.Nj + 1 : b.Nk + 1;
}
__device__ __forceinline__ long halo_cell(const GamBox& b, int d, int pos, int u, int v) {
    return d == 0 ? lidx(b, pos, u, v) : (d == 1 ? lidx(b, u, pos, v) : lidx(b, u, v, pos));
}
template <class R>
__global__ void __launch_bounds__(256) k_halo(GamBox b, StateBuf<R> S, R* __restrict__ buf, int d, int side,
                                              int unpack, int copyB, const GamScalars* sc) {
    if (sc->halted) return;  // a failed step keeps its state, ghosts included
    long nu, nv;
    halo_extents(b, d, nu, nv);
    const long t = blockIdx.x * (long)blockDim.x + threadIdx.x;
    if (t >= 4 * nu * nv) return;
    const int u = (int)(t % nu), v = (int)((t / nu) % nv), l = (int)(t / (nu * nv));
    const long fs = b.fs;
    for (int q = 0; q < 11; q++) {
        if (unpack && q >= 8 && !copyB) break;
        const long c = halo_cell(b, d, halo_pos(b, d, side, unpack != 0, q, l), u, v);
        GAM_BOX_CHECK(c, c, 15);
        const long e = ((long)(q * 4 + l) * nv + v) * nu + u;
        R* p = halo_ptr(S, fs, q);
        if (unpack)
            p[c] = buf[e];
        else
            buf[e] = p[c];
    }
}
// Bxyz of the unpacked ghost cells from their faces (the final bFlux2Fld)
template <class R>
__global__ void __launch_bounds__(256) k_halo_bxyz(GamBox b, Geo<R> g, StateBuf<R> S, int d, int side,
                                                   const GamScalars* sc, RingData ring) {
    if (sc->halted) return;
    const long nu = d == 0 ? b.Nj : b.Ni, nv = d == 2 ? b.Nj : b.Nk;  // cell extents
    const long t = blockIdx.x * (long)blockDim.x + threadIdx.x;
    if (t >= 4 * nu * nv) return;
    const int u = (int)(t % nu), v = (int)((t / nu) % nv), l = (int)(t / (nu * nv));
    const int Nd = d == 0 ? b.Nip : (d == 1 ? b.Njp : b.Nkp);
    const int pos = side == 0 ? l : GAM_NG + Nd + l;
    const long fs = b.fs, c = halo_cell(b, d, pos, u, v);
    // a ghost across the LFM pole takes its conjugate's field
    const int ic = d == 0 ? pos : u;
    int jc = d == 1 ? pos : (d == 0 ? u : v), kc = d == 2 ? pos : v;
    const long cb = (ring.on && ring_conj_cc(b, ring, jc, kc)) ? lidx(b, ic, jc, kc) : c;
    GAM_BOX_CHECK(cb, cb + b.sk, 15);
    R B[3];
    cell_bxyz(b, g, cb, S.mf[cb], S.mf[cb + 1], S.mf[fs + cb], S.mf[fs + cb + b.sx], S.mf[2 * fs + cb],
              S.mf[2 * fs + cb + b.sk], B);
#pragma unroll
    for (int x = 0; x < 3; x++) S.B[x * fs + c] = B[x];
}
// dside = side + 2 d
template <class R> void launch_halo(const Ctx<R>& C, int cur, cudaStream_t s, int dside, int unpack, int copyB, void* buf) {
    const GamBox& b = C.b;
    const int d = dside >> 1, side = dside & 1;
    const StateBuf<R> S = C.st[cur];
    long nu, nv;
    halo_extents(b, d, nu, nv);
    const long n = 4L * nu * nv;
    k_halo<R><<<(unsigned)((n + 255) / 256), 256, 0, s>>>(b, S, (R*)buf, d, side, unpack, copyB, C.sc);
    if (unpack && !copyB && C.P.doMHD) {
        const long m = 4L * (d == 0 ? b.Nj : b.Ni) * (d == 2 ? b.Nj : b.Nk);
        k_halo_bxyz<R><<<(unsigned)((m + 255) / 256), 256, 0, s>>>(b, C.g, S, d, side, C.sc, C.P.ring);
    }
}

#endif  // GAM_GEO_TABLES

}  // namespace GAM_NS
