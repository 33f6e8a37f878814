// pm_pair_math.cuh -- what the pair kernels share: the registered combinations
// of terms, the FP32 and FP64 arithmetic of one pair, and the dispatch of a
// combination to a kernel template.
//
// Per pair (OneAtomPair::doOneAtomPair / OneAtomPairTwo::doOneAtomPair,
// forces/OneAtomPair.h:127-188, forces/OneAtomPairTwo.h:131-199):
//   cutoff test r^2 > rc^2 -> skip (rc = largest switching cutoff);
//   exclusion check only for atoms of the same molecule (FULL -> skip,
//   MODIFIED -> A14/B14 and coulombScalingFactor);
//   potentials, switching F = F S - E dS, E = E S when any switch modifies;
//   f_i -= d F, f_j += d F (d = x_j - x_i), energies into the LJ / Coulomb
//   slots, virial addVirial(d F, d) (base/ScalarStructure.cpp:41-62).
//
// Mixed precision: a pair whose FP32 r^2 lies within a relative guard band of
// a cutoff is re-decided in FP64 with the reference's own minimalDifference
// arithmetic on the original positions, so the pair set is the reference's
// bit for bit.  Potentials and switching in FP32.  FP64: the reference's
// formulas on the FP64 positions; 1/r from one reciprocal square root.
#pragma once

#include <algorithm>

#include "pm_kernels.h"
#include "../../include/pmgpu.h"

namespace pm {

// ------------------------------------------------------------------ combos
#define LJ PMGPU_POT_LENNARD_JONES
#define CO PMGPU_POT_COULOMB
#define EW PMGPU_POT_EWALD_REAL
#define NP PMGPU_POT_NONE
#define SCUT PMGPU_SW_CUTOFF
#define SC1 PMGPU_SW_C1
#define SC2 PMGPU_SW_C2
#define SSH PMGPU_SW_SHIFT
#define SUN PMGPU_SW_UNIVERSAL
#define LJT PMGPU_POT_LENNARD_JONES_TABLE
#define COT PMGPU_POT_COULOMB_TABLE
#define EWT PMGPU_POT_EWALD_REAL_TABLE

__host__ __device__ constexpr bool pot_table(int p) { return p == LJT || p == COT || p == EWT; }
// the ScalarStructure slot of a potential's energy
__host__ __device__ constexpr bool pot_lj_slot(int p) { return p == LJ || p == LJT; }

__host__ __device__ constexpr bool sw_modifies(int s) { return s == SC1 || s == SC2 || s == SSH; }
__host__ __device__ constexpr bool pot_r2(int p) { return p == LJ || p == CO; }

// ---------------------------------------------------------------- shared
// ExclusionTable::check for a pair of the same molecule; returns the class
__device__ __forceinline__ int excl_class(const PairArgs& p, int oi, int oj)
{
    return excl_lookup(p.xfull, p.xmod, p.xrow, p.xent, oi, oj);
}

// ---------------------------------------------------------------- FP32 math
// FP32 hi part and remainder of a double constant
#define PM_HI(x) ((float)(x))
#define PM_LO(x) ((float)((x) - (double)(float)(x)))

// e^-x for x >= 0 as 2^(-x log2 e) on the hardware base-2 exponential
// (ex2.approx: relative error ~2^-22); the rounding of the scaled argument
// adds |x| log2(e) 2^-24 relative, the same order as the rounding of x itself
__device__ __forceinline__ float exp_neg(float x)
{
    float y;
    const float a = x * -1.4426950408889634f;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(a));
    return y;
}

// 1/x: the hardware approximation and one Newton-Raphson step
// (y' = y + y (1 - x y)), faithful to ~1 ulp for normal x
__device__ __forceinline__ float rcp_nr(float x)
{
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));      // (no denormal arguments here)
    float e = fmaf(-x, y, 1.0f);
    return fmaf(y, e, y);
}

__device__ __forceinline__ float poly5f(float ar)
{
    // poly5 (base/mathutilities.cpp:29-40), Abramowitz & Stegun 7.1.26.  The
    // coefficients are the same for every pair, so their FP32 rounding is
    // compensated (hi + lo) instead of biasing the real-space Ewald sum.
    const double E1 = 0.254829592, E2 = -0.284496736, E3 = 1.421413741,
                 E4 = -1.453152027, E5 = 1.061405429, PP = 0.3275911;
    float t = rcp_nr(fmaf(PM_HI(PP), ar, fmaf(PM_LO(PP), ar, 1.0f)));
    // each remainder is added after the O(1) partial result it corrects
    float h = fmaf(t, PM_HI(E5), PM_HI(E4)) + fmaf(t, PM_LO(E5), PM_LO(E4));
    h = fmaf(t, h, PM_HI(E3)) + PM_LO(E3);
    h = fmaf(t, h, PM_HI(E2)) + PM_LO(E2);
    h = fmaf(t, h, PM_HI(E1)) + PM_LO(E1);
    return t * h;
}

// qq is the compensated charge product (hi*hi exact inside the FMA plus the
// hi*lo cross terms), so the FP32 rounding of each atom's charge cancels
template <int POT>
__device__ __forceinline__ void pot_f32(const PairArgs& p, const TermF& t, float r2, float rd2, float rinv,
                                        float qq, int ti, int tj, int excl, float& e, float& f)
{
    if (POT == LJ) {
        const float4* tab = excl == PMGPU_EXCL_MODIFIED ? p.ljm : p.ljn;
        float4 par = __ldg(tab + (ti * p.n_types + tj));   // A_hi, B_hi, A_lo, B_lo
        float r6 = rd2 * rd2 * rd2;
        float r12 = r6 * r6;
        float r6B = fmaf(par.y, r6, par.w * r6);
        float r12A = fmaf(par.x, r12, par.z * r12);
        e = r12A - r6B;
        f = __fmul_rn(fmaf(12.0f, r12A, -__fmul_rn(6.0f, r6B)), rd2);
    } else if (POT == CO) {
        e = __fmul_rn(qq, rinv);
        e = excl == PMGPU_EXCL_MODIFIED ? __fmul_rn(e, p.csf) : e;
        f = __fmul_rn(e, rd2);
    } else if (POT == EW) {
        qq = excl == PMGPU_EXCL_MODIFIED ? qq * p.csf : qq;
        float r = r2 * rinv;
        float ar = fmaf(t.alpha, r, t.alpha_lo * r);     // compensated alpha
        float ex = qq * exp_neg(ar * ar);
        e = __fmul_rn(poly5f(ar) * ex, rinv);
        f = __fmul_rn(fmaf(t.two_alpha_pi, ex, fmaf(t.two_alpha_pi_lo, ex, e)) * rinv, rinv);
    } else if (pot_table(POT)) {
        // LookUpTableBase::index on the FP32 r^2 (its top exponent and PRE
        // mantissa bits pick the entry) and the cubic of ::interpolate
        // (base/LookUpTableBase.h:243-272) in FP32 on the FP32 copy of the
        // table; out of range -> the first / last entry with dt = 0
        const unsigned u = __float_as_uint(r2);
        int k = (int)(u >> t.tab_shift) * t.tab_step - t.tab_first;
        const bool clamp = k < 0 || k > t.tab_last;
        k = k < 0 ? 0 : (k > t.tab_last ? t.tab_last : k);
        const float dt = clamp ? 0.f : r2 - __uint_as_float(u & ~((1u << t.tab_shift) - 1u));
        const float4* T = reinterpret_cast<const float4*>(t.tab + k);
        float a, b, c, d;
        if (POT == LJT) {
            // A part and B part of the entry; compensated A, B
            const float4* tab = excl == PMGPU_EXCL_MODIFIED ? p.ljm : p.ljn;
            const float4 par = __ldg(tab + (ti * p.n_types + tj));   // A_hi, B_hi, A_lo, B_lo
            const float4 ta = __ldg(T), tb = __ldg(T + 1);
            a = fmaf(par.x, ta.x, __fmul_rn(par.z, ta.x)) + fmaf(par.y, tb.x, __fmul_rn(par.w, tb.x));
            b = fmaf(par.x, ta.y, __fmul_rn(par.z, ta.y)) + fmaf(par.y, tb.y, __fmul_rn(par.w, tb.y));
            c = fmaf(par.x, ta.z, __fmul_rn(par.z, ta.z)) + fmaf(par.y, tb.z, __fmul_rn(par.w, tb.z));
            d = fmaf(par.x, ta.w, __fmul_rn(par.z, ta.w)) + fmaf(par.y, tb.w, __fmul_rn(par.w, tb.w));
        } else {
            const float q = excl == PMGPU_EXCL_MODIFIED ? qq * p.csf : qq;
            const float4 tc = __ldg(T);
            a = __fmul_rn(tc.x, q); b = __fmul_rn(tc.y, q); c = __fmul_rn(tc.z, q); d = __fmul_rn(tc.w, q);
        }
        e = fmaf(fmaf(fmaf(dt, d, c), dt, b), dt, a);
        f = __fmul_rn(-2.0f, fmaf(fmaf(__fmul_rn(3.0f, dt), d, __fmul_rn(2.0f, c)), dt, b));
    } else {
        e = 0.f; f = 0.f;
    }
}

// switching functions as selects (no branches: the two pair evaluations of
// a lane interleave); OUT: a pair may lie outside this term's cutoff
template <int SW, bool OUT = true>
__device__ __forceinline__ void sw_f32(const TermF& t, float r2, float rinv, bool inside, float& v, float& d)
{
    if (SW == SC2) {
        const float c2 = t.cut2 - r2;
        const float c4 = __fmul_rn(c2, fmaf(2.0f, r2, t.s2));
        const float c24 = __fmul_rn(c2, c4);
        const float dd = fmaf(c2, c2, -c4);
        const bool out = OUT && r2 > t.cut2, mid = r2 >= t.on2;
        v = out ? 0.f : (mid ? fmaf(t.s1, c24, __fmul_rn(t.s1_lo, c24)) : 1.f);
        d = (out || !mid) ? 0.f : fmaf(t.s3, dd, __fmul_rn(t.s3_lo, dd));
    } else if (SW == SC1) {
        const float dist = r2 * rinv;
        const float in = fmaf(-r2, t.c1_05_3, t.c1_15_1) + fmaf(-r2, t.c1_05_3_lo, t.c1_15_1_lo);
        const bool out = OUT && r2 > t.cut2;
        v = out ? 0.f : fmaf(-dist, in, 1.0f);
        d = out ? 0.f : fmaf(dist, t.c1_15_3, -t.c1_15_1 * rinv) + fmaf(dist, t.c1_15_3_lo, -t.c1_15_1_lo * rinv);
    } else if (SW == SSH) {
        const float x = fmaf(-r2, t.sh_a_lo, fmaf(-r2, t.sh_a, 1.0f));
        const bool out = OUT && r2 > t.cut2;
        v = out ? 0.f : __fmul_rn(x, x);
        d = out ? 0.f : fmaf(t.sh_b, x, t.sh_b_lo * x);
    } else if (SW == SCUT) {
        d = 0.f;
        v = inside ? 1.f : 0.f;
    } else {
        v = 1.f; d = 0.f;
    }
}

// exact FP64 squared distance of two atoms (reference minimalDifference)
__device__ __forceinline__ double exact_d2(const PairArgs& p, int oi, int oj)
{
    const double* pi = p.pos + 3 * (size_t)oi;
    const double* pj = p.pos + 3 * (size_t)oj;
    double dx, dy, dz;
    return pbc_min_diff(p.pbc, pi[0], pi[1], pi[2], pj[0], pj[1], pj[2], dx, dy, dz);
}


// ---------------------------------------------------------------- FP64 math
template <int POT>
__device__ __forceinline__ void pot_f64(const PairArgs& p, const TermD& t, double d2, double rd2, double rinv,
                                        double qi, double qj, int ti, int tj, int excl, double& e, double& f)
{
    if (POT == LJ) {
        // LennardJonesForce::operator() (forces/LennardJonesForce.h:37-74)
        double4 par = p.ljd[(size_t)ti * p.n_types + tj];
        double A = excl == PMGPU_EXCL_MODIFIED ? par.z : par.x;
        double B = excl == PMGPU_EXCL_MODIFIED ? par.w : par.y;
        double r6 = rd2 * rd2 * rd2;
        double r12 = r6 * r6;
        double r6B = B * r6;
        double r12A = A * r12;
        e = r12A - r6B;
        f = 12.0 * r12A * rd2 - 6.0 * r6B * rd2;
    } else if (POT == CO) {
        // CoulombForce::operator() (forces/CoulombForce.h:41-57)
        e = qi * qj * rinv;
        if (excl == PMGPU_EXCL_MODIFIED) e *= p.csfd;
        f = e * rd2;
    } else if (POT == EW) {
        // CoulombEwaldRealForce::operator() (forces/CoulombEwaldRealForce.h:45-73)
        double qq = qi * qj;
        if (p.csfd != 1.0 && excl == PMGPU_EXCL_MODIFIED) qq *= p.csfd;
        double rr = rinv;
        // r from the reciprocal root, with its rounding put right
        const double h = d2 * rr;
        double ar = t.alpha * fma(0.5 * rr, fma(-h, h, d2), h);
        double ex = qq * exp(-ar * ar);
        const double E1 = 0.254829592, E2 = -0.284496736, E3 = 1.421413741,
                     E4 = -1.453152027, E5 = 1.061405429, PP = 0.3275911;
        double tt = 1.0 / (1.0 + PP * ar);
        double poly = tt * (E1 + tt * (E2 + tt * (E3 + tt * (E4 + tt * E5))));
        e = poly * ex * rr;
        f = ((e + t.two_alpha_pi * ex) * rr * rr);
    } else if (pot_table(POT)) {
        // LookUpTableBase::index / ::interpolate (base/LookUpTableBase.h:243-272)
        // with LennardJonesTableForce::operator() (forces/LennardJonesTableForce.h:81-101),
        // CoulombTableForce::operator() (CoulombTableForce.h:83-108) and
        // CoulombEwaldRealTableForce::operator() (CoulombEwaldRealTableForce.h:85-107)
        const long long u = __double_as_longlong(d2);
        long long k = (u >> t.tab_shift) * t.tab_step - t.tab_first;
        double dt = 0.0;
        if (k < 0) k = 0;
        else if (k > t.tab_last) k = t.tab_last;
        else dt = d2 - __longlong_as_double(u & ~((1ll << t.tab_shift) - 1ll));
        const double4* T = reinterpret_cast<const double4*>(t.tab + k);
        double a, b, c, d;
        if (POT == LJT) {
            const double4 par = p.ljd[(size_t)ti * p.n_types + tj];
            const double A = excl != PMGPU_EXCL_MODIFIED ? par.x : par.z;
            const double B = excl != PMGPU_EXCL_MODIFIED ? par.y : par.w;
            const double4 ta = T[0], tb = T[1];
            a = ta.x * A + tb.x * B;
            b = ta.y * A + tb.y * B;
            c = ta.z * A + tb.z * B;
            d = ta.w * A + tb.w * B;
        } else {
            const double q = qi * qj * ((p.csfd != 1.0 && excl == PMGPU_EXCL_MODIFIED) ? p.csfd : 1.0);
            const double4 tc = T[0];
            a = tc.x * q; b = tc.y * q; c = tc.z * q; d = tc.w * q;
        }
        e = ((dt * d + c) * dt + b) * dt + a;
        f = -2.0 * ((3.0 * dt * d + 2.0 * c) * dt + b);
    } else {
        e = 0.0; f = 0.0;
    }
}

template <int SW>
__device__ __forceinline__ void sw_f64(const TermD& t, double d2, double& v, double& d)
{
    if (SW == SC2) {           // C2SwitchingFunction.h:64-82
        d = 0.0;
        if (d2 > t.cut2) v = 0.0;
        else if (d2 >= t.on2) {
            double c2 = t.cut2 - d2;
            double c4 = c2 * (t.s2 + 2.0 * d2);
            v = t.s1 * (c2 * c4);
            d = t.s3 * (c2 * c2 - c4);
        } else v = 1.0;
    } else if (SW == SC1) {    // C1SwitchingFunction.h:64-75
        if (d2 > t.cut2) { v = 0.0; d = 0.0; return; }
        double dist = sqrt(d2);
        v = 1.0 - dist * (t.c1_15_1 - d2 * t.c1_05_3);
        d = -t.c1_15_1 / dist + dist * t.c1_15_3;
    } else if (SW == SSH) {    // ShiftSwitchingFunction.h
        if (d2 > t.cut2) { v = 0.0; d = 0.0; return; }
        double x = (1.0 - d2 * t.sh_a);
        v = x * x;
        d = t.sh_b * x;
    } else if (SW == SCUT) {   // CutoffSwitchingFunction.h:64-68
        d = 0.0;
        v = (d2 > t.cut2 ? 0.0 : 1.0);
    } else {
        v = 1.0; d = 0.0;
    }
}

// the terms of one pair: force factor (F_j = d ft) and energies
template <int NT, int P0, int S0, int P1, int S1>
__device__ __forceinline__ void pair_f64(const PairArgs& p, double d2, double qi, double qj, int ti, int tj, int excl,
                                         double& ft, double& e0, double& e1)
{
    constexpr bool kMod = sw_modifies(S0) || (NT > 1 && sw_modifies(S1));
    constexpr bool kRoot = P0 == CO || P0 == EW || (NT > 1 && (P1 == CO || P1 == EW));
    constexpr bool kR2 = pot_r2(P0) || (NT > 1 && pot_r2(P1));
    const double rinv = kRoot ? rsqrt(d2) : 0.0;
    double rd2 = kRoot ? rinv * rinv : (kR2 ? 1.0 / d2 : 1.0);
    // (one Newton step: the square of a rounded root alone is 2.5 ulp off, and a
    // Lennard-Jones term takes its sixth power)
    if (kRoot && kR2) rd2 = fma(rd2, fma(-d2, rd2, 1.0), rd2);
    double f0, f1 = 0.0;
    e1 = 0.0;
    pot_f64<P0>(p, p.td[0], d2, rd2, rinv, qi, qj, ti, tj, excl, e0, f0);
    if (NT > 1) pot_f64<P1>(p, p.td[1], d2, rd2, rinv, qi, qj, ti, tj, excl, e1, f1);
    if (kMod) {
        double sv, sd;
        sw_f64<S0>(p.td[0], d2, sv, sd);
        f0 = f0 * sv - e0 * sd;
        e0 = e0 * sv;
        if (NT > 1) {
            sw_f64<S1>(p.td[1], d2, sv, sd);
            f1 = f1 * sv - e1 * sd;
            e1 = e1 * sv;
        }
    }
    ft = NT > 1 ? f0 + f1 : f0;
}

// the registered combinations: X(ARG, id, number of terms, potential and switch
// of each), the ids in order from 0
#define PM_COMBOS(X, ARG) \
    X(ARG, 0, 1, CO, SC1, NP, SUN) \
    X(ARG, 1, 1, CO, SC2, NP, SUN) \
    X(ARG, 2, 1, CO, SCUT, NP, SUN) \
    X(ARG, 3, 1, CO, SSH, NP, SUN) \
    X(ARG, 4, 1, EW, SCUT, NP, SUN) \
    X(ARG, 5, 1, LJ, SC1, NP, SUN) \
    X(ARG, 6, 1, LJ, SC2, NP, SUN) \
    X(ARG, 7, 1, LJ, SCUT, NP, SUN) \
    X(ARG, 8, 1, LJ, SSH, NP, SUN) \
    X(ARG, 9, 2, LJ, SC1, EW, SCUT) \
    X(ARG, 10, 2, LJ, SC1, CO, SSH) \
    X(ARG, 11, 2, LJ, SC2, CO, SC1) \
    X(ARG, 12, 2, LJ, SC2, EW, SCUT) \
    X(ARG, 13, 2, LJ, SC2, CO, SCUT) \
    X(ARG, 14, 2, LJ, SC2, CO, SSH) \
    X(ARG, 15, 2, LJ, SCUT, EW, SCUT) \
    X(ARG, 16, 2, LJ, SC2, CO, SC2) \
    X(ARG, 17, 1, LJT, SUN, NP, SUN) \
    X(ARG, 18, 1, COT, SUN, NP, SUN) \
    X(ARG, 19, 1, EWT, SUN, NP, SUN) \
    X(ARG, 20, 2, LJ, SC1, EWT, SUN) \
    X(ARG, 21, 2, LJ, SC2, EWT, SUN) \
    X(ARG, 22, 2, LJ, SCUT, EWT, SUN) \
    X(ARG, 23, 2, LJT, SUN, EWT, SUN) \
    X(ARG, 24, 2, LJT, SUN, COT, SUN)

// inside switch (combo): a kernel of the combination launched on its blocks, or
// a function of it called
#define PM_COMBO_LAUNCH(KERNEL, ID, ...) case ID: KERNEL<__VA_ARGS__><<<blocks, 128, 0, s>>>(a); break;
#define PM_COMBO_RETURN(FUNCTION, ID, ...) case ID: return FUNCTION<__VA_ARGS__>(a, s, launches);
#define PM_COMBO_SWITCH(CASE, WHAT) \
    switch (combo) { \
    PM_COMBOS(CASE, WHAT) \
    default: return (int)cudaErrorInvalidValue; \
    }

}  // namespace pm
