// collide_fp64.cuh -- the plain FP64 collision, operation for operation as the reference.
//
// Bit-for-bit parity with the reference's FP64 CPU build rests on three facts:
//  (1) the reference is compiled by GCC in ISO C++17 mode, which does not contract a*b+c into an
//      FMA; every file that includes this header is compiled with nvcc --fmad=false, so each
//      multiply and add below is one correctly rounded IEEE operation as on the CPU;
//  (2) the sequence of rounded operations is the reference's:
//        calcula         LBM_functions.cpp:3518-3589
//        dist_eq         LBM_functions.cpp:2945-3000
//        coll_Ext_Reg    Collision_operators.cpp:1182-1307  (Pi accumulation, f1, f_gt1, update)
//        coll_Reg        Collision_operators.cpp:860-967
//        coll_BGK        Collision_operators.cpp:12-49
//        coll_MRT        Collision_operators.cpp:583-699 (D2Q9)
//  (3) the only operations left out are exact ones: products by the velocity components
//      c in {-1, 0, +1}, sums with +-0 (the terms whose coefficient is zero), and the source
//      term S of source() (LBM_functions.cpp:5646-5716), which is +-0 for every finite state
//      because all programs pass zero acceleration.  Leaving these out can change only the sign
//      of an exactly zero intermediate, which no later operation turns into a different
//      non-zero value, so finite results are identical.  A non-finite state may carry Inf where
//      the reference carries NaN; both are "non-finite" to every stability check.
//
// Sharing between opposite directions is exact too: c.u of direction opp(i) is the exact negation
// of that of i, so (0.5 cv) cv is identical and 1 + 3 cv becomes 1 - 3 cv.
//
// The kernels are bound by the FP64 pipe (about 1.7 unfused operations per clock and SM), so products by
// powers of two, which are exact, are not spent on it:
//  - ((0.5 cv) cv) 3 rounds the same real number as 1.5 (cv cv), because halving commutes with rounding;
//    cv cv is then the square the velocity's modulus uses as well.  The same for (0.5 vq) 3 = 1.5 vq.
//  - s +- 2 p is one fused multiply-add: 2 p is exact, so the fma rounds once, as the add does.
//  - the sum from 0.0 starts with its first term.
// (Subnormal and overflowing intermediates round differently under a halving; the first are absorbed by
// the 1 they are added to, the second belong to a state that is non-finite one operation later.)
// D2Q9 E-RLBM: 169 -> 160 operations per update, 79 of them on the FP64 pipe where the integer forms below apply.
#pragma once

#include "fp64_int.cuh"
#include "lattice.cuh"

namespace erlbm {
namespace exact {

// Reference constants, formed with the reference's own operations (calc_Q: Q = c c - c_s^2 delta;
// one_over_2cs4 = 0.5 * 3 * 3; f1 prefactor one_over_2cs4 * w_i).
constexpr double CS2 = 1. / 3.;
constexpr double QA = 1.0 * 1.0 - CS2;  // Q_aa for c_a = +-1
constexpr double QB = 0.0 * 0.0 - CS2;  // Q_aa for c_a = 0
constexpr double O2CS4 = 0.5 * 3. * 3.;

// Equilibrium of one opposite pair from cv = c_i.u of its first member and cv2 = cv cv.
__device__ __forceinline__ void feq_pair(double cv, double cv2, double wr, double C, double &fa, double &fb)
{
    const double t3 = cv * 3.;
    const double B = (1.5 * cv2) * 3.;
    fa = wr * (((1.0 + t3) + B) - C);
    fb = wr * (((1.0 - t3) + B) - C);
}

// ------------------------------------------------------------------------------------------------
// D2Q9
// ------------------------------------------------------------------------------------------------

// calcula: rho summed in velocity order from 0.0; momenta summed in velocity order.
__device__ __forceinline__ void moments9(const double f[9], double &rho, double &ux, double &uy)
{
    double r = f[0];
#pragma unroll
    for (int i = 1; i < 9; i++) r = r + f[i];
    const double mx = ((((f[1] - f[2]) + f[5]) - f[6]) + f[7]) - f[8];
    const double my = ((((f[3] - f[4]) + f[5]) - f[6]) - f[7]) + f[8];
    if (r != 0.0) {
        const double inv = 1.0 / r;
        ux = mx * inv;
        uy = my * inv;
    } else {
        ux = 0.;
        uy = 0.;
    }
    rho = r;
}

// dist_eq for D2Q9 (vz = 0).
__device__ __forceinline__ void equilibrium9(double rho, double ux, double uy, double feq[9])
{
    const double xx = ux * ux, yy = uy * uy;
    const double C = 1.5 * (xx + yy);
    const double sp = ux + uy, sm = ux - uy;
    const double wr0 = (4. / 9.) * rho, wr1 = (1. / 9.) * rho, wr2 = (1. / 36.) * rho;
    feq[0] = wr0 * (1.0 - C);
    feq_pair(ux, xx, wr1, C, feq[1], feq[2]);
    feq_pair(uy, yy, wr1, C, feq[3], feq[4]);
    feq_pair(sp, sp * sp, wr2, C, feq[5], feq[6]);
    feq_pair(sm, sm * sm, wr2, C, feq[7], feq[8]);
}

// The same for the collision: where the velocity is below the bound of fp64int::eq_pair (Mach 0.28) the sums of
// the pairs' polynomials run on the integer pipes, nine FP64 operations less per pair.
// A form of the update that needs a range of operands is taken where every lane of the warp is in it: a warp with lanes
// on both sides would go through both forms, and a Taylor-Green run above Mach 0.28 has such warps in every step.  All
// forms give the same bits.  FP64 Taylor-Green map, 80 runs of 600 steps 21.4 -> 16.3 ms (17.4 without integer forms),
// 1200 runs 80 -> 69.5; obstacle map of 600 runs of 1000 steps 84.4 -> 76.7; single lattices of smooth flows as before.
__device__ __forceinline__ bool warp_agrees(bool in_range) { return __all_sync(__activemask(), in_range); }

__device__ __forceinline__ uint32_t abs_hi(double x) { return (uint32_t)__double2hiint(x) & 0x7fffffffu; }

__device__ __forceinline__ void feq_pair_int(double cv, double cv2, double wr, uint64_t C62, double &fa, double &fb)
{
    double a, b;
    fp64int::eq_pair(cv, cv2, C62, a, b);
    fa = wr * a;
    fb = wr * b;
}

__device__ __forceinline__ void equilibrium9_int(double rho, double ux, double uy, double feq[9])
{
    const double sp = ux + uy, sm = ux - uy;
    if (!warp_agrees(max(abs_hi(sp), abs_hi(sm)) < fp64int::EQ_MAX_HI)) {  // |ux|, |uy| <= max(|sp|, |sm|)
        equilibrium9(rho, ux, uy, feq);
        return;
    }
    const double xx = ux * ux, yy = uy * uy;
    const double C = 1.5 * (xx + yy);
    const uint64_t C62 = fp64int::fixed62(C);
    const double wr1 = (1. / 9.) * rho, wr2 = (1. / 36.) * rho;
    feq[0] = ((4. / 9.) * rho) * (1.0 - C);
    feq_pair_int(ux, xx, wr1, C62, feq[1], feq[2]);
    feq_pair_int(uy, yy, wr1, C62, feq[3], feq[4]);
    feq_pair_int(sp, sp * sp, wr2, C62, feq[5], feq[6]);
    feq_pair_int(sm, sm * sm, wr2, C62, feq[7], feq[8]);
}

// Whether all Q populations have the fixed-point form of fp64int.
template <int Q>
__device__ __forceinline__ bool fixed_form(const double *f)
{
    uint32_t most = 0;
#pragma unroll
    for (int i = 0; i < Q; i++) most = max(most, fp64int::fix_range(f[i]));
    return most < (Q == 9 ? fp64int::FIX_SPAN : fp64int::FIX_SPAN_HALF);
}

// moments9 with its sums in fixed point (fixed_form holds), every partial sum rounded as the FP64 add rounds it:
// 18 FP64 operations less.  F: the populations in fixed point.
__device__ __forceinline__ void moments9_fixed(const double f[9], int64_t F[9], double &rho, double &ux, double &uy)
{
    using fp64int::round53;
#pragma unroll
    for (int i = 0; i < 9; i++) F[i] = fp64int::to_fixed(f[i]);
    int64_t r = F[0];
#pragma unroll
    for (int i = 1; i < 9; i++) r = round53(r + F[i]);
    int64_t mx = round53(F[1] - F[2]), my = round53(F[3] - F[4]);
    mx = round53(round53(round53(round53(mx + F[5]) - F[6]) + F[7]) - F[8]);
    my = round53(round53(round53(round53(my + F[5]) - F[6]) - F[7]) + F[8]);
    rho = fp64int::to_double(r);
    const double inv = fp64int::reciprocal(rho);
    ux = fp64int::to_double(mx) * inv;
    uy = fp64int::to_double(my) * inv;
}

// D_i = f_i - feq_i in fixed point, exact.  False when a feq has no fixed-point form.  shared: every |D_i| is small
// enough that sums of up to 10 of them (6 for nine populations) stay below 2^53 units: then the D_i are FP64 numbers,
// and their sums are exact in any order, so that the terms the sums share are added once.  Otherwise D_i is rounded as
// the FP64 difference is, and so is every partial sum in the reference's order (low viscosity: most nodes of the
// obstacle map's lower rows; those took 55 FP64 operations more).
template <int Q>
__device__ __forceinline__ bool fixed_parts(const int64_t *F, const double *feq, int64_t *D, bool &shared)
{
    if (!warp_agrees(fixed_form<Q>(feq))) return false;
    uint32_t most = 0;
#pragma unroll
    for (int i = 0; i < Q; i++) {
        D[i] = F[i] - fp64int::to_fixed(feq[i]);
        const int32_t h = (int32_t)fp64int::hi32((uint64_t)D[i]);
        most = max(most, (uint32_t)(h ^ (h >> 31)));
    }
    shared = warp_agrees(most < (1u << 21) / (Q == 9 ? 6 : 10) - 1);
    if (!shared) {
#pragma unroll
        for (int i = 0; i < Q; i++) D[i] = fp64int::round53(D[i]);
    }
    return true;
}

// D[I0] + D[I] + ... in order, every sum rounded; a negative index -I stands for - D[I].
template <int I0, int... I>
__device__ __forceinline__ int64_t rounded_sum(const int64_t *D)
{
    int64_t s = D[I0];
    ((s = fp64int::round53(I > 0 ? s + D[I > 0 ? I : -I] : s - D[I > 0 ? I : -I])), ...);
    return s;
}

// Row ROW of the MRT transform applied to f: the reference sums M[ROW][i] * f[i] from 0.0 in
// column order.  Terms with M = 0 add +-0 and are left out; products by +-1 are exact.
template <int ROW>
__device__ __forceinline__ double mrt9_row(const double f[9])
{
    double acc = 0.0;
    bool first = true;
#pragma unroll
    for (int i = 0; i < 9; i++) {
        const int m = mrt9_m(ROW, i);
        if (m == 0) continue;
        // m = +-1, +-2, +-4: the product is exact, so the fused form rounds once, as product and add do
        acc = first ? (double)m * f[i] : (m == 1 ? acc + f[i] : (m == -1 ? acc - f[i] : __fma_rn((double)m, f[i], acc)));
        first = false;
    }
    return acc;
}

// Population I from the moments: sum over c of M^-1[I][c] * m[c] from 0.0, M^-1[I][c] =
// M[c][I] / |row c|^2 (a correctly rounded quotient, the value of the reference's literal).
template <int I>
__device__ __forceinline__ double mrt9_back(const double m[9])
{
    double acc = 0.0;
    bool first = true;
#pragma unroll
    for (int c = 0; c < 9; c++) {
        const int a = mrt9_m(c, I);
        if (a == 0) continue;
        const double t = ((double)a / (double)mrt9_norm2(c)) * m[c];
        acc = first ? t : acc + t;
        first = false;
    }
    return acc;
}

// coll_MRT, D2Q9: moments m = M f and m_eq = M f_eq; m <- m - s (m - m_eq) on the non-conserved
// rows (the conserved rows have s = 0, and the force moments are those of a zero force); f = M^-1 m.
__device__ __forceinline__ void collide9_mrt(double f[9], const Relax &R, const double feq[9])
{
    double m[9];
    m[0] = mrt9_row<0>(f);
    m[3] = mrt9_row<3>(f);
    m[5] = mrt9_row<5>(f);
    m[1] = mrt9_row<1>(f);
    m[1] = m[1] - MRT9_SE * (m[1] - mrt9_row<1>(feq));
    m[2] = mrt9_row<2>(f);
    m[2] = m[2] - MRT9_SEPS * (m[2] - mrt9_row<2>(feq));
    m[4] = mrt9_row<4>(f);
    m[4] = m[4] - MRT9_SQ * (m[4] - mrt9_row<4>(feq));
    m[6] = mrt9_row<6>(f);
    m[6] = m[6] - MRT9_SQ * (m[6] - mrt9_row<6>(feq));
    m[7] = mrt9_row<7>(f);
    m[7] = m[7] - R.inv_tau * (m[7] - mrt9_row<7>(feq));
    m[8] = mrt9_row<8>(f);
    m[8] = m[8] - R.inv_tau * (m[8] - mrt9_row<8>(feq));
    f[0] = mrt9_back<0>(m);
    f[1] = mrt9_back<1>(m);
    f[2] = mrt9_back<2>(m);
    f[3] = mrt9_back<3>(m);
    f[4] = mrt9_back<4>(m);
    f[5] = mrt9_back<5>(m);
    f[6] = mrt9_back<6>(m);
    f[7] = mrt9_back<7>(m);
    f[8] = mrt9_back<8>(m);
}

// Whether every sum of up to 2^M of the d_i = f_i - feq_i, i >= 1, is exact in any order: all of them are multiples
// of the last place 2^(e-52) of the smallest f_i or feq_i (exponent e), and with every |d_i| < 2^(e-M+1) no sum
// exceeds 2^53 of those.  Then the terms that the sums of d share are added once.
template <int Q, int M>
__device__ __forceinline__ bool exact_sums(const double *f, const double *feq, const double *d)
{
    int least = __double2hiint(f[1]);  // negative for a negative value
    unsigned most = 0;
#pragma unroll
    for (int i = 1; i < Q; i++) {
        least = min(least, min(__double2hiint(f[i]), __double2hiint(feq[i])));
        most = max(most, abs_hi(d[i]));
    }
    return (int)(most >> 20) + M <= (least >> 20);
}

// The collision keeps a node's density up to its rounding.  Where the populations, equilibria and non-equilibrium
// parts are in the ranges of fixed_parts or exact_sums, every rounding is below 2^-52 of the density times a
// relaxation coefficient, so the density after the collision differs from the one before by less than 2^-21 of it
// for coefficients below 2^10: two units of its upper word.  A density check that has seen a greater density needs no
// sum of such a node (18 FP64 operations).  The hint is the upper word of the density, or NO_HINT.
constexpr uint32_t NO_HINT = 0xffffffffu;
__device__ __forceinline__ uint32_t density_hint(double rho, const Relax &R)
{
    const uint32_t h = (uint32_t)__double2hiint(rho);
    return max(abs_hi(R.omega_1), abs_hi(R.omega_gt1)) < 0x40900000u ? h : NO_HINT;
}
// Whether a node's density after the collision is less than a density with the upper word `known`.
__device__ __forceinline__ bool density_below(uint32_t hint, uint32_t known) { return known > 2 && hint < known - 2; }

template <int OP, bool FIXED>
__device__ __forceinline__ void collide9(double f[9], const Relax &R, uint32_t &hint)
{
    double rho, ux, uy, feq[9];
    int64_t F[9];
    const bool fixed = FIXED && warp_agrees(fixed_form<9>(f));
    if (fixed)
        moments9_fixed(f, F, rho, ux, uy);
    else
        moments9(f, rho, ux, uy);
    equilibrium9_int(rho, ux, uy, feq);
    if constexpr (OP == OP_MRT) {
        collide9_mrt(f, R, feq);
        return;
    }
    if (OP == OP_BGK) {
#pragma unroll
        for (int i = 0; i < 9; i++) f[i] = f[i] + (feq[i] - f[i]) * R.inv_tau;
        return;
    }
    double d[9], pxx, pyy, pxy;
    int64_t D[9];
    bool shared;
    if (fixed && fixed_parts<9>(F, feq, D, shared)) {
        hint = density_hint(rho, R);
        int64_t xx, yy, xy;
        if (shared) {
            const int64_t s56 = D[5] + D[6], s78 = D[7] + D[8], t = s56 + s78;
            xx = (D[1] + D[2]) + t;
            yy = (D[3] + D[4]) + t;
            xy = s56 - s78;
        } else {
            xx = rounded_sum<1, 2, 5, 6, 7, 8>(D);
            yy = rounded_sum<3, 4, 5, 6, 7, 8>(D);
            xy = rounded_sum<5, 6, -7, -8>(D);
        }
        pxx = fp64int::to_double(xx);
        pyy = fp64int::to_double(yy);
        pxy = fp64int::to_double(xy);
#pragma unroll
        for (int i = 0; i < 9; i++) d[i] = fp64int::to_double(D[i]);
    } else {
#pragma unroll
        for (int i = 0; i < 9; i++) d[i] = f[i] - feq[i];
        if (!FIXED && warp_agrees(exact_sums<9, 3>(f, feq, d))) {
            if (__double2hiint(f[0]) > 0) hint = density_hint(rho, R);
            const double s56 = d[5] + d[6], s78 = d[7] + d[8], t = s56 + s78;
            pxx = (d[1] + d[2]) + t;
            pyy = (d[3] + d[4]) + t;
            pxy = s56 - s78;
        } else {
            pxx = ((((d[1] + d[2]) + d[5]) + d[6]) + d[7]) + d[8];
            pyy = ((((d[3] + d[4]) + d[5]) + d[6]) + d[7]) + d[8];
            pxy = ((d[5] + d[6]) - d[7]) - d[8];
        }
    }
    const double xa = QA * pxx, xb = QB * pxx, ya = QA * pyy, yb = QB * pyy;
    const double dd = xa + ya;
    double f1[9];
    f1[0] = (O2CS4 * (4. / 9.)) * (xb + yb);
    f1[1] = f1[2] = (O2CS4 * (1. / 9.)) * (xa + yb);
    f1[3] = f1[4] = (O2CS4 * (1. / 9.)) * (xb + ya);
    f1[5] = f1[6] = (O2CS4 * (1. / 36.)) * __fma_rn(2., pxy, dd);
    f1[7] = f1[8] = (O2CS4 * (1. / 36.)) * __fma_rn(-2., pxy, dd);
    if (OP == OP_REG) {
#pragma unroll
        for (int i = 0; i < 9; i++) f[i] = feq[i] + R.omega_1 * f1[i];
        return;
    }
#pragma unroll
    for (int i = 0; i < 9; i++) {
        const double gt1 = d[i] - f1[i];
        f[i] = (feq[i] + R.omega_1 * f1[i]) + R.omega_gt1 * gt1;
    }
}

// ------------------------------------------------------------------------------------------------
// D3Q19
// ------------------------------------------------------------------------------------------------

__device__ __forceinline__ void moments19(const double f[19], double &rho, double &ux, double &uy, double &uz)
{
    double r = f[0];
#pragma unroll
    for (int i = 1; i < 19; i++) r = r + f[i];
    const double mx = ((((((((f[1] - f[2]) + f[7]) - f[8]) + f[9]) - f[10]) + f[11]) - f[12]) + f[13]) - f[14];
    const double my = ((((((((f[3] - f[4]) + f[7]) - f[8]) - f[9]) + f[10]) - f[15]) + f[16]) - f[17]) + f[18];
    const double mz = ((((((((f[5] - f[6]) + f[11]) - f[12]) - f[13]) + f[14]) - f[15]) + f[16]) + f[17]) - f[18];
    if (r != 0.0) {
        const double inv = 1.0 / r;
        ux = mx * inv;
        uy = my * inv;
        uz = mz * inv;
    } else {
        ux = 0.;
        uy = 0.;
        uz = 0.;
    }
    rho = r;
}

__device__ __forceinline__ void equilibrium19(double rho, double ux, double uy, double uz, double feq[19])
{
    const double xx = ux * ux, yy = uy * uy, zz = uz * uz;
    const double C = 1.5 * ((xx + yy) + zz);
    const double xpy = ux + uy, xmy = ux - uy, xpz = ux + uz, xmz = ux - uz, ypz = uy + uz, zmy = uz - uy;
    const double wr0 = (1. / 3.) * rho, wr1 = (1. / 18.) * rho, wr2 = (1. / 36.) * rho;
    feq[0] = wr0 * (1.0 - C);
    feq_pair(ux, xx, wr1, C, feq[1], feq[2]);
    feq_pair(uy, yy, wr1, C, feq[3], feq[4]);
    feq_pair(uz, zz, wr1, C, feq[5], feq[6]);
    feq_pair(xpy, xpy * xpy, wr2, C, feq[7], feq[8]);
    feq_pair(xmy, xmy * xmy, wr2, C, feq[9], feq[10]);
    feq_pair(xpz, xpz * xpz, wr2, C, feq[11], feq[12]);
    feq_pair(xmz, xmz * xmz, wr2, C, feq[13], feq[14]);
    // direction 16 is (0,1,1) and 15 its opposite; 17 is (0,-1,1) and 18 its opposite
    feq_pair(ypz, ypz * ypz, wr2, C, feq[16], feq[15]);
    feq_pair(zmy, zmy * zmy, wr2, C, feq[17], feq[18]);
}

// moments19 in fixed point, as moments9_fixed: 45 FP64 operations less.
__device__ __forceinline__ void moments19_fixed(const double f[19], int64_t F[19], double &rho, double &ux, double &uy,
                                                double &uz)
{
    using fp64int::round53;
#pragma unroll
    for (int i = 0; i < 19; i++) F[i] = fp64int::to_fixed(f[i]);
    int64_t r = F[0];
#pragma unroll
    for (int i = 1; i < 19; i++) r = round53(r + F[i]);
    int64_t mx = round53(F[1] - F[2]), my = round53(F[3] - F[4]), mz = round53(F[5] - F[6]);
#pragma unroll
    for (int i = 7; i < 19; i++) {
        if (Lat<19>::cx(i)) mx = round53(Lat<19>::cx(i) > 0 ? mx + F[i] : mx - F[i]);
        if (Lat<19>::cy(i)) my = round53(Lat<19>::cy(i) > 0 ? my + F[i] : my - F[i]);
        if (Lat<19>::cz(i)) mz = round53(Lat<19>::cz(i) > 0 ? mz + F[i] : mz - F[i]);
    }
    rho = fp64int::to_double(r);
    const double inv = 1.0 / rho;
    ux = fp64int::to_double(mx) * inv;
    uy = fp64int::to_double(my) * inv;
    uz = fp64int::to_double(mz) * inv;
}

__device__ __forceinline__ void equilibrium19_int(double rho, double ux, double uy, double uz, double feq[19])
{
    const double xpy = ux + uy, xmy = ux - uy, xpz = ux + uz, xmz = ux - uz, ypz = uy + uz, zmy = uz - uy;
    const uint32_t most = max(max(max(abs_hi(xpy), abs_hi(xmy)), max(abs_hi(xpz), abs_hi(xmz))),
                              max(abs_hi(ypz), abs_hi(zmy)));
    if (!warp_agrees(most < fp64int::EQ_MAX_HI)) {
        equilibrium19(rho, ux, uy, uz, feq);
        return;
    }
    const double xx = ux * ux, yy = uy * uy, zz = uz * uz;
    const double C = 1.5 * ((xx + yy) + zz);
    const uint64_t C62 = fp64int::fixed62(C);
    const double wr1 = (1. / 18.) * rho, wr2 = (1. / 36.) * rho;
    feq[0] = ((1. / 3.) * rho) * (1.0 - C);
    // A loop, not nine copies: unrolled, a step of the exact D3Q19 update is some 80 KB of instructions, and warps
    // wait for their fetch (obstacle map 87.4 -> 84.8 ms, 64^3 5.07 -> 4.83 ms for 30 steps with their copies; three
    // pairs at a time is slower than either).  The pairs' arrays live in local memory, where the LSU has room.
    const double cv[9] = {ux, uy, uz, xpy, xmy, xpz, xmz, -ypz, zmy};  // of directions 1, 3, ... 17
#pragma unroll 1
    for (int p = 0; p < 9; p++) {
        const double w = p < 3 ? wr1 : wr2;
        feq_pair_int(cv[p], cv[p] * cv[p], w, C62, feq[2 * p + 1], feq[2 * p + 2]);
    }
}

template <int OP, bool FIXED>
__device__ __forceinline__ void collide19(double f[19], const Relax &R, uint32_t &hint)
{
    double rho, ux, uy, uz, feq[19];
    int64_t F[19];
    const bool fixed = FIXED && warp_agrees(fixed_form<19>(f));
    if (fixed)
        moments19_fixed(f, F, rho, ux, uy, uz);
    else
        moments19(f, rho, ux, uy, uz);
    equilibrium19_int(rho, ux, uy, uz, feq);
    if (OP == OP_BGK) {
#pragma unroll
        for (int i = 0; i < 19; i++) f[i] = f[i] + (feq[i] - f[i]) * R.inv_tau;
        return;
    }
    double d[19], pxx, pyy, pzz, pxy, pxz, pyz;
    int64_t D[19];
    bool shared;
    if (fixed && fixed_parts<19>(F, feq, D, shared)) {
        hint = density_hint(rho, R);
        int64_t xx, yy, zz, xy, xz, yz;
        if (shared) {
            const int64_t a = D[7] + D[8], b = D[9] + D[10], ab = a + b;
            const int64_t g = D[11] + D[12], h = D[13] + D[14], gh = g + h;
            const int64_t m = D[15] + D[16], n = D[17] + D[18], mn = m + n;
            xx = (D[1] + D[2]) + (ab + gh);
            yy = (D[3] + D[4]) + (ab + mn);
            zz = (D[5] + D[6]) + (gh + mn);
            xy = a - b;
            xz = g - h;
            yz = m - n;
        } else {
            xx = rounded_sum<1, 2, 7, 8, 9, 10, 11, 12, 13, 14>(D);
            yy = rounded_sum<3, 4, 7, 8, 9, 10, 15, 16, 17, 18>(D);
            zz = rounded_sum<5, 6, 11, 12, 13, 14, 15, 16, 17, 18>(D);
            xy = rounded_sum<7, 8, -9, -10>(D);
            xz = rounded_sum<11, 12, -13, -14>(D);
            yz = rounded_sum<15, 16, -17, -18>(D);
        }
        pxx = fp64int::to_double(xx);
        pyy = fp64int::to_double(yy);
        pzz = fp64int::to_double(zz);
        pxy = fp64int::to_double(xy);
        pxz = fp64int::to_double(xz);
        pyz = fp64int::to_double(yz);
#pragma unroll
        for (int i = 0; i < 19; i++) d[i] = fp64int::to_double(D[i]);
    } else {
#pragma unroll
        for (int i = 0; i < 19; i++) d[i] = f[i] - feq[i];
        if (!FIXED && warp_agrees(exact_sums<19, 4>(f, feq, d))) {
            if (__double2hiint(f[0]) > 0) hint = density_hint(rho, R);
            const double a = d[7] + d[8], b = d[9] + d[10], ab = a + b;
            const double g = d[11] + d[12], h = d[13] + d[14], gh = g + h;
            const double m = d[15] + d[16], n = d[17] + d[18], mn = m + n;
            pxx = (d[1] + d[2]) + (ab + gh);
            pyy = (d[3] + d[4]) + (ab + mn);
            pzz = (d[5] + d[6]) + (gh + mn);
            pxy = a - b;
            pxz = g - h;
            pyz = m - n;
        } else {
            pxx = ((((((((d[1] + d[2]) + d[7]) + d[8]) + d[9]) + d[10]) + d[11]) + d[12]) + d[13]) + d[14];
            pyy = ((((((((d[3] + d[4]) + d[7]) + d[8]) + d[9]) + d[10]) + d[15]) + d[16]) + d[17]) + d[18];
            pzz = ((((((((d[5] + d[6]) + d[11]) + d[12]) + d[13]) + d[14]) + d[15]) + d[16]) + d[17]) + d[18];
            pxy = ((d[7] + d[8]) - d[9]) - d[10];
            pxz = ((d[11] + d[12]) - d[13]) - d[14];
            pyz = ((d[15] + d[16]) - d[17]) - d[18];
        }
    }
    const double xa = QA * pxx, xb = QB * pxx;
    const double ya = QA * pyy, yb = QB * pyy;
    const double za = QA * pzz, zb = QB * pzz;
    const double kr = O2CS4 * (1. / 3.), k1 = O2CS4 * (1. / 18.), k2 = O2CS4 * (1. / 36.);
    double f1[19];
    f1[0] = kr * ((xb + yb) + zb);
    f1[1] = f1[2] = k1 * ((xa + yb) + zb);
    f1[3] = f1[4] = k1 * ((xb + ya) + zb);
    f1[5] = f1[6] = k1 * ((xb + yb) + za);
    const double bxy = (xa + ya) + zb;
    f1[7] = f1[8] = k2 * __fma_rn(2., pxy, bxy);
    f1[9] = f1[10] = k2 * __fma_rn(-2., pxy, bxy);
    const double bxz = (xa + yb) + za;
    f1[11] = f1[12] = k2 * __fma_rn(2., pxz, bxz);
    f1[13] = f1[14] = k2 * __fma_rn(-2., pxz, bxz);
    const double byz = (xb + ya) + za;
    f1[15] = f1[16] = k2 * __fma_rn(2., pyz, byz);
    f1[17] = f1[18] = k2 * __fma_rn(-2., pyz, byz);
    if (OP == OP_REG) {
#pragma unroll
        for (int i = 0; i < 19; i++) f[i] = feq[i] + R.omega_1 * f1[i];
        return;
    }
#pragma unroll
    for (int i = 0; i < 19; i++) {
        const double gt1 = d[i] - f1[i];
        f[i] = (feq[i] + R.omega_1 * f1[i]) + R.omega_gt1 * gt1;
    }
}

template <int Q, int OP, bool FIXED = true>
__device__ __forceinline__ uint32_t collide(double *f, const Relax &R)
{
    static_assert(Q == 9 || OP != OP_MRT, "MRT is a D2Q9 operator");
    uint32_t hint = NO_HINT;
    if constexpr (Q == 9)
        collide9<OP, FIXED>(f, R, hint);
    else
        collide19<OP, FIXED>(f, R, hint);
    return hint;
}

// calcula velocity of one node (for kinectic_energy, Other_functions.cpp:100-115):
// returns 0.5 * (vx*vx + vy*vy + vz*vz) with vz = 0 for D2Q9.
template <int Q>
__device__ __forceinline__ double node_energy(const double *f)
{
    if constexpr (Q == 9) {
        double rho, ux, uy;
        moments9(f, rho, ux, uy);
        return 0.5 * ((ux * ux + uy * uy) + 0.0 * 0.0);
    } else {
        double rho, ux, uy, uz;
        moments19(f, rho, ux, uy, uz);
        return 0.5 * ((ux * ux + uy * uy) + uz * uz);
    }
}

// density (LBM_functions.cpp:5544-5552)
template <int Q>
__device__ __forceinline__ double node_density(const double *f)
{
    double r = f[0];
#pragma unroll
    for (int i = 1; i < Q; i++) r = r + f[i];
    return r;
}

// ZouHeD3Q19_vx_x, left-plane branch (Boundary_conditions.cpp:370-403) with vy = vz = 0, applied
// to one node's post-stream populations.  The right-plane branch (:404-436) mirrors it.  The terms with
// vy and vz are +-0; x / 6 is half of x / 3, so that 0.5 ty and rho vx / 6 enter by fused multiply-adds by exact
// halves; a quotient by a constant of the run is fp64int::quotient.  About 50 FP64 operations instead of 90.
struct ZouHe {
    double vx, y, z;  // y = 1 - vx; z = 1 / y, or 0 where no reciprocal was formed
};

__device__ __forceinline__ double zou_he_quotient(double a, const ZouHe &c)
{
    return c.z != 0.0 && fp64int::quotient_range(a) ? fp64int::quotient(a, c.y, c.z) : a / c.y;
}

__device__ __forceinline__ double third(double a) { return fp64int::quotient_range(a) ? fp64int::quotient3(a) : a / 3.0; }

__device__ __forceinline__ void zou_he_left(double f[19], const ZouHe &c)
{
    const double s_minus = (((f[1] + f[7]) + f[9]) + f[11]) + f[13];
    const double s_zero = (((((((f[0] + f[3]) + f[4]) + f[5]) + f[6]) + f[15]) + f[16]) + f[17]) + f[18];
    const double rho = zou_he_quotient(__fma_rn(2.0, s_minus, s_zero), c);
    const double ty = (((((f[18] + f[3]) + f[16]) - f[15]) - f[4]) - f[17]);
    const double tz = (((((f[17] + f[5]) + f[16]) - f[15]) - f[6]) - f[18]);
    const double a3 = third(rho * c.vx);
    f[1] = f[1] + a3;
    f[7] = __fma_rn(-0.5, ty, __fma_rn(0.5, a3, f[7]));
    f[9] = __fma_rn(0.5, ty, __fma_rn(0.5, a3, f[9]));
    f[11] = __fma_rn(-0.5, tz, __fma_rn(0.5, a3, f[11]));
    f[13] = __fma_rn(0.5, tz, __fma_rn(0.5, a3, f[13]));
}

__device__ __forceinline__ void zou_he_right(double f[19], const ZouHe &c)
{
    const double s_plus = (((f[2] + f[8]) + f[10]) + f[12]) + f[14];
    const double s_zero = (((((((f[0] + f[3]) + f[4]) + f[5]) + f[6]) + f[15]) + f[16]) + f[17]) + f[18];
    const double rho = zou_he_quotient(__fma_rn(2.0, s_plus, s_zero), c);
    const double ty = (((((f[18] + f[3]) + f[16]) - f[15]) - f[4]) - f[17]);
    const double tz = (((((f[17] + f[5]) + f[16]) - f[15]) - f[6]) - f[18]);
    const double a3 = third(rho * c.vx);
    f[2] = f[2] - a3;
    f[10] = __fma_rn(-0.5, ty, __fma_rn(-0.5, a3, f[10]));
    f[8] = __fma_rn(0.5, ty, __fma_rn(-0.5, a3, f[8]));
    f[14] = __fma_rn(-0.5, tz, __fma_rn(-0.5, a3, f[14]));
    f[12] = __fma_rn(0.5, tz, __fma_rn(-0.5, a3, f[12]));
}

// ZouHeD2Q9_vx_x (Boundary_conditions.cpp:710-744), also the node update of parabolic_D2Q9_x
// (:748-800) with the profile's velocity: the +x movers from the closure density.
__device__ __forceinline__ void zou_he_d2q9(double f[9], double vx)
{
    const double rho = (((f[0] + f[3]) + f[4]) + 2 * ((f[2] + f[8]) + f[6])) / (1. - vx);
    const double p = (1.0 + 3.0 * vx) + 3.0 * vx * vx;
    f[1] = (rho / 9.0) * p;
    f[5] = (rho / 36.0) * p;
    f[7] = (rho / 36.0) * p;
}

// Node update of parabolic_D3Q19_x (Boundary_conditions.cpp:456-530): the +x movers from their
// opposites, rho from the closure (vy = vz = 0).
__device__ __forceinline__ void parabolic_d3q19(double f[19], double vx)
{
    const double vy = 0.0, vz = 0.0;
    const double s_minus = (((f[2] + f[8]) + f[10]) + f[12]) + f[14];
    const double s_zero = (((((((f[0] + f[3]) + f[4]) + f[5]) + f[6]) + f[15]) + f[16]) + f[17]) + f[18];
    const double rho = (2.0 * s_minus + s_zero) / (1.0 - vx);
    const double ty = (((((f[18] + f[3]) + f[16]) - f[15]) - f[4]) - f[17]);
    const double tz = (((((f[17] + f[5]) + f[16]) - f[15]) - f[6]) - f[18]);
    const double a3 = rho * vx / 3.0, a6 = rho * vx / 6.0;
    f[1] = f[2] + a3;
    f[7] = ((f[8] + a6) + 0.5 * rho * vy) - 0.5 * ty;
    f[9] = ((f[10] + a6) - 0.5 * rho * vy) + 0.5 * ty;
    f[11] = ((f[12] + a6) + 0.5 * rho * vz) - 0.5 * tz;
    f[13] = ((f[14] + a6) - 0.5 * rho * vz) + 0.5 * tz;
}

}  // namespace exact
}  // namespace erlbm
