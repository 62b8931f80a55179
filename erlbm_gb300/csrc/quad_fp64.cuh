// quad_fp64.cuh -- the exact FP64 collision of one node by four lanes, for lattices of few nodes.
//
// A warp's FP64 instruction holds its scheduler's pipe for some 80 cycles, whether its operands are independent or
// not and however few lanes take part.  A lattice of a few thousand nodes gives the GPU's 608 schedulers less than
// a warp each, and its step lasts as long as one thread's chain of FP64 operations.  Here a node's direction pairs
// are spread over four lanes, which shortens the chain from 262 operations to 109 (D3Q19) and from 140 to 65 (D2Q9),
// every one of them the operation collide19 / collide9 (collide_fp64.cuh) does for that population, in its order.
//  - moments: lane 0 sums the density, lanes 1 to 3 the momenta, as fused multiply-adds by 0 and +-1 (exact);
//  - D3Q19: lane 0 has the axis pairs, lanes 1, 2, 3 the diagonal pairs of the xy, xz and yz planes, lane 1 the rest
//    population too; D2Q9: a pair each, the rest population in every lane;
//  - the sums of the non-equilibrium parts go over shuffles where they are exact in any order (exact_sums), and
//    otherwise every lane forms them from all parts in the reference's order.
#pragma once

#include "collide_fp64.cuh"

namespace erlbm {
namespace quad {

using exact::abs_hi;

// Four lanes that share a node: this lane's number and the first lane's.
struct Team {
    int sub, base;
    __device__ __forceinline__ double from(double v, int lane) const { return __shfl_sync(0xffffffffu, v, base + lane); }
    __device__ __forceinline__ double pick(double a, double b, double c, double d) const
    {
        const double x = sub & 1 ? b : a, y = sub & 1 ? d : c;
        return sub & 2 ? y : x;
    }
    template <class T>
    __device__ __forceinline__ T first(T a, T other) const { return sub == 0 ? a : other; }
};

// Bit i: direction i's component along this lane's moment (lane 0: the density) is +1 (plus) or -1 (minus).
template <int Q>
__device__ __forceinline__ void moment_signs(int sub, uint32_t &plus, uint32_t &minus)
{
    uint32_t p[4] = {}, m[4] = {};
#pragma unroll
    for (int i = 0; i < Q; i++) {
        p[0] |= 1u << i;
        p[1] |= (uint32_t)(Lat<Q>::cx(i) > 0) << i;
        m[1] |= (uint32_t)(Lat<Q>::cx(i) < 0) << i;
        p[2] |= (uint32_t)(Lat<Q>::cy(i) > 0) << i;
        m[2] |= (uint32_t)(Lat<Q>::cy(i) < 0) << i;
        p[3] |= (uint32_t)(Lat<Q>::cz(i) > 0) << i;
        m[3] |= (uint32_t)(Lat<Q>::cz(i) < 0) << i;
    }
    plus = sub == 0 ? p[0] : (sub == 1 ? p[1] : (sub == 2 ? p[2] : p[3]));
    minus = sub == 0 ? m[0] : (sub == 1 ? m[1] : (sub == 2 ? m[2] : m[3]));
}

template <int Q>
__device__ __forceinline__ void moments(const double *f, const Team &t, double &rho, double &ux, double &uy, double &uz)
{
    uint32_t plus, minus;
    moment_signs<Q>(t.sub, plus, minus);
    double s = 0.0;
#pragma unroll
    for (int i = 0; i < Q; i++) {
        const uint32_t c = (plus >> i & 1u ? 0x3ff00000u : 0u) | (minus >> i & 1u ? 0xbff00000u : 0u);
        s = __fma_rn(__hiloint2double((int)c, 0), f[i], s);
    }
    rho = t.from(s, 0);
    const double u = rho != 0.0 ? s * (1.0 / rho) : 0.0;
    ux = t.from(u, 1);
    uy = t.from(u, 2);
    uz = Q == 19 ? t.from(u, 3) : 0.0;
}

// The polynomials ((1 +- 3 cv) + 4.5 cv^2) - C of a pair.
__device__ __forceinline__ void polynomials(double cv, double cv2, double C, uint64_t C62, bool small, double &a, double &b)
{
    if (small) {
        fp64int::eq_pair(cv, cv2, C62, a, b);
    } else {
        const double t3 = cv * 3., B = (1.5 * cv2) * 3.;
        a = ((1.0 + t3) + B) - C;
        b = ((1.0 - t3) + B) - C;
    }
}

// Collision of the team's node.  f: its populations, the same in the four lanes.  out: this lane's share, a pair in
// out[2 s], out[2 s + 1] for each of its slots (population<Q>); hint as exact::collide.
template <int Q>
constexpr int SLOTS = Q == 19 ? 3 : 2;

// The population in member m (0, 1) of slot s of lane `sub`, -1 for none.
template <int Q>
__host__ __device__ constexpr int population(int sub, int s, int m)
{
    if (Q == 9) return s == 0 ? 1 + 2 * sub + m : (sub == 0 && m == 0 ? 0 : -1);
    if (s == 2) return sub == 0 ? 5 + m : (sub == 1 && m == 0 ? 0 : -1);
    if (sub == 0) return 1 + 2 * s + m;
    if (sub == 3 && s == 0) return 16 - m;  // direction 16 is (0,1,1) and 15 its opposite
    return 3 + 4 * sub + 2 * s + m;
}

// Value of population i, from the share of the lane that has it.
template <int Q>
__device__ __forceinline__ double gathered(const double *share, const Team &t, int i)
{
    double v = 0.0;
#pragma unroll
    for (int k = 0; k < 4 * 2 * SLOTS<Q>; k++) {
        const int sub = k / (2 * SLOTS<Q>), s = k / 2 % SLOTS<Q>, m = k % 2;
        if (population<Q>(sub, s, m) == i) v = t.from(share[2 * s + m], sub);
    }
    return v;
}

template <int Q, int OP>
__device__ __forceinline__ uint32_t collide(const double *f, const Team &t, const Relax &R, double *out)
{
    constexpr int S = SLOTS<Q>;
    const int sub = t.sub;
    double rho, ux, uy, uz;
    moments<Q>(f, t, rho, ux, uy, uz);
    // this lane's populations and velocities
    double g[2 * S], cv[S];
    if constexpr (Q == 19) {
        g[0] = t.pick(f[1], f[7], f[11], f[16]), g[1] = t.pick(f[2], f[8], f[12], f[15]);
        g[2] = t.pick(f[3], f[9], f[13], f[17]), g[3] = t.pick(f[4], f[10], f[14], f[18]);
        g[4] = t.first(f[5], f[0]), g[5] = t.first(f[6], f[0]);
        const double a = sub == 3 ? uz : ux, b = sub & 1 ? uy : uz;  // the lane's plane: ux uy, ux uz, uz uy
        const double sp = a + b, sm = a - b;
        cv[0] = t.first(ux, sp), cv[1] = t.first(uy, sm), cv[2] = uz;
    } else {
        g[0] = t.pick(f[1], f[3], f[5], f[7]), g[1] = t.pick(f[2], f[4], f[6], f[8]);
        g[2] = g[3] = f[0];
        const double s = sub == 3 ? ux - uy : ux + uy;
        cv[0] = sub == 0 ? ux : (sub == 1 ? uy : s);
    }
    const double xx = ux * ux, yy = uy * uy;
    const double C = Q == 19 ? 1.5 * ((xx + yy) + uz * uz) : 1.5 * (xx + yy);
    const double k1 = Q == 19 ? 1. / 18. : 1. / 9., k2 = 1. / 36., kr = Q == 19 ? 1. / 3. : 4. / 9.;
    const bool axis = Q == 19 ? sub == 0 : sub < 2;
    const double wr = (axis ? k1 : k2) * rho;
    double q[2 * S];
    {
        uint32_t most = abs_hi(cv[0]);
        if (Q == 19) most = max(most, max(abs_hi(cv[1]), abs_hi(cv[2])));
        const bool small = most < fp64int::EQ_MAX_HI && abs_hi(C) < 0x3fbc28f5u;  // C < 0.11
        const uint64_t C62 = small ? fp64int::fixed62(C) : 0;
        const double rest = 1.0 - C;
        double a, b;
        polynomials(cv[0], cv[0] * cv[0], C, C62, small, a, b);
        q[0] = wr * a, q[1] = wr * b;
        if constexpr (Q == 19) {
            polynomials(cv[1], cv[1] * cv[1], C, C62, small, a, b);
            q[2] = wr * a, q[3] = wr * b;
            const double w2 = t.first(k1, kr) * rho;
            polynomials(cv[2], cv[2] * cv[2], C, C62, small, a, b);
            q[4] = w2 * t.first(a, rest), q[5] = w2 * t.first(b, rest);
        } else {
            q[2] = q[3] = (kr * rho) * rest;
        }
    }
    constexpr int N = Q == 19 ? 6 : 3;  // populations a lane updates (D2Q9: its pair and the rest population)
    if constexpr (OP == OP_BGK) {
#pragma unroll
        for (int i = 0; i < N; i++) out[i] = g[i] + (q[i] - g[i]) * R.inv_tau;
        return exact::NO_HINT;
    }
    double d[2 * S];
#pragma unroll
    for (int i = 0; i < N; i++) d[i] = g[i] - q[i];
    if (N < 2 * S) d[2 * S - 1] = d[2 * S - 2];
    // exact_sums over the team
    int least = min(__double2hiint(g[0]), __double2hiint(q[0]));
    unsigned most = abs_hi(d[0]);
#pragma unroll
    for (int i = 1; i < N; i++) {
        least = min(least, min(__double2hiint(g[i]), __double2hiint(q[i])));
        most = max(most, abs_hi(d[i]));
    }
#pragma unroll
    for (int o = 1; o < 4; o <<= 1) {
        least = min(least, __shfl_xor_sync(0xffffffffu, least, o));
        most = max(most, __shfl_xor_sync(0xffffffffu, most, o));
    }
    const bool any_order = (int)(most >> 20) + (Q == 19 ? 4 : 3) <= (least >> 20);
    const uint32_t hint = any_order ? exact::density_hint(rho, R) : exact::NO_HINT;
    double pxx, pyy, pzz = 0.0, pab;
    if (__all_sync(0xffffffffu, any_order)) {
        const double s0 = d[0] + d[1];
        if constexpr (Q == 19) {
            const double s1 = d[2] + d[3], s2 = d[4] + d[5], sum = s0 + s1;
            pab = s0 - s1;
            const double ab = t.from(sum, 1), gh = t.from(sum, 2), mn = t.from(sum, 3);
            pxx = t.from(s0, 0) + (ab + gh);
            pyy = t.from(s1, 0) + (ab + mn);
            pzz = t.from(s2, 0) + (gh + mn);
        } else {
            const double s56 = t.from(s0, 2), s78 = t.from(s0, 3), both = s56 + s78;
            pxx = t.from(s0, 0) + both;
            pyy = t.from(s0, 1) + both;
            pab = s56 - s78;
        }
    } else {
        double D[Q];
#pragma unroll
        for (int i = 1; i < Q; i++) D[i] = gathered<Q>(d, t, i);
        if constexpr (Q == 19) {
            pxx = ((((((((D[1] + D[2]) + D[7]) + D[8]) + D[9]) + D[10]) + D[11]) + D[12]) + D[13]) + D[14];
            pyy = ((((((((D[3] + D[4]) + D[7]) + D[8]) + D[9]) + D[10]) + D[15]) + D[16]) + D[17]) + D[18];
            pzz = ((((((((D[5] + D[6]) + D[11]) + D[12]) + D[13]) + D[14]) + D[15]) + D[16]) + D[17]) + D[18];
            const double a = t.pick(D[7], D[7], D[11], D[15]), b = t.pick(D[8], D[8], D[12], D[16]);
            const double c = t.pick(D[9], D[9], D[13], D[17]), e = t.pick(D[10], D[10], D[14], D[18]);
            pab = ((a + b) - c) - e;
        } else {
            pxx = ((((D[1] + D[2]) + D[5]) + D[6]) + D[7]) + D[8];
            pyy = ((((D[3] + D[4]) + D[5]) + D[6]) + D[7]) + D[8];
            pab = ((D[5] + D[6]) - D[7]) - D[8];
        }
    }
    using namespace exact;
    const double xa = QA * pxx, xb = QB * pxx, ya = QA * pyy, yb = QB * pyy;
    const double f1k = axis ? O2CS4 * k1 : O2CS4 * k2;
    double f1[S];
    if constexpr (Q == 19) {
        const double za = QA * pzz, zb = QB * pzz;
        const double b0 = ((sub == 3 ? xb : xa) + (sub & 1 ? ya : yb)) + (sub < 2 ? zb : za);
        // lane 1: xa ya zb; 2: xa yb za; 3: xb ya za; lane 0, X: xa yb zb
        const double b1 = (xb + ya) + zb;
        const double b2 = (xb + yb) + t.first(za, zb);
        const double h0 = __fma_rn(2., pab, b0), h1 = __fma_rn(-2., pab, b0);
        f1[0] = f1k * t.first(b0, h0);
        f1[1] = f1k * t.first(b1, h1);
        f1[2] = t.first(O2CS4 * k1, O2CS4 * kr) * b2;
    } else {
        const double b0 = (sub == 1 ? xb : xa) + (sub == 0 ? yb : ya);
        const double h = __fma_rn(sub == 3 ? -2. : 2., pab, b0);
        f1[0] = f1k * (axis ? b0 : h);
        f1[1] = (O2CS4 * kr) * (xb + yb);
    }
#pragma unroll
    for (int s = 0; s < S; s++) {
        const double w1 = R.omega_1 * f1[s];
#pragma unroll
        for (int m = 0; m < 2; m++) {
            const int i = 2 * s + m;
            if (i >= N) continue;
            if (OP == OP_REG)
                out[i] = q[i] + w1;
            else
                out[i] = (q[i] + w1) + R.omega_gt1 * (d[i] - f1[s]);
        }
    }
    return hint;
}

}  // namespace quad
}  // namespace erlbm
