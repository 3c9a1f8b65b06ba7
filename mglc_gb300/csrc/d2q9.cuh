// d2q9.cuh -- the D2Q9 MRT collision of the reference's 2-D codes, bit for bit
// (Lid_driven_cavity/fortran/2d/2d_revised/mpi_blocked/evolution.f90:16-68 and
// Micro_particles/fortran/case4/mpi_particle/fluid.F90:14-64), shared by the
// 2-D cavity and the 2-D particle kernels.  Both are bound by the FP64 pipe (a
// warp's instruction holds the SM's unit for 16 clocks or more), so the fast
// path writes the statements with as few FP64 instructions as give the same bits:
// 108 a node with the quotients of the macro (ncu), where the statements as written
// took about 190 (2-D cavity, 1024^2: 404 us a step as written, 331 with
// the first three of these, 221 with all; 22 are its bytes):
//  * products by 2, 4, 1/2 and 1/4 are exact, so a sum with one is a single
//    fused multiply-add with the same rounding, and a chain of sums of doubled
//    terms is twice the chain of the terms;
//  * the conserved moments relax at s = 0: m - 0 (m - meq) is m for finite
//    values other than -0;
//  * x/18 = 2 (x/36) and x/12 = (x/6)/2 exactly, so eight quotients serve all;
//    a quotient by 6, 9, 18 or 36 is one multiply and one fused multiply-add
//    (div_const), and two quotients by rho share one reciprocal (div_pair);
//  * the fifty additions of the moments, and most of that reciprocal, run on
//    integers, each rounded as FP64 rounds (Fix9), in issue slots that are empty.
// A node whose values are outside the ranges that these need (fast_ok) takes
// the statements as the reference writes them.
// Include only in files compiled with -fmad=false: the contractions are the
// explicit __fma_rn.
#pragma once
#include <cuda_runtime.h>

#include "fix61.cuh"

namespace mglc {

// Quotients by the collision's constant divisors d = 6, 9, 18, 36, rounded
// exactly as IEEE division rounds them, from one multiply and one fused
// multiply-add: x/d = RN(x*h + RN(x*l)) with h = 1/d rounded down and
// l = 1/d - h rounded to nearest (a two-term reciprocal; Brisebarre, Muller and
// Raina, "Accelerating correctly rounded floating-point division when the
// divisor is known in advance", IEEE Trans. Computers 53(8), 2004).  Why the
// rounding is the division's: d = 3*2^k or 9*2^k, so for normal x the exact
// x/d lies at least ulp(x/d)/18 from every rounding midpoint (d times a
// midpoint is an odd multiple of 2^(e-53), x an even one), while h + l is 1/d
// to about 2^-106 relative, putting x*h + RN(x*l) within ~2^-104 relative of
// x/d: no midpoint between them.  Zeros keep their signs because l > 0; inputs
// below 2^-900 in magnitude (x*l could lose bits to underflow) are outside.
constexpr double INV6_H = 0x1.5555555555555p-3, INV6_L = 0x1.5555555555555p-57;
constexpr double INV9_H = 0x1.c71c71c71c71cp-4, INV9_L = 0x1.c71c71c71c71cp-58;
constexpr double INV18_H = 0x1.c71c71c71c71cp-5, INV18_L = 0x1.c71c71c71c71cp-59;
constexpr double INV36_H = 0x1.c71c71c71c71cp-6, INV36_L = 0x1.c71c71c71c71cp-60;

__device__ __forceinline__ double div_const(double x, double h, double l) {
    return __fma_rn(x, h, __dmul_rn(x, l));
}

// 2^-900 <= |x| < 2^901, or a zero of either sign
__device__ __forceinline__ bool mid_or_zero(double x) {
    const unsigned h = (unsigned)__double2hiint(x);
    return ((h >> 20) & 0x7ffu) - 123u <= 1800u || ((h << 1) | (unsigned)__double2loint(x)) == 0u;
}
// the same, without -0
__device__ __forceinline__ bool mid_or_pzero(double x) {
    const unsigned h = (unsigned)__double2hiint(x);
    return ((h >> 20) & 0x7ffu) - 123u <= 1800u || (h | (unsigned)__double2loint(x)) == 0u;
}
// a density whose reciprocal div_pair may share: 2^-15 <= r < 2^16 (so r > 0)
// and a significand that is not all ones
__device__ __forceinline__ bool den_ok(double r) {
    const unsigned h = (unsigned)__double2hiint(r);
    return (h >> 20) - 1008u <= 30u &&
           !((h & 0xfffffu) == 0xfffffu && (unsigned)__double2loint(r) == 0xffffffffu);
}

// a/r and b/r, correctly rounded, from one reciprocal (Markstein, "Computation
// of elementary functions on the IBM RISC System/6000 processor", IBM J. Res.
// Dev. 34(1), 1990): Newton steps from a single-precision seed (relative error
// 2^-23 -> 2^-46 -> below one ulp), one more gives 1/r correctly rounded unless
// r's significand is all ones; then with q = RN(a y) and the exact remainder
// a - q r, RN(q + rem y) is a/r correctly rounded.  For den_ok(r) and
// mid_or_pzero(a), mid_or_pzero(b): no remainder leaves the normal range, and
// a zero quotient is +0.
__device__ __forceinline__ void div_pair(double a, double b, double r, double& qa, double& qb) {
    double y = (double)__frcp_rn((float)r);
    y = __fma_rn(__fma_rn(-r, y, 1.0), y, y);
    y = __fma_rn(__fma_rn(-r, y, 1.0), y, y);
    y = __fma_rn(__fma_rn(-r, y, 1.0), y, y);
    const double ta = __dmul_rn(a, y), tb = __dmul_rn(b, y);
    qa = __fma_rn(__fma_rn(-r, ta, a), y, ta);
    qb = __fma_rn(__fma_rn(-r, tb, b), y, tb);
}

// Sums of populations, each addition rounded as FP64's: populations in [2^-6, 1/2)
// are exact in units of 2^-58, and there an addition is an integer one followed
// by the rounding of the sum to 53 significant bits (rn53), bit for bit.
__device__ __forceinline__ bool d2q9_fix_ok(const double (&f)[9]) {
    unsigned worst = 0;
#pragma unroll
    for (int q = 1; q < 9; q++)
        worst = max(worst, (unsigned)__double2hiint(f[q]) - 0x3F900000u);  // 2^-6
    return worst < 0x00400000u &&                                          // below 1/4
           (unsigned)__double2hiint(f[0]) - 0x3F900000u < 0x00500000u;     // below 1/2
}
struct Fix9 {
    long long v;
};
__device__ __forceinline__ Fix9 operator+(Fix9 a, Fix9 b) { return {rn53(a.v + b.v)}; }
__device__ __forceinline__ Fix9 operator-(Fix9 a, Fix9 b) { return {rn53(a.v - b.v)}; }
// s a + b, one rounding
__device__ __forceinline__ Fix9 fma9(int s, Fix9 a, Fix9 b) { return {rn53(s * a.v + b.v)}; }
__device__ __forceinline__ double fma9(int s, double a, double b) { return __fma_rn((double)s, a, b); }
__device__ __forceinline__ Fix9 neg9(Fix9 a) { return {-a.v}; }
__device__ __forceinline__ double neg9(double a) { return -a; }
__device__ __forceinline__ void d2q9_fix_load(const double (&f)[9], Fix9 (&F)[9]) {
#pragma unroll
    for (int q = 0; q < 9; q++) {
        const unsigned hi = (unsigned)__double2hiint(f[q]), lo = (unsigned)__double2loint(f[q]);
        const unsigned s = (hi >> 20) - 1017u;
        const unsigned mh = (hi & 0xFFFFFu) | 0x100000u;
        F[q].v = (long long)(((unsigned long long)__funnelshift_l(lo, mh, s) << 32) | (lo << s));
    }
}

// moments of the macro (evolution.f90:103-107, fluid.F90:164-184)
template <class T>
__device__ __forceinline__ void d2q9_sums(const T (&f)[9], T& r, T& jx, T& jy) {
    r = f[0] + f[1] + f[2] + f[3] + f[4] + f[5] + f[6] + f[7] + f[8];
    jx = f[1] - f[3] + f[5] - f[6] - f[7] + f[8];
    jy = f[2] - f[4] + f[5] + f[6] - f[7] - f[8];
}
// and of the collision.  GROUPED: m1 and m2 sum the equal terms first
// (evolution.f90:17-18, case1 fluid.F90:15-16), else term by term (case4 fluid.F90)
template <bool GROUPED, class T>
__device__ __forceinline__ void d2q9_moments(const T (&f)[9], T (&m)[9]) {
    d2q9_sums(f, m[0], m[3], m[5]);
    T m1 = fma9(-4, f[0], neg9(f[1])) - f[2] - f[3] - f[4], m2;
    if (GROUPED) {
        m1 = fma9(2, f[5] + f[6] + f[7] + f[8], m1);
        m2 = fma9(2, f[0], neg9(f[1] + f[2] + f[3] + f[4]));  // half of 4 f0 - 2 (...)
    } else {
        m1 = fma9(2, f[5], m1);
        m1 = fma9(2, f[6], m1);
        m1 = fma9(2, f[7], m1);
        m1 = fma9(2, f[8], m1);
        m2 = fma9(2, f[0], neg9(f[1])) - f[2] - f[3] - f[4];
    }
    m[1] = m1;
    m[2] = fma9(2, m2, f[5]) + f[6] + f[7] + f[8];
    m[4] = fma9(2, f[3] - f[1], f[5]) - f[6] - f[7] + f[8];
    m[6] = fma9(2, f[4] - f[2], f[5]) + f[6] - f[7] - f[8];
    m[7] = f[1] - f[2] + f[3] - f[4];
    m[8] = f[5] - f[6] + f[7] - f[8];
}

// velocity from the sums as doubles
__device__ __forceinline__ void d2q9_velocity(double r, double jx, double jy, double& u, double& v) {
    if (den_ok(r) && mid_or_pzero(jx) && mid_or_pzero(jy)) {
        div_pair(jx, jy, r, u, v);
    } else {
        u = jx / r;
        v = jy / r;
    }
}
// and for a density of R >= 1/4 in units of 2^-58 (sums in range, so below 2.75): the
// reciprocal to 2^-60 on integers, rounded, then div_pair's last step
__device__ __forceinline__ void d2q9_velocity(long long R, double r, double jx, double jy,
                                              double& u, double& v) {
    if (R >= (1LL << 56) && den_ok(r)) {
        double y = fix_out<60>(rn53(fix_recip(R << 3, fix_dig(R << 3))));
        y = __fma_rn(__fma_rn(-r, y, 1.0), y, y);
        const double ta = __dmul_rn(jx, y), tb = __dmul_rn(jy, y);
        u = __fma_rn(__fma_rn(-r, ta, jx), y, ta);
        v = __fma_rn(__fma_rn(-r, tb, jy), y, tb);
    } else {
        u = jx / r;
        v = jy / r;
    }
}

__device__ __forceinline__ void d2q9_macro(const double (&f)[9], double& r, double& u, double& v) {
    double jx, jy;
    if (d2q9_fix_ok(f)) {
        Fix9 F[9], R, X, Y;
        d2q9_fix_load(f, F);
        d2q9_sums(F, R, X, Y);
        r = fix_out<58>(R.v);
        jx = fix_out<58>(X.v);
        jy = fix_out<58>(Y.v);
        d2q9_velocity(R.v, r, jx, jy, u, v);
    } else {
        d2q9_sums(f, r, jx, jy);
        d2q9_velocity(r, jx, jy, u, v);
    }
}

// the collision as the reference writes it; GROUPED: m1 and m2 sum the equal
// terms first (evolution.f90:17-18, case1 fluid.F90:15-16), else term by term
// (case4 fluid.F90)
template <bool GROUPED>
__device__ __noinline__ void d2q9_collide_plain(const double* f, double rho, double u, double v,
                                                double snu, double sq, double* fp) {
    double m[9], meq[9], s[9], mp[9];
    m[0] = f[0] + f[1] + f[2] + f[3] + f[4] + f[5] + f[6] + f[7] + f[8];
    if (GROUPED) {
        m[1] = -4.0 * f[0] - f[1] - f[2] - f[3] - f[4] + 2.0 * (f[5] + f[6] + f[7] + f[8]);
        m[2] = 4.0 * f[0] - 2.0 * (f[1] + f[2] + f[3] + f[4]) + f[5] + f[6] + f[7] + f[8];
    } else {
        m[1] = -4.0 * f[0] - f[1] - f[2] - f[3] - f[4] + 2.0 * f[5] + 2.0 * f[6] + 2.0 * f[7] + 2.0 * f[8];
        m[2] = 4.0 * f[0] - 2.0 * f[1] - 2.0 * f[2] - 2.0 * f[3] - 2.0 * f[4] + f[5] + f[6] + f[7] + f[8];
    }
    m[3] = f[1] - f[3] + f[5] - f[6] - f[7] + f[8];
    m[4] = -2.0 * f[1] + 2.0 * f[3] + f[5] - f[6] - f[7] + f[8];
    m[5] = f[2] - f[4] + f[5] + f[6] - f[7] - f[8];
    m[6] = -2.0 * f[2] + 2.0 * f[4] + f[5] + f[6] - f[7] - f[8];
    m[7] = f[1] - f[2] + f[3] - f[4];
    m[8] = f[5] - f[6] + f[7] - f[8];
    meq[0] = rho;
    meq[1] = rho * (-2.0 + 3.0 * (u * u + v * v));
    meq[2] = rho * (1.0 - 3.0 * (u * u + v * v));
    meq[3] = rho * u;
    meq[4] = -meq[3];
    meq[5] = rho * v;
    meq[6] = -meq[5];
    meq[7] = rho * (u * u - v * v);
    meq[8] = rho * (u * v);
    s[0] = 0.0; s[1] = snu; s[2] = snu; s[3] = 0.0; s[4] = sq; s[5] = 0.0; s[6] = sq;
    s[7] = snu; s[8] = snu;
    for (int a = 0; a < 9; a++) mp[a] = m[a] - s[a] * (m[a] - meq[a]);
    fp[0] = (mp[0] - mp[1] + mp[2]) / 9.0;
    fp[1] = mp[0] / 9.0 - mp[1] / 36.0 - mp[2] / 18.0 + mp[3] / 6.0 - mp[4] / 6.0 + mp[7] * 0.25;
    fp[2] = mp[0] / 9.0 - mp[1] / 36.0 - mp[2] / 18.0 + mp[5] / 6.0 - mp[6] / 6.0 - mp[7] * 0.25;
    fp[3] = mp[0] / 9.0 - mp[1] / 36.0 - mp[2] / 18.0 - mp[3] / 6.0 + mp[4] / 6.0 + mp[7] * 0.25;
    fp[4] = mp[0] / 9.0 - mp[1] / 36.0 - mp[2] / 18.0 - mp[5] / 6.0 + mp[6] / 6.0 - mp[7] * 0.25;
    fp[5] = mp[0] / 9.0 + mp[1] / 18.0 + mp[2] / 36.0 + mp[3] / 6.0 + mp[4] / 12.0 + mp[5] / 6.0 +
            mp[6] / 12.0 + mp[8] * 0.25;
    fp[6] = mp[0] / 9.0 + mp[1] / 18.0 + mp[2] / 36.0 - mp[3] / 6.0 - mp[4] / 12.0 + mp[5] / 6.0 +
            mp[6] / 12.0 - mp[8] * 0.25;
    fp[7] = mp[0] / 9.0 + mp[1] / 18.0 + mp[2] / 36.0 - mp[3] / 6.0 - mp[4] / 12.0 - mp[5] / 6.0 -
            mp[6] / 12.0 + mp[8] * 0.25;
    fp[8] = mp[0] / 9.0 + mp[1] / 18.0 + mp[2] / 36.0 + mp[3] / 6.0 + mp[4] / 12.0 - mp[5] / 6.0 -
            mp[6] / 12.0 - mp[8] * 0.25;
}

// post-collision populations fp of one node from its populations and rho, u, v
// (MACRO: which it forms first)
template <bool GROUPED, bool MACRO>
__device__ __forceinline__ void d2q9_collide(const double (&f)[9], double& rho, double& u, double& v,
                                             double snu, double sq, double (&fp)[9]) {
    double m[9];
    if (d2q9_fix_ok(f)) {
        Fix9 F[9], M[9];
        d2q9_fix_load(f, F);
        d2q9_moments<GROUPED>(F, M);
#pragma unroll
        for (int a = 0; a < 9; a++) m[a] = fix_out<58>(M[a].v);
        if (MACRO) d2q9_velocity(M[0].v, m[0], m[3], m[5], u, v);
    } else {
        // A density that is not finite: the conserved moment relaxes to m0 - 0 (m0 - rho),
        // a NaN, and every population takes it (a cavity of NaN ran at 0.57 of the speed that
        // the statements as written had, without this).
        const double m0 = f[0] + f[1] + f[2] + f[3] + f[4] + f[5] + f[6] + f[7] + f[8];
        if (!isfinite(m0)) {
            if (MACRO) rho = m0;
#pragma unroll
            for (int a = 0; a < 9; a++) fp[a] = __longlong_as_double(0x7ff8000000000000LL);
            return;
        }
        d2q9_moments<GROUPED>(f, m);
        if (MACRO) d2q9_velocity(m[0], m[3], m[5], u, v);
    }
    if (MACRO) rho = m[0];
    const double m0 = m[0], m1 = m[1], m2 = m[2], m3 = m[3], m4 = m[4], m5 = m[5], m6 = m[6],
                 m7 = m[7], m8 = m[8];
    const double u2 = u * u, v2 = v * v, t3 = 3.0 * (u2 + v2);
    const double ru = rho * u, rv = rho * v;
    const double p1 = m1 - snu * (m1 - rho * (-2.0 + t3));
    const double p2 = m2 - snu * (m2 - rho * (1.0 - t3));
    const double p4 = m4 - sq * (m4 + ru);
    const double p6 = m6 - sq * (m6 + rv);
    const double p7 = m7 - snu * (m7 - rho * (u2 - v2));
    const double p8 = m8 - snu * (m8 - rho * (u * v));
    const double p0 = m0 - p1 + p2;
    const bool fast = mid_or_pzero(m0) && mid_or_pzero(m3) && mid_or_pzero(m5) && mid_or_zero(rho) &&
                      mid_or_zero(ru) && mid_or_zero(rv) && mid_or_zero(p1) && mid_or_zero(p2) &&
                      mid_or_zero(p4) && mid_or_zero(p6) && mid_or_zero(p7) && mid_or_zero(p8) &&
                      mid_or_zero(p0);
    if (fast) {
        const double q0 = div_const(m0, INV9_H, INV9_L), q1 = div_const(p1, INV36_H, INV36_L),
                     q2 = div_const(p2, INV18_H, INV18_L), q3 = div_const(m3, INV6_H, INV6_L),
                     q4 = div_const(p4, INV6_H, INV6_L), q5 = div_const(m5, INV6_H, INV6_L),
                     q6 = div_const(p6, INV6_H, INV6_L);
        fp[0] = div_const(p0, INV9_H, INV9_L);
        const double B = q0 - q1 - q2;
        fp[1] = __fma_rn(0.25, p7, B + q3 - q4);
        fp[2] = __fma_rn(-0.25, p7, B + q5 - q6);
        fp[3] = __fma_rn(0.25, p7, B - q3 + q4);
        fp[4] = __fma_rn(-0.25, p7, B - q5 + q6);
        const double E = __fma_rn(0.5, q2, __fma_rn(2.0, q1, q0));
        const double P = __fma_rn(0.5, q4, E + q3), M = __fma_rn(-0.5, q4, E - q3);
        fp[5] = __fma_rn(0.25, p8, __fma_rn(0.5, q6, P + q5));
        fp[6] = __fma_rn(-0.25, p8, __fma_rn(0.5, q6, M + q5));
        fp[7] = __fma_rn(0.25, p8, __fma_rn(-0.5, q6, M - q5));
        fp[8] = __fma_rn(-0.25, p8, __fma_rn(-0.5, q6, P - q5));
    } else {
        double g[9], o[9];
        for (int a = 0; a < 9; a++) g[a] = f[a];
        d2q9_collide_plain<GROUPED>(g, rho, u, v, snu, sq, o);
        for (int a = 0; a < 9; a++) fp[a] = o[a];
    }
}

}  // namespace mglc
