// fix61.cuh -- the FP64 collision on the integer pipe.
//
// GB300 issues two FP64 instructions per clock and SM, 64 lanes' worth of
// integer ones in the same time, and the FP64 step is bound by that pipe: 141
// FP64 instructions a lid cell are 256 ps of it, while 304 bytes are 45 ps of
// HBM and nine tenths of the issue slots stay empty.  The pair form (PairK,
// lbm_common.cuh) is therefore computed on 64-bit integers holding value * 2^61:
//  * a population in [2^-8, 1/2) is exact in 2^-61, so loading rounds nothing;
//    sums and differences are exact;
//  * a product keeps 2^-61, rounded to nearest;
//  * each stored value is rounded once, to nearest even.
// 2^-61 is finer than an FP64 ulp from 2^-8 up, so every result lies closer to
// the exact collision than the FP64 evaluation's, whose sums and products round
// on the way (tests/test_fix61_host.py; velocity error after six steps of 384^3
// 2.1e-13 against 3.3e-13).  1554 instructions a lid cell, twelve of them FP64 (ncu):
// 384^3 in 3.26 ms a step (17.4 GLUPS, 78% of HBM) against 15.7 ms in FP64;
// the heated cavity at 128^3, temperature populations on integers too, in units of
// their own (fix_heat; 235 with those in FP64), in 205 us (10.2 GLUPS) against 813.
// Cells outside its range (a population outside [2^-8, 1/8), the rest
// population outside [1/8, 1/2), negative and non-finite ones among them, rho
// below 1/4 or a velocity component of 1/2 or more) take the FP64 form; inside,
// every intermediate stays below 2^63.
#pragma once
#include <cstdint>

#include "lbm_common.cuh"

namespace mglc {

constexpr double FIX_ONE = 2305843009213693952.0;  // 2^61

// every population in range, from the high words of their bit patterns
__device__ __forceinline__ bool fix61_ok(const double (&f)[Q19]) {
    unsigned worst = 0;
#pragma unroll
    for (int q = 1; q < Q19; q++)
        worst = max(worst, (unsigned)__double2hiint(f[q]) - 0x3F700000u);  // 2^-8
    return worst < 0x00500000u &&                                          // below 2^-3
           (unsigned)__double2hiint(f[0]) - 0x3FC00000u < 0x00200000u;     // [2^-3, 1/2)
}

// x in [2^-8, 1/2) as x * 2^61: the significand shifted left by 0..8
__device__ __forceinline__ long long fix61_load(double x) {
    const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
    const unsigned s = (hi >> 20) - 1014u;
    const unsigned mh = (hi & 0xFFFFFu) | 0x100000u;
    return (long long)(((unsigned long long)__funnelshift_l(lo, mh, s) << 32) | (lo << s));
}

// v * 2^-61 rounded to nearest even, for 2^53 <= v < 2^63
__device__ __forceinline__ double fix61_store(long long v) {
    const unsigned hi = (unsigned)((unsigned long long)v >> 32);
    const int lz = __clz((int)hi), r = 11 - lz;  // 1 <= r <= 10 bits to drop
    const unsigned odd = (unsigned)((unsigned long long)v >> r) & 1u;
    const unsigned long long w = (unsigned long long)v + ((1u << (r - 1)) - 1u) + odd;
    // exponent field 1023 + 63 - lz - 61, less one for the implicit bit
    const unsigned long long m = w >> r;
    return __longlong_as_double((long long)(m + ((unsigned long long)(unsigned)(1024 - lz) << 52)));
}
// v * 2^-Q for any v, on the FP64 unit
template <int Q = 61>
__device__ __forceinline__ double fix61_store_any(long long v) {
    const long long b = __double_as_longlong((double)v);
    return __longlong_as_double(v ? b - ((long long)Q << 52) : 0LL);
}

// v rounded to 53 significant bits, to nearest even; |v| < 2^63
__device__ __forceinline__ long long rn53(long long v) {
    const int hi = (int)(v >> 32);
    const int r = max(11 - __clz(hi ^ (hi >> 31)), 0);
    const unsigned m = (1u << r) - 1u;  // the bits to drop
    const unsigned odd = (unsigned)(v >> r) & m & 1u;
    return (v + (long long)(m >> 1) + (long long)odd) & ~(long long)m;
}

// the same for v >= 0
__device__ __forceinline__ long long rn53_pos(long long v) {
    const int r = max(11 - __clz((int)(v >> 32)), 0);
    const unsigned m = (1u << r) - 1u;
    const unsigned odd = (unsigned)(v >> r) & m & 1u;
    return (v + (long long)(m >> 1) + (long long)odd) & ~(long long)m;
}

// v * 2^-Q for a v of at most 53 significant bits, with integer operations
template <int Q>
__device__ __forceinline__ double fix_out(long long v) {
    const long long sg = v >> 63;
    const unsigned long long a = (unsigned long long)((v ^ sg) - sg);
    const int lz = __clzll((long long)a);
    const unsigned long long m = a << (lz & 63) >> 11;  // the leading bit at bit 52
    const unsigned long long b = m + ((unsigned long long)(unsigned)(1022 + 63 - Q - lz) << 52);
    return __longlong_as_double((long long)(a ? b | ((unsigned long long)sg << 63) : 0ull));
}

// v = h * 2^32 + l in balanced digits
struct FixD {
    int h, l;
};
__device__ __forceinline__ FixD fix_dig(long long v) {
    FixD d;
    d.l = (int)v;
    d.h = (int)(v >> 32) + (int)((unsigned)d.l >> 31);
    return d;
}
__device__ __forceinline__ long long join(FixD d) { return ((long long)d.h << 32) + d.l; }
// a + (v * c) / 2^64, the product rounded to nearest
__device__ __forceinline__ long long fix_mad(FixD v, FixC c, long long a) {
    long long x = (long long)v.h * c.l + (0x80000000LL + __mulhi(v.l, c.l));
    x += (long long)v.l * c.h;
    return (long long)v.h * c.h + (a + (long long)(int)(x >> 32));
}
__device__ __forceinline__ long long fix_mad(long long v, FixC c, long long a) {
    return fix_mad(fix_dig(v), c, a);
}
// (v * w) / 2^S, rounded to nearest, 58 <= S <= 64
template <int S>
__device__ __forceinline__ long long fix_mul(FixD v, FixD w) {
    long long x = (long long)v.h * w.l + ((1LL << (S - 33)) + __mulhi(v.l, w.l));
    x += (long long)v.l * w.h;
    const long long t = (long long)v.h * w.h;
    return S == 64 ? t + (long long)(int)(x >> 32) : (t << (64 - S)) + (x >> (S - 32));
}

// 1/rho in units of 2^-60 for rho in [1/4, 2.75) (units of 2^-61): a
// single-precision seed and two Newton steps, the first to 2^-43 on one digit,
// the second with the exact residual (within 1.5 units)
__device__ __forceinline__ long long fix_recip(long long rho, FixD rd) {
    const float rf = (float)(int)(rho >> 32) * 0x1p-29f;
    const int xh = __float2int_rn(__frcp_rn(rf) * 0x1p28f);  // units of 2^-28
    // e = 1 - rho x, units of 2^-61, below 2^-21
    const long long e = (1LL << 61) - (((long long)rd.h * xh << 4) + ((long long)rd.l * xh >> 28));
    const long long x1 = ((long long)xh << 32) + ((long long)xh * (int)(e >> 10) >> 19);
    const int e1 = (int)((1LL << 61) - fix_mul<60>(rd, fix_dig(x1)));  // below 2^-42
    return x1 + (((long long)(int)(x1 >> 32) * e1 + (1LL << 28)) >> 29);
}

__device__ __forceinline__ void fix_pair(long long* F, int a, int b, const FixK& k, long long E,
                                         long long O) {
    const long long p = fix_mad(F[a] + F[b], k.c1, E), m = fix_mad(F[a] - F[b], k.c2, O);
    F[a] = p + m;
    F[b] = p - m;
}

// integer populations to doubles, the first NFP of them on the FP64 unit, the
// others with integer operations (all on the FP64 unit when one is below 2^-8 or
// negative, which is rare): the lid kernels, which need that unit for nothing
// else, run best with 10 (3309 us a step at 384^3; 3456 with none, 3326 with all),
// the heated ones, which store their temperature populations through it too, with 5
// (205 us at 128^3; 208 with none, 209 with 10)
template <int NFP>
__device__ __forceinline__ void fix61_store_all(const long long (&F)[Q19], double (&f)[Q19]) {
    int least = 0x7fffffff;
#pragma unroll
    for (int q = 0; q < Q19; q++) least = min(least, (int)(F[q] >> 32));
    if (least >= 0x200000) {
#pragma unroll
        for (int q = 0; q < Q19; q++)
            f[q] = q < NFP ? fix61_store_any(F[q]) : fix61_store(F[q]);
    } else {
#pragma unroll
        for (int q = 0; q < Q19; q++) f[q] = fix61_store_any(F[q]);
    }
}

// Density, momentum and velocity of a cell, as the collision takes them.
struct FixFlow {
    long long r;                // density
    FixD rd, Jx, Jy, Jz;        // and rho u
    FixD ux, uy, uz;            // velocity, units of 2^-63
    long long ex, ey, ez, d19;  // 2 (j - rho u); FIRST: Snu/19 (sum f - rho)
};
// From the populations and half the force carried from the previous step
// (hx, hy, hz; rho u = j + Fp/2), or, FIRST (the step after initial or load),
// from the macro arrays; false when the density or the velocity is out of range.
template <bool FIRST>
__device__ __forceinline__ bool fix61_flow(const long long (&F)[Q19], const FixK& k, long long hx,
                                           long long hy, long long hz, double rho0, double u0,
                                           double v0, double w0, FixFlow& o) {
    long long r, jx, jy, jz;
    moments0(F, r, jx, jy, jz);
    if (FIRST) {
        if (!(rho0 >= 0.25 && rho0 < 2.75 && fabs(u0) < 0.5 && fabs(v0) < 0.5 && fabs(w0) < 0.5))
            return false;
        o.r = __double2ll_rn(rho0 * FIX_ONE);
        o.rd = fix_dig(o.r);
        o.ux = fix_dig(__double2ll_rn(u0 * (4.0 * FIX_ONE)));
        o.uy = fix_dig(__double2ll_rn(v0 * (4.0 * FIX_ONE)));
        o.uz = fix_dig(__double2ll_rn(w0 * (4.0 * FIX_ONE)));
        const long long Jx = fix_mul<63>(o.rd, o.ux), Jy = fix_mul<63>(o.rd, o.uy),
                        Jz = fix_mul<63>(o.rd, o.uz);
        o.Jx = fix_dig(Jx);
        o.Jy = fix_dig(Jy);
        o.Jz = fix_dig(Jz);
        o.ex = 2 * (jx - Jx);
        o.ey = 2 * (jy - Jy);
        o.ez = 2 * (jz - Jz);
        o.d19 = fix_mad(r - o.r, k.l19, 0);
        return true;
    }
    jx += hx;
    jy += hy;
    jz += hz;
    const long long half = r >> 1;
    if (!(r >= (1LL << 59) && jx < half && -jx < half && jy < half && -jy < half && jz < half &&
          -jz < half))
        return false;
    o.r = r;
    o.rd = fix_dig(r);
    o.Jx = fix_dig(jx);
    o.Jy = fix_dig(jy);
    o.Jz = fix_dig(jz);
    const FixD di = fix_dig(fix_recip(r, o.rd));
    o.ux = fix_dig(fix_mul<58>(o.Jx, di));
    o.uy = fix_dig(fix_mul<58>(o.Jy, di));
    o.uz = fix_dig(fix_mul<58>(o.Jz, di));
    o.ex = -2 * hx;
    o.ey = -2 * hy;
    o.ez = -2 * hz;
    o.d19 = 0;
    return true;
}

// The collision in place of a cell's populations as integers.
// LID: the lid operator's quirk (pair_collide_lid).  FORCE: 0 none, 1 F_z only,
// 2 all components (pair_collide_forced; fx, fy, fz this step's force); DF: the
// force changes from step to step.
template <bool LID, int FORCE, bool FIRST, bool DF>
__device__ __forceinline__ void fix61_collide(long long (&F)[Q19], const FixK& k, const FixFlow& o,
                                              long long fx, long long fy, long long fz) {
    // Snu/8 V in units of 2^-62, V = rho u + (1 - Snu/2)/(Snu/2) F
    long long vx = fix_mad(o.Jx, k.l8, 0), vy = fix_mad(o.Jy, k.l8, 0), vz = fix_mad(o.Jz, k.l8, 0);
    // Sq/12 W, W = rho u + (1 - Sq/2)/Sq F
    long long gx = fix_mad(o.Jx, k.l6, 0), gy = fix_mad(o.Jy, k.l6, 0), gz = fix_mad(o.Jz, k.l6, 0);
    if (FORCE == 2) {
        const FixD dx = fix_dig(fx), dy = fix_dig(fy);
        vx = fix_mad(dx, k.kv, vx);
        vy = fix_mad(dy, k.kv, vy);
        gx = fix_mad(dx, k.kw, gx);
        gy = fix_mad(dy, k.kw, gy);
    }
    if (FORCE) {
        const FixD dz = fix_dig(fz);
        vz = fix_mad(dz, k.kv, vz);
        gz = fix_mad(dz, k.kw, gz);
    }
    const FixD kx = fix_dig(vx), ky = fix_dig(vy), kz = fix_dig(vz);
    const long long X = fix_mul<64>(kx, o.ux), Y = fix_mul<64>(ky, o.uy), Z = fix_mul<64>(kz, o.uz);
    // u_a V_b + u_b V_a: equal products where neither component has a force
    const long long cxy = FORCE == 2 ? fix_mul<64>(kx, o.uy) + fix_mul<64>(ky, o.ux)
                                     : 2 * fix_mul<64>(kx, o.uy);
    const long long cxz = FORCE ? fix_mul<64>(kx, o.uz) + fix_mul<64>(kz, o.ux)
                                : 2 * fix_mul<64>(kx, o.uz);
    const long long cyz = FORCE ? fix_mul<64>(ky, o.uz) + fix_mul<64>(kz, o.uy)
                                : 2 * fix_mul<64>(ky, o.uz);
    const long long S = X + Y + Z;
    const long long b = fix_mad(o.rd, k.l18, fix_mad(S, k.third, 0));
    const long long b2 = 2 * b + o.d19, be = b + o.d19;
    // what the conserved momentum leaves in the odd part: Sq/20 (2 (j - rho u) + F)
    long long ox = gx, oy = gy, oz = gz;
    if (FIRST || (DF && FORCE == 2)) {
        ox = fix_mad(o.ex + (FORCE == 2 ? fx : 0), k.l20, gx);
        oy = fix_mad(o.ey + (FORCE == 2 ? fy : 0), k.l20, gy);
    }
    if (FIRST || (DF && FORCE)) oz = fix_mad(o.ez + (FORCE ? fz : 0), k.l20, gz);
    long long bxy = be + X + Y, bxz = be + X + Z, q = 0;
    const long long byz = be + Y + Z;
    if (LID) {  // (Y - Z)(1 - 1/rho)/3, half of it on the edges
        const long long w = (1LL << 60) - fix_recip(o.r, o.rd);
        const long long qh = fix_mul<60>(fix_dig(fix_mad(Y - Z, k.sixth, 0)), fix_dig(w));
        q = 2 * qh;
        bxy += qh;
        bxz -= qh;
    }
    F[0] = 2 * fix_mad(F[0], k.c1, fix_mad(o.rd, k.l0, -2 * S)) + o.d19;
    fix_pair(F, 1, 2, k, b2 + 2 * X, gx + ox);
    fix_pair(F, 3, 4, k, b2 - q + 2 * Y, gy + oy);
    fix_pair(F, 5, 6, k, b2 + q + 2 * Z, gz + oz);
    fix_pair(F, 7, 10, k, bxy + cxy, ox + oy);
    fix_pair(F, 9, 8, k, bxy - cxy, ox - oy);
    fix_pair(F, 11, 14, k, bxz + cxz, ox + oz);
    fix_pair(F, 13, 12, k, bxz - cxz, ox - oz);
    fix_pair(F, 15, 18, k, byz + cyz, oy + oz);
    fix_pair(F, 17, 16, k, byz - cyz, oy - oz);
}

// The temperature part.  Its populations are of either sign, down to zero and of
// whatever scale the walls set, so each cell has units of its own: the largest of its
// seven populations lies in [2^(59 - head), 2^(60 - head)) units, smaller ones are
// rounded to a unit, at most 2^-57 of the largest, where FP64's own half ulp of it is
// 2^-54.  head leaves |T| below 2^61 (FixHeatK: from the equilibrium weights).  In fixed
// units of 2^-61 a temperature of 1e-6 was 5e4 times less accurate than in FP64, and
// walls of 1 and 0 put populations out of range.
struct HeatUnit {
    int top;  // exponent field of the largest population, plus head
};
// false: a population that is not finite, or all of them below 2^-959 but not zero
__device__ __forceinline__ bool fix_heat_unit(const double (&g)[Q7], const FixHeatK& k,
                                              HeatUnit& o) {
    unsigned worst = 0;
#pragma unroll
    for (int q = 0; q < Q7; q++) worst = max(worst, (unsigned)__double2hiint(g[q]) & 0x7fffffffu);
    o.top = (int)(worst >> 20) + k.head;
    if (worst < 64u << 20) {
        unsigned any = 0;
#pragma unroll
        for (int q = 0; q < Q7; q++)
            any |= (unsigned)__double2hiint(g[q]) << 1 | (unsigned)__double2loint(g[q]);
        o.top = 1023;
        return any == 0;
    }
    return worst < 2040u << 20;
}
// x in the cell's units, rounded to nearest
__device__ __forceinline__ long long fix_heat_load(double x, HeatUnit k) {
    const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
    const int s = min(k.top + 2 - (int)((hi >> 20) & 0x7ffu), 63);
    const unsigned long long m =
        ((unsigned long long)((hi & 0xFFFFFu) | 0x100000u) << 32 | lo) << 10;
    const long long v = (long long)(((m >> s) + 1) >> 1), sg = (int)hi >> 31;
    return (v ^ sg) - sg;
}
__device__ __forceinline__ double fix_heat_store(long long v, HeatUnit k) {
    const double b = (double)v;
    // units of 2^(top - 1082)
    return v ? __hiloint2double(__double2hiint(b) + (k.top - 1082) * (1 << 20), __double2loint(b)) : 0.0;
}
// D3Q7 collision (pair_collide_t) in place, |T| < 2^61 units
__device__ __forceinline__ void fix_heat(long long (&G)[Q7], long long T, const FixHeatK& k,
                                         const FixFlow& o) {
    const FixD t = fix_dig(T);
    const long long E = fix_mad(t, k.gE, 0);
    const FixD h = fix_dig(2 * fix_mad(t, k.hd, 0));
    G[0] = 2 * fix_mad(G[0], k.g1, 2 * fix_mad(t, k.c0, 0));
    const FixD u[3] = {o.ux, o.uy, o.uz};
#pragma unroll
    for (int a = 0; a < 3; a++) {
        const int q = 2 * a + 1;
        const long long p = fix_mad(G[q] + G[q + 1], k.g1, E);
        const long long m = fix_mad(G[q] - G[q + 1], k.g2, fix_mul<63>(h, u[a]));
        G[q] = p + m;
        G[q + 1] = p - m;
    }
}

}  // namespace mglc
