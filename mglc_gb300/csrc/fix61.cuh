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
// 2.1e-13 against 3.3e-13).  About a thousand integer instructions a lid cell:
// 384^3 in 3.31 ms a step (17.1 GLUPS, 77% of HBM) against 15.7 ms in FP64.
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
// the same for any v, on the FP64 unit
__device__ __forceinline__ double fix61_store_any(long long v) {
    const long long b = __double_as_longlong((double)v);
    return __longlong_as_double(v ? b - (61LL << 52) : 0LL);
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

// populations converted back on the FP64 unit (the others with integer
// operations), balancing the two
#ifndef FIX_CVT_OUT
#define FIX_CVT_OUT 10
#endif

__device__ __forceinline__ void fix_pair(long long* F, int a, int b, const FixK& k, long long E,
                                         long long O) {
    const long long p = fix_mad(F[a] + F[b], k.c1, E), m = fix_mad(F[a] - F[b], k.c2, O);
    F[a] = p + m;
    F[b] = p - m;
}

// integer populations to doubles; v below 2^-8 or negative (rare): the FP64 unit
__device__ __forceinline__ void fix61_store_all(const long long (&F)[Q19], double (&f)[Q19]) {
    int least = 0x7fffffff;
#pragma unroll
    for (int q = 0; q < Q19; q++) least = min(least, (int)(F[q] >> 32));
    if (least >= 0x200000) {
#pragma unroll
        for (int q = 0; q < Q19; q++)
            f[q] = q < FIX_CVT_OUT ? fix61_store_any(F[q]) : fix61_store(F[q]);
    } else {
#pragma unroll
        for (int q = 0; q < Q19; q++) f[q] = fix61_store_any(F[q]);
    }
}

// The lid collision (pair_collide_lid) in place of a cell's populations as
// integers; false, with nothing changed, when the density or the velocity is
// out of range.  rho: the density of the equilibrium.  FIRST (the step after
// initial or load): rho and u come from the macro arrays (rho0, u0, v0, w0),
// and the projections of the populations on the conserved density and momentum
// are taken back out (trt_collide_lid, CONS).
template <bool FIRST>
__device__ __forceinline__ bool fix61_collide_lid(long long (&F)[Q19], const FixK& k,
                                                  long long& rho, double rho0 = 0.0,
                                                  double u0 = 0.0, double v0 = 0.0,
                                                  double w0 = 0.0) {
    long long r, jx, jy, jz;
    moments0(F, r, jx, jy, jz);
    FixD rd, dx, dy, dz, di, ux, uy, uz;
    long long inv, hx = 0, hy = 0, hz = 0, d19 = 0;
    if (FIRST) {
        if (!(rho0 >= 0.25 && rho0 < 2.75 && fabs(u0) < 0.5 && fabs(v0) < 0.5 && fabs(w0) < 0.5))
            return false;
        const long long rf = r, ax = jx, ay = jy, az = jz;
        r = __double2ll_rn(rho0 * FIX_ONE);
        ux = fix_dig(__double2ll_rn(u0 * (4.0 * FIX_ONE)));
        uy = fix_dig(__double2ll_rn(v0 * (4.0 * FIX_ONE)));
        uz = fix_dig(__double2ll_rn(w0 * (4.0 * FIX_ONE)));
        rd = fix_dig(r);
        inv = fix_recip(r, rd);
        di = fix_dig(inv);
        jx = fix_mul<63>(rd, ux);
        jy = fix_mul<63>(rd, uy);
        jz = fix_mul<63>(rd, uz);
        dx = fix_dig(jx);
        dy = fix_dig(jy);
        dz = fix_dig(jz);
        d19 = fix_mad(rf - r, k.l19, 0);
        hx = fix_mad(ax - jx, k.l10, 0);
        hy = fix_mad(ay - jy, k.l10, 0);
        hz = fix_mad(az - jz, k.l10, 0);
    } else {
        const long long half = r >> 1;
        if (!(r >= (1LL << 59) && jx < half && -jx < half && jy < half && -jy < half &&
              jz < half && -jz < half))
            return false;
        rd = fix_dig(r);
        dx = fix_dig(jx);
        dy = fix_dig(jy);
        dz = fix_dig(jz);
        inv = fix_recip(r, rd);
        di = fix_dig(inv);
        // u in units of 2^-63
        ux = fix_dig(fix_mul<58>(dx, di));
        uy = fix_dig(fix_mul<58>(dy, di));
        uz = fix_dig(fix_mul<58>(dz, di));
    }
    rho = r;
    // Snu/8 rho u in units of 2^-62
    const FixD kx = fix_dig(fix_mad(dx, k.l8, 0)), ky = fix_dig(fix_mad(dy, k.l8, 0)),
               kz = fix_dig(fix_mad(dz, k.l8, 0));
    const long long X = fix_mul<64>(kx, ux), Y = fix_mul<64>(ky, uy), Z = fix_mul<64>(kz, uz);
    const long long cxy = 2 * fix_mul<64>(kx, uy), cxz = 2 * fix_mul<64>(kx, uz),
                    cyz = 2 * fix_mul<64>(ky, uz);
    // half the lid quirk's term, (Y - Z)(1 - 1/rho)/6
    const long long qh = fix_mul<60>(fix_dig(fix_mad(Y - Z, k.sixth, 0)), fix_dig((1LL << 60) - inv));
    const long long S = X + Y + Z;
    const long long b = fix_mad(rd, k.l18, fix_mad(S, k.third, 0)), b2 = 2 * b + d19, be = b + d19;
    const long long gx = fix_mad(dx, k.l6, 0), gy = fix_mad(dy, k.l6, 0), gz = fix_mad(dz, k.l6, 0);
    const long long ox = gx + hx, oy = gy + hy, oz = gz + hz;
    const long long q = 2 * qh;
    const long long bxy = be + qh + X + Y, bxz = be - qh + X + Z, byz = be + Y + Z;
    F[0] = 2 * fix_mad(F[0], k.c1, fix_mad(rd, k.l0, -2 * S)) + d19;
    fix_pair(F, 1, 2, k, b2 + 2 * X, gx + ox);
    fix_pair(F, 3, 4, k, b2 - q + 2 * Y, gy + oy);
    fix_pair(F, 5, 6, k, b2 + q + 2 * Z, gz + oz);
    fix_pair(F, 7, 10, k, bxy + cxy, ox + oy);
    fix_pair(F, 9, 8, k, bxy - cxy, ox - oy);
    fix_pair(F, 11, 14, k, bxz + cxz, ox + oz);
    fix_pair(F, 13, 12, k, bxz - cxz, ox - oz);
    fix_pair(F, 15, 18, k, byz + cyz, oy + oz);
    fix_pair(F, 17, 16, k, byz - cyz, oy - oz);
    return true;
}

}  // namespace mglc
