// macro64.cuh -- the FP64 density and momentum of a cell (macro.f90:6-25,
// bouyancy3d_mpi.F90:986-1010), for the getters' kernels.
//
// Those are bound by the FP64 pipe when every addition runs on it (FP64 storage:
// 45 additions and three divisions a cell; the reduced forms: 19 conversions and
// multiply-adds besides), two to four times the time of their memory traffic.
//  * FP64 storage: the fields are the reference's bit for bit, so each
//    addition has to round as FP64's; with the populations exact in units of
//    2^-61 (fix61.cuh) an addition is an integer one followed by the rounding
//    of the sum to 53 significant bits, to nearest even.
//  * reduced forms: the stored deviations, rho0 and half the force are summed in
//    units of 2^-60, exactly but for what lies below 2^-60 (the temperature
//    populations in units of their own scale), and the velocity is a product with the integer reciprocal,
//    to 2^-61: closer to the exact quotient of the stored values than the FP64
//    sums with w rho0, which round at 2^-54.  Four conversions a cell remain of
//    33 FP64 instructions.
//  * FP64 storage: the three quotients by rho share one reciprocal, taken from
//    integers where the density is one (div_by).
// FP16 256^3 1028 -> 479 us (174 are its bytes), FP32 97x63x129 60 -> 29, heated and
// rotating 81x97x72 67 -> 29.
#pragma once
#include <cmath>

#include "d2q9.cuh"
#include "fix61.cuh"

namespace mglc {

// sum f and sum f e in the order of the populations, in FP64
__device__ __forceinline__ void sums_fp64(const double (&f)[Q19], double& r, double& jx, double& jy,
                                          double& jz) {
    r = f[0];
#pragma unroll
    for (int q = 1; q < Q19; q++) r = __dadd_rn(r, f[q]);
    jx = f[1];
    jy = f[3];
    jz = f[5];
#pragma unroll
    for (int q = 2; q < Q19; q++) {
        if (ex19(q)) jx = __dadd_rn(jx, ex19(q) * f[q]);
        if (ey19(q) && q != 3) jy = __dadd_rn(jy, ey19(q) * f[q]);
        if (ez19(q) && q != 5) jz = __dadd_rn(jz, ez19(q) * f[q]);
    }
}

// sum f and sum f e in the order of the populations, each addition rounded as
// FP64 rounds it
// (R: the density times 2^61, 0 where the sums ran in FP64).  Z64: the z momentum on
// the FP64 unit, which the lid's kernel leaves idle otherwise (256^3 with a 134 MB
// copy: 800 us so, 918 all on integers, 850 with the quotients there instead; heated
// 128^3, with sums of its own: 145 without).
template <bool Z64>
__device__ __forceinline__ void macro_sums(const double (&f)[Q19], double& r, double& jx,
                                           double& jy, double& jz, long long& R) {
    R = 0;
    if (fix61_ok(f)) {
        long long J[3] = {0, 0, 0};
#pragma unroll
        for (int q = 0; q < Q19; q++) {
            const long long F = fix61_load(f[q]);
            R = q ? rn53_pos(R + F) : F;
            if (ex19(q)) J[0] = rn53(ex19(q) > 0 ? J[0] + F : J[0] - F);
            if (ey19(q)) J[1] = rn53(ey19(q) > 0 ? J[1] + F : J[1] - F);
            if (!Z64 && ez19(q)) J[2] = rn53(ez19(q) > 0 ? J[2] + F : J[2] - F);
        }
        r = fix_out<61>(R);
        jx = fix_out<61>(J[0]);
        jy = fix_out<61>(J[1]);
        if (Z64) {
            jz = f[5];
#pragma unroll
            for (int q = 6; q < Q19; q++)
                if (ez19(q)) jz = __dadd_rn(jz, ez19(q) * f[q]);
        } else {
            jz = fix_out<61>(J[2]);
        }
        return;
    }
    sums_fp64(f, r, jx, jy, jz);
}

// in the reference's order, from stored deviations f = (f_abs - w rho0) / inv
__device__ __forceinline__ void macro_sums_ordered(const float (&f)[Q19], double inv, double rho0,
                                                   double& r, double& jx, double& jy, double& jz) {
    double a[Q19];
#pragma unroll
    for (int q = 0; q < Q19; q++) a[q] = (double)f[q] * inv + w19(q) * rho0;
    sums_fp64(a, r, jx, jy, jz);
}

// h + x = h' + error, the error added to l
__device__ __forceinline__ void two_sum(float& h, float& l, float x) {
    const float s = h + x, b = s - h;
    l += (h - (s - b)) + (x - b);
    h = s;
}
// x 2^e2 in units of 2^-60, cut towards zero, for |x| 2^e2 < 2^(L - 127); `worst` takes
// the exponent field, above L - 1 where x is out of range (infinities and NaN too)
template <int L>
__device__ __forceinline__ long long fix60_load(float x, int e2, int& worst) {
    const int b = __float_as_int(x);
    const int e = ((b >> 23) & 0xff) + e2;
    // (a subnormal, taken for a normal of the least exponent, is below 2^-60 too)
    worst = max(worst, ((b >> 23) & 0xff) == 0xff ? 0x7fff : e);
    const unsigned m = ((unsigned)b & 0x7fffffu) | 0x800000u;
    // the significand at the place of exponent L - 1, then down
    constexpr int TOP = L - 1 - 150 + 60;
    const long long v = (long long)(((unsigned long long)m << TOP) >> min(max(L - 1 - e, 0), 63));
    const long long sg = b >> 31;
    return (v ^ sg) - sg;
}

// The sum of temperature populations of any scale: in units of 2^-60 of the power of two
// above the largest, so cut at 2^-59 of it or less (an FP64 sum rounds at 2^-53).  false:
// one is not finite, or all are below 2^-65 but not zero
__device__ __forceinline__ bool fix60_temperature(const float (&g)[Q7], double& t) {
    unsigned big = 0;
#pragma unroll
    for (int q = 0; q < Q7; q++) big = max(big, (unsigned)__float_as_int(g[q]) & 0x7fffffffu);
    const int e = (int)(big >> 23);
    int worst = 0;
    long long v = 0;
#pragma unroll
    for (int q = 0; q < Q7; q++) v += fix60_load<127>(g[q], 126 - e, worst);
    const double b = (double)v;
    t = v && big ? __hiloint2double(__double2hiint(b) + (e - 126 - 60) * (1 << 20), __double2loint(b))
                 : 0.0;
    return big == 0 || (e >= 62 && e < 255);
}

// Scale, rho0 and range of the reduced forms' sums; on: rho0 in [0, 4) and a
// power-of-two scale.
struct Fix60K {
    int on, e2;
    long long rho0;
};
inline Fix60K make_fix60(double rho0, double inv) {
    Fix60K k{};
    int e = 0;
    const bool pow2 = inv > 0.0 && std::frexp(inv, &e) == 0.5;
    k.on = pow2 && e > -60 && e < 60 && rho0 >= 0.0 && rho0 < 4.0;
    k.e2 = e - 1;
    if (k.on) k.rho0 = std::llrint(std::ldexp(rho0, 60));
    return k;
}

// rho and the momenta of stored deviations (units of 2^-60); false: a population of
// 1/8 or more (19 of them and rho0 stay below 8), or not finite
__device__ __forceinline__ bool fix60_sums(const float (&f)[Q19], const Fix60K& k, long long& r,
                                           long long (&j)[3]) {
    int worst = 0;
    r = k.rho0;
    j[0] = j[1] = j[2] = 0;
#pragma unroll
    for (int q = 0; q < Q19; q++) {
        const long long v = fix60_load<124>(f[q], k.e2, worst);
        r += v;
        if (ex19(q)) j[0] = ex19(q) > 0 ? j[0] + v : j[0] - v;
        if (ey19(q)) j[1] = ey19(q) > 0 ? j[1] + v : j[1] - v;
        if (ez19(q)) j[2] = ez19(q) > 0 ? j[2] + v : j[2] - v;
    }
    return k.on && worst < 124;
}
// rho (units of 2^-60) has an integer reciprocal and the momenta are below it
__device__ __forceinline__ bool fix60_flow(long long r, const long long (&j)[3]) {
    return r >= (1LL << 58) && r < (11LL << 58) && j[0] < r && -j[0] < r && j[1] < r && -j[1] < r &&
           j[2] < r && -j[2] < r;
}

// 1/r, correctly rounded, for r of significand not all ones (den_ok) and R = r 2^61 in
// [2^59, 11 2^59): the integer reciprocal, rounded, and one Newton step
__device__ __forceinline__ double recip_of(long long R, double r) {
    const double y = fix_out<60>(rn53(fix_recip(R, fix_dig(R))));
    return __fma_rn(__fma_rn(-r, y, 1.0), y, y);
}

// a/r, b/r and c/r, correctly rounded (div_pair, d2q9.cuh); R: r 2^61 where it is known
// as an integer, else 0
__device__ __forceinline__ void div_by(double a, double b, double c, double r, double& qa,
                                       double& qb, double& qc, long long R = 0) {
    if (den_ok(r) && mid_or_pzero(a) && mid_or_pzero(b) && mid_or_pzero(c)) {
        double y;
        if (R >= (1LL << 59) && R < (11LL << 59)) {
            y = recip_of(R, r);
        } else {
            y = (double)__frcp_rn((float)r);
            y = __fma_rn(__fma_rn(-r, y, 1.0), y, y);
            y = __fma_rn(__fma_rn(-r, y, 1.0), y, y);
            y = __fma_rn(__fma_rn(-r, y, 1.0), y, y);
        }
        const double ta = __dmul_rn(a, y), tb = __dmul_rn(b, y), tc = __dmul_rn(c, y);
        qa = __fma_rn(__fma_rn(-r, ta, a), y, ta);
        qb = __fma_rn(__fma_rn(-r, tb, b), y, tb);
        qc = __fma_rn(__fma_rn(-r, tc, c), y, tc);
    } else {
        qa = __ddiv_rn(a, r);
        qb = __ddiv_rn(b, r);
        qc = __ddiv_rn(c, r);
    }
}

}  // namespace mglc
