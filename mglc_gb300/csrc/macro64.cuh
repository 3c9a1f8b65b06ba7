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
//  * reduced forms: the stored deviations are summed in pairs of FP32 values
//    (Knuth's TwoSum), good to 2^-45 of the largest, below the rounding of the
//    FP64 sum with w rho0; scale and rho0 come in at the end.
//  * the three quotients by rho share one reciprocal (div_by).
#pragma once
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
__device__ __forceinline__ void macro_sums(const double (&f)[Q19], double& r, double& jx,
                                           double& jy, double& jz) {
    if (fix61_ok(f)) {
        long long R = 0, J[3] = {0, 0, 0};
#pragma unroll
        for (int q = 0; q < Q19; q++) {
            const long long F = fix61_load(f[q]);
            R = q ? rn53(R + F) : F;
            if (ex19(q)) J[0] = rn53(ex19(q) > 0 ? J[0] + F : J[0] - F);
            if (ey19(q)) J[1] = rn53(ey19(q) > 0 ? J[1] + F : J[1] - F);
            if (ez19(q)) J[2] = rn53(ez19(q) > 0 ? J[2] + F : J[2] - F);
        }
        r = fix61_store_any(R);
        jx = fix61_store_any(J[0]);
        jy = fix61_store_any(J[1]);
        jz = fix61_store_any(J[2]);
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
// the same sums of stored deviations f = (f_abs - w rho0) / inv (inv a power of
// two); not finite or huge: in FP64 as the populations would be
__device__ __forceinline__ void macro_sums(const float (&f)[Q19], float inv, double rho0,
                                           double& r, double& jx, double& jy, double& jz) {
    float h = f[0], l = 0.0f, H[3] = {f[1], f[3], f[5]}, L[3] = {0.0f, 0.0f, 0.0f};
#pragma unroll
    for (int q = 1; q < Q19; q++) {
        two_sum(h, l, f[q]);
        if (ex19(q) && q != 1) two_sum(H[0], L[0], ex19(q) > 0 ? f[q] : -f[q]);
        if (ey19(q) && q != 3) two_sum(H[1], L[1], ey19(q) > 0 ? f[q] : -f[q]);
        if (ez19(q) && q != 5) two_sum(H[2], L[2], ez19(q) > 0 ? f[q] : -f[q]);
    }
    const float big = fabsf(h) + fabsf(H[0]) + fabsf(H[1]) + fabsf(H[2]);
    if (big < 1e30f) {
        const double s = (double)inv;
        r = fma((double)h + (double)l, s, rho0);
        jx = ((double)H[0] + (double)L[0]) * s;
        jy = ((double)H[1] + (double)L[1]) * s;
        jz = ((double)H[2] + (double)L[2]) * s;
        return;
    }
    macro_sums_ordered(f, (double)inv, rho0, r, jx, jy, jz);
}

// a/r, b/r and c/r, correctly rounded (div_pair, d2q9.cuh)
__device__ __forceinline__ void div_by(double a, double b, double c, double r, double& qa,
                                       double& qb, double& qc) {
    if (den_ok(r) && mid_or_pzero(a) && mid_or_pzero(b) && mid_or_pzero(c)) {
        double y = (double)__frcp_rn((float)r);
        y = __fma_rn(__fma_rn(-r, y, 1.0), y, y);
        y = __fma_rn(__fma_rn(-r, y, 1.0), y, y);
        y = __fma_rn(__fma_rn(-r, y, 1.0), y, y);
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
