// k_aux.cu -- macroscopic fields, equilibrium initialisation, layout
// conversion between the reference's AoS arrays and the device SoA planes,
// and deterministic FP64 reductions (residual, totals).
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <type_traits>

#include "kernels.cuh"
#include "cell_map.cuh"
#include "launch.cuh"
#include "macro64.cuh"

namespace mglc {

template <typename S>
__device__ __forceinline__ double to_d(S v);
template <>
__device__ __forceinline__ double to_d<double>(double v) { return v; }
template <>
__device__ __forceinline__ double to_d<float>(float v) { return (double)v; }
template <>
__device__ __forceinline__ double to_d<__half>(__half v) { return (double)__half2float(v); }
template <>
__device__ __forceinline__ double to_d<__nv_bfloat16>(__nv_bfloat16 v) {
    return (double)__bfloat162float(v);
}
template <typename S>
__device__ __forceinline__ S from_d(double v);
template <>
__device__ __forceinline__ double from_d<double>(double v) { return v; }
template <>
__device__ __forceinline__ float from_d<float>(double v) { return (float)v; }
template <>
__device__ __forceinline__ __half from_d<__half>(double v) { return __float2half_rn((float)v); }
template <>
__device__ __forceinline__ __nv_bfloat16 from_d<__nv_bfloat16>(double v) {
    return __float2bfloat16_rn((float)v);
}

// ------------------------------------------------------------- macro() --
// Reference order: rho = sum over alpha from 0..18 sequentially, momentum in
// the order of the alpha loop (macro.f90:6-25 / bouyancy3d_mpi.F90:986-1010),
// with the thermal half-force shift; every operation rounds as IEEE FP64 does,
// so that for FP64 storage the fields equal the reference's.
// storage type of the temperature populations for a given f storage type
template <typename S> struct GType { using T = float; };
template <> struct GType<double> { using T = double; };

// stored population of a reduced form, in its arithmetic type
__device__ __forceinline__ float to_f(float v) { return v; }
__device__ __forceinline__ float to_f(__half v) { return __half2float(v); }
__device__ __forceinline__ float to_f(__nv_bfloat16 v) { return __bfloat162float(v); }

// macro64.cuh: 384^3 FP64 in 2.6 ms (its traffic is 1.5 ms of HBM), 11 ms with every
// addition on the FP64 pipe; 256^3 FP16 0.48 ms against 1.03
// ORDERED (reduced forms): every addition in FP64 and in the reference's order,
// for the fields that the first step after a load starts from (another rounding
// of them, however small, and the 16-bit stores round otherwise from there on)
template <typename S, bool THERMAL, bool ORDERED>
__global__ void __launch_bounds__(256) k_macro(const S* f,
                        const typename GType<S>::T* gt, const void* Fv,
                        Geom g, double rho0, double inv_scale, Fix60K fk, double* rho, double* u,
                        double* v, double* w, double* T) {
    after_previous();
    const long long n = g.plane;
    for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < n;
         c += (long long)gridDim.x * blockDim.x) {
        double r, jx, jy, jz;
        long long R = 0;
        if constexpr (std::is_same<S, double>::value) {
            double fq[Q19];
#pragma unroll
            for (int q = 0; q < Q19; q++) fq[q] = f[q * n + c];
            macro_sums<!THERMAL>(fq, r, jx, jy, jz, R);
        } else {
            float fq[Q19];
#pragma unroll
            for (int q = 0; q < Q19; q++) fq[q] = to_f(f[q * n + c]);
            if constexpr (!ORDERED) {
                float F[3] = {0.0f, 0.0f, 0.0f}, gq[Q7];
                if (THERMAL) {
#pragma unroll
                    for (int a = 0; a < 3; a++) F[a] = ((const float*)Fv)[a * n + c];
#pragma unroll
                    for (int q = 0; q < Q7; q++) gq[q] = gt[q * n + c];
                }
                long long r60, j[3];
                bool ok = fix60_sums(fq, fk, r60, j);
                double t = 0.0;
                if (THERMAL) {
                    int worst = 0;
#pragma unroll
                    for (int a = 0; a < 3; a++) j[a] += fix60_load<124>(F[a], -1, worst);
                    ok = fix60_temperature(gq, t) && ok && worst < 124;  // forces below 1/4
                }
                if (ok && fix60_flow(r60, j)) {
                    const FixD y = fix_dig(fix_recip(2 * r60, fix_dig(2 * r60)));
                    rho[c] = fix61_store_any<60>(r60);
                    u[c] = fix61_store_any<60>(fix_mul<60>(fix_dig(j[0]), y));
                    v[c] = fix61_store_any<60>(fix_mul<60>(fix_dig(j[1]), y));
                    w[c] = fix61_store_any<60>(fix_mul<60>(fix_dig(j[2]), y));
                    if (THERMAL) T[c] = t;
                    continue;
                }
            }
            macro_sums_ordered(fq, inv_scale, rho0, r, jx, jy, jz);
        }
        if (THERMAL) {
            double Fx, Fy, Fz;
            if (std::is_same<S, double>::value) {
                const double* F = (const double*)Fv;
                Fx = F[c]; Fy = F[n + c]; Fz = F[2 * n + c];
            } else {
                const float* F = (const float*)Fv;
                Fx = F[c]; Fy = F[n + c]; Fz = F[2 * n + c];
            }
            jx = __dadd_rn(jx, __dmul_rn(0.5, Fx));
            jy = __dadd_rn(jy, __dmul_rn(0.5, Fy));
            jz = __dadd_rn(jz, __dmul_rn(0.5, Fz));
            double t = (double)gt[c];
#pragma unroll
            for (int q = 1; q < Q7; q++) t = __dadd_rn(t, (double)gt[q * n + c]);
            T[c] = t;
        }
        rho[c] = r;
        double uu, vv, ww;
        div_by(jx, jy, jz, r, uu, vv, ww, R);
        u[c] = uu;
        v[c] = vv;
        w[c] = ww;
    }
}

static int grid_for(long long n, int block) {
    long long b = (n + block - 1) / block;
    if (b > 152 * 32) b = 152 * 32;
    if (b < 1) b = 1;
    return (int)b;
}

template <typename S>
static cudaError_t macro_go(bool thermal, const Geom& g, const void* f, const void* gt,
                            const void* F, double rho0, double inv, double* rho, double* u,
                            double* v, double* w, double* T, bool ordered, cudaStream_t s) {
    int gr = grid_for(g.plane, 256);
    using G = typename GType<S>::T;
    constexpr bool kRed = !std::is_same<S, double>::value;
    const Fix60K fk = make_fix60(rho0, inv);
    if (thermal && ordered && kRed)
        launch_next(k_macro<S, true, kRed>, gr, 256, 0, s, (const S*)f, (const G*)gt, F, g, rho0, inv, fk, rho, u, v, w, T);
    else if (thermal)
        launch_next(k_macro<S, true, false>, gr, 256, 0, s, (const S*)f, (const G*)gt, F, g, rho0, inv, fk, rho, u, v, w, T);
    else if (ordered && kRed)
        launch_next(k_macro<S, false, kRed>, gr, 256, 0, s, (const S*)f, nullptr, nullptr, g, rho0, inv, fk, rho, u, v, w, T);
    else
        launch_next(k_macro<S, false, false>, gr, 256, 0, s, (const S*)f, nullptr, nullptr, g, rho0, inv, fk, rho, u, v, w, T);
    return cudaGetLastError();
}

cudaError_t launch_macro(int form, bool thermal, const Geom& g, const void* f, const void* gt,
                         const void* F, double rho0, float inv_scale, double* rho, double* u,
                         double* v, double* w, double* T, bool ordered, cudaStream_t s) {
    switch (form) {
        case FORM_FP64: return macro_go<double>(thermal, g, f, gt, F, rho0, 1.0, rho, u, v, w, T, ordered, s);
        case FORM_FP32: return macro_go<float>(thermal, g, f, gt, F, rho0, 1.0, rho, u, v, w, T, ordered, s);
        case FORM_FP16: return macro_go<__half>(thermal, g, f, gt, F, rho0, inv_scale, rho, u, v, w, T, ordered, s);
        case FORM_BF16: return macro_go<__nv_bfloat16>(thermal, g, f, gt, F, rho0, 1.0, rho, u, v, w, T, ordered, s);
    }
    return cudaErrorInvalidValue;
}

// ------------------------------------------------------ equilibrium init --
// f = rho*omega*(1 + 3 un + 4.5 un^2 - 1.5 us2)   (initial.f90:67-72)
// g = omegaT*T*(1 + 21/(6+paraA) un)               (bouyancy3d_mpi.F90:586-589)
// IEEE-rounded operations in the reference's order (bit-equal for FP64).
template <typename S, bool THERMAL>
__global__ void k_equilibrium(Geom g, const double* rho, const double* u, const double* v,
                              const double* w, const double* T, double para_a, double rho0,
                              double scale, S* f, typename GType<S>::T* gt) {
    const long long n = g.plane;
    const bool shifted = !std::is_same<S, double>::value;
    for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < n;
         c += (long long)gridDim.x * blockDim.x) {
        const double uu = u[c], vv = v[c], ww = w[c], r = rho[c];
        const double us2 = __dadd_rn(__dadd_rn(__dmul_rn(uu, uu), __dmul_rn(vv, vv)), __dmul_rn(ww, ww));
#pragma unroll
        for (int q = 0; q < Q19; q++) {
            double un = __dadd_rn(__dadd_rn(__dmul_rn(uu, (double)ex19(q)), __dmul_rn(vv, (double)ey19(q))),
                                  __dmul_rn(ww, (double)ez19(q)));
            double poly = __dsub_rn(__dadd_rn(__dadd_rn(1.0, __dmul_rn(3.0, un)),
                                              __dmul_rn(__dmul_rn(4.5, un), un)),
                                    __dmul_rn(1.5, us2));
            double fe = __dmul_rn(__dmul_rn(r, w19(q)), poly);
            if (shifted) fe = (fe - w19(q) * rho0) * scale;
            f[q * n + c] = from_d<S>(fe);
        }
        if (THERMAL) {
            const double t = T[c];
            const double wt0 = (1.0 - para_a) / 7.0, wt = (para_a + 6.0) / 42.0;
            const double coef = 21.0 / (6.0 + para_a);
#pragma unroll
            for (int q = 0; q < Q7; q++) {
                double un = __dadd_rn(__dadd_rn(__dmul_rn(uu, (double)ex19(q)), __dmul_rn(vv, (double)ey19(q))),
                                      __dmul_rn(ww, (double)ez19(q)));
                double ge = __dmul_rn(__dmul_rn(q == 0 ? wt0 : wt, t), __dadd_rn(1.0, __dmul_rn(coef, un)));
                gt[q * n + c] = (typename GType<S>::T)ge;
            }
        }
    }
}

template <typename S>
static cudaError_t eq_go(bool thermal, const Geom& g, const double* rho, const double* u,
                         const double* v, const double* w, const double* T, double para_a,
                         double rho0, double scale, void* f, void* gt, cudaStream_t s) {
    int gr = grid_for(g.plane, 256);
    if (thermal)
        k_equilibrium<S, true><<<gr, 256, 0, s>>>(g, rho, u, v, w, T, para_a, rho0, scale, (S*)f,
                                                  (typename GType<S>::T*)gt);
    else
        k_equilibrium<S, false><<<gr, 256, 0, s>>>(g, rho, u, v, w, T, para_a, rho0, scale, (S*)f, nullptr);
    return cudaGetLastError();
}

cudaError_t launch_equilibrium(int form, bool thermal, const Geom& g, const double* rho,
                               const double* u, const double* v, const double* w,
                               const double* T, double para_a, double rho0, float scale, void* f,
                               void* gt, cudaStream_t s) {
    switch (form) {
        case FORM_FP64: return eq_go<double>(thermal, g, rho, u, v, w, T, para_a, rho0, 1.0, f, gt, s);
        case FORM_FP32: return eq_go<float>(thermal, g, rho, u, v, w, T, para_a, rho0, 1.0, f, gt, s);
        case FORM_FP16: return eq_go<__half>(thermal, g, rho, u, v, w, T, para_a, rho0, scale, f, gt, s);
        case FORM_BF16: return eq_go<__nv_bfloat16>(thermal, g, rho, u, v, w, T, para_a, rho0, 1.0, f, gt, s);
    }
    return cudaErrorInvalidValue;
}

// ------------------------------------------------------ layout conversion --
template <typename S>
__global__ void k_aos_to_soa(int Q, long long plane, long long cell0, long long ncells,
                             const double* __restrict__ aos, S* __restrict__ soa, double rho0,
                             double scale, bool shifted) {
    for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < ncells;
         c += (long long)gridDim.x * blockDim.x) {
        for (int q = 0; q < Q; q++) {
            double v = aos[(long long)Q * c + q];
            if (shifted) v = (v - w19(q) * rho0) * scale;
            soa[q * plane + cell0 + c] = from_d<S>(v);
        }
    }
}
template <typename S>
__global__ void k_soa_to_aos(int Q, long long plane, long long cell0, long long ncells,
                             const S* __restrict__ soa, double* __restrict__ aos, double rho0,
                             double inv_scale, bool shifted) {
    for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < ncells;
         c += (long long)gridDim.x * blockDim.x) {
        for (int q = 0; q < Q; q++) {
            double v = to_d<S>(soa[q * plane + cell0 + c]);
            if (shifted) v = v * inv_scale + w19(q) * rho0;
            aos[(long long)Q * c + q] = v;
        }
    }
}

cudaError_t launch_aos_to_soa(int form, int Q, const Geom& g, long long cell0, long long ncells,
                              const double* aos, void* soa, double rho0, float scale,
                              bool shifted, cudaStream_t s) {
    int gr = grid_for(ncells, 256);
    switch (form) {
        case FORM_FP64: k_aos_to_soa<double><<<gr, 256, 0, s>>>(Q, g.plane, cell0, ncells, aos, (double*)soa, rho0, 1.0, false); break;
        case FORM_FP32: k_aos_to_soa<float><<<gr, 256, 0, s>>>(Q, g.plane, cell0, ncells, aos, (float*)soa, rho0, 1.0, shifted); break;
        case FORM_FP16: k_aos_to_soa<__half><<<gr, 256, 0, s>>>(Q, g.plane, cell0, ncells, aos, (__half*)soa, rho0, scale, shifted); break;
        case FORM_BF16: k_aos_to_soa<__nv_bfloat16><<<gr, 256, 0, s>>>(Q, g.plane, cell0, ncells, aos, (__nv_bfloat16*)soa, rho0, 1.0, shifted); break;
        default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

cudaError_t launch_soa_to_aos(int form, int Q, const Geom& g, long long cell0, long long ncells,
                              const void* soa, double* aos, double rho0, float inv_scale,
                              bool shifted, cudaStream_t s) {
    int gr = grid_for(ncells, 256);
    switch (form) {
        case FORM_FP64: k_soa_to_aos<double><<<gr, 256, 0, s>>>(Q, g.plane, cell0, ncells, (const double*)soa, aos, rho0, 1.0, false); break;
        case FORM_FP32: k_soa_to_aos<float><<<gr, 256, 0, s>>>(Q, g.plane, cell0, ncells, (const float*)soa, aos, rho0, 1.0, shifted); break;
        case FORM_FP16: k_soa_to_aos<__half><<<gr, 256, 0, s>>>(Q, g.plane, cell0, ncells, (const __half*)soa, aos, rho0, inv_scale, shifted); break;
        case FORM_BF16: k_soa_to_aos<__nv_bfloat16><<<gr, 256, 0, s>>>(Q, g.plane, cell0, ncells, (const __nv_bfloat16*)soa, aos, rho0, 1.0, shifted); break;
        default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

// ------------------------------------------------------------ reductions --
constexpr int RED_BLOCK = 256;
constexpr int RED_MAX_BLOCKS = 152 * 8;

int reduce_blocks(long long n) {
    long long b = (n + RED_BLOCK - 1) / RED_BLOCK;
    if (b > RED_MAX_BLOCKS) b = RED_MAX_BLOCKS;
    if (b < 1) b = 1;
    return (int)b;
}

// block-wide sum of NV values, warp shuffles then shared memory; fixed order
// Each of the NV (3 or 4) sums by the pairwise tree over the lanes, then over the warps in
// order.  Over the first two levels a lane gives half of its values away and keeps the
// other half: six additions a warp instead of twenty, each of which holds the SM's
// FP64 unit for 16 clocks.
template <int NV>
__device__ __forceinline__ void block_sum(double (&v)[NV], double* out) {
    __shared__ double sh[RED_BLOCK / 32][NV];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    double x[4];
#pragma unroll
    for (int k = 0; k < 4; k++) x[k] = k < NV ? v[k] : 0.0;
#pragma unroll
    for (int n = 2, o = 16; n > 0; n >>= 1, o >>= 1) {
        const bool up = (lane & o) != 0;
#pragma unroll
        for (int i = 0; i < n; i++) {
            const double give = up ? x[i] : x[i + n];
            x[i] = (up ? x[i + n] : x[i]) + __shfl_xor_sync(0xffffffffu, give, o);
        }
    }
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) x[0] += __shfl_xor_sync(0xffffffffu, x[0], o);
    const int mine = ((lane >> 4) & 1) * 2 + ((lane >> 3) & 1);
    if ((lane & 7) == 0 && mine < NV) sh[wid][mine] = x[0];
    __syncthreads();
    if (threadIdx.x < NV) {
        double t = 0.0;
        for (int wv = 0; wv < RED_BLOCK / 32; wv++) t += sh[wv][threadIdx.x];
        out[threadIdx.x] = t;
    }
}

__global__ void __launch_bounds__(RED_BLOCK)
    k_residual(long long n, const double* u, const double* v, const double* w, const double* T,
               double* up, double* vp, double* wp, double* Tp, bool with_w, double* partials) {
    after_previous();
    double acc[4] = {0.0, 0.0, 0.0, 0.0};
    for (long long c = blockIdx.x * (long long)RED_BLOCK + threadIdx.x; c < n;
         c += (long long)gridDim.x * RED_BLOCK) {
        const double uu = u[c], vv = v[c], ww = w[c];
        const double a = uu - up[c], b = vv - vp[c], cw = ww - wp[c];
        acc[0] += a * a + b * b + (with_w ? cw * cw : 0.0);
        acc[1] += uu * uu + vv * vv + ww * ww;
        up[c] = uu;
        vp[c] = vv;
        wp[c] = ww;
        if (T) {
            const double t = T[c];
            acc[2] += fabs(t - Tp[c]);
            acc[3] += fabs(t);
            Tp[c] = t;
        }
    }
    block_sum<4>(acc, partials + 4 * blockIdx.x);
}

// one warp per value: each lane sums a strided subset in order, eight loads in
// flight, then a fixed tree (one warp for all, a load at a time: 16 us for 1216
// blocks)
template <int NV>
__global__ void k_finish(int nblocks, const double* partials, double* out) {
    after_previous();
    const int lane = threadIdx.x & 31, k = threadIdx.x >> 5;
    double acc = 0.0;
    for (int b0 = lane; b0 < nblocks; b0 += 8 * 32) {
        double x[8];
#pragma unroll
        for (int q = 0; q < 8; q++) x[q] = b0 + 32 * q < nblocks ? partials[NV * (b0 + 32 * q) + k] : 0.0;
#pragma unroll
        for (int q = 0; q < 8; q++)
            if (b0 + 32 * q < nblocks) acc += x[q];
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
    if (lane == 0) out[k] = acc;
}

cudaError_t launch_residual(long long n, const double* u, const double* v, const double* w,
                            const double* T, double* up, double* vp, double* wp, double* Tp,
                            bool with_w, double* partials, double* out4, cudaStream_t s) {
    int nb = reduce_blocks(n);
    launch_next(k_residual, nb, RED_BLOCK, 0, s, n, u, v, w, T, up, vp, wp, Tp, with_w, partials);
    launch_next(k_finish<4>, 1, 4 * 32, 0, s, nb, partials, out4);
    return cudaGetLastError();
}

__global__ void __launch_bounds__(RED_BLOCK)
    k_totals(long long n, const double* rho, const double* u, const double* v, const double* w,
             const double* T, double* partials) {
    after_previous();
    double acc[3] = {0.0, 0.0, 0.0};
    for (long long c = blockIdx.x * (long long)RED_BLOCK + threadIdx.x; c < n;
         c += (long long)gridDim.x * RED_BLOCK) {
        const double r = rho[c], uu = u[c], vv = v[c], ww = w[c];
        acc[0] += r;
        acc[1] += 0.5 * r * (uu * uu + vv * vv + ww * ww);
        if (T) acc[2] += T[c];
    }
    block_sum<3>(acc, partials + 3 * blockIdx.x);
}

cudaError_t launch_totals(long long n, const double* rho, const double* u, const double* v,
                          const double* w, const double* T, double* partials, double* out3,
                          cudaStream_t s) {
    int nb = reduce_blocks(n);
    launch_next(k_totals, nb, RED_BLOCK, 0, s, n, rho, u, v, w, T, partials);
    launch_next(k_finish<3>, 1, 3 * 32, 0, s, nb, partials, out3);
    return cudaGetLastError();
}

// calNuRe (mpi_blocked/RaNu.F90:13-47) sums plus the wall-gradient sums of the
// hot/cold wall Nusselt numbers.  The wall sits half a cell outside the first
// node, so dT/dn|wall = (9 T_1 - T_2 - 8 T_wall)/3 (second order).
__global__ void __launch_bounds__(RED_BLOCK)
    k_thermal_stats(Geom g, DivBy byx, DivBy byy, const double* u, const double* v, const double* w,
                    const double* T, int wall_axis, double* partials) {
    after_previous();
    double acc[4] = {0.0, 0.0, 0.0, 0.0};
    const long long n = g.plane;
    const long long sxy = (long long)g.nx * g.ny;
    const long long step = (long long)gridDim.x * RED_BLOCK;
    long long c = blockIdx.x * (long long)RED_BLOCK + threadIdx.x;
    double nu = 0.0, nv = 0.0, nw = 0.0, nt = 0.0;  // the next cell's, loaded ahead
    if (c < n) nu = u[c], nv = v[c], nw = w[c], nt = T[c];
    for (; c < n; c += step) {
        const double uu = nu, vv = nv, ww = nw, t = nt;
        if (c + step < n) nu = u[c + step], nv = v[c + step], nw = w[c + step], nt = T[c + step];
        acc[0] += ww * t;
        acc[1] += uu * uu + vv * vv + ww * ww;
        if (wall_axis == 1) {
            int j;  // by multiplication below 2^31 cells
            if (n < (1LL << 31)) {
                const unsigned row = byx((unsigned)c);
                j = (int)(row - byy(row) * (unsigned)g.ny);
            } else {
                j = (int)((c / g.nx) % g.ny);
            }
            if (j == 0) acc[2] += 9.0 * t - T[c + g.nx];
            if (j == g.ny - 1) acc[3] += 9.0 * t - T[c - g.nx];
        } else if (wall_axis == 2) {
            if (c < sxy) acc[2] += 9.0 * t - T[c + sxy];
            if (c >= n - sxy) acc[3] += 9.0 * t - T[c - sxy];
        }
    }
    block_sum<4>(acc, partials + 4 * blockIdx.x);
}

cudaError_t launch_thermal_stats(const Geom& g, const double* u, const double* v, const double* w,
                                 const double* T, int wall_axis, double* partials, double* out4,
                                 cudaStream_t s) {
    int nb = reduce_blocks(g.plane);
    launch_next(k_thermal_stats, nb, RED_BLOCK, 0, s, g, make_div(g.nx), make_div(g.ny), u, v, w, T, wall_axis, partials);
    launch_next(k_finish<4>, 1, 4 * 32, 0, s, nb, partials, out4);
    return cudaGetLastError();
}

}  // namespace mglc
