// k_particle.cu -- moving spheres in a D3Q19 channel (periodic x, no-slip y/z
// walls): the 3-D generalisation of the reference's Micro_particles step
// (MPI/Micro_particles/fortran/case4/mpi_particle, main.F90:35-73).
//
// Per time step:
//   k_pbulk     fluid cells: macro, forced MRT collision, push to the
//               neighbours (x wraps, y/z walls bounce back in place);
//               solid cells do nothing.  Block partials of sum rho and of
//               the post-collision mass feed the average density.
//   k_pfinish   fixed-order sums -> rho_avg (particle_bounceback.F90:15-35)
//   k_plinks    PART_NSLAB CTAs per particle: every fluid node x with a neighbour
//               x+e inside the particle is a boundary link.  The
//               post-collision values the quadratic interpolated bounce-back
//               needs (particle_bounceback.F90:65-75) are read from the
//               streamed array: fp(a,y) sits in f(a, y+e_a) after the push
//               (including solid destination cells, which only fluid pushes
//               write).  Writes f(abar,x) and accumulates the Wen 2014
//               momentum exchange (particle_force.F90:59-66)
//   k_pmark     springs, gravity and body force (:96-190), the particle's motion
//               (particle_update.F90:26-50) and the owner mask of its new
//               centre (:80-93), cleared by k_pbulk
//   k_pphase    density bookkeeping of nodes that change phase and the list of
//               nodes that left a particle
//   k_prefill   refill of those nodes (:134-193), two phases per particle (all
//               reads, then all writes), and the particle's new state.
// Six launches a step instead of twelve.
// Any kernel that detects a failure (no owner, q out of range, overlap, wall
// penetration) writes a status code; every kernel returns at once while the
// status is set, so the state freezes at the failing step and the host
// reports MGLC_ERR_PARTICLE.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <atomic>
#include <cmath>

#include "fix61.cuh"
#include "launch.cuh"
#include "macro64.cuh"
#include "particles.cuh"

namespace mglc {

constexpr int PB = 256;             // threads of the per-particle kernels
constexpr int NSLAB = PART_NSLAB;   // CTAs per particle in k_plinks

template <typename S>
struct PSt;
template <>
struct PSt<double> {
    static constexpr bool SHIFT = false;
    __device__ static double ld(const double* p) { return *p; }
    __device__ static void st(double* p, double v) { *p = v; }
};
template <>
struct PSt<float> {
    static constexpr bool SHIFT = true;
    __device__ static double ld(const float* p) { return (double)*p; }
    __device__ static void st(float* p, double v) { *p = (float)v; }
};

// absolute population value (FP64) of a stored slot
template <typename S>
__device__ __forceinline__ double pabs(const S* f, long long idx, int q, double rho0) {
    double v = PSt<S>::ld(f + idx);
    return PSt<S>::SHIFT ? v + w19(q) * rho0 : v;
}
template <typename S>
__device__ __forceinline__ void pset(S* f, long long idx, int q, double v, double rho0) {
    PSt<S>::st(f + idx, PSt<S>::SHIFT ? v - w19(q) * rho0 : v);
}

// Signed x separation with the nearest periodic image.  Centres stay in
// [0.5, nx + 0.5) and nodes in [1, nx], so one shift by L brings d into
// [-L/2, L/2]; a larger |d| (a centre that jumped, which k_pmark reports)
// takes the closed form d - L rint(d/L).  A non-finite d is returned as is:
// no loop depends on it.
__device__ __forceinline__ double dxp(double a, double b, const PartParams& p) {
    double d = a - b;
    if (p.periodic_x && isfinite(d)) {
        const double L = (double)p.nx, h = 0.5 * L;
        if (d > h) d -= L;
        else if (d < -h) d += L;
        if (d > h || d < -h) d -= L * rint(d / L);
    }
    return d;
}
// ((x-xc)^2 + (y-yc)^2 + (z-zc)^2) <= R^2 with IEEE-rounded operations
__device__ __forceinline__ bool inside(double x, double y, double z, const double* X, double R,
                                       const PartParams& p) {
    const double a = dxp(x, X[0], p), b = y - X[1], c = z - X[2];
    double d = __dadd_rn(__dadd_rn(__dmul_rn(a, a), __dmul_rn(b, b)), __dmul_rn(c, c));
    return d <= __dmul_rn(R, R);
}
__device__ __forceinline__ int wrapx(int i, int nx) { return i < 0 ? i + nx : (i >= nx ? i - nx : i); }

// par: which owner buffer holds the mask that the state is frozen with (before
// the particles move this step's, in the refill the new one)
__device__ __forceinline__ void pfail(const PartDev& d, int code, int c, int other, int par) {
    if (atomicCAS(d.status, 0, code) == 0) {
        d.status[1] = c;
        d.status[2] = other;
        d.status[3] = par;
    }
}

// Has a step failed?  One answer for the whole block, so that it leaves together:
// other blocks of the same launch may be setting the status, and warps that read it
// late would leave the others to barriers and shared values that they never wrote.
__device__ __forceinline__ bool stopped(const PartDev& d) { return __syncthreads_or(d.status[0]); }

template <int NV>
__device__ __forceinline__ void block_sum_to(double (&v)[NV], double* out, int stride) {
    __shared__ double sh[32][NV];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
#pragma unroll
    for (int k = 0; k < NV; k++)
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v[k] += __shfl_down_sync(0xffffffffu, v[k], o);
    if (lane == 0)
#pragma unroll
        for (int k = 0; k < NV; k++) sh[wid][k] = v[k];
    __syncthreads();
    if (threadIdx.x == 0)
        for (int k = 0; k < NV; k++) {
            double t = 0.0;
            for (int q = 0; q < nw; q++) t += sh[q][k];
            out[k * stride] = t;
        }
    __syncthreads();
}

// ------------------------------------------------------------- bulk step --
// compute type: FP64 for FP64 storage; FP32 (on deviations f - w rho0) for
// FP32 storage
template <typename S> struct PC { using C = double; };
template <> struct PC<float> { using C = float; };

// per-step constants of the bulk kernel in its arithmetic type (converted
// once on the host: double -> float conversions are slow on the device)
template <typename C> struct PBulkK {
    C rho0, ax, ay, az;
    MrtCoef<C> cd;
};
static PBulkK<float> bulk_k(const PartParams& p, float) {
    return {(float)p.rho0, (float)p.body_force[0], (float)p.body_force[1], (float)p.body_force[2],
            cast_coef<float>(make_mrt_coef(p.snu, p.sq))};
}
static PBulkK<double> bulk_k(const PartParams& p, double) {
    return {p.rho0, p.body_force[0], p.body_force[1], p.body_force[2], make_mrt_coef(p.snu, p.sq)};
}

// The fluid collision of one cell: f in place; rho_m the density as stored
// (less rho0 for deviations).
template <bool FIRST>
__device__ __forceinline__ void pcollide(float (&f)[Q19], const PBulkK<float>& k, float& rho_m) {
    float rho, ux, uy, uz;
    if (FIRST) {  // the reference's initial fields: rho0, u = 0
        rho = k.rho0;
        rho_m = 0.0f;
        ux = uy = uz = 0.0f;
    } else {
        float jx, jy, jz;
        moments0(f, rho_m, jx, jy, jz);
        rho = k.rho0 + rho_m;
        // u = (sum f e + F/2)/rho with F = rho*a (thermal macro form)
        const float inv = __frcp_rn(rho);
        ux = (jx + 0.5f * (rho * k.ax)) * inv;
        uy = (jy + 0.5f * (rho * k.ay)) * inv;
        uz = (jz + 0.5f * (rho * k.az)) * inv;
    }
    mrt_collide<float, true, false>(f, rho_m, rho, ux, uy, uz, rho * k.ax, rho * k.ay, rho * k.az,
                                    k.cd);
}
// The FP64 form's torques nearly cancel, so the rounding of every population
// shows in them and the collision keeps the operations of the moment form.  It
// is bound by the FP64 pipe (a warp's instruction holds the unit for 16 clocks),
// while nine tenths of the issue slots are empty; so the additions of the
// forward transform, a third of its operations, run on integers: populations in
// [2^-6, 1/2) are exact in units of 2^-58, and an integer addition followed by
// rounding to 53 significant bits (rn53) is the FP64 addition bit for bit.
struct Fix58 {
    long long v;
};
__device__ __forceinline__ Fix58 operator+(Fix58 a, Fix58 b) { return {rn53(a.v + b.v)}; }
__device__ __forceinline__ Fix58 operator-(Fix58 a, Fix58 b) { return {rn53(a.v - b.v)}; }
__device__ __forceinline__ bool fix58_ok(const double (&f)[Q19]) {
    unsigned worst = 0;
#pragma unroll
    for (int q = 1; q < Q19; q++)
        worst = max(worst, (unsigned)__double2hiint(f[q]) - 0x3F900000u);  // 2^-6
    return worst < 0x00300000u &&                                          // below 2^-3
           (unsigned)__double2hiint(f[0]) - 0x3F900000u < 0x00500000u;     // below 1/2
}
__device__ __forceinline__ void fix58_moments(const double (&f)[Q19], MrtMom<double>& o,
                                              double& rho, double& jx, double& jy, double& jz,
                                              long long& R) {
    Fix58 F[Q19];
#pragma unroll
    for (int q = 0; q < Q19; q++) F[q].v = fix61_load(f[q]) >> 3;  // exact
    Fix58 r, x, y, z;
    moments0(F, r, x, y, z);
    const Fix58 s1 = F[1] + F[2], d1 = F[1] - F[2], s2 = F[3] + F[4], d2 = F[3] - F[4];
    const Fix58 s3 = F[5] + F[6], d3 = F[5] - F[6], s4 = F[7] + F[10], d4 = F[7] - F[10];
    const Fix58 s5 = F[9] + F[8], d5 = F[9] - F[8], s6 = F[11] + F[14], d6 = F[11] - F[14];
    const Fix58 s7 = F[13] + F[12], d7 = F[13] - F[12], s8 = F[15] + F[18], d8 = F[15] - F[18];
    const Fix58 s9 = F[17] + F[16], d9 = F[17] - F[16];
    const Fix58 sa = s1 + s2 + s3, se = (s4 + s5) + (s6 + s7) + (s8 + s9);
    // the roundings of mrt_energy; the other products of mrt_moments are by powers of
    // two, exact, so that fused or not each sum rounds once
    o.m1 = fix_out<58>(rn53(-30 * F[0].v + rn53(8 * se.v + rn53(-11 * sa.v))));
    o.m2 = fix_out<58>(rn53(12 * F[0].v + rn53(-4 * sa.v + se.v)));
    const Fix58 a45 = d4 + d5, b45 = d4 - d5, a67 = d6 + d7, b67 = d6 - d7, a89 = d8 + d9,
                b89 = d8 - d9;
    o.m4 = fix_out<58>(rn53(-4 * d1.v + (a45 + a67).v));
    o.m6 = fix_out<58>(rn53(-4 * d2.v + (b45 + a89).v));
    o.m8 = fix_out<58>(rn53(-4 * d3.v + (b67 + b89).v));
    const Fix58 sxy = s4 + s5, sxz = s6 + s7, syz = s8 + s9, s23 = s2 + s3, t23 = s2 - s3;
    const Fix58 sp = sxy + sxz, sm = sxy - sxz;
    o.m9 = fix_out<58>(rn53((Fix58{rn53(2 * s1.v - s23.v)} + sp).v - 2 * syz.v));
    o.m10 = fix_out<58>(rn53((Fix58{rn53(-4 * s1.v + 2 * s23.v)} + sp).v - 2 * syz.v));
    o.m11 = fix_out<58>((t23 + sm).v);
    o.m12 = fix_out<58>(rn53(-2 * t23.v + sm.v));
    o.m13 = fix_out<58>((s4 - s5).v);
    o.m14 = fix_out<58>((s8 - s9).v);
    o.m15 = fix_out<58>((s6 - s7).v);
    o.m16 = fix_out<58>((a45 - a67).v);
    o.m17 = fix_out<58>(rn53(-b45.v + a89.v));
    o.m18 = fix_out<58>((b67 - b89).v);
    rho = fix_out<58>(r.v);
    R = r.v < (11LL << 56) ? r.v << 3 : 0;  // in units of 2^-61
    jx = fix_out<58>(x.v);
    jy = fix_out<58>(y.v);
    jz = fix_out<58>(z.v);
}
template <bool FIRST>
__device__ __forceinline__ void pcollide(double (&f)[Q19], const PBulkK<double>& k, double& rho) {
    double ux = 0.0, uy = 0.0, uz = 0.0;
    MrtMom<double> m;
    if (FIRST) {
        rho = k.rho0;
        m = mrt_moments(f);
    } else {
        double jx, jy, jz;
        long long R = 0;
        if (fix58_ok(f)) {
            fix58_moments(f, m, rho, jx, jy, jz, R);
        } else {
            moments0(f, rho, jx, jy, jz);
            m = mrt_moments(f);
        }
        // u = (sum f e + F/2)/rho with F = rho*a (thermal macro form)
        div_by(jx + 0.5 * (rho * k.ax), jy + 0.5 * (rho * k.ay), jz + 0.5 * (rho * k.az), rho, ux,
               uy, uz, R);
    }
    mrt_relax<double, true, false>(f, m, rho, rho, ux, uy, uz, rho * k.ax, rho * k.ay, rho * k.az,
                                   k.cd);
}

// The mass of the collided populations, added in their order.  FP64: where they are
// exact in units of 2^-61, integer additions rounded as FP64 rounds, bit for bit (the
// unit that the collision waits for stays free: 18 additions a cell on it against
// none).  The density before the collision is not that mass: the first step's
// density is rho0, whatever the populations are.
__device__ __forceinline__ float pmass(const float (&f)[Q19]) {
    float m = 0.0f;
#pragma unroll
    for (int q = 0; q < Q19; q++) m += f[q];
    return m;
}
__device__ __forceinline__ double pmass(const double (&f)[Q19]) {
    if (fix61_ok(f)) {
        long long R = fix61_load(f[0]);
#pragma unroll
        for (int q = 1; q < Q19; q++) R = rn53_pos(R + fix61_load(f[q]));
        return fix_out<61>(R);
    }
    double m = f[0];
#pragma unroll
    for (int q = 1; q < Q19; q++) m = __dadd_rn(m, f[q]);
    return m;
}

// One thread per node of an x-row segment.  Fluid nodes collide and push
// their populations (walls at y, z and, unless periodic, x bounce them back in
// place); solid nodes do nothing.  Each warp writes its partial sums of the
// fluid density before collision and of the post-collision mass to its own
// slot, so no block barrier is needed and the totals are added in a fixed
// order by k_pfinish.  The FP32 form writes its two FP32 sums and its count of
// fluid nodes and leaves FP64 to k_pfinish (a warp's FP64 instruction holds the
// unit for 16 clocks, and there were seven for every 32 cells).
// The owner mask that the next positions will be marked in is cleared on the
// way.
// resident 128-thread blocks per SM the bulk kernel holds its registers to
#ifndef MGLC_PBULK_MINB
#define MGLC_PBULK_MINB 8
#endif
#ifndef MGLC_PBULK_MINB64
#define MGLC_PBULK_MINB64 4
#endif
template <typename S, bool FIRST, typename IDX>
__global__ void __launch_bounds__(128, (sizeof(S) == 4 ? MGLC_PBULK_MINB : MGLC_PBULK_MINB64))
    k_pbulk(const S* fin, S* __restrict__ fout, const int* owner,
            int* __restrict__ owner_new, PartParams p, PBulkK<typename PC<S>::C> bk,
            double* partials, const int* status) {
    after_previous();
    using C = typename PC<S>::C;
    if (status[0]) return;
    const int nx = p.nx, ny = p.ny, nz = p.nz;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y, k = blockIdx.z;
    const IDX P = (IDX)nx * ny * nz;
    C cacc[2] = {C(0), C(0)};  // per-cell sums, added over the warp in the arithmetic type
    const bool active = i < nx;
    const IDX cell = (IDX)i + (IDX)nx * ((IDX)j + (IDX)ny * k);
    // the populations are loaded before the mask answers (solid cells read
    // in-bounds values they do not use), so both loads are in flight together
    C f[Q19];
    if (active) {
#pragma unroll
        for (int q = 0; q < Q19; q++) f[q] = (C)fin[q * P + cell];
    }
    const bool fluid = active && owner[cell] < 0;
    if (active) owner_new[cell] = -1;
    if (fluid) {
        pcollide<FIRST>(f, bk, cacc[0]);
        cacc[1] = pmass(f);
        const IDX sy = nx, sz = (IDX)nx * ny;
        // asked of the warp's fluid nodes together: apart, a row's two end warps
        // would store twice
        const bool edge = i == 0 || i == nx - 1 || j == 0 || j == ny - 1 || k == 0 || k == nz - 1;
        if (!__any_sync(__activemask(), edge)) {
            // every population streams, no wrap
#pragma unroll
            for (int q = 0; q < Q19; q++)
                fout[q * P + cell + (IDX)ex19(q) + (IDX)ey19(q) * sy + (IDX)ez19(q) * sz] = (S)f[q];
        } else {
#pragma unroll
            for (int q = 0; q < Q19; q++) {
                const int dx = ex19(q), dy = ey19(q), dz = ez19(q);
                const int jj = j + dy, kk = k + dz, ir = i + dx;
                const bool xwall = !p.periodic_x && (ir < 0 || ir >= nx);
                const bool wall = xwall || jj < 0 || jj >= ny || kk < 0 || kk >= nz;
                // no-slip wall: back into the node's opposite slot
                const IDX to = wall ? opp19(q) * P + cell
                                    : q * P + ((IDX)wrapx(ir, nx) + sy * jj + sz * kk);
                fout[to] = (S)f[q];
            }
        }
    }
    // both sums by the pairwise tree over the lanes, five additions for the two: the lower
    // half of the warp keeps the first, the upper half the second (FP64 128x64x64 277 us a
    // step; 283 with ten additions)
    const bool up = (threadIdx.x & 16) != 0;
    C acc = up ? cacc[1] : cacc[0];
    acc += __shfl_xor_sync(0xffffffffu, up ? cacc[0] : cacc[1], 16);
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    // fluid cells of this warp (deviation storage adds rho0 for each of them)
    const unsigned fl = __ballot_sync(0xffffffffu, fluid);
    if ((threadIdx.x & 15) == 0) {  // the first lane of either half
        const int nw = blockDim.x >> 5;
        const int b = blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * blockIdx.z);
        const int slot = b * nw + (threadIdx.x >> 5);
        const int nslot = gridDim.x * gridDim.y * gridDim.z * nw;
        if constexpr (sizeof(C) == 4) {
            ((float*)partials)[2 * slot + up] = acc;
            if (!up) ((int*)(partials + nslot))[slot] = __popc(fl);
        } else {
            partials[(up ? nslot : 0) + slot] = acc;
        }
    }
}

// blocks: the FP64 form's torques nearly cancel and show the rounding of the
// average, so its ranges stay 32 (7 us for 16384 partials); the FP32 form, whose
// partials are eight times as many in the channel, spreads over the SMs
template <typename S>
constexpr int FINISH_BLOCKS = PSt<S>::SHIFT ? 128 : 32;

// rho_avg at bounce-back and the post-collision mass from the bulk partials:
// FINISH_BLOCKS contiguous ranges; the last block to finish adds their sums by
// a fixed shuffle tree (as two launches: 14 + 4 us)
template <typename S>
__global__ void __launch_bounds__(256) k_pfinish(PartDev d, int nblocks, double rho0) {
    after_previous();
    if (stopped(d)) return;
    __shared__ int last;
    constexpr int NB = FINISH_BLOCKS<S>;
    const int per = (nblocks + NB - 1) / NB;
    const int b0 = blockIdx.x * per, b1 = min(nblocks, b0 + per);
    double* part = d.partials + 2 * (size_t)nblocks;
    double acc[2] = {0.0, 0.0};
#pragma unroll 4
    for (int b = b0 + threadIdx.x; b < b1; b += blockDim.x) {
        if constexpr (PSt<S>::SHIFT) {
            const float2 v = ((const float2*)d.partials)[b];
            const double nf = (double)((const int*)(d.partials + nblocks))[b] * rho0;
            acc[0] += (double)v.x + nf;
            acc[1] += (double)v.y + nf;
        } else {
            acc[0] += d.partials[b];
            acc[1] += d.partials[nblocks + b];
        }
    }
    __shared__ double out[2];
    block_sum_to<2>(acc, out, 1);
    if (threadIdx.x == 0) {
        part[blockIdx.x] = out[0];
        part[NB + blockIdx.x] = out[1];
        __threadfence();
        last = atomicAdd(d.done, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last || threadIdx.x >= 32) return;
    __threadfence();
    double a0 = 0.0, a1 = 0.0;
#pragma unroll
    for (int q = 0; q < NB; q += 32) {
        a0 += __ldcg(part + q + threadIdx.x);
        a1 += __ldcg(part + NB + q + threadIdx.x);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        a0 += __shfl_down_sync(0xffffffffu, a0, o);
        a1 += __shfl_down_sync(0xffffffffu, a1, o);
    }
    if (threadIdx.x == 0) {
        d.rho_avg[0] = a0 / (double)d.n_fluid[0];
        d.rho_avg[2] = a1;
        *d.done = 0;
    }
}
// --------------------------------------------------- boundary links (IBB) --
// Deviation f - w rho0 of the post-collision value fp(q, c) of node c
// (coordinates as 0-based indices), read from the streamed array; nodes
// outside the walls hold the reference's ghost value omega*rho0 (deviation 0).
// L: arithmetic type of the population work (FP64 for FP64 storage, FP32 for
// FP32 storage).
template <typename S, typename L>
__device__ __forceinline__ L fp_dev(const S* f, int q, int i, int j, int k, const PartParams& p) {
    const int nx = p.nx, ny = p.ny, nz = p.nz;
    if (j < 0 || j >= ny || k < 0 || k >= nz) return L(0);
    if (!p.periodic_x && (i < 0 || i >= nx)) return L(0);
    const long long P = (long long)nx * ny * nz;
    i = wrapx(i, nx);
    const int jj = j + ey19(q), kk = k + ez19(q), ir = i + ex19(q);
    long long idx;
    int qq = q;
    if (jj < 0 || jj >= ny || kk < 0 || kk >= nz || (!p.periodic_x && (ir < 0 || ir >= nx))) {
        qq = opp19(q);  // bounced back into slot opp(q) of c (w_q = w_opp(q))
        idx = qq * P + (i + (long long)nx * (j + (long long)ny * k));
    } else {
        idx = q * P + (wrapx(ir, nx) + (long long)nx * (jj + (long long)ny * kk));
    }
    if (PSt<S>::SHIFT) return (L)f[idx];
    return (L)((double)f[idx] - w19(qq) * p.rho0);
}

// Direction components for a direction index held in a register: 2-bit
// fields (component + 1) of one 64-bit constant per axis, so no compare chain.
__host__ __device__ constexpr unsigned long long pack_e(int axis) {
    unsigned long long v = 0;
    for (int a = 0; a < Q19; a++) {
        const int e = axis == 0 ? ex19(a) : (axis == 1 ? ey19(a) : ez19(a));
        v |= (unsigned long long)(e + 1) << (2 * a);
    }
    return v;
}
__device__ __forceinline__ int e_rt(unsigned long long pack, int a) {
    return (int)((pack >> (2 * a)) & 3ull) - 1;
}
constexpr unsigned long long EX_PACK = pack_e(0), EY_PACK = pack_e(1), EZ_PACK = pack_e(2);
__host__ __device__ constexpr int opp_rt(int a) {
    // 1<->2, 3<->4, 5<->6; 7<->10, 8<->9, 11<->14, 12<->13, 15<->18, 16<->17
    return a <= 6 ? (a & 1 ? a + 1 : a - 1) : ((a - 7) & 3) == 0 ? a + 3 : ((a - 7) & 3) == 3 ? a - 3
                                            : ((a - 7) & 3) == 1 ? a + 1 : a - 1;
}

constexpr bool opp_rt_ok() {
    for (int a = 1; a < Q19; a++)
        if (opp_rt(a) != opp19(a)) return false;
    return true;
}
static_assert(opp_rt_ok(), "opp_rt must match opp19");

// largest owner tile k_plinks stages in dynamic shared memory (beside its
// ~38 KB of static shared memory); bigger spheres read the mask from global
constexpr size_t TILE_MAX_BYTES = 160 * 1024;

// Link-list capacity of k_plinks: one scan round adds at most PB * 18 links,
// so the list is processed as soon as fewer than that many slots are free.
constexpr int LINK_CAP = PB * 27;
// Nodes that a list spans at most: an entry is the node's distance from the list's first
// scan round, and its direction, in 31 bits (a slab has 2^26 nodes from radius 320).
constexpr int LINK_SPAN = 1 << 26;

// Is node (i, j, k) (0-based, x unwrapped) a fluid node, or a ghost beyond a
// wall?  Only those have a post-collision value of this step.
__device__ __forceinline__ bool node_avail(int i, int j, int k, const PartParams& p,
                                           const int* owner) {
    if (j < 0 || j >= p.ny || k < 0 || k >= p.nz) return true;
    if (i < 0 || i >= p.nx) {
        if (!p.periodic_x) return true;
        i = wrapx(i, p.nx);
    }
    return owner[i + (long long)p.nx * (j + (long long)p.ny * k)] < 0;
}

// The interpolation weights of the quadratic bounce-back sum to one, so it is
// applied to deviations directly.  The momentum exchange of a link,
//   (e - u_w) fp - (-e - u_w) f_new = 2 e w rho0 + (e - u_w) dfp + (e + u_w) df_new,
// splits into a constant part and a small variable part.  The constant parts
// are summed exactly as integers: with m = 2 (axis links, w = 1/18) or 1
// (diagonal links, w = 1/36),
//   sum 2 e w rho0        = rho0/18 * sum m e
//   sum r x (2 e w rho0)  = rho0/18 * (sum m n x e - X x sum m e)
// because r = o + q e gives r x e = o x e, and o = n - X with n the node's
// (unwrapped) coordinates.  The variable parts use the population arithmetic
// type; q (calQ2) is computed in FP64 for the FP64 form and, from the FP64
// |x - X|^2 - R^2, in FP32 for the FP32 form.
// TILE: the owner ids of the slab's box plus a one-node halo are staged in
// dynamic shared memory (walls and, without periodicity, the x faces as -2),
// so the scan's 19 lookups per node stay on chip.
// FP64 instructions are what the FP32 form spends its time on if they are left
// in (each holds the SM's unit for 16 clocks or more, whatever lanes are
// active), so: the centre's conversions are one warp's; the node's distance to
// the surface is an exact fixed-point one; the few links that need an FP64 root
// are collected and take it together; the slab's sums are integers and triples
// of FP32 values (Sum3).  A link's values and masks are loaded before any is used
// (one latency a link instead of three), after the roots, so that the warps need
// no barrier between their links.  200 spheres of radius 5, FP32: 95 -> 48 us
// (1.3 waves of blocks, a quarter of the issue slots waiting at barriers);
// blocks of 128 threads, one wave: 69 us.  24 spheres, FP64: 59 -> 46 us, the
// FP64 unit of the 96 SMs that have a block.
// A sum of FP32 values as three of them, errors kept by TwoSum: good to about 2^-70 of
// the largest partial sum (FP64: 2^-53).
struct Sum3 {
    float h, m, l;
    __device__ __forceinline__ Sum3 from_lane(int o) const {  // the one of lane ^ o
        return {__shfl_xor_sync(0xffffffffu, h, o), __shfl_xor_sync(0xffffffffu, m, o),
                __shfl_xor_sync(0xffffffffu, l, o)};
    }
    __device__ __forceinline__ void operator+=(Sum3 x) {
        float e1 = 0.0f, e2 = 0.0f;
        two_sum(h, e1, x.h);
        two_sum(m, e2, x.m);
        two_sum(m, e2, e1);
        l += x.l + e2;
    }
};
struct Sum64 {
    double h;
    __device__ __forceinline__ Sum64 from_lane(int o) const { return {__shfl_xor_sync(0xffffffffu, h, o)}; }
    __device__ __forceinline__ void operator+=(Sum64 x) { h += x.h; }
};
// Eight sums over the warp, each by the pairwise tree over the lanes' bits 4 to 0: at the
// first three levels a lane gives half of its values away and keeps the other half,
// nine additions instead of forty.  Lane l ends with sum 4 b4 + 2 b3 + b2 of its bits.
template <class T>
__device__ __forceinline__ T warp_sum8(T (&v)[8], int lane) {
#pragma unroll
    for (int n = 4, o = 16; n > 0; n >>= 1, o >>= 1) {
        const bool up = (lane & o) != 0;
#pragma unroll
        for (int i = 0; i < n; i++) {
            const T give = up ? v[i] : v[i + n];
            T keep = up ? v[i + n] : v[i];
            keep += give.from_lane(o);
            v[i] = keep;
        }
    }
    v[0] += v[0].from_lane(2);
    v[0] += v[0].from_lane(1);
    return v[0];
}

// The exact sum over the warp of integers of 32 bits, from their halves.  A slab's torque
// sum is about 14 R^2 x, past 32 bits in lattices of some 6e8 nodes; a thread's share,
// a few links in a thousand, stays below them in any lattice that fits the device.
__device__ __forceinline__ long long warp_sum64(int v) {
    const unsigned lo = __reduce_add_sync(0xffffffffu, (unsigned)v & 0xffffu);
    const int hi = __reduce_add_sync(0xffffffffu, v >> 16);
    return (long long)hi * 65536 + (long long)lo;
}

// What a block of k_plinks needs of its particle's centre, converted once.
template <typename L>
struct LinkCentre {
    double X0, X1, X2;
    L ox, oy, oz;           // spin
    L ux, uy, uz, ravg;     // velocity, average density
    float xf0, xf1, xf2, reach2;
    // FP32 form: floor of the centre, its fraction in units of 2^-52, R^2 in
    // units of 2^-(2 sh - 64); sh: shift that takes distances below R + 2 to 62
    // bits (0: the centre is not a multiple of 2^-52, or R is too large)
    int fi, fj, fk, sh;
    long long qi, qj, qk, r2;
};

// |v| * |v| / 2^64
__device__ __forceinline__ long long sq_hi(long long v) {
    const unsigned long long a = (unsigned long long)(v < 0 ? -v : v);
    return (long long)__umul64hi(a, a);
}

// resident blocks per SM the FP32 link kernel holds its registers to
#ifndef MGLC_PLINKS_MINB
#define MGLC_PLINKS_MINB 4
#endif
template <typename S, bool TILE>
__global__ void __launch_bounds__(PB, sizeof(S) == 4 ? MGLC_PLINKS_MINB : 2)
    k_plinks(S* __restrict__ f, PartParams p, PartDev d) {
    after_previous();
    using L = typename PC<S>::C;
    if (stopped(d)) return;
    __shared__ LinkCentre<L> s_c;
    __shared__ int s_box[3];
    __shared__ int s_list[LINK_CAP];  // (box index - tb) * 32 + direction
    __shared__ int s_wsum[2][PB / 32];
    __shared__ Sum3 s_sum[PB / 32][7];
    __shared__ double s_av[PB / 32][7], s_out[13];
    __shared__ int s_nf[PB / 32][3];
    __shared__ long long s_nt[PB / 32][3];
    __shared__ int s_def[PB], s_nd;  // listed links that take the FP64 root,
    __shared__ float s_q[PB];        // and the roots
    extern __shared__ int s_own[];
    const int c = blockIdx.x, slab = blockIdx.y;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const double R = p.radius;
    const int nx = p.nx, ny = p.ny, nz = p.nz;
    const long long P = (long long)nx * ny * nz;
    // box of nodes within R+2 of the centre (1-based coordinate = index + 1)
    if (threadIdx.x < 3) s_box[threadIdx.x] = (int)floor(d.xc[3 * c + threadIdx.x]);
    if (threadIdx.x == 0) s_nd = 0;
    const int h = (int)ceil(R) + 2;
    __syncthreads();
    const int ci = s_box[0] - 1, cj = s_box[1] - 1, ck = s_box[2] - 1;
    const int bw = 2 * h + 2;
    const int kz0 = slab * bw / NSLAB, kz1 = (slab + 1) * bw / NSLAB;
    const int nbox = bw * bw * (kz1 - kz0);
    const int TX = bw + 2, TY = bw + 2, TZ = kz1 - kz0 + 2;
    if (TILE) {
        // a thread walks the tile in strides of PB without divisions, TU loads in flight
        int ti = (int)threadIdx.x % TX, tj = (int)threadIdx.x / TX % TY, tk = (int)threadIdx.x / (TX * TY);
        const int ai = PB % TX, aj = PB / TX % TY, ak = PB / (TX * TY), nt_ = TX * TY * TZ;
        constexpr int TU = 6;
        for (int e = threadIdx.x; e < nt_; e += TU * PB) {
            int o[TU];
#pragma unroll
            for (int u = 0; u < TU; u++) {
                int i = ci - h + ti - 1;
                const int j = cj - h + tj - 1, k = ck - h + kz0 + tk - 1;
                if (p.periodic_x) i = i < 0 ? i + nx : (i >= nx ? i - nx : i);
                const bool in = e + u * PB < nt_ && j >= 0 && j < ny && k >= 0 && k < nz && i >= 0 && i < nx;
                o[u] = in ? d.owner_cur[i + (long long)nx * (j + (long long)ny * k)] : -2;
                ti += ai;
                int carry = ti >= TX;
                if (carry) ti -= TX;
                tj += aj + carry;
                carry = tj >= TY;
                if (carry) tj -= TY;
                tk += ak + carry;
            }
#pragma unroll
            for (int u = 0; u < TU; u++)
                if (e + u * PB < nt_) s_own[e + u * PB] = o[u];
        }
    }
    if (wid == PB / 32 - 1) {
        const double X0 = d.xc[3 * c], X1 = d.xc[3 * c + 1], X2 = d.xc[3 * c + 2];
        LinkCentre<L> v;
        v.X0 = X0; v.X1 = X1; v.X2 = X2;
        v.ux = (L)d.uc[3 * c]; v.uy = (L)d.uc[3 * c + 1]; v.uz = (L)d.uc[3 * c + 2];
        v.ox = (L)d.om[3 * c]; v.oy = (L)d.om[3 * c + 1]; v.oz = (L)d.om[3 * c + 2];
        v.ravg = (L)d.rho_avg[0];
        v.reach2 = (float)((R + 1.8) * (R + 1.8));  // |x - X| <= R + sqrt(2) for a link
        v.xf0 = (float)X0; v.xf1 = (float)X1; v.xf2 = (float)X2;
        v.sh = 0;
        if (sizeof(L) == 4) {
            const double one = 4503599627370496.0;  // 2^52
            const double f0 = floor(X0), f1 = floor(X1), f2 = floor(X2);
            const double q0 = (X0 - f0) * one, q1 = (X1 - f1) * one, q2 = (X2 - f2) * one;
            const int bits = 32 - __clz(h);  // distances below 2^bits
            if (q0 == floor(q0) && q1 == floor(q1) && q2 == floor(q2) && bits <= 9) {
                v.fi = s_box[0]; v.fj = s_box[1]; v.fk = s_box[2];
                v.qi = (long long)q0; v.qj = (long long)q1; v.qk = (long long)q2;
                v.sh = 62 - bits;
                v.r2 = __double2ll_rn(ldexp(R * R, 2 * v.sh - 64));
            }
        }
        if (lane == 0) s_c = v;
    }
    __syncthreads();
    const double X0 = s_c.X0, X1 = s_c.X1, X2 = s_c.X2;
    const L Ux = s_c.ux, Uy = s_c.uy, Uz = s_c.uz, Ox = s_c.ox, Oy = s_c.oy, Oz = s_c.oz;
    const L ravg = s_c.ravg;
    const float reach2f = s_c.reach2, Xf0 = s_c.xf0, Xf1 = s_c.xf1, Xf2 = s_c.xf2, Lf = (float)p.nx;
    const int sh = s_c.sh;
    int nf[3] = {0, 0, 0};  // sum m e
    int nt[3] = {0, 0, 0};  // sum m (n x e)
    L av[7] = {L(0), L(0), L(0), L(0), L(0), L(0), L(0)};  // variable force, torque, mass change
    auto own_at = [&](int bi, int bj, int bk) {  // box coordinates, bk absolute in the box
        return s_own[(bi + 1) + TX * ((bj + 1) + TY * (bk - kz0 + 1))];
    };
    int tb = 0;  // box index that the list counts from
    // The fraction q of listed link le: ray-sphere root from the node (calQ2,
    // particle_bounceback.F90:144-185), FP64 (false: out of range, status set).
    // The node lies within R + 1.8 < nx / 2 of the centre: the unwrapped difference
    // is the periodic minimum image.
    auto root64 = [&](int le, double& qd) {
        const int tt = tb + (le >> 5), a = le & 31;
        const int ea = e_rt(EX_PACK, a), eb = e_rt(EY_PACK, a), ec = e_rt(EZ_PACK, a);
        const double ox = (double)(ci - h + tt % bw + 1) - X0, oy = (double)(cj - h + tt / bw % bw + 1) - X1,
                     oz = (double)(ck - h + kz0 + tt / (bw * bw) + 1) - X2;
        const double sx = ea > 0 ? ox : (ea < 0 ? -ox : 0.0);
        const double sy = eb > 0 ? oy : (eb < 0 ? -oy : 0.0);
        const double sz = ec > 0 ? oz : (ec < 0 ? -oz : 0.0);
        const double cc = ox * ox + oy * oy + oz * oz - R * R;
        const double cb = 2.0 * (sx + sy + sz);
        const double delta = cb * cb - (a <= 6 ? 4.0 : 8.0) * cc;
        if (delta < 0) { pfail(d, PS_Q_RANGE, c, 0, d.par); return false; }
        qd = (-cb - sqrt(delta)) * (a <= 6 ? 0.5 : 0.25);  // /(2 |e|^2), exact
        if (qd > 1.0 || qd < 0.0) { pfail(d, PS_Q_RANGE, c, 0, d.par); return false; }
        return true;
    };
    // FP32 form: |x - X|^2 - R^2 (the cancelling part) beyond FP32, the root in FP32.
    // Its error grows where the ray is nearly tangent (small delta) and matters
    // where q is near 0 or 1, the ends the range check tests: those links (false)
    // take the FP64 root, so the FP32 and FP64 forms accept and reject the same links.
    auto root32 = [&](int le, float& ox, float& oy, float& oz, float& q) {
        const int tt = tb + (le >> 5), a = le & 31;
        const int iu = ci - h + tt % bw, j = cj - h + tt / bw % bw, k = ck - h + kz0 + tt / (bw * bw);
        const int ea = e_rt(EX_PACK, a), eb = e_rt(EY_PACK, a), ec = e_rt(EZ_PACK, a);
        float cbf, ccf;
        if (sh) {
            // x - X exactly, in units of 2^-52, and its square to 2^-52 or so
            const long long wx = ((long long)(iu + 1 - s_c.fi) << 52) - s_c.qi;
            const long long wy = ((long long)(j + 1 - s_c.fj) << 52) - s_c.qj;
            const long long wz = ((long long)(k + 1 - s_c.fk) << 52) - s_c.qk;
            const long long w = wx * ea + wy * eb + wz * ec;
            const int up = sh - 52;
            const long long cc = sq_hi(wx << up) + sq_hi(wy << up) + sq_hi(wz << up) - s_c.r2;
            ox = (float)wx * 0x1p-52f;
            oy = (float)wy * 0x1p-52f;
            oz = (float)wz * 0x1p-52f;
            cbf = 2.0f * ((float)w * 0x1p-52f);
            ccf = (float)cc * __int_as_float((127 - (2 * sh - 64)) << 23);
        } else {
            const double x = (double)(iu + 1) - X0, y = (double)(j + 1) - X1, z = (double)(k + 1) - X2;
            const double sx = ea > 0 ? x : (ea < 0 ? -x : 0.0);
            const double sy = eb > 0 ? y : (eb < 0 ? -y : 0.0);
            const double sz = ec > 0 ? z : (ec < 0 ? -z : 0.0);
            ox = (float)x;
            oy = (float)y;
            oz = (float)z;
            cbf = 2.0f * (float)(sx + sy + sz);
            ccf = (float)(x * x + y * y + z * z - R * R);
        }
        const float delta = cbf * cbf - (a <= 6 ? 4.0f : 8.0f) * ccf;
        q = (-cbf - sqrtf(fmaxf(delta, 0.0f))) * (a <= 6 ? 0.5f : 0.25f);
        return delta > 1e-2f * cbf * cbf + 1e-3f && q > 1e-3f && q < 1.0f - 1e-3f;
    };
    // Links are listed (box index, direction) over the scan rounds of PB box
    // nodes, in a deterministic order, and processed one per thread once the
    // list is nearly full or the box is done.
    int nl = 0;  // listed so far, the same in every thread
    int par = 0;
    for (int t0 = 0; t0 < nbox; t0 += PB, par ^= 1) {
        unsigned my_dirs = 0;  // bit a: direction a is a boundary link of my node
        const int t = t0 + threadIdx.x;
        if (t < nbox) {
            const int bi = t % bw, bj = (t / bw) % bw, bk = kz0 + t / (bw * bw);
            int i = ci - h + bi;
            const int j = cj - h + bj, k = ck - h + bk;
            bool ok = !(j < 0 || j >= ny || k < 0 || k >= nz);
            if (ok) {
                // a filter only: every link node lies within R + sqrt(2) of the
                // centre, well inside the R + 1.8 kept here, so FP32 suffices
                float ox = (float)(i + 1) - Xf0;
                if (p.periodic_x) {
                    if (ox > 0.5f * Lf) ox -= Lf;
                    else if (ox < -0.5f * Lf) ox += Lf;
                }
                const float oy = (float)(j + 1) - Xf1, oz = (float)(k + 1) - Xf2;
                ok = ox * ox + oy * oy + oz * oz <= reach2f;
            }
            if (ok) {
                if (p.periodic_x) i = wrapx(i, nx);
                else ok = i >= 0 && i < nx;
            }
            if (TILE) {
                if (ok && own_at(bi, bj, bk) < 0) {
#pragma unroll
                    for (int a = 1; a < Q19; a++)
                        if (own_at(bi + ex19(a), bj + ey19(a), bk + ez19(a)) == c) my_dirs |= 1u << a;
                }
            } else if (ok && d.owner_cur[i + (long long)nx * (j + (long long)ny * k)] < 0) {
                for (int a = 1; a < Q19; a++) {
                    const int jn = j + ey19(a), kn = k + ez19(a);
                    if (jn < 0 || jn >= ny || kn < 0 || kn >= nz) continue;
                    int in = i + ex19(a);
                    if (p.periodic_x) in = wrapx(in, nx);
                    else if (in < 0 || in >= nx) continue;
                    if (d.owner_cur[in + (long long)nx * (jn + (long long)ny * kn)] != c) continue;
                    my_dirs |= 1u << a;
                }
            }
        }
        // deterministic slots: exclusive prefix sum of the per-thread link counts
        const int cnt = __popc(my_dirs);
        int incl = cnt;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += v;
        }
        if (lane == 31) s_wsum[par][wid] = incl;
        __syncthreads();
        int slot = nl + incl - cnt;
#pragma unroll
        for (int q = 0; q < PB / 32; q++) {
            const int v = s_wsum[par][q];
            if (q < wid) slot += v;
            nl += v;
        }
        for (unsigned m = my_dirs; m; m &= m - 1) s_list[slot++] = (t - tb) * 32 + __ffs(m) - 1;
        // uniform over the block
        if (nl <= LINK_CAP - PB * 18 && t0 + PB < nbox && t0 + 2 * PB - tb <= LINK_SPAN) continue;
        __syncthreads();
        if constexpr (sizeof(L) == 4) {
            // the links that need it take their FP64 root together, over the
            // whole list, before any is processed (s_def full: where they are)
            for (int e = threadIdx.x; e < nl; e += PB) {
                const int le = s_list[e];
                float ox, oy, oz, q;
                if (root32(le, ox, oy, oz, q)) continue;
                const int slot = atomicAdd(&s_nd, 1);
                if (slot < PB) {
                    s_def[slot] = le;
                    s_list[e] = -1 - slot;
                }
            }
            __syncthreads();
            if (threadIdx.x < s_nd) {
                const int le = s_def[threadIdx.x];
                double qd;
                s_q[threadIdx.x] = root64(le, qd) ? (float)qd : -1.0f;
            }
            __syncthreads();
            if (threadIdx.x == 0) s_nd = 0;
        }
        for (int e = threadIdx.x; e < nl; e += PB) {
            int le = s_list[e];
            L ox, oy, oz, q;
            if constexpr (sizeof(L) == 4) {
                bool have = false;
                if (le < 0) {
                    q = s_q[-1 - le];
                    le = s_def[-1 - le];
                    have = true;
                    if (q < 0.0f) continue;
                }
                float qf;
                const bool near = root32(le, ox, oy, oz, qf);
                if (!have) q = qf;
                if (!have && !near) {
                    double qd;
                    if (!root64(le, qd)) continue;
                    q = (float)qd;
                }
            } else {
                if (!root64(le, q)) continue;
            }
            const int tt = tb + (le >> 5), a = le & 31;
            const int bi = tt % bw, bj = (tt / bw) % bw, bk = kz0 + tt / (bw * bw);
            const int iu = ci - h + bi, j = cj - h + bj, k = ck - h + bk;  // iu: unwrapped
            const int i = p.periodic_x ? wrapx(iu, nx) : iu;
            const int ea = e_rt(EX_PACK, a), eb = e_rt(EY_PACK, a), ec = e_rt(EZ_PACK, a);
            const int m = a <= 6 ? 2 : 1;
            if constexpr (sizeof(L) == 8) {
                ox = (double)(iu + 1) - X0;
                oy = (double)(j + 1) - X1;
                oz = (double)(k + 1) - X2;
            }
            // interpolation nodes inside a solid have no post-collision value
            // of this step: fall back to the linear IBB, then to simple
            // bounce-back (nodes beyond the walls are ghosts and available).
            // All values are loaded before any is used.
            const int ra = opp_rt(a);
            const bool lo = q < L(0.5);
            const bool av1 = TILE ? own_at(bi - ea, bj - eb, bk - ec) < 0
                                  : node_avail(i - ea, j - eb, k - ec, p, d.owner_cur);
            const L dpa = fp_dev<S, L>(f, a, i, j, k, p);
            const int s1 = lo ? 1 : 0, qs = lo ? a : ra;
            L v1 = L(0), v2 = L(0);
            bool av2 = false;
            if (lo ? av1 : true) v1 = fp_dev<S, L>(f, qs, i - s1 * ea, j - s1 * eb, k - s1 * ec, p);
            if (av1) {
                const int s2 = s1 + 1;
                v2 = fp_dev<S, L>(f, qs, i - s2 * ea, j - s2 * eb, k - s2 * ec, p);
                av2 = !lo || node_avail(i - 2 * ea, j - 2 * eb, k - 2 * ec, p, d.owner_cur);
            }
            // constant parts (integers)
            const int n0 = iu + 1, n1 = j + 1, n2 = k + 1;
            nf[0] += m * ea;
            nf[1] += m * eb;
            nf[2] += m * ec;
            nt[0] += m * (n1 * ec - n2 * eb);
            nt[1] += m * (n2 * ea - n0 * ec);
            nt[2] += m * (n0 * eb - n1 * ea);
            // wall point relative to the centre and its velocity U + Omega x r
            const L rx = (L)ox + q * (L)ea, ry = (L)oy + q * (L)eb, rz = (L)oz + q * (L)ec;
            const L uw0 = Ux + (Oy * rz - Oz * ry);
            const L uw1 = Uy + (Oz * rx - Ox * rz);
            const L uw2 = Uz + (Ox * ry - Oy * rx);
            const L w = a <= 6 ? L(1.0 / 18.0) : L(1.0 / 36.0);
            const L mv = L(6) * w * ravg * (-(L)ea * uw0 - (L)eb * uw1 - (L)ec * uw2);  // moving wall
            L dn;
            if (lo) {
                if (av1 && av2) {
                    const L c0 = q * (L(1) + L(2) * q), c1 = L(1) - L(4) * q * q,
                            c2 = q * (L(1) - L(2) * q);
                    dn = c0 * dpa + c1 * v1 - c2 * v2 + mv;
                } else if (av1) {  // case1/mpi_complete/particle_bounceback.F90:66-69
                    dn = L(2) * q * dpa + (L(1) - L(2) * q) * v1 + mv;
                } else {
                    dn = dpa + mv;
                }
            } else if (av1) {
                const L iq = L(1) / q, i2 = L(1) / (L(1) + L(2) * q), a2 = L(2) * q - L(1);
                dn = (iq * i2) * dpa + (a2 * iq) * v1 - (a2 * i2) * v2 + (iq * i2) * mv;
            } else {  // case1/mpi_complete/particle_bounceback.F90:70-73
                const L h = L(0.5) / q;
                dn = h * dpa + (L(1) - h) * v1 + h * mv;
            }
            const long long fslot = ra * P + (i + (long long)nx * (j + (long long)ny * k));
            if (PSt<S>::SHIFT) {
                f[fslot] = (S)dn;
                dn = (L)f[fslot];  // as stored
            } else {
                const double wd = a <= 6 ? 1.0 / 18.0 : 1.0 / 36.0;
                f[fslot] = (S)((double)dn + wd * p.rho0);
                dn = (L)((double)f[fslot] - wd * p.rho0);
            }
            // Wen et al. 2014 Galilean-invariant momentum exchange, variable part
            const L F0 = ((L)ea - uw0) * dpa + ((L)ea + uw0) * dn;
            const L F1 = ((L)eb - uw1) * dpa + ((L)eb + uw1) * dn;
            const L F2 = ((L)ec - uw2) * dpa + ((L)ec + uw2) * dn;
            av[0] += F0;
            av[1] += F1;
            av[2] += F2;
            av[3] += ry * F2 - rz * F1;
            av[4] += rz * F0 - rx * F2;
            av[5] += rx * F1 - ry * F0;
            av[6] += dn - dpa;
        }
        __syncthreads();
        nl = 0;
        tb = t0 + PB;
    }
    // the warp's sums: exact integers, and the variable parts
#pragma unroll
    for (int q = 0; q < 3; q++) {
        const int a = __reduce_add_sync(0xffffffffu, nf[q]);
        const long long b = warp_sum64(nt[q]);
        if (lane == 0) {
            s_nf[wid][q] = a;
            s_nt[wid][q] = b;
        }
    }
    {
        const int sum = ((lane >> 4) & 1) * 4 + ((lane >> 3) & 1) * 2 + ((lane >> 2) & 1);
        if constexpr (sizeof(L) == 4) {
            Sum3 v[8];
#pragma unroll
            for (int q = 0; q < 8; q++) v[q] = {q < 7 ? av[q] : 0.0f, 0.0f, 0.0f};
            const Sum3 t = warp_sum8(v, lane);
            if ((lane & 3) == 0 && sum < 7) s_sum[wid][sum] = t;
        } else {
            Sum64 v[8];
#pragma unroll
            for (int q = 0; q < 8; q++) v[q].h = q < 7 ? av[q] : 0.0;
            const Sum64 t = warp_sum8(v, lane);
            if ((lane & 3) == 0 && sum < 7) s_av[wid][sum] = t.h;
        }
    }
    __syncthreads();
    if (wid == 0) {
        if constexpr (sizeof(L) == 4) {
            // 8 lanes per sum add the warps' parts
#pragma unroll
            for (int r = 0; r < 2; r++) {
                const int q = min(4 * r + (lane >> 3), 6), w = lane & 7;
                Sum3 v = s_sum[w][q];
#pragma unroll
                for (int o = 4; o > 0; o >>= 1) v += v.from_lane(o);
                if (w == 0) s_out[q] = (double)v.h + ((double)v.m + (double)v.l);
            }
        } else if (lane < 7) {  // the warps' parts in order
            double v = 0.0;
#pragma unroll
            for (int w = 0; w < PB / 32; w++) v += s_av[w][lane];
            s_out[lane] = v;
        }
        if (lane < 6) {
            long long v = 0;
#pragma unroll
            for (int w = 0; w < PB / 32; w++) v += lane < 3 ? (long long)s_nf[w][lane] : s_nt[w][lane - 3];
            s_out[7 + lane] = (double)v;  // exact: far below 2^53
        }
        __syncwarp();
        const double* out = s_out;
        if (lane == 0) {
            const double k0 = p.rho0 / 18.0;
            const double NF0 = out[7], NF1 = out[8], NF2 = out[9];
            const double fc[3] = {k0 * NF0, k0 * NF1, k0 * NF2};
            const double tc[3] = {k0 * (out[10] - (X1 * NF2 - X2 * NF1)),
                                  k0 * (out[11] - (X2 * NF0 - X0 * NF2)),
                                  k0 * (out[12] - (X0 * NF1 - X1 * NF0))};
            const int sl = c * NSLAB + slab;  // per-slab partials, summed in slab order
            for (int q = 0; q < 3; q++) {
                d.flink[3 * sl + q] = fc[q] + out[q];
                d.tlink[3 * sl + q] = tc[q] + out[3 + q];
            }
            d.corr[sl] = out[6];
        }
    }
}

// The node t = bi + bw (bj + bw bk) of a particle's box, walked by one thread
// in strides of PB without divisions: PB's digits in base bw are added with
// carries (the same nodes, in the same order, as t % bw, (t / bw) % bw, ...).
struct BoxWalk {
    int bi, bj, bk, ai, aj, ak, bw;
    __device__ BoxWalk(long long t0, int bw_) : bw(bw_) {
        if (bw_ < 1024) {  // 32-bit divisions
            const int t = (int)t0, b2 = bw_ * bw_;
            bi = t % bw_;
            bj = t / bw_ % bw_;
            bk = t / b2;
            ai = PB % bw_;
            aj = PB / bw_ % bw_;
            ak = PB / b2;
            return;
        }
        const long long b2 = (long long)bw_ * bw_;
        bi = (int)(t0 % bw_);
        bj = (int)((t0 / bw_) % bw_);
        bk = (int)(t0 / b2);
        ai = PB % bw_;
        aj = (int)(((long long)PB / bw_) % bw_);
        ak = (int)((long long)PB / b2);
    }
    __device__ void next() {
        bi += ai;
        int carry = 0;
        if (bi >= bw) { bi -= bw; carry = 1; }
        bj += aj + carry;
        carry = 0;
        if (bj >= bw) { bj -= bw; carry = 1; }
        bk += ak + carry;
    }
};

// ------------------------------------------- force, motion, new mask --------
// mass, volume and moment of inertia of a sphere
struct SphereK {
    double vol, M, I;
};
inline SphereK sphere_k(const PartParams& p) {
    const double R0 = p.radius;
    SphereK k;
    k.vol = 4.0 / 3.0 * p.pi * R0 * R0 * R0;
    k.M = p.rho_solid * 4.0 / 3.0 * p.pi * R0 * R0 * R0;
    k.I = 0.4 * k.M * R0 * R0;
    return k;
}

// The FP64 value *x cut to FP32, on integers (2^-20 relative; tiny values 0,
// huge ones, infinities and NaN: NaN)
__device__ __forceinline__ float top32(const double* x) {
    const int2 w = *reinterpret_cast<const int2*>(x);
    const int e = (w.y >> 20) & 0x7ff;
    const unsigned m = ((unsigned)(e - 896) << 23) | ((unsigned)(w.y & 0xfffff) << 3);
    if (e >= 896 + 255) return __int_as_float(0x7fc00000);
    return e <= 896 ? 0.0f : __int_as_float((int)(m | ((unsigned)w.y & 0x80000000u)));
}

// Force, torque (particle_force.F90:96-190 in 3-D) and motion
// (particle_update.F90:26-50) of particle c by one block; the new centre is left
// in Xn and d.*_new, the state moves on once every particle has done so.  false:
// the particle has left the range a step may take.
__device__ bool pmotion(const PartParams& p, const SphereK& sk, const PartDev& d, int c, double* Xn) {
    __shared__ double fij[3];
    __shared__ int s_ok;
    const int np = p.np;
    const double R0 = p.radius, Rc = p.radius;
    const double* X = d.xc + 3 * c;
    // FP64 only for the pairs whose top 20 bits do not rule them out: y and z are
    // below 2^16 (a difference off by 2^-3), x below 2 nx
    const float xt[3] = {top32(X), top32(X + 1), top32(X + 2)}, Lf = (float)p.nx;
    const float far = (float)(Rc + R0 + p.thr_part) * 1.001f + 0.3f + 4e-6f * Lf;
    // the spring force of particle c2 added to fp; false: out of range
    auto spring = [&](int c2, double (&fp)[3]) {
        if (c2 == c) return false;
        const double* X2 = d.xc + 3 * c2;
        float g0 = top32(X2) - xt[0];
        if (p.periodic_x) {
            if (g0 > 0.5f * Lf) g0 -= Lf;
            else if (g0 < -0.5f * Lf) g0 += Lf;
        }
        if (fabsf(g0) > far || fabsf(top32(X2 + 1) - xt[1]) > far || fabsf(top32(X2 + 2) - xt[2]) > far)
            return false;  // certainly (not taken for a NaN)
        const double d0 = dxp(X[0], X2[0], p), d1 = X[1] - X2[1], d2 = X[2] - X2[2];
        const double thr = p.thr_part;
        const double reach = Rc + R0 + thr;
        if (fabs(d0) >= reach || fabs(d1) >= reach || fabs(d2) >= reach) return false;
        const double dij = sqrt(d0 * d0 + d1 * d1 + d2 * d2);
        if (dij >= Rc + R0 + thr) return false;
        if (dij >= Rc + R0) {
            const double t = (dij - Rc - R0 - thr) / thr;
            fp[0] = fp[0] + p.scale_part * (t * t) * d0 / dij;
            fp[1] = fp[1] + p.scale_part * (t * t) * d1 / dij;
            fp[2] = fp[2] + p.scale_part * (t * t) * d2 / dij;
            return true;
        }
        pfail(d, PS_OVERLAP, c, c2, d.par);
        return false;
    };
    // The whole block looks for contacts; their forces, which are rare, are one
    // warp's: a lane adds every 32nd particle's, then the tree over the lanes, so that
    // the sums do not depend on how many threads look.
    bool hit = false;
    double none[3] = {0.0, 0.0, 0.0};
    for (int c2 = threadIdx.x; c2 < np; c2 += PB) hit = spring(c2, none) || hit;
    const bool any = __syncthreads_or(hit);
    if (threadIdx.x < 32) {
        double fp[3] = {0.0, 0.0, 0.0};
        if (any) {
            for (int c2 = threadIdx.x; c2 < np; c2 += 32) spring(c2, fp);
#pragma unroll
            for (int q = 0; q < 3; q++)
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) fp[q] += __shfl_down_sync(0xffffffffu, fp[q], o);
        }
        if (threadIdx.x == 0)
            for (int q = 0; q < 3; q++) fij[q] = fp[q];
    }
    __syncthreads();
    if (threadIdx.x < 32) {  // lane q: component q
        const int q = min((int)threadIdx.x, 2);
        const double ravg = d.rho_avg[0], thw = p.thr_wall;
        double fw = 0.0;
        if (q > 0 || !p.periodic_x) {
            const int nax = q == 0 ? p.nx : (q == 1 ? p.ny : p.nz);
            double dw = X[q] - Rc - 1.0;
            if (dw < 0) pfail(d, PS_WALL, c, 0, d.par);
            else if (dw < thw) fw = fw + p.scale_wall * ((dw - thw) / thw) * ((dw - thw) / thw);
            dw = (double)nax - X[q] - Rc;
            if (dw < 0) pfail(d, PS_WALL, c, 0, d.par);
            else if (dw < thw) fw = fw - p.scale_wall * ((dw - thw) / thw) * ((dw - thw) / thw);
        }
        double fl = 0.0, tl = 0.0;
#pragma unroll
        for (int sl = 0; sl < NSLAB; sl++) {
            fl += d.flink[3 * (c * NSLAB + sl) + q];
            tl += d.tlink[3 * (c * NSLAB + sl) + q];
        }
        double tot = fl + (p.rho_solid - ravg) * sk.vol * (q == 0 ? p.gravity[0] : q == 1 ? p.gravity[1] : p.gravity[2]) + fij[q] + fw;
        tot = tot + ravg * sk.vol * (q == 0 ? p.body_force[0] : q == 1 ? p.body_force[1] : p.body_force[2]);
        const double a = tot / sk.M;
        const double u = d.uc[3 * c + q] + a, om = d.om[3 * c + q] + tl / sk.I;
        double x = X[q] + d.uc[3 * c + q] + 0.5 * a;
        bool ok = isfinite(x) && isfinite(u) && isfinite(om);
        if (q == 0 && p.periodic_x) {
            // one wrap per step is enough only while the step moves the centre by
            // less than half the periodic length
            const double L = (double)p.nx;
            ok = ok && fabs(x - X[0]) < 0.5 * L;
            if (x >= L + 0.5) x -= L;
            if (x < 0.5) x += L;
        }
        ok = __all_sync(0xffffffffu, ok);
        if (threadIdx.x < 3) {
            d.ftot[3 * c + q] = tot;
            d.ttot[3 * c + q] = tl;
            d.xc_new[3 * c + q] = x;
            d.uc_new[3 * c + q] = u;
            d.om_new[3 * c + q] = om;
            Xn[q] = x;
        }
        if (threadIdx.x == 0) s_ok = ok;
    }
    __syncthreads();
    return s_ok;
}

// MOVE: the particle's force and motion first (as a launch of its own, a warp per
// particle and one block that moved them all, 46 us for 200 spheres; in
// k_plinks's last block, longer still, waiting in the fence for that SM's
// scattered stores).
template <bool MOVE>
__global__ void __launch_bounds__(PB) k_pmark(int* owner, PartParams p, SphereK sk, PartDev d) {
    after_previous();
    if (MOVE && stopped(d)) return;
    const int c = blockIdx.x;
    __shared__ double X[3];
    if constexpr (MOVE) {
        if (!pmotion(p, sk, d, c, X)) {
            if (threadIdx.x == 0) atomicCAS(d.done + 1, 0u, (unsigned)c + 1u);
            return;
        }
    } else {
        if (threadIdx.x < 3) X[threadIdx.x] = d.xc[3 * c + threadIdx.x];
        __syncthreads();
    }
    __shared__ int s_c[3];
    __shared__ float s_f[3];
    if (threadIdx.x < 3) {
        s_c[threadIdx.x] = (int)floor(X[threadIdx.x]) - 1;
        s_f[threadIdx.x] = (float)X[threadIdx.x];
    }
    __syncthreads();
    const double R = p.radius;
    const int h = (int)ceil(R) + 1;
    const int ci = s_c[0], cj = s_c[1], ck = s_c[2];
    const int bw = 2 * h + 2;
    const long long nbox = (long long)bw * bw * bw;
    const float Xf0 = s_f[0], Xf1 = s_f[1], Xf2 = s_f[2], Lf = (float)p.nx;
    const float Xmax = fmaxf(fabsf(Xf0), fmaxf(fabsf(Xf1), fabsf(Xf2))) + Lf;  // wrapped nodes too
    const float r2 = (float)(R * R);
    BoxWalk bw_it(threadIdx.x, bw);
    for (long long t = threadIdx.x; t < nbox; t += PB, bw_it.next()) {
        const int bi = bw_it.bi, bj = bw_it.bj, bk = bw_it.bk;
        int i = ci - h + bi;
        const int j = cj - h + bj, k = ck - h + bk;
        if (j < 0 || j >= p.ny || k < 0 || k >= p.nz) continue;
        if (p.periodic_x) i = wrapx(i, p.nx);
        else if (i < 0 || i >= p.nx) continue;
        // FP32 decides far from the surface; nodes within tol of it use the
        // IEEE-rounded FP64 test.  tol bounds the FP32 error of d2 (the centre
        // rounded to FP32, then the differences, squares and sums) at least
        // twice over, so wherever FP32 decides, its decision is the FP64 test's.
        float fx = (float)(i + 1) - Xf0;
        if (p.periodic_x) {
            if (fx > 0.5f * Lf) fx -= Lf;
            else if (fx < -0.5f * Lf) fx += Lf;
        }
        const float fy = (float)(j + 1) - Xf1, fz = (float)(k + 1) - Xf2;
        const float d2 = fx * fx + fy * fy + fz * fz;
        const float tol = 1e-3f * r2 + 4e-6f * (float)(h + 1) * (Xmax + (float)(h + 1)) + 1e-6f * d2;
        bool in;
        if (fabsf(d2 - r2) > tol) in = d2 < r2;
        else in = inside((double)(i + 1), (double)(j + 1), (double)(k + 1), X, R, p);
        if (in) owner[i + (long long)p.nx * (j + (long long)p.ny * k)] = c;
    }
}

// Nodes that change phase: the density bookkeeping of the average used by the
// refill, and each particle's list of nodes to refill.  PREP_SLAB blocks per
// particle walk a z slab of its old box and, where that differs, of its new one;
// the last block to finish forms the average: (mass after bounce-back + link
// corrections + phase changes) / (fluid count + its change).  (As three
// launches, the boxes walked three times by one block each: 17 + 8 + 15 us.)
constexpr int PREP_SLAB = PART_NSLAB;
#ifndef MGLC_PU
#define MGLC_PU 2
#endif
constexpr int PU = MGLC_PU;
template <typename S>
__global__ void __launch_bounds__(PB) k_pphase(const S* f, PartParams p, PartDev d) {
    after_previous();
    if (stopped(d)) return;
    const int c = blockIdx.x, slab = blockIdx.y;
    if (d.done[1]) {  // a particle went out of range: the state moves and freezes
        if (c == 0 && slab == 0 && threadIdx.x == 0) pfail(d, PS_DIVERGED, (int)d.done[1] - 1, 0, d.par);
        return;
    }
    const long long P = (long long)p.nx * p.ny * p.nz;
    double sum = 0.0;
    int cnt = 0;
    __shared__ int s_c[6];  // corner node of the old and the new box, less h
    if (threadIdx.x < 6)
        s_c[threadIdx.x] = (int)floor(threadIdx.x < 3 ? d.xc[3 * c + threadIdx.x] : d.xc_new[3 * c + threadIdx.x - 3]) - 1;
    __syncthreads();
    // the second box only where it is another one; the first pass then looks for
    // entering nodes too
    const bool same = s_c[0] == s_c[3] && s_c[1] == s_c[4] && s_c[2] == s_c[5];
    const int h = (int)ceil(p.radius) + 1;
    for (int pass = 0; pass < (same ? 1 : 2); pass++) {
        const int ci = s_c[3 * pass], cj = s_c[3 * pass + 1], ck = s_c[3 * pass + 2];
        const int bw = 2 * h + 2;
        const int k0 = slab * bw / PREP_SLAB, k1 = (slab + 1) * bw / PREP_SLAB;
        const long long t1 = (long long)bw * bw * k1;
        BoxWalk bw_it((long long)bw * bw * k0 + threadIdx.x, bw);
        for (long long t = (long long)bw * bw * k0 + threadIdx.x; t < t1; t += PU * PB) {
            // PU nodes' masks in flight
            long long cell[PU];
            int oc[PU], on[PU];
#pragma unroll
            for (int u = 0; u < PU; u++, bw_it.next()) {
                int i = ci - h + bw_it.bi;
                const int j = cj - h + bw_it.bj, k = ck - h + bw_it.bk;
                bool in = t + u * PB < t1 && j >= 0 && j < p.ny && k >= 0 && k < p.nz;
                if (p.periodic_x) i = wrapx(i, p.nx);
                else in = in && i >= 0 && i < p.nx;
                cell[u] = i + (long long)p.nx * (j + (long long)p.ny * k);
                oc[u] = in ? d.owner_cur[cell[u]] : c;  // outside: no change of phase
                on[u] = in ? d.owner_new[cell[u]] : c;
            }
#pragma unroll
            for (int u = 0; u < PU; u++) {
                if (pass == 0 && oc[u] == c && on[u] < 0) {  // leaves particle c: counted with rho_solid
                    sum += p.rho_solid;
                    cnt += 1;
                    const int slot = atomicAdd(d.rf_count + c, 1);
                    if (slot < PART_REFILL) d.rf_list[(size_t)c * PART_REFILL + slot] = cell[u];
                }
                if ((pass == 1 || same) && oc[u] < 0 && on[u] == c) {  // enters particle c: drop its density
                    double r = 0.0;
                    for (int q = 0; q < Q19; q++) r += pabs<S>(f, q * P + cell[u], q, p.rho0);
                    sum -= r;
                    cnt -= 1;
                }
            }
        }
    }
    // most blocks have nothing to add
    __shared__ double out[2];
    __shared__ int last;
    if (__syncthreads_or(cnt != 0 || sum != 0.0)) {
        double acc[2] = {sum, (double)cnt};
        block_sum_to<2>(acc, out, 1);
    } else if (threadIdx.x == 0) {
        out[0] = out[1] = 0.0;
    }
    if (threadIdx.x == 0) {
        d.prep_sum[c * PREP_SLAB + slab] = out[0];
        d.prep_cnt[c * PREP_SLAB + slab] = (int)llround(out[1]);
        __threadfence();
        last = atomicAdd(d.done + 2, 1u) == gridDim.x * gridDim.y - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    double acc[2] = {0.0, 0.0};
    for (int q = threadIdx.x; q < p.np * PREP_SLAB; q += PB) {
        acc[0] += __ldcg(d.corr + q) + __ldcg(d.prep_sum + q);
        acc[1] += (double)__ldcg(d.prep_cnt + q);
    }
    block_sum_to<2>(acc, out, 1);
    for (int q = threadIdx.x; q < p.np; q += PB)
        if (__ldcg(d.rf_count + q) > PART_REFILL) pfail(d, PS_REFILL_FULL, q, 0, d.par ^ 1);
    if (threadIdx.x == 0) {
        const long long n1 = d.n_fluid[0] + llround(out[1]);
        d.rho_avg[1] = (d.rho_avg[2] + out[0]) / (double)n1;
        d.n_fluid[0] = n1;
        d.done[2] = 0;
    }
}

// D3Q19 forward moments and inverse in the reference's basis, FP64
__device__ void moments19d(const double* f, double* m) {
    m[0] = f[0] + f[1] + f[2] + f[3] + f[4] + f[5] + f[6] + f[7] + f[8] + f[9] + f[10] + f[11] +
           f[12] + f[13] + f[14] + f[15] + f[16] + f[17] + f[18];
    m[1] = -30.0 * f[0] - 11.0 * (f[1] + f[2] + f[3] + f[4] + f[5] + f[6]) +
           8.0 * (f[7] + f[8] + f[9] + f[10] + f[11] + f[12] + f[13] + f[14] + f[15] + f[16] + f[17] + f[18]);
    m[2] = 12.0 * f[0] - 4.0 * (f[1] + f[2] + f[3] + f[4] + f[5] + f[6]) + f[7] + f[8] + f[9] +
           f[10] + f[11] + f[12] + f[13] + f[14] + f[15] + f[16] + f[17] + f[18];
    m[3] = f[1] - f[2] + f[7] - f[8] + f[9] - f[10] + f[11] - f[12] + f[13] - f[14];
    m[4] = -4.0 * (f[1] - f[2]) + f[7] - f[8] + f[9] - f[10] + f[11] - f[12] + f[13] - f[14];
    m[5] = f[3] - f[4] + f[7] + f[8] - f[9] - f[10] + f[15] - f[16] + f[17] - f[18];
    m[6] = -4.0 * (f[3] - f[4]) + f[7] + f[8] - f[9] - f[10] + f[15] - f[16] + f[17] - f[18];
    m[7] = f[5] - f[6] + f[11] + f[12] - f[13] - f[14] + f[15] + f[16] - f[17] - f[18];
    m[8] = -4.0 * (f[5] - f[6]) + f[11] + f[12] - f[13] - f[14] + f[15] + f[16] - f[17] - f[18];
    m[9] = 2.0 * (f[1] + f[2]) - f[3] - f[4] - f[5] - f[6] + f[7] + f[8] + f[9] + f[10] + f[11] +
           f[12] + f[13] + f[14] - 2.0 * (f[15] + f[16] + f[17] + f[18]);
    m[10] = -4.0 * (f[1] + f[2]) + 2.0 * (f[3] + f[4] + f[5] + f[6]) + f[7] + f[8] + f[9] + f[10] +
            f[11] + f[12] + f[13] + f[14] - 2.0 * (f[15] + f[16] + f[17] + f[18]);
    m[11] = f[3] + f[4] - f[5] - f[6] + f[7] + f[8] + f[9] + f[10] - (f[11] + f[12] + f[13] + f[14]);
    m[12] = -2.0 * (f[3] + f[4] - f[5] - f[6]) + (f[7] + f[8] + f[9] + f[10]) - (f[11] + f[12] + f[13] + f[14]);
    m[13] = f[7] - f[8] - f[9] + f[10];
    m[14] = f[15] - f[16] - f[17] + f[18];
    m[15] = f[11] - f[12] - f[13] + f[14];
    m[16] = f[7] - f[8] + f[9] - f[10] - f[11] + f[12] - f[13] + f[14];
    m[17] = -f[7] - f[8] + f[9] + f[10] + f[15] - f[16] + f[17] - f[18];
    m[18] = f[11] + f[12] - f[13] - f[14] - f[15] - f[16] + f[17] + f[18];
}
// f = M^-1 m with M^-1 = M^T diag(1/|M_k|^2)
__device__ void inverse19d(const double* m, double* f) {
    const double a0 = m[0] / 19.0, a1 = m[1] / 2394.0, a2 = m[2] / 252.0;
    const double b3 = m[3] / 10.0, b4 = m[4] / 40.0, b5 = m[5] / 10.0, b6 = m[6] / 40.0,
                 b7 = m[7] / 10.0, b8 = m[8] / 40.0;
    const double c9 = m[9] / 36.0, c10 = m[10] / 72.0, c11 = m[11] / 12.0, c12 = m[12] / 24.0;
    const double d13 = m[13] / 4.0, d14 = m[14] / 4.0, d15 = m[15] / 4.0;
    const double e16 = m[16] / 8.0, e17 = m[17] / 8.0, e18 = m[18] / 8.0;
    f[0] = a0 - 30.0 * a1 + 12.0 * a2;
    const double ax = a0 - 11.0 * a1 - 4.0 * a2, ed = a0 + 8.0 * a1 + a2;
    f[1] = ax + (b3 - 4.0 * b4) + (2.0 * c9 - 4.0 * c10);
    f[2] = ax - (b3 - 4.0 * b4) + (2.0 * c9 - 4.0 * c10);
    f[3] = ax + (b5 - 4.0 * b6) - c9 + 2.0 * c10 + c11 - 2.0 * c12;
    f[4] = ax - (b5 - 4.0 * b6) - c9 + 2.0 * c10 + c11 - 2.0 * c12;
    f[5] = ax + (b7 - 4.0 * b8) - c9 + 2.0 * c10 - c11 + 2.0 * c12;
    f[6] = ax - (b7 - 4.0 * b8) - c9 + 2.0 * c10 - c11 + 2.0 * c12;
    const double E = ed + c9 + c10;
    f[7] = E + c11 + c12 + d13 + (b3 + b4 + b5 + b6) + e16 - e17;
    f[10] = E + c11 + c12 + d13 - (b3 + b4 + b5 + b6) - e16 + e17;
    f[9] = E + c11 + c12 - d13 + (b3 + b4 - b5 - b6) + e16 + e17;
    f[8] = E + c11 + c12 - d13 - (b3 + b4 - b5 - b6) - e16 - e17;
    f[11] = E - c11 - c12 + d15 + (b3 + b4 + b7 + b8) - e16 + e18;
    f[14] = E - c11 - c12 + d15 - (b3 + b4 + b7 + b8) + e16 - e18;
    f[13] = E - c11 - c12 - d15 + (b3 + b4 - b7 - b8) - e16 - e18;
    f[12] = E - c11 - c12 - d15 - (b3 + b4 - b7 - b8) + e16 + e18;
    const double Ez = ed - 2.0 * c9 - 2.0 * c10;
    f[15] = Ez + d14 + (b5 + b6 + b7 + b8) + e17 - e18;
    f[18] = Ez + d14 - (b5 + b6 + b7 + b8) - e17 + e18;
    f[17] = Ez - d14 + (b5 + b6 - b7 - b8) + e17 + e18;
    f[16] = Ez - d14 - (b5 + b6 - b7 - b8) - e17 - e18;
}

// refill (particle_update.F90:134-193 in 3-D): extrapolate along the lattice
// direction closest to the outward normal, then reset the momentum moments to
// rho_avg times the wall velocity.  All of a particle's refills read before
// any of them is written.
template <typename S>
__global__ void __launch_bounds__(PB) k_prefill(S* __restrict__ f, PartParams p, PartDev d) {
    after_previous();
    const int c = blockIdx.x;
    // the particle moves on, with an error too if that came after the motion
    // (status from an earlier step: the values are those of now)
    const int code = d.status[0];
    if (threadIdx.x < 3 && (!code || code == PS_REFILL_FULL || code == PS_NO_REFILL_DIR || code == PS_DIVERGED)) {
        const int q = 3 * c + threadIdx.x;
        d.xc[q] = d.xc_new[q];
        d.uc[q] = d.uc_new[q];
        d.om[q] = d.om_new[q];
    }
    if (__syncthreads_or(code)) return;
    const int n = d.rf_count[c];  // at most PART_REFILL: k_pphase has failed where more
    if (n == 0) return;
    const long long P = (long long)p.nx * p.ny * p.nz;
    __shared__ double s_val[PART_REFILL][Q19];
    const double s_ravg = d.rho_avg[1];
    const double* X = d.xc_new + 3 * c;
    const double* U = d.uc_new + 3 * c;
    const double* O = d.om_new + 3 * c;
    for (int slot = threadIdx.x; slot < n; slot += PB) {
        const long long cell = d.rf_list[(size_t)c * PART_REFILL + slot];
        const int i = (int)(cell % p.nx), j = (int)(cell / p.nx % p.ny),
                  k = (int)(cell / ((long long)p.nx * p.ny));
        const double rx = dxp((double)(i + 1), X[0], p), ry = (double)(j + 1) - X[1],
                     rz = (double)(k + 1) - X[2];
        double out = 0.0;
        int ec = 0;
        const double rn = __dsqrt_rn(__dadd_rn(__dadd_rn(__dmul_rn(rx, rx), __dmul_rn(ry, ry)), __dmul_rn(rz, rz)));
        for (int a = 1; a < Q19; a++) {
            const double tn = __ddiv_rn(__dadd_rn(__dadd_rn(__dmul_rn(rx, (double)ex19(a)), __dmul_rn(ry, (double)ey19(a))),
                                                  __dmul_rn(rz, (double)ez19(a))), rn);
            if (tn > out) {
                out = tn;
                ec = a;
            }
        }
        if (ec == 0) {
            pfail(d, PS_NO_REFILL_DIR, c, 0, d.par ^ 1);
            continue;
        }
        const int e0 = ex19(ec), e1 = ey19(ec), e2 = ez19(ec);
        double fl[Q19], m[Q19];
        for (int a = 0; a < Q19; a++) {
            double fv[3];
            for (int s = 1; s <= 3; s++) {
                const int ii = p.periodic_x ? wrapx(i + s * e0, p.nx) : i + s * e0;
                const int jj = j + s * e1, kk = k + s * e2;
                if (ii < 0 || ii >= p.nx || jj < 0 || jj >= p.ny || kk < 0 || kk >= p.nz)
                    fv[s - 1] = w19(a) * p.rho0;  // ghost value
                else
                    fv[s - 1] = pabs<S>(f, a * P + (ii + (long long)p.nx * (jj + (long long)p.ny * kk)), a, p.rho0);
            }
            // 3 f(x+e) - 3 f(x+2e) + f(x+3e) (particle_update.F90:157-159)
            fl[a] = __dadd_rn(__dsub_rn(__dmul_rn(3.0, fv[0]), __dmul_rn(3.0, fv[1])), fv[2]);
        }
        moments19d(fl, m);
        const double x0 = X[0] + rx, y0 = (double)(j + 1), z0 = (double)(k + 1);
        const double qx = x0 - X[0], qy = y0 - X[1], qz = z0 - X[2];
        m[3] = s_ravg * (U[0] + (O[1] * qz - O[2] * qy));
        m[5] = s_ravg * (U[1] + (O[2] * qx - O[0] * qz));
        m[7] = s_ravg * (U[2] + (O[0] * qy - O[1] * qx));
        inverse19d(m, fl);
        for (int a = 0; a < Q19; a++) s_val[slot][a] = fl[a];
    }
    // a node without a direction has set the status: nothing is written
    __syncthreads();
    if (threadIdx.x == 0) d.rf_count[c] = 0;
    if (__ldcg(d.status)) return;
    for (int t = threadIdx.x; t < n * Q19; t += PB) {
        const int slot = t / Q19, a = t % Q19;
        pset<S>(f, a * P + d.rf_list[(size_t)c * PART_REFILL + slot], a, s_val[slot][a], p.rho0);
    }
}

// ------------------------------------------------------------ initialise --
template <typename S>
__global__ void k_pinit_f(S* f, const int* owner, PartParams p) {
    const long long P = (long long)p.nx * p.ny * p.nz;
    for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < P;
         c += (long long)gridDim.x * blockDim.x) {
        const bool fluid = owner[c] < 0;
        for (int q = 0; q < Q19; q++) pset<S>(f, q * P + c, q, fluid ? w19(q) * (1.0 + 0.0) : 0.0, p.rho0);
    }
}
__global__ void k_pcount(const int* owner, long long n, long long* out) {
    long long cnt = 0;
    for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < n;
         c += (long long)gridDim.x * blockDim.x)
        cnt += owner[c] < 0;
    double acc[1] = {(double)cnt};
    __shared__ double o[1];
    block_sum_to<1>(acc, o, 1);
    if (threadIdx.x == 0) out[0] = llround(o[0]);
}

template <typename S>
__global__ void k_pmacro(const S* f, const int* owner, PartParams p, Fix60K fk, bool first, double* rho,
                         double* u, double* v, double* w) {
    after_previous();
    const long long P = (long long)p.nx * p.ny * p.nz;
    for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < P;
         c += (long long)gridDim.x * blockDim.x) {
        if (owner[c] >= 0) {
            rho[c] = p.rho_solid;
            u[c] = v[c] = w[c] = 0.0;
            continue;
        }
        if (first) {
            rho[c] = p.rho0;
            u[c] = v[c] = w[c] = 0.0;
            continue;
        }
        double r, jx, jy, jz, uu, vv, ww;
        typename PC<S>::C fq[Q19];
#pragma unroll
        for (int q = 0; q < Q19; q++) fq[q] = f[q * P + c];
        long long R = 0;
        if constexpr (PSt<S>::SHIFT) {
            long long j[3];
            if (fix60_sums(fq, fk, R, j)) {
                r = fix61_store_any<60>(R);
                jx = fix61_store_any<60>(j[0]);
                jy = fix61_store_any<60>(j[1]);
                jz = fix61_store_any<60>(j[2]);
                R *= 2;
            } else {
                macro_sums_ordered(fq, 1.0, p.rho0, r, jx, jy, jz);
                R = 0;
            }
        } else {
            macro_sums<false>(fq, r, jx, jy, jz, R);
        }
        div_by(jx + 0.5 * (r * p.body_force[0]), jy + 0.5 * (r * p.body_force[1]),
               jz + 0.5 * (r * p.body_force[2]), r, uu, vv, ww, R);
        rho[c] = r;
        u[c] = uu;
        v[c] = vv;
        w[c] = ww;
    }
}

// ---------------------------------------------------------------- launch --
static dim3 pblock(int nx) {
    int bx = ((nx + 31) / 32) * 32;
    return dim3(bx > 128 ? 128 : bx, 1, 1);
}
// number of per-warp partial slots of the bulk kernel
int particle_bulk_blocks(const PartParams& p) {
    dim3 b = pblock(p.nx);
    return ((p.nx + b.x - 1) / b.x) * p.ny * p.nz * (int)(b.x / 32);
}

template <typename S>
static cudaError_t pstep_go(bool first, const void* fin, void* fout, const PartParams& p,
                            const PartDev& d, cudaStream_t s) {
    using C = typename PC<S>::C;
    dim3 b = pblock(p.nx), g((p.nx + b.x - 1) / b.x, p.ny, p.nz);
    const PBulkK<C> bk = bulk_k(p, C());
    // 32-bit indices while every population index (and the +-1 neighbour
    // offsets) fits in int
    const bool i32 = (long long)p.nx * p.ny * p.nz * (Q19 + 1) < (1LL << 31);
    const S* fi = (const S*)fin;
    S* fo = (S*)fout;
    if (first && i32) launch_next(k_pbulk<S, true, int>, g, b, 0, s, fi, fo, d.owner_cur, d.owner_new, p, bk, d.partials, d.status);
    else if (first) launch_next(k_pbulk<S, true, long long>, g, b, 0, s, fi, fo, d.owner_cur, d.owner_new, p, bk, d.partials, d.status);
    else if (i32) launch_next(k_pbulk<S, false, int>, g, b, 0, s, fi, fo, d.owner_cur, d.owner_new, p, bk, d.partials, d.status);
    else launch_next(k_pbulk<S, false, long long>, g, b, 0, s, fi, fo, d.owner_cur, d.owner_new, p, bk, d.partials, d.status);
    launch_next(k_pfinish<S>, FINISH_BLOCKS<S>, 256, 0, s, d, d.nblocks, p.rho0);
    if (p.np > 0) {
        const int bw = 2 * ((int)ceil(p.radius) + 2) + 2;
        const size_t tile = sizeof(int) * (size_t)(bw + 2) * (bw + 2) * ((bw + NSLAB - 1) / NSLAB + 2);
        if (tile <= TILE_MAX_BYTES) {
            // the shared-memory opt-in is a per-device attribute of the kernel
            static std::atomic<unsigned long long> opted{0};  // bit = device ordinal
            int dev = 0;
            cudaGetDevice(&dev);
            const unsigned long long bit = 1ull << (dev & 63);
            if (!(opted.load() & bit)) {
                cudaError_t e = cudaFuncSetAttribute(k_plinks<S, true>,
                                                     cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                     (int)TILE_MAX_BYTES);
                if (e != cudaSuccess) return e;
                opted.fetch_or(bit);
            }
            launch_next(k_plinks<S, true>, dim3(p.np, NSLAB), PB, tile, s, (S*)fout, p, d);
        } else {
            launch_next(k_plinks<S, false>, dim3(p.np, NSLAB), PB, 0, s, (S*)fout, p, d);
        }
        launch_next(k_pmark<true>, p.np, PB, 0, s, d.owner_new, p, sphere_k(p), d);
        launch_next(k_pphase<S>, dim3(p.np, PREP_SLAB), PB, 0, s, (const S*)fout, p, d);
        launch_next(k_prefill<S>, p.np, PB, 0, s, (S*)fout, p, d);
    }
    return cudaGetLastError();
}

cudaError_t launch_particle_step(int form, bool first, const void* fin, void* fout,
                                 const PartParams& p, const PartDev& d, cudaStream_t s) {
    if (form == FORM_FP64) return pstep_go<double>(first, fin, fout, p, d, s);
    if (form == FORM_FP32) return pstep_go<float>(first, fin, fout, p, d, s);
    return cudaErrorInvalidValue;
}

cudaError_t launch_particle_init(int form, void* f, const PartParams& p, const PartDev& d,
                                 cudaStream_t s) {
    const long long n = (long long)p.nx * p.ny * p.nz;
    cudaError_t e = cudaMemsetAsync(d.owner_cur, 0xFF, sizeof(int) * (size_t)n, s);
    if (e != cudaSuccess) return e;
    if (p.np > 0) launch_next(k_pmark<false>, p.np, PB, 0, s, d.owner_cur, p, sphere_k(p), d);
    int gb = (int)std::min<long long>((n + 255) / 256, 152 * 16);
    if (form == FORM_FP64) k_pinit_f<double><<<gb, 256, 0, s>>>((double*)f, d.owner_cur, p);
    else k_pinit_f<float><<<gb, 256, 0, s>>>((float*)f, d.owner_cur, p);
    k_pcount<<<1, 1024, 0, s>>>(d.owner_cur, n, d.n_fluid);
    return cudaGetLastError();
}

cudaError_t launch_particle_macro(int form, bool first, const void* f, const PartParams& p,
                                  const PartDev& d, double* rho, double* u, double* v, double* w,
                                  cudaStream_t s) {
    const long long n = (long long)p.nx * p.ny * p.nz;
    int gb = (int)std::min<long long>((n + 255) / 256, 152 * 16);
    if (form == FORM_FP64)
        launch_next(k_pmacro<double>, gb, 256, 0, s, (const double*)f, d.owner_cur, p, make_fix60(p.rho0, 1.0), first, rho, u, v, w);
    else
        launch_next(k_pmacro<float>, gb, 256, 0, s, (const float*)f, d.owner_cur, p, make_fix60(p.rho0, 1.0), first, rho, u, v, w);
    return cudaGetLastError();
}

}  // namespace mglc
