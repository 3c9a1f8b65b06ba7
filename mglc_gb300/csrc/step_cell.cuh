// step_cell.cuh -- per-cell bodies of the fused lattice-Boltzmann steps,
// shared by the one-solve kernels (k_step.cu) and the multi-solve tile-queue
// kernel of the solve server (k_serve.cu).
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <type_traits>

#include "fix61.cuh"
#include "kernels.cuh"

namespace mglc {

// ---------------------------------------------------------------- storage --
template <typename S>
struct St;
// SCALED (16-bit types): the cell bodies compute in units of the storage
// scale (a power of two, so every product with it is exact and the results
// are bitwise those of unscaled arithmetic); cvt_s / st_s / st_sr_s convert
// without the scale multiply.
template <>
struct St<double> {
    using C = double;
    static constexpr bool SHIFT = false;
    static constexpr bool SCALED = false;
    __device__ static C cvt_s(double v) { return v; }
    __device__ static void st_s(double* p, C v) { *p = v; }
    __device__ static void st_sr_s(double* p, C v, unsigned) { *p = v; }
    __device__ static C ld(const double* p, float) { return __ldg(p); }
    // raw: a two-buffer step's load, from L2 (coherent, as launch.cuh asks; through L1 FP32
    // 97^3 took 25.2 us a step against 23.8, eight served solves 23.2 ms against 22.3);
    // raw_rw: for a buffer that the same kernel also writes (in place FP32 128^3 51.8 us
    // through L1, 53.1 from L2)
    __device__ static double raw(const double* p) { return __ldcg(p); }
    __device__ static double raw_rw(const double* p) { return *p; }
    __device__ static void st_sr(double* p, C v, float, unsigned) { *p = v; }
    __device__ static C cvt(double v, float) { return v; }
    __device__ static void st(double* p, C v, float) { *p = v; }
};
template <>
struct St<float> {
    using C = float;
    static constexpr bool SHIFT = true;
    static constexpr bool SCALED = false;
    __device__ static C cvt_s(float v) { return v; }
    __device__ static void st_s(float* p, C v) { *p = v; }
    __device__ static void st_sr_s(float* p, C v, unsigned) { *p = v; }
    __device__ static C ld(const float* p, float) { return __ldg(p); }
    __device__ static float raw(const float* p) { return __ldcg(p); }
    __device__ static float raw_rw(const float* p) { return *p; }
    __device__ static void st_sr(float* p, C v, float, unsigned) { *p = v; }
    __device__ static C cvt(float v, float) { return v; }
    __device__ static void st(float* p, C v, float) { *p = v; }
};
template <>
struct St<__half> {
    using C = float;
    static constexpr bool SHIFT = true;
    static constexpr bool SCALED = true;
    __device__ static C cvt_s(__half v) { return __half2float(v); }
    __device__ static void st_s(__half* p, C v) { *p = __float2half_rn(v); }
    __device__ static void st_sr_s(__half* p, C v, unsigned r) {
        *p = __float2half_rz(__uint_as_float(__float_as_uint(v) + (r >> 19)));
    }
    // two values rounded stochastically by the conversion itself (cvt.rs):
    // a into the high half, b into the low half, each with its own 16 bits
    // of r; NaN and infinities convert as themselves
    __device__ static unsigned pack_sr(float a, float b, unsigned r) {
        unsigned d;
        asm("cvt.rs.f16x2.f32 %0, %1, %2, %3;" : "=r"(d) : "f"(a), "f"(b), "r"(r));
        return d;
    }
    __device__ static void st_bits(__half* p, unsigned short v) { *p = __ushort_as_half(v); }
    __device__ static C ld(const __half* p, float inv) { return __half2float(__ldg(p)) * inv; }
    __device__ static __half raw(const __half* p) { return __ldcg(p); }
    __device__ static __half raw_rw(const __half* p) { return *p; }
    // stochastic rounding: 13 uniform bits added below the 10 kept mantissa
    // bits, then truncation (unbiased; rounding errors do not correlate from
    // step to step, so they do not accumulate into a drift)
    // (finite values only: adding to a NaN pattern could wrap into the sign
    // bit; the cell bodies round to nearest in cells whose rho or u is not finite)
    __device__ static void st_sr(__half* p, C v, float sc, unsigned r) {
        *p = __float2half_rz(__uint_as_float(__float_as_uint(v * sc) + (r >> 19)));
    }
    __device__ static C cvt(__half v, float inv) { return __half2float(v) * inv; }
    __device__ static void st(__half* p, C v, float sc) { *p = __float2half_rn(v * sc); }
};
template <>
struct St<__nv_bfloat16> {
    using C = float;
    static constexpr bool SHIFT = true;
    static constexpr bool SCALED = true;
    __device__ static C cvt_s(__nv_bfloat16 v) { return __bfloat162float(v); }
    __device__ static void st_s(__nv_bfloat16* p, C v) { *p = __float2bfloat16_rn(v); }
    __device__ static void st_sr_s(__nv_bfloat16* p, C v, unsigned r) {
        *p = __float2bfloat16_rz(__uint_as_float(__float_as_uint(v) + (r >> 16)));
    }
    __device__ static unsigned pack_sr(float a, float b, unsigned r) {
        unsigned d;
        asm("cvt.rs.bf16x2.f32 %0, %1, %2, %3;" : "=r"(d) : "f"(a), "f"(b), "r"(r));
        return d;
    }
    __device__ static void st_bits(__nv_bfloat16* p, unsigned short v) {
        *p = __ushort_as_bfloat16(v);
    }
    __device__ static C ld(const __nv_bfloat16* p, float inv) {
        return __bfloat162float(__ldg(p)) * inv;
    }
    __device__ static __nv_bfloat16 raw(const __nv_bfloat16* p) { return __ldcg(p); }
    __device__ static __nv_bfloat16 raw_rw(const __nv_bfloat16* p) { return *p; }
    __device__ static void st_sr(__nv_bfloat16* p, C v, float sc, unsigned r) {
        *p = __float2bfloat16_rz(__uint_as_float(__float_as_uint(v * sc) + (r >> 16)));
    }
    __device__ static C cvt(__nv_bfloat16 v, float inv) { return __bfloat162float(v) * inv; }
    __device__ static void st(__nv_bfloat16* p, C v, float sc) { *p = __float2bfloat16_rn(v * sc); }
};

// ----------------------------------------------------- bounds checking --
// Built with MGLC_BOUNDS_CHECK (mglc_gb300/build.py, environment variable of
// the same name), every global access of the cell bodies below checks its
// element index against its array's extent; an index outside is counted
// (per translation unit, read by the host through mglc_debug_bounds_hits)
// and the access is skipped: a diagnostic build that cannot fault on a bad
// index.  Without the macro the checks compile to nothing.
#ifdef MGLC_BOUNDS_CHECK
static __device__ unsigned long long g_oob_hits;
template <typename IDX>
__device__ __forceinline__ bool oob(IDX idx, IDX limit) {
    if ((long long)idx < 0 || idx >= limit) {
        atomicAdd(&g_oob_hits, 1ull);
        return true;
    }
    return false;
}
#define MGLC_OOB_READER(NAME)                                                  \
    extern "C" unsigned long long NAME() {                                     \
        unsigned long long h = 0;                                              \
        if (cudaMemcpyFromSymbol(&h, mglc::g_oob_hits, sizeof h) != cudaSuccess) {\
            cudaGetLastError();                                                \
            return ~0ull;                                                      \
        }                                                                      \
        return h;                                                              \
    }
#else
template <typename IDX>
__device__ __forceinline__ bool oob(IDX, IDX) {
    return false;
}
#define MGLC_OOB_READER(NAME)
#endif
// checked store p[idx] = v (skipped when idx is outside [0, limit))
template <typename T, typename V, typename IDX>
__device__ __forceinline__ void st_chk(T* p, IDX idx, IDX limit, V v) {
    if (!oob(idx, limit)) p[idx] = v;
}

// No cell of the warp touches a wall?  Asked of the warp, not of the cell: the
// lanes of a warp that has one take the general stores together (an address
// selected per population); apart, the warp stores twice, as a quarter of the
// warps of a 256-cell row did.  us a step, apart and together: FP16 with stochastic
// rounding 256^3 322 / 295, FP32 256^3 407 / 391, 97^3 28.4 / 26.6, heated 128^3
// 77.3 / 72.0, FP64 32^3 8.5 / 6.5, 384^3 3349 / 3265, heated 128^3 235 / 237.
__device__ __forceinline__ bool warp_interior(unsigned bm) {
    return !__any_sync(__activemask(), bm != 0);
}

// Reciprocal of the density (rho is within a few percent of 1 in every
// cavity flow).  FP32: the hardware reciprocal; FP64: recip64.
__device__ __forceinline__ float recip(float x) { return __frcp_rn(x); }
__device__ __forceinline__ double recip(double x) { return recip64(x); }

// Minimum resident blocks of 128 threads per SM for the lid step kernels.  The
// FP64 kernels, on the integer pipe, ran best at 5 (100 registers): 384^3 in
// 3309 us a step, 3348 at 6 and 3557 at 4 (most populations converted back on
// the FP64 unit); the other forms keep the compiler's choice (0: no bound; a
// bound of 12 or 16 blocks slowed the 16-bit kernels by 7-30%).
template <typename S>
struct LidMinBlocks {
    static constexpr int value = std::is_same<S, double>::value ? 5 : 0;
};

// and for the heated cavity's (128^3 FP64: 205 us a step at 4, 211 at 3, 234 at 5)
template <typename S>
struct ThermalMinBlocks {
    static constexpr int value = std::is_same<S, double>::value ? 4 : 0;
};

// Scalar constants converted once on the host to the arithmetic type.
template <typename C>
struct StepK {
    int nx, ny, nz;
    C u0, rho0;
    float scale, inv_scale;
    unsigned seed;  // one-solve kernels: the step index (stochastic rounding)
    int sr;         // 1: 16-bit stores round stochastically, 0: to nearest
    MrtCoef<C> c;
    // thermal
    C gbeta, omega_rot, t_ref, para_a, qd, qnu, chot, ccold;
    int bc_y, bc_z;
    PairK<C> pk;  // FP64 only
};

template <typename C>
inline StepK<C> make_k(const Geom& g, const MrtCoef<double>& cd, double u0, double rho0,
                       float scale, float inv_scale) {
    StepK<C> k{};
    k.nx = g.nx; k.ny = g.ny; k.nz = g.nz;
    k.u0 = (C)u0; k.rho0 = (C)rho0;
    k.scale = scale; k.inv_scale = inv_scale;
    k.c = cast_coef<C>(cd);
    k.pk = make_pair_k<C>(cd.snu, 2.0 * cd.lo);
    return k;
}

// The range box of FX64: |f| < 1, 1/4 <= rho < 2, |u| < 1/2; a cell outside it,
// or holding a NaN or an infinity, writes NaN.
__device__ __forceinline__ bool out_of_box(double rho, double ux, double uy, double uz) {
    return !(rho >= 0.25 && rho < 2.0 && fabs(ux) < 0.5 && fabs(uy) < 0.5 && fabs(uz) < 0.5);
}
template <int N>
__device__ __forceinline__ bool beyond_one(const double (&f)[N]) {  // |f| >= 1, or not finite
    unsigned worst = 0;
#pragma unroll
    for (int q = 0; q < N; q++) worst = max(worst, (unsigned)__double2hiint(f[q]) & 0x7fffffffu);
    return worst >= 0x3FF00000u;
}
// A density that is not finite makes every population NaN (each takes a term with
// rho, and u is NaN); said here, not computed, as a diverged solve is all such cells.
__device__ __forceinline__ bool not_finite(double r) {
    return ((unsigned)__double2hiint(r) & 0x7ff00000u) == 0x7ff00000u;
}
template <int N>
__device__ __forceinline__ void set_nan(double (&f)[N]) {
#pragma unroll
    for (int q = 0; q < N; q++) f[q] = __longlong_as_double(0x7ff8000000000000LL);
}

// Face mask of a cell: bit 0/1 = low/high x face, 2/3 = y, 4/5 = z.
__device__ __forceinline__ unsigned face_mask(int i, int j, int k, int nx, int ny, int nz) {
    return (unsigned)(i == 0) | ((unsigned)(i == nx - 1) << 1) | ((unsigned)(j == 0) << 2) |
           ((unsigned)(j == ny - 1) << 3) | ((unsigned)(k == 0) << 4) |
           ((unsigned)(k == nz - 1) << 5);
}
// does direction (dx,dy,dz) leave the domain from a cell with face mask m
__host__ __device__ constexpr unsigned leave_bits(int dx, int dy, int dz) {
    return (dx < 0 ? 1u : 0u) | (dx > 0 ? 2u : 0u) | (dy < 0 ? 4u : 0u) | (dy > 0 ? 8u : 0u) |
           (dz < 0 ? 16u : 0u) | (dz > 0 ? 32u : 0u);
}

// Uniform bits for the stochastic rounding of 16-bit stores: one integer
// hash (lowbias32 finaliser) of (cell, step) per cell, then the high bits of
// its product with a distinct odd constant per population.
__device__ __forceinline__ unsigned sr_hash(unsigned x) {
    x ^= x >> 16;
    x *= 0x7FEB352Du;
    x ^= x >> 15;
    x *= 0x846CA68Bu;
    x ^= x >> 16;
    return x;
}
__device__ __forceinline__ unsigned sr_cell(unsigned cell, unsigned step) {
    return sr_hash(cell * 0x9E3779B1u ^ sr_hash(step + 0x632BE5ABu));
}
__device__ __forceinline__ unsigned sr_pop(unsigned h, int q) {
    return h * (0x2545F491u + 2u * 0x9E3779B9u * (unsigned)q);
}
// Random bits of population pair p (populations 2p and 2p+1, rounded by one
// cvt.rs): the cell hash times a distinct odd constant per pair, plus its
// high half so that the low 16 bits depend on every bit of the hash.
__device__ __forceinline__ unsigned sr_pair(unsigned h, unsigned hh, int p) {
    return h * (0x2545F491u + 2u * 0x9E3779B9u * (unsigned)p) + hh;
}
constexpr int NPAIR19 = (Q19 + 1) / 2;

// Stochastically rounded 16-bit words of f[19], two populations per
// conversion (population 2p in the high half of w[p], 2p+1 in the low half).
template <typename S, typename C>
__device__ __forceinline__ void sr_pack19(const C (&f)[Q19], unsigned cell, unsigned seed,
                                          unsigned (&w)[NPAIR19]) {
    const unsigned h0 = sr_cell(cell, seed), hh = h0 >> 16;
#pragma unroll
    for (int p = 0; p < NPAIR19; p++)
        w[p] = St<S>::pack_sr(f[2 * p], 2 * p + 1 < Q19 ? f[2 * p + 1] : C(0), sr_pair(h0, hh, p));
}
__device__ __forceinline__ unsigned short sr_half(const unsigned (&w)[NPAIR19], int q) {
    return (unsigned short)((q & 1) ? (w[q >> 1] & 0xFFFFu) : (w[q >> 1] >> 16));
}

// ------------------------------------------------------------ lid kernel --
// IDX: 32-bit element indices when Q*cells < 2^31, 64-bit otherwise.
// lid_cell_from: collide and push one cell whose 19 stored populations are
// already in registers (raw); lid_cell: load them, then the same.  SR: the
// 16-bit stores round stochastically (a compile-time choice, so the
// round-to-nearest kernels carry none of its code).
//
// In-place (AA) pattern, one population buffer: an even step reads the
// cell's own slots and writes each post-collision population q into the
// cell's own slot opp(q) (SWAP_STORE); an odd step reads population q from
// slot opp(q) of the upstream cell x - e_q (or, when that cell is outside,
// from the cell's own slot q, which the even step filled with the reflected
// value) and writes like the push kernel, into slot q of x + e_q or, at a
// wall, into the cell's own slot opp(q).  Every slot is read and then written
// by one thread only, so a step needs no second buffer.  Wall reflections
// and the lid term are applied when a population is written, with that
// step's rho, exactly as in the push kernel: the arithmetic, and so every
// bit of the result, is the push kernel's.  After an odd step the buffer
// holds the post-stream populations (the push layout); after an even step a
// pairwise swap (k_aa_swap) restores that layout.
template <typename S, bool FIRST, typename IDX, bool SR = false, bool SWAP_STORE = false>
__device__ __forceinline__ void lid_cell_from(int i, int j, int k, const S (&raw)[Q19],
                                              S* __restrict__ fout,
                                              const StepK<typename St<S>::C>& K, IDX P,
                                              const double* mrho,
                                              const double* mu,
                                              const double* mv,
                                              const double* mw, unsigned seed) {
    using C = typename St<S>::C;
    const int nx = K.nx, ny = K.ny, nz = K.nz;
    const IDX cell = (IDX)i + (IDX)nx * ((IDX)j + (IDX)ny * (IDX)k);
    // f, rho_m and the momenta in units of the storage scale sc (1 unless
    // SCALED); rho and u are unscaled, rhos = sc * rho
    const C sc = St<S>::SCALED ? (C)K.scale : C(1);
    C f[Q19];
#pragma unroll
    for (int q = 0; q < Q19; q++) f[q] = St<S>::cvt_s(raw[q]);
    C rho, rhos;
    if constexpr (std::is_same<S, double>::value) {
        // in range: on the integer pipe (fix61.cuh); else the FP64 pair form
        bool ok = K.pk.fix.on && fix61_ok(f);
        if (ok) {
            long long F[Q19];
#pragma unroll
            for (int q = 0; q < Q19; q++) F[q] = fix61_load(f[q]);
            FixFlow fl;
            if (FIRST)
                ok = fix61_flow<true>(F, K.pk.fix, 0, 0, 0, mrho[cell], mu[cell], mv[cell],
                                      mw[cell], fl);
            else
                ok = fix61_flow<false>(F, K.pk.fix, 0, 0, 0, 0.0, 0.0, 0.0, 0.0, fl);
            if (ok) fix61_collide<true, 0, FIRST, false>(F, K.pk.fix, fl, 0, 0, 0);
            rho = fix61_store_any(fl.r);
            fix61_store_all<10>(F, f);  // (out of range after all: the same values back)
            if (K.pk.box && rho >= 2.0) set_nan(f);
        }
        if (!ok) {
            C jx, jy, jz, ux, uy, uz;
            const bool bad = K.pk.box && beyond_one(f);
            moments0(f, rho, jx, jy, jz);
            if (!FIRST && (bad || not_finite(rho))) {
                set_nan(f);
            } else if (FIRST) {
                const double rf = rho;
                rho = mrho[cell];
                ux = mu[cell];
                uy = mv[cell];
                uz = mw[cell];
                trt_collide_lid<C, true>(f, rho, rho, ux, uy, uz, K.c, C(1), rf - rho,
                                         jx - rho * ux, jy - rho * uy, jz - rho * uz);
            } else {
                const C inv = recip(rho);
                ux = jx * inv;
                uy = jy * inv;
                uz = jz * inv;
                pair_collide_lid(f, rho, jx, jy, jz, inv, ux, uy, uz, K.pk);
            }
            if (K.pk.box && (bad || out_of_box(rho, ux, uy, uz))) set_nan(f);
        }
        rhos = rho;
    } else {
        C rho_m, ux, uy, uz, jx, jy, jz, inv;
        if (FIRST) {
            rho = (C)mrho[cell];
            ux = (C)mu[cell];
            uy = (C)mv[cell];
            uz = (C)mw[cell];
            rho_m = St<S>::SHIFT ? (rho - K.rho0) * sc : rho;
        } else {
            moments0(f, rho_m, jx, jy, jz);
            rho = St<S>::SHIFT ? K.rho0 + (St<S>::SCALED ? rho_m * (C)K.inv_scale : rho_m) : rho_m;
            inv = St<S>::SCALED ? recip(rho) * (C)K.inv_scale : recip(rho);
            ux = jx * inv;
            uy = jy * inv;
            uz = jz * inv;
        }
        rhos = St<S>::SCALED ? rho * sc : rho;
        // The pair form rounds the equilibrium itself (error ~ eps |feq|, where
        // the moment form rounds only m - meq), and that rounding leaks into the
        // conserved density and momentum step after step.  In FP64 the leak is
        // ~1e-15 relative and in the 16-bit forms far below the storage error,
        // but FP32 storage keeps 1e-7 of the FP64 result only with the moment
        // form (64^3, Re = 400, 2000 steps: velocity 4e-6 with the pair form).
        // The first step after initial or load takes rho and u from the macro
        // arrays, so the pair form adds back what its relaxation would take from
        // the conserved sums of f (zero when the arrays agree with f).
        if constexpr (std::is_same<S, float>::value) {
            mrt_collide<C, false, true>(f, rho_m, rhos, ux, uy, uz, C(0), C(0), C(0), K.c, sc);
        } else if constexpr (FIRST) {
            C rf;
            moments0(f, rf, jx, jy, jz);
            trt_collide_lid<C, true>(f, rho_m, rhos, ux, uy, uz, K.c, sc, rf - rho_m,
                                     jx - rhos * ux, jy - rhos * uy, jz - rhos * uz);
        } else {
            trt_collide_lid<C>(f, rho_m, rhos, ux, uy, uz, K.c, sc);
        }
    }
    // moving lid: f(14) = f_post(11) - rho/6*U0, f(13) = f_post(12) + rho/6*U0
    // (bounce_back.f90:77-78).  On the top layer populations 11 and 12 always
    // leave through the lid (the lid face is written last, so it wins on
    // edges); the term is applied to them before the stores.
    if (k == nz - 1) {
        const C lid = rhos / C(6) * K.u0;
        f[11] = f[11] - lid;
        f[12] = f[12] + lid;
    }
    const IDX sy = (IDX)nx, sz = (IDX)nx * (IDX)ny;
    const unsigned bm = face_mask(i, j, k, nx, ny, nz);
    unsigned w[NPAIR19];
    if constexpr (SR) sr_pack19<S>(f, (unsigned)cell, seed, w);
    auto put = [&](IDX idx, int q) {
        if (oob(idx, (IDX)Q19 * P)) return;
        if constexpr (SR) St<S>::st_bits(fout + idx, sr_half(w, q));
        else St<S>::st_s(fout + idx, f[q]);
    };
    if (SWAP_STORE) {  // in-place even step: own cell, slot opp(q)
#pragma unroll
        for (int q = 0; q < Q19; q++) put((IDX)opp19(q) * P + cell, q);
        return;
    }
    if (warp_interior(bm)) {  // every population streams
#pragma unroll
        for (int q = 0; q < Q19; q++) {
            const int dx = ex19(q), dy = ey19(q), dz = ez19(q);
            put((IDX)q * P + cell + (IDX)(dx + dy * (int)sy) + (IDX)dz * sz, q);
        }
        return;
    }
#pragma unroll
    for (int q = 0; q < Q19; q++) {
        const int dx = ex19(q), dy = ey19(q), dz = ez19(q);
        const IDX to = (bm & leave_bits(dx, dy, dz)) == 0
                           ? (IDX)q * P + cell + (IDX)(dx + dy * (int)sy) + (IDX)dz * sz
                           : (IDX)opp19(q) * P + cell;
        put(to, q);
    }
}

template <typename S, typename IDX>
__device__ __forceinline__ void lid_load(int i, int j, int k, const S* fin, int nx,
                                         int ny, IDX P, S (&raw)[Q19]) {
    const IDX cell = (IDX)i + (IDX)nx * ((IDX)j + (IDX)ny * (IDX)k);
#pragma unroll
    for (int q = 0; q < Q19; q++) {
        const IDX idx = (IDX)q * P + cell;
        raw[q] = oob(idx, (IDX)Q19 * P) ? S() : St<S>::raw(fin + idx);
    }
}

// in-place pattern loads (plain loads: the buffer is written by the same kernel).
// ODD: population q from slot opp(q) of the upstream cell, or from the cell's
// own slot q where the upstream cell is outside the domain.
template <typename S, typename IDX, bool ODD>
__device__ __forceinline__ void lid_load_aa(int i, int j, int k, const S* f, int nx, int ny,
                                            int nz, IDX P, S (&raw)[Q19]) {
    const IDX cell = (IDX)i + (IDX)nx * ((IDX)j + (IDX)ny * (IDX)k);
    auto ldaa = [&](IDX idx) -> S { return oob(idx, (IDX)Q19 * P) ? S() : St<S>::raw_rw(f + idx); };
    if (!ODD) {
#pragma unroll
        for (int q = 0; q < Q19; q++) raw[q] = ldaa((IDX)q * P + cell);
        return;
    }
    const IDX sy = (IDX)nx, sz = (IDX)nx * (IDX)ny;
    const unsigned bm = face_mask(i, j, k, nx, ny, nz);
    if (bm == 0) {  // interior cell: every upstream cell is inside
#pragma unroll
        for (int q = 0; q < Q19; q++) {
            const int dx = ex19(q), dy = ey19(q), dz = ez19(q);
            raw[q] = ldaa((IDX)opp19(q) * P + cell - (IDX)(dx + dy * (int)sy) -
                                        (IDX)dz * sz);
        }
        return;
    }
#pragma unroll
    for (int q = 0; q < Q19; q++) {
        const int dx = ex19(q), dy = ey19(q), dz = ez19(q);
        if ((bm & leave_bits(-dx, -dy, -dz)) != 0)
            raw[q] = ldaa((IDX)q * P + cell);
        else
            raw[q] = ldaa((IDX)opp19(q) * P + cell - (IDX)(dx + dy * (int)sy) -
                                        (IDX)dz * sz);
    }
}

template <typename S, bool FIRST, typename IDX, bool SR = false>
__device__ __forceinline__ void lid_cell(int i, int j, int k, const S* fin,
                                         S* __restrict__ fout, const StepK<typename St<S>::C>& K,
                                         IDX P, const double* mrho,
                                         const double* mu,
                                         const double* mv,
                                         const double* mw, unsigned seed) {
    S raw[Q19];  // every load is issued before the first conversion
    lid_load<S, IDX>(i, j, k, fin, K.nx, K.ny, P, raw);
    lid_cell_from<S, FIRST, IDX, SR>(i, j, k, raw, fout, K, P, mrho, mu, mv, mw, seed);
}

// -------------------------------------------------------- thermal kernel --
// Temperature populations are kept in the arithmetic type (FP64, or FP32 for
// the reduced forms): g_0 ~ 0.7 T has a 16-bit ulp (~2e-4) far above the
// per-step diffusive increments, so 16-bit g would stagnate.
// thermal_cell_from: collide and push one cell whose populations and carried
// force are already loaded (f converted to the arithmetic type, g, fp =
// F_x, F_y, F_z of the previous step; load_carried); SWAP_STORE: the in-place
// even step (own cell, slot opp(q), reflected and anti-bounce-back values
// formed as the push kernel forms them).  thermal_cell: load, then the same.
// The carried force is loaded with the populations, not where it is used: a
// load left inside the cell body has been issued only after the population
// loads were consumed in some builds (a second memory round trip per cell,
// halving the 16-bit forms' speed).
template <typename C, bool ROT, typename IDX>
__device__ __forceinline__ void load_carried(const C* F, IDX P, IDX cell, IDX fz_off,
                                             C (&fp)[3]) {
    fp[0] = fp[1] = C(0);
    if (ROT) {
        fp[0] = oob(P + cell, (IDX)3 * P) ? C(0) : F[cell];
        fp[1] = oob(P + cell, (IDX)3 * P) ? C(0) : F[P + cell];
    }
    fp[2] = oob(fz_off + cell, fz_off + P) ? C(0) : F[fz_off + cell];
}

template <typename S, bool FIRST, bool ROT, typename IDX, bool SR = false, bool SWAP_STORE = false>
__device__ __forceinline__ void thermal_cell_from(
    int i, int j, int k, typename St<S>::C (&f)[Q19], typename St<S>::C (&g)[Q7],
    const typename St<S>::C (&fp)[3], S* __restrict__ fout, typename St<S>::C* __restrict__ gout,
    typename St<S>::C* __restrict__ F, const StepK<typename St<S>::C>& K, IDX P,
    const double* mrho, const double* mu, const double* mv,
    const double* mw, const double* mT, IDX fz_off, unsigned seed) {
    // F holds F_x, F_y at planes 0 and 1 (rotation only) and F_z at element offset fz_off
    using C = typename St<S>::C;
    const int nx = K.nx, ny = K.ny, nz = K.nz;
    const IDX cell = (IDX)i + (IDX)nx * ((IDX)j + (IDX)ny * (IDX)k);
    // f (as loaded by the caller), rho_m and the momenta in units of the
    // storage scale sc (1 unless SCALED); rho, u, T and the carried force are
    // unscaled
    const C sc = St<S>::SCALED ? (C)K.scale : C(1);
    const C fxp = fp[0], fyp = fp[1], fzp = fp[2];  // carried from the previous step
    auto force = [&](C rho, C ux, C uy, C temp, C& fx, C& fy, C& fz) {
        // body force from (rho,u,T) of the previous macro (bouyancy3d_mpi.F90:743-745)
        fx = fy = C(0);
        if (ROT) {
            fx = C(-2) * rho * uy * K.omega_rot;
            fy = C(2) * rho * ux * K.omega_rot;
            if (!oob(P + cell, (IDX)3 * P)) {
                F[cell] = fx;
                F[P + cell] = fy;
            }
        }
        fz = rho * K.gbeta * (temp - K.t_ref);
        if (!oob(fz_off + cell, fz_off + P)) F[fz_off + cell] = fz;
    };
    if constexpr (std::is_same<S, double>::value) {
        // in range on the integer pipe (fix61.cuh), else the FP64 pair forms
        constexpr int FO = ROT ? 2 : 1;
        const double small = 0.125;
        double temp;
        long long G[Q7], T = 0;
        HeatUnit hu;
        bool hot = !FIRST && K.pk.heat.on && fix_heat_unit(g, K.pk.heat, hu);
        if (hot) {
#pragma unroll
            for (int q = 0; q < Q7; q++) {
                G[q] = fix_heat_load(g[q], hu);
                T += G[q];
            }
            hot = T < (1LL << 61) && -T < (1LL << 61);
            temp = fix_heat_store(T, hu);
        } else {
            temp = FIRST ? mT[cell] : ((g[0] + g[1]) + (g[2] + g[3])) + ((g[4] + g[5]) + g[6]);
        }
        double rho, ux, uy, uz, fx, fy, fz;
        bool ok = K.pk.fix.on && fix61_ok(f) && fabs(fxp) < small && fabs(fyp) < small &&
                  fabs(fzp) < small, bad = false, none = false;
        long long L[Q19];
        FixFlow fl;
        if (ok) {
#pragma unroll
            for (int q = 0; q < Q19; q++) L[q] = fix61_load(f[q]);
            if (FIRST) {
                ok = fix61_flow<true>(L, K.pk.fix, 0, 0, 0, mrho[cell], mu[cell], mv[cell],
                                      mw[cell], fl);
            } else {
                const double h = 0.5 * FIX_ONE;
                ok = fix61_flow<false>(L, K.pk.fix, ROT ? __double2ll_rn(fxp * h) : 0,
                                       ROT ? __double2ll_rn(fyp * h) : 0, __double2ll_rn(fzp * h),
                                       0.0, 0.0, 0.0, 0.0, fl);
            }
        }
        if (ok) {
            rho = fix61_store_any(fl.r);
            if (FIRST || ROT || K.pk.box || !hot) {
                ux = FIRST ? mu[cell] : fix61_store_any<63>(join(fl.ux));
                uy = FIRST ? mv[cell] : fix61_store_any<63>(join(fl.uy));
                uz = FIRST ? mw[cell] : fix61_store_any<63>(join(fl.uz));
            } else {
                ux = uy = uz = 0.0;  // used as integers only
            }
        } else if (FIRST) {
            rho = mrho[cell];
            ux = mu[cell];
            uy = mv[cell];
            uz = mw[cell];
        } else {
            moments0(f, rho, ux, uy, uz);
            none = not_finite(rho);
            const double inv = none ? rho - rho : recip(rho);  // (NaN)
            // u^n = (sum f e + F^n/2)/rho^n with the force carried from the previous step
            ux = (ux + 0.5 * fxp) * inv;
            uy = (uy + 0.5 * fyp) * inv;
            uz = (uz + 0.5 * fzp) * inv;
        }
        force(rho, ux, uy, temp, fx, fy, fz);
        if (ok && fabs(fx) < small && fabs(fy) < small && fabs(fz) < small) {
            fix61_collide<false, FO, FIRST, true>(
                L, K.pk.fix, fl, ROT ? __double2ll_rn(fx * FIX_ONE) : 0,
                ROT ? __double2ll_rn(fy * FIX_ONE) : 0, __double2ll_rn(fz * FIX_ONE));
            fix61_store_all<5>(L, f);
        } else if (none) {
            bad = true;
            set_nan(f);
        } else {
            bad = beyond_one(f);
            double rf, jx, jy, jz;
            moments0(f, rf, jx, jy, jz);
            if (!FIRST && ok) {  // (a force of 1/8 or more)
                ux = fix61_store_any<63>(join(fl.ux));
                uy = fix61_store_any<63>(join(fl.uy));
                uz = fix61_store_any<63>(join(fl.uz));
            }
            if (FIRST) {
                // rho, u from the macro arrays: the odd term is e.(2 (j - rho u) + F)/10
                // and the density projection goes back in (trt_collide_forced)
                trt_collide_forced<C, ROT, true>(f, rho, rho, ux, uy, uz, fx, fy, fz,
                                                 fx + 2.0 * (jx - rho * ux),
                                                 fy + 2.0 * (jy - rho * uy),
                                                 fz + 2.0 * (jz - rho * uz), K.c, rf - rho);
            } else {
                pair_collide_forced<ROT>(f, rho, jx + 0.5 * fxp, jy + 0.5 * fyp,
                                               jz + 0.5 * fzp, ux, uy, uz, fx, fy, fz, fx - fxp,
                                               fy - fyp, fz - fzp, K.pk);
            }
        }
        if (K.pk.box) {  // FX64's range box, with |g| and |T| below 2
#pragma unroll
            for (int q = 0; q < Q7; q++) bad |= !(fabs(g[q]) < 2.0);
            bad = bad || !(fabs(temp) < 2.0) || out_of_box(rho, ux, uy, uz);
        }
        if (K.pk.box && bad) {
            set_nan(f);
            set_nan(g);
        } else if (ok && hot) {
            fix_heat(G, T, K.pk.heat, fl);
#pragma unroll
            for (int q = 0; q < Q7; q++) g[q] = fix_heat_store(G[q], hu);
        } else if (FIRST) {
            const double sg = ((g[0] + g[1]) + (g[2] + g[3])) + ((g[4] + g[5]) + g[6]);
            trt_collide_t<C, true>(g, temp, ux, uy, uz, K.para_a, K.qd, K.qnu, sg - temp);
        } else {
            pair_collide_t(g, temp, ux, uy, uz, K.pk);
        }
    } else {
        C rho_m, rho, ux, uy, uz, temp, jx, jy, jz;
        if (FIRST) {
            rho = (C)mrho[cell];
            ux = (C)mu[cell];
            uy = (C)mv[cell];
            uz = (C)mw[cell];
            temp = (C)mT[cell];
            rho_m = St<S>::SHIFT ? (rho - K.rho0) * sc : rho;
        } else {
            moments0(f, rho_m, jx, jy, jz);
            if (St<S>::SCALED) {
                jx = jx * (C)K.inv_scale;
                jy = jy * (C)K.inv_scale;
                jz = jz * (C)K.inv_scale;
            }
            rho = St<S>::SHIFT ? K.rho0 + (St<S>::SCALED ? rho_m * (C)K.inv_scale : rho_m) : rho_m;
            const C inv = recip(rho);
            // u^n = (sum f e + F^n/2)/rho^n with the force carried from the previous step
            ux = (jx + C(0.5) * fxp) * inv;
            uy = (jy + C(0.5) * fyp) * inv;
            uz = (jz + C(0.5) * fzp) * inv;
            temp = ((g[0] + g[1]) + (g[2] + g[3])) + ((g[4] + g[5]) + g[6]);
        }
        C fx, fy, fz;
        force(rho, ux, uy, temp, fx, fy, fz);
        // the pair form where its equilibrium rounding stays below the storage
        // error (the 16-bit forms; see lid_cell_from)
        if constexpr (std::is_same<S, float>::value) {
            mrt_collide<C, true, false>(f, rho_m, rho, ux, uy, uz, fx, fy, fz, K.c);
        } else if constexpr (FIRST) {
            // rho, u from the macro arrays, as above
            C rf;
            moments0(f, rf, jx, jy, jz);
            const C rhos = rho * sc;
            trt_collide_forced<C, ROT, true>(
                f, rho_m, rhos, ux, uy, uz, fx * sc, fy * sc, fz * sc,
                fx * sc + C(2) * (jx - rhos * ux), fy * sc + C(2) * (jy - rhos * uy),
                fz * sc + C(2) * (jz - rhos * uz), K.c, rf - rho_m);
        } else {
            trt_collide_forced<C, ROT>(f, rho_m, rho * sc, ux, uy, uz, fx * sc, fy * sc, fz * sc,
                                       (fx - fxp) * sc, (fy - fyp) * sc, (fz - fzp) * sc, K.c);
        }
        // D3Q7: the FP32 temperature populations of the reduced forms keep the
        // moment form (its rounding does not leak into the conserved sum of g; see
        // lid_cell_from for the FP32 measurement)
        mrt_collide_t<C>(g, temp, ux, uy, uz, K.para_a, K.qd, K.qnu);
    }

    const IDX sy = (IDX)nx, sz = (IDX)nx * (IDX)ny;
    const unsigned bm = face_mask(i, j, k, nx, ny, nz);
    unsigned w[NPAIR19];
    if constexpr (SR) sr_pack19<S>(f, (unsigned)cell, seed, w);
    auto put = [&](IDX idx, int q) {
        if (oob(idx, (IDX)Q19 * P)) return;
        if constexpr (SR) St<S>::st_bits(fout + idx, sr_half(w, q));
        else St<S>::st_s(fout + idx, f[q]);
    };
    if (SWAP_STORE) {  // in-place even step: own cell, slot opp(q)
#pragma unroll
        for (int q = 0; q < Q19; q++) put((IDX)opp19(q) * P + cell, q);
#pragma unroll
        for (int q = 0; q < Q7; q++) {
            const int dy = ey19(q), dz = ez19(q);
            C val = g[q];
            if ((bm & leave_bits(ex19(q), dy, dz)) != 0) {
                if (dy != 0 && K.bc_y) val = -val + (dy < 0 ? K.chot : K.ccold);
                if (dz != 0 && K.bc_z) val = -val + (dz < 0 ? K.chot : K.ccold);
            }
            st_chk(gout, (IDX)((IDX)opp19(q) * P + cell), (IDX)Q7 * P, val);
        }
        return;
    }
    if (warp_interior(bm)) {
#pragma unroll
        for (int q = 0; q < Q19; q++) {
            const int dx = ex19(q), dy = ey19(q), dz = ez19(q);
            put((IDX)q * P + cell + (IDX)(dx + dy * (int)sy) + (IDX)dz * sz, q);
        }
#pragma unroll
        for (int q = 0; q < Q7; q++) {
            const int dx = ex19(q), dy = ey19(q), dz = ez19(q);
            st_chk(gout, (IDX)((IDX)q * P + cell + (IDX)(dx + dy * (int)sy) + (IDX)dz * sz), (IDX)Q7 * P, g[q]);
        }
        return;
    }
#pragma unroll
    for (int q = 0; q < Q19; q++) {
        const int dx = ex19(q), dy = ey19(q), dz = ez19(q);
        const IDX to = (bm & leave_bits(dx, dy, dz)) == 0
                           ? (IDX)q * P + cell + (IDX)(dx + dy * (int)sy) + (IDX)dz * sz
                           : (IDX)opp19(q) * P + cell;
        put(to, q);
    }
    // D3Q7: adiabatic walls reflect, constant-T walls anti-bounce-back
    // g_in = -g_out + (6+paraA)/21 * T_wall (bouyancy3d_mpi.F90:1101-1210)
#pragma unroll
    for (int q = 0; q < Q7; q++) {
        const int dx = ex19(q), dy = ey19(q), dz = ez19(q);
        IDX to = (IDX)((IDX)q * P + cell + (IDX)(dx + dy * (int)sy) + (IDX)dz * sz);
        C val = g[q];
        if ((bm & leave_bits(dx, dy, dz)) != 0) {
            if (dy != 0 && K.bc_y) val = -val + (dy < 0 ? K.chot : K.ccold);
            if (dz != 0 && K.bc_z) val = -val + (dz < 0 ? K.chot : K.ccold);
            to = (IDX)((IDX)opp19(q) * P + cell);
        }
        st_chk(gout, to, (IDX)Q7 * P, val);
    }
}


template <typename S, bool FIRST, bool ROT, typename IDX, bool SR = false>
__device__ __forceinline__ void thermal_cell(
    int i, int j, int k, const S* fin, S* __restrict__ fout,
    const typename St<S>::C* gin, typename St<S>::C* __restrict__ gout,
    typename St<S>::C* __restrict__ F, const StepK<typename St<S>::C>& K, IDX P,
    const double* mrho, const double* mu, const double* mv,
    const double* mw, const double* mT, IDX fz_off, unsigned seed) {
    using C = typename St<S>::C;
    const IDX cell = (IDX)i + (IDX)K.nx * ((IDX)j + (IDX)K.ny * (IDX)k);
    // every load is issued before the first conversion (as in lid_cell):
    // left to itself the scheduler has interleaved them with the arithmetic
    // in some builds of the 16-bit forms, halving their speed
    S raw[Q19];
    C f[Q19], g[Q7], fp[3];
#pragma unroll
    for (int q = 0; q < Q19; q++)
        raw[q] = oob((IDX)q * P + cell, (IDX)Q19 * P) ? S() : St<S>::raw(fin + ((IDX)q * P + cell));
#pragma unroll
    for (int q = 0; q < Q7; q++)
        g[q] = oob((IDX)q * P + cell, (IDX)Q7 * P) ? C(0) : St<C>::raw(gin + ((IDX)q * P + cell));
    load_carried<C, ROT, IDX>(F, P, cell, fz_off, fp);
#pragma unroll
    for (int q = 0; q < Q19; q++) f[q] = St<S>::cvt_s(raw[q]);
    thermal_cell_from<S, FIRST, ROT, IDX, SR>(i, j, k, f, g, fp, fout, gout, F, K, P, mrho, mu,
                                              mv, mw, mT, fz_off, seed);
}

// in-place pattern loads of a heated-cavity cell (plain loads; ODD: from the
// upstream cells' opposite slots, or the own slot where upstream is outside)
template <typename S, typename IDX, bool ODD, bool ROT = false>
__device__ __forceinline__ void thermal_load_aa(int i, int j, int k, const S* f,
                                                const typename St<S>::C* g,
                                                const typename St<S>::C* F, IDX fz_off,
                                                const StepK<typename St<S>::C>& K, IDX P,
                                                typename St<S>::C (&fv)[Q19],
                                                typename St<S>::C (&gv)[Q7],
                                                typename St<S>::C (&fp)[3]) {
    const int nx = K.nx, ny = K.ny, nz = K.nz;
    const IDX cell = (IDX)i + (IDX)nx * ((IDX)j + (IDX)ny * (IDX)k);
    const IDX sy = (IDX)nx, sz = (IDX)nx * (IDX)ny;
    const unsigned bm = face_mask(i, j, k, nx, ny, nz);
    // an interior cell (bm == 0) reads every population from upstream
    auto src = [&](int q) -> IDX {
        const int dx = ex19(q), dy = ey19(q), dz = ez19(q);
        if (!ODD || (bm != 0 && (bm & leave_bits(-dx, -dy, -dz)) != 0)) return (IDX)q * P + cell;
        return (IDX)opp19(q) * P + cell - (IDX)(dx + dy * (int)sy) - (IDX)dz * sz;
    };
    S raw[Q19];
#pragma unroll
    for (int q = 0; q < Q19; q++) raw[q] = oob(src(q), (IDX)Q19 * P) ? S() : St<S>::raw_rw(f + src(q));
    // g through L2 only (ld.global.cg, coherent): measured 1.3x faster for the
    // stochastically rounded 16-bit form, neutral for the others
#pragma unroll
    for (int q = 0; q < Q7; q++)
        gv[q] = oob(src(q), (IDX)Q7 * P) ? typename St<S>::C(0) : __ldcg(g + src(q));
    load_carried<typename St<S>::C, ROT, IDX>(F, P, cell, fz_off, fp);
#pragma unroll
    for (int q = 0; q < Q19; q++) fv[q] = St<S>::cvt_s(raw[q]);  // in units of the storage scale
}

}  // namespace mglc
