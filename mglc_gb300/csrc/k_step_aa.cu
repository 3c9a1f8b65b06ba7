// k_step_aa.cu -- the lid-driven cavity step in place (AA pattern): one
// population buffer instead of two, the arithmetic of the push kernel.
//
// A step alternates between two kernels (step_cell.cuh, lid_load_aa and the
// SWAP_STORE path of lid_cell_from): the even kernel reads and writes each
// cell's own slots, the odd kernel reads upstream slots and writes
// downstream ones.  k_aa_swap turns the buffer left by an even step into the
// post-stream layout (the reference's f), which getters and checkpoints read.
// Same reference routines as k_step.cu (mpi_3d_blocked/{collision.f90:15-202,
// streaming.f90:8-20, bounce_back.f90:6-83, macro.f90:6-25}).
#include "cell_map.cuh"
#include "launch.cuh"
#include "step_cell.cuh"

namespace mglc {

template <typename S, bool FIRST, typename IDX, bool SR, bool ODD, class MAP>
__global__ void __launch_bounds__(128, LidMinBlocks<S>::value)
    k_lid_step_aa(S* f, StepK<typename St<S>::C> K, MAP map, IDX P, const double* mrho,
                  const double* mu, const double* mv,
                  const double* mw) {
    after_previous();
    int i, j, k;
    if (!map.at(K.nx, K.ny, P, i, j, k)) return;
    S raw[Q19];  // every load is issued before the first store
    lid_load_aa<S, IDX, ODD>(i, j, k, f, K.nx, K.ny, K.nz, P, raw);
    lid_cell_from<S, FIRST, IDX, SR, !ODD>(i, j, k, raw, f, K, P, mrho, mu, mv, mw, K.seed);
}

// Heated cavity in place: flow and temperature populations each on one
// buffer; the carried force is the cell's own (read, then written).
template <typename S, bool FIRST, bool ROT, typename IDX, bool SR, bool ODD, class MAP>
__global__ void __launch_bounds__(128, ThermalMinBlocks<S>::value)
    k_thermal_step_aa(S* f, typename St<S>::C* g, typename St<S>::C* __restrict__ F,
                      StepK<typename St<S>::C> K, MAP map, IDX P, const double* mrho,
                      const double* mu, const double* mv,
                      const double* mw, const double* mT) {
    after_previous();
    using C = typename St<S>::C;
    int i, j, k;
    if (!map.at(K.nx, K.ny, P, i, j, k)) return;
    C fv[Q19], gv[Q7], fp[3];  // every load is issued before the first store
    thermal_load_aa<S, IDX, ODD, ROT>(i, j, k, f, g, F, (IDX)2 * P, K, P, fv, gv, fp);
    thermal_cell_from<S, FIRST, ROT, IDX, SR, !ODD>(i, j, k, fv, gv, fp, f, g, F, K, P, mrho, mu,
                                                    mv, mw, mT, (IDX)2 * P, K.seed);
}

// Pairwise exchange (q, x) <-> (opp(q), x - e_q) for the directions with
// opp(q) > q (nine of D3Q19, three of D3Q7): the streaming half of a step,
// without collision.  The pair is owned by the thread of x, so the exchange
// is race-free; where x - e_q is outside, slot q of x already holds the
// reflected population.
template <typename S, int Q, typename IDX, class MAP>
__global__ void __launch_bounds__(128) k_aa_swap(S* f, int nx, int ny, int nz, MAP map, IDX P) {
    after_previous();
    int i, j, k;
    if (!map.at(nx, ny, P, i, j, k)) return;
    const IDX cell = (IDX)i + (IDX)nx * ((IDX)j + (IDX)ny * (IDX)k);
    const IDX sy = (IDX)nx, sz = (IDX)nx * (IDX)ny;
    const unsigned bm = face_mask(i, j, k, nx, ny, nz);
#pragma unroll
    for (int q = 1; q < Q; q++) {
        if (opp19(q) < q) continue;
        const int dx = ex19(q), dy = ey19(q), dz = ez19(q);
        if ((bm & leave_bits(-dx, -dy, -dz)) != 0) continue;
        const IDX ia = (IDX)q * P + cell;
        const IDX ib = (IDX)opp19(q) * P + cell - (IDX)(dx + dy * (int)sy) - (IDX)dz * sz;
        if (oob(ia, (IDX)Q * P) || oob(ib, (IDX)Q * P)) continue;
        S* a = f + ia;
        S* b = f + ib;
        const S t = *a;
        *a = *b;
        *b = t;
    }
}

namespace {

template <typename S>
cudaError_t lid_go_aa(bool first, bool odd, void* f, const LidStepArgs& a, cudaStream_t s,
                      bool box = false) {
    using C = typename St<S>::C;
    StepK<C> K = make_k<C>(a.g, a.cd, a.u0, a.rho0, a.scale, a.inv_scale);
    set_box(K.pk, box);
    K.seed = a.seed;
    K.sr = a.sr;
    const CellLaunch l(a.g);
    const bool small = index32(a.g);
    constexpr bool kHalf = sizeof(S) == 2;  // stochastic rounding: 16-bit storage only
    const bool sr = kHalf && a.sr;
    S* fp = (S*)f;
#define AA_LAUNCH(FI, IT, SRV, OD, MAP)                                       \
    launch_next(k_lid_step_aa<S, FI, IT, SRV, OD, MAP>, l.grid, l.block, 0, s,   \
        fp, K, MAP(a.g), (IT)a.g.plane, a.rho, a.u, a.v, a.w)
#define AA_PICK(IT, MAP)                                                   \
    if (odd) {                                                             \
        if (sr) AA_LAUNCH(false, IT, kHalf, true, MAP);                    \
        else AA_LAUNCH(false, IT, false, true, MAP);                       \
    } else if (first) {                                                    \
        if (sr) AA_LAUNCH(true, IT, kHalf, false, MAP);                    \
        else AA_LAUNCH(true, IT, false, false, MAP);                       \
    } else {                                                               \
        if (sr) AA_LAUNCH(false, IT, kHalf, false, MAP);                   \
        else AA_LAUNCH(false, IT, false, false, MAP);                      \
    }
    if (linear_cells(a.g)) {
        AA_PICK(unsigned, CellMap)
    } else if (small) {
        AA_PICK(unsigned, RowMap)
    } else {
        AA_PICK(long long, RowMap)
    }
#undef AA_PICK
#undef AA_LAUNCH
    return cudaGetLastError();
}

template <typename S, int Q>
cudaError_t swap_go(const Geom& g, void* f, cudaStream_t s) {
    const CellLaunch l(g);
    if (linear_cells(g))
        launch_next(k_aa_swap<S, Q, unsigned, CellMap>, l.grid, l.block, 0, s, (S*)f, g.nx, g.ny, g.nz, CellMap(g), (unsigned)g.plane);
    else if (index32(g))
        launch_next(k_aa_swap<S, Q, unsigned, RowMap>, l.grid, l.block, 0, s, (S*)f, g.nx, g.ny, g.nz, RowMap(g), (unsigned)g.plane);
    else
        launch_next(k_aa_swap<S, Q, long long, RowMap>, l.grid, l.block, 0, s, (S*)f, g.nx, g.ny, g.nz, RowMap(g), (long long)g.plane);
    return cudaGetLastError();
}

template <typename S>
cudaError_t th_go_aa(bool first, bool odd, void* f, void* g, void* F, const ThermalStepArgs& a,
                     cudaStream_t s, bool box = false) {
    using C = typename St<S>::C;
    StepK<C> K = make_k<C>(a.g, a.cd, 0.0, a.rho0, a.scale, a.inv_scale);
    K.seed = a.seed;
    K.sr = a.sr;
    K.gbeta = (C)a.gbeta; K.omega_rot = (C)a.omega_rot; K.t_ref = (C)a.t_ref;
    K.para_a = (C)a.para_a; K.qd = (C)a.qd; K.qnu = (C)a.qnu;
    K.chot = (C)((6.0 + a.para_a) / 21.0 * a.t_hot);
    K.ccold = (C)((6.0 + a.para_a) / 21.0 * a.t_cold);
    K.bc_y = a.bc_y; K.bc_z = a.bc_z;
    pair_k_heat(K.pk, a.para_a, a.qd, a.qnu);
    set_box(K.pk, box);
    const CellLaunch l(a.g);
    const bool rot = a.omega_rot != 0.0;
    const bool small = index32(a.g);
    constexpr bool kHalf = sizeof(S) == 2;
    const bool sr = kHalf && a.sr;
    S* fp = (S*)f;
    C* gp = (C*)g;
    C* Fp = (C*)F;
#define TA_LAUNCH(FI, RO, IT, SRV, OD, MAP)                                      \
    launch_next(k_thermal_step_aa<S, FI, RO, IT, SRV, OD, MAP>, l.grid, l.block, 0, s,    \
        fp, gp, Fp, K, MAP(a.g), (IT)a.g.plane, a.rho, a.u, a.v, a.w, a.T)
#define TA_SR(FI, RO, IT, OD, MAP)                        \
    do {                                                  \
        if (sr) TA_LAUNCH(FI, RO, IT, kHalf, OD, MAP);    \
        else TA_LAUNCH(FI, RO, IT, false, OD, MAP);       \
    } while (0)
#define TA_PICK(RO, IT, MAP)                              \
    if (odd) TA_SR(false, RO, IT, true, MAP);             \
    else if (first) TA_SR(true, RO, IT, false, MAP);      \
    else TA_SR(false, RO, IT, false, MAP);
    if (linear_cells(a.g)) {
        if (rot) { TA_PICK(true, unsigned, CellMap) } else { TA_PICK(false, unsigned, CellMap) }
    } else if (small) {
        if (rot) { TA_PICK(true, unsigned, RowMap) } else { TA_PICK(false, unsigned, RowMap) }
    } else {
        if (rot) { TA_PICK(true, long long, RowMap) } else { TA_PICK(false, long long, RowMap) }
    }
#undef TA_PICK
#undef TA_SR
#undef TA_LAUNCH
    return cudaGetLastError();
}

}  // namespace

// first: the step reads the stored macroscopic fields (after initial/load; the
// layout is then the post-stream one, so first implies an even step)
cudaError_t launch_lid_step_aa(int form, bool first, bool odd, void* f, const LidStepArgs& a,
                               cudaStream_t s) {
    if (first && odd) return cudaErrorInvalidValue;
    switch (form) {
        case FORM_FX64: return lid_go_aa<double>(first, odd, f, a, s, true);
        case FORM_FP64: return lid_go_aa<double>(first, odd, f, a, s);
        case FORM_FP32: return lid_go_aa<float>(first, odd, f, a, s);
        case FORM_FP16: return lid_go_aa<__half>(first, odd, f, a, s);
        case FORM_BF16: return lid_go_aa<__nv_bfloat16>(first, odd, f, a, s);
    }
    return cudaErrorInvalidValue;
}

cudaError_t launch_thermal_step_aa(int form, bool first, bool odd, void* f, void* g, void* F,
                                   const ThermalStepArgs& a, cudaStream_t s) {
    if (first && odd) return cudaErrorInvalidValue;
    switch (form) {
        case FORM_FX64: return th_go_aa<double>(first, odd, f, g, F, a, s, true);
        case FORM_FP64: return th_go_aa<double>(first, odd, f, g, F, a, s);
        case FORM_FP32: return th_go_aa<float>(first, odd, f, g, F, a, s);
        case FORM_FP16: return th_go_aa<__half>(first, odd, f, g, F, a, s);
        case FORM_BF16: return th_go_aa<__nv_bfloat16>(first, odd, f, g, F, a, s);
    }
    return cudaErrorInvalidValue;
}

// g (heated cavity): D3Q7 populations in the arithmetic type (FP64 or FP32)
cudaError_t launch_aa_swap(int form, const Geom& g, void* f, void* gt, cudaStream_t s) {
    cudaError_t e = cudaErrorInvalidValue;
    switch (form) {
        case FORM_FP64: e = swap_go<double, Q19>(g, f, s); break;
        case FORM_FP32: e = swap_go<float, Q19>(g, f, s); break;
        case FORM_FP16: e = swap_go<__half, Q19>(g, f, s); break;
        case FORM_BF16: e = swap_go<__nv_bfloat16, Q19>(g, f, s); break;
    }
    if (e != cudaSuccess || !gt) return e;
    return form == FORM_FP64 ? swap_go<double, Q7>(g, gt, s) : swap_go<float, Q7>(g, gt, s);
}

}  // namespace mglc

MGLC_OOB_READER(mglc_oob_hits_k_step_aa)
