// k_step.cu -- fused lattice-Boltzmann step kernels (lid and thermal cavities).
//
// One thread per lattice cell, push scheme: a thread reads its own cell's
// post-stream populations (coalesced SoA loads), derives rho and u (the
// reference macro), collides, and writes each post-collision population to
// the neighbour it streams to.  Populations that would leave the domain are
// reflected in place (halfway bounce-back), which replaces the reference's
// halo exchange + bounceback sweep; the moving-lid term uses the cell's own
// rho, which is the reference's rho(i,j,nz) from the previous macro().
//
// Reference routines fused here (paths relative to the MGLC repository):
//   lid:     mpi_3d_blocked/{collision.f90:15-202, streaming.f90:8-20,
//            bounce_back.f90:6-83, macro.f90:6-25}
//   thermal: bouyancy3d_mpi.F90 collision :641-864, streaming :867-892,
//            bounceback :895-983, collisionT :1014-1070, streamingT :1073-1098,
//            bouncebackT :1101-1210, macro :986-1010, macroT :1215-1231
#include "cell_map.cuh"
#include "launch.cuh"
#include "step_cell.cuh"

namespace mglc {

template <typename S, bool FIRST, typename IDX, bool SR, class MAP>
__global__ void __launch_bounds__(128, LidMinBlocks<S>::value)
    k_lid_step(const S* fin, S* __restrict__ fout, StepK<typename St<S>::C> K,
               MAP map, IDX P, const double* mrho, const double* mu,
               const double* mv, const double* mw) {
    after_previous();
    int i, j, k;
    if (!map.at(K.nx, K.ny, P, i, j, k)) return;
    lid_cell<S, FIRST, IDX, SR>(i, j, k, fin, fout, K, P, mrho, mu, mv, mw, K.seed);
}

template <typename S, bool FIRST, bool ROT, typename IDX, bool SR, class MAP>
__global__ void __launch_bounds__(128, ThermalMinBlocks<S>::value)
    k_thermal_step(const S* fin, S* __restrict__ fout,
                   const typename St<S>::C* gin, typename St<S>::C* __restrict__ gout,
                   typename St<S>::C* __restrict__ F, StepK<typename St<S>::C> K, MAP map, IDX P,
                   const double* mrho, const double* mu,
                   const double* mv, const double* mw,
                   const double* mT) {
    after_previous();
    int i, j, k;
    if (!map.at(K.nx, K.ny, P, i, j, k)) return;
    thermal_cell<S, FIRST, ROT, IDX, SR>(i, j, k, fin, fout, gin, gout, F, K, P, mrho, mu, mv, mw,
                                         mT, (IDX)2 * P, K.seed);
}

// --------------------------------------------------------------- launch --
template <typename S>
static cudaError_t lid_go(bool first, const void* fin, void* fout, const LidStepArgs& a,
                          cudaStream_t s, bool box = false) {
    using C = typename St<S>::C;
    StepK<C> K = make_k<C>(a.g, a.cd, a.u0, a.rho0, a.scale, a.inv_scale);
    set_box(K.pk, box);
    K.seed = a.seed;
    K.sr = a.sr;
    const CellLaunch l(a.g);
    const bool small = index32(a.g);
    // stochastic rounding exists for the 16-bit storage types only
    constexpr bool kHalf = sizeof(S) == 2;
#define LID_LAUNCH(FI, IT, SRV, MAP)                                                              \
    launch_next(k_lid_step<S, FI, IT, SRV, MAP>, l.grid, l.block, 0, s, (const S*)fin, (S*)fout, K, MAP(a.g), \
                                                               (IT)a.g.plane, a.rho, a.u, a.v, a.w)
#define LID_SR(FI, IT, MAP)                              \
    if (kHalf && a.sr) LID_LAUNCH(FI, IT, kHalf, MAP);   \
    else LID_LAUNCH(FI, IT, false, MAP);
    if (linear_cells(a.g)) {
        if (first) { LID_SR(true, unsigned, CellMap) } else { LID_SR(false, unsigned, CellMap) }
    } else if (small) {
        if (first) { LID_SR(true, unsigned, RowMap) } else { LID_SR(false, unsigned, RowMap) }
    } else {
        if (first) { LID_SR(true, long long, RowMap) } else { LID_SR(false, long long, RowMap) }
    }
#undef LID_SR
#undef LID_LAUNCH
    return cudaGetLastError();
}

cudaError_t launch_lid_step(int form, bool first, const void* fin, void* fout,
                            const LidStepArgs& a, cudaStream_t s) {
    switch (form) {
        case FORM_FX64: return lid_go<double>(first, fin, fout, a, s, true);
        case FORM_FP64: return lid_go<double>(first, fin, fout, a, s);
        case FORM_FP32: return lid_go<float>(first, fin, fout, a, s);
        case FORM_FP16: return lid_go<__half>(first, fin, fout, a, s);
        case FORM_BF16: return lid_go<__nv_bfloat16>(first, fin, fout, a, s);
    }
    return cudaErrorInvalidValue;
}

template <typename S>
static cudaError_t th_go(bool first, const void* fin, void* fout, const void* gin, void* gout,
                         void* F, const ThermalStepArgs& a, cudaStream_t s, bool box = false) {
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
#define TH_LAUNCH2(FI, RO, IT, SRV, MAP)                                                     \
    launch_next(k_thermal_step<S, FI, RO, IT, SRV, MAP>, l.grid, l.block, 0, s,                \
        (const S*)fin, (S*)fout, (const C*)gin, (C*)gout, (C*)F, K, MAP(a.g), (IT)a.g.plane, \
        a.rho, a.u, a.v, a.w, a.T)
#define TH_LAUNCH(FI, RO, IT, MAP)                              \
    do {                                                        \
        if (kHalf && a.sr) TH_LAUNCH2(FI, RO, IT, kHalf, MAP);  \
        else TH_LAUNCH2(FI, RO, IT, false, MAP);                \
    } while (0)
#define TH_ROT(IT, MAP)                                  \
    if (first && rot) TH_LAUNCH(true, true, IT, MAP);     \
    else if (first) TH_LAUNCH(true, false, IT, MAP);      \
    else if (rot) TH_LAUNCH(false, true, IT, MAP);        \
    else TH_LAUNCH(false, false, IT, MAP);
    if (linear_cells(a.g)) {
        TH_ROT(unsigned, CellMap)
    } else if (small) {
        TH_ROT(unsigned, RowMap)
    } else {
        TH_ROT(long long, RowMap)
    }
#undef TH_ROT
#undef TH_LAUNCH
#undef TH_LAUNCH2
    return cudaGetLastError();
}

cudaError_t launch_thermal_step(int form, bool first, const void* fin, void* fout,
                                const void* gin, void* gout, void* F, const ThermalStepArgs& a,
                                cudaStream_t s) {
    switch (form) {
        case FORM_FX64: return th_go<double>(first, fin, fout, gin, gout, F, a, s, true);
        case FORM_FP64: return th_go<double>(first, fin, fout, gin, gout, F, a, s);
        case FORM_FP32: return th_go<float>(first, fin, fout, gin, gout, F, a, s);
        case FORM_FP16: return th_go<__half>(first, fin, fout, gin, gout, F, a, s);
        case FORM_BF16: return th_go<__nv_bfloat16>(first, fin, fout, gin, gout, F, a, s);
    }
    return cudaErrorInvalidValue;
}

}  // namespace mglc

MGLC_OOB_READER(mglc_oob_hits_k_step)
