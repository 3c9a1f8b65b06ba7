// k_particle2d.cu -- D2Q9 moving circles, the reference's case4 step
// (MPI/Micro_particles/fortran/case4/mpi_particle, main.F90:35-73) and, as the
// P2_SHEAR variant, its case1 step (MPI/Micro_particles/fortran/case1/
// mpi_complete, main.F90:34-67: a circle carried through the shear between
// two moving walls, periodic in x, both compile-time frames and both
// interpolation orders).  The case4 routines are:
//
//   collision (fluid.F90:14-64, solid nodes skipped), streaming from fluid
//   sources (:97-108), four halfway-bounce-back walls (:115-161),
//   bounceback_particle (particle_bounceback.F90:15-97, calQ :101-141 or
//   calQ2 :144-185), macro (fluid.F90:164-184), calForce (particle_force.F90:
//   35-190), updateCenter and refill (particle_update.F90:26-193).
//
// Layout: one plane per population with two ghost layers each side, the
// reference's arrays (-1..nx+2 filled with omega*rho0; one more zero layer).
// Everything is FP64 and this file is compiled without FMA contraction, so
// each expression rounds as the reference's statement does (d2q9.cuh writes
// the collision with fewer operations that give the same bits).  Steps whose
// order matters in the reference keep its loop order: the density averages
// are exact parallel replays of the sequential sum (the k_gs_* kernels), each
// circle's link terms are evaluated one per thread and added in loop order,
// and the refill sweep refills its sorted node list on one thread; the rest
// is one thread per node or per link.
//
// One step (8 launches and two density averages of two each):
//   k2_collide      every fluid node but the ones that just     context stream
//                   left a circle
//   gs              the average over the new mask: its first    side stream,
//                   kernel lists the nodes that left a circle,  beside k2_collide
//                   its last block refills and collides them
//   gs              the average for the bounce-back             side stream
//   k2_stream       pull, walls, and macro where no neighbour is solid; the
//                   other fluid nodes are listed; the next mask cleared
//   k2_boundary     a block per listed node: calQ, the interpolated bounce-back
//                   and momentum exchange of its links, then its macro
//   k2_force        a block per circle; the last one moves the circles
//   k2_mark         the new mask, a block per circle
// The first average belongs to the previous step's end; only a node that left
// a circle needs it, so the other nodes collide meanwhile (the last step of a
// call runs it before the call returns).
// FP64 instructions are dear here (a warp's instruction takes the FP64 unit
// for 16 clocks or more, whether one lane is active or 32), so what is chained
// or scattered is compacted first and decided on integers.
// Case4 at 400x800 with three circles: 1118 us a step before (19 launches:
// the node-wise collision 210, the averages 2 x 140, bounce-back 187 and links
// 169 with calQ's bisections one after another in a thread, the forces 203 on
// one warp a circle), 198 us now: k2_collide 64 (FP64 pipe), k2_stream 24,
// k2_boundary 17, k2_force 29 (190 dependent adds at ~90 clocks), k2_mark 7; the
// two averages, 7 + 32 each, run beside k2_collide and k2_stream.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>

#include "mglc.h"
#include "d2q9.cuh"
#include "launch.cuh"
#include "particles2d.cuh"

namespace mglc {

namespace {

__device__ __constant__ int c_ex[9] = {0, 1, 0, -1, 0, 1, -1, -1, 1};
__device__ __constant__ int c_ey[9] = {0, 0, 1, 0, -1, 1, 1, -1, -1};
__device__ __constant__ int c_r[9] = {0, 3, 4, 1, 2, 7, 8, 5, 6};
__device__ __constant__ double c_w[9] = {4.0 / 9.0, 1.0 / 9.0, 1.0 / 9.0, 1.0 / 9.0, 1.0 / 9.0,
                                         1.0 / 36.0, 1.0 / 36.0, 1.0 / 36.0, 1.0 / 36.0};

// what a listed boundary node keeps: the owner of each of its eight links, and
// each link's F_x, F_y and torque.  Any fluid node may be listed (circles of one
// node three apart list eight of nine), so the arrays hold every node.
constexpr int NODE_LINKS = 8, LINK_TERMS = 3, NODE_TERMS = NODE_LINKS * LINK_TERMS;

enum { S_NO_OWNER = 1, S_Q = 2, S_OVERLAP = 3, S_WALL = 4, S_NO_DIR = 5 };

// Records of one ordered density sum (GsPiece below): per chunk of addends its
// plain partial sum and count, then its pieces and their number.
struct GsPiece;
struct GsBuf {
    double* part;
    int* cnt;
    GsPiece* piece;  // GS_PIECES per chunk
    int* np;         // pieces of a chunk; 0: it has to be added the plain way
    unsigned* done;  // blocks that have finished (k_gs_map)
};

struct D2 {
    P2Params p;
    int X;      // padded row length nx + 6
    size_t C;   // padded cells: elements between population planes
    int par;    // which of the two mask buffers ob is
    double *f, *fp, *rho, *u, *v;
    int *ob, *on;  // solid mask of this step, and the next one's (swapped every step)
    double *xc, *uc, *om, *xco, *uco, *omo, *force, *torque;  // np x 3
    double* ravg;  // average density: [0] over ob (bounce-back, forces), [1] over on (refill)
    int* status;   // [0] code, [1] particle, [2] mask buffer that holds the frozen state's mask
    // fluid nodes with a solid neighbour (k2_stream): their list, each node's
    // place in it (-1: not listed), and per (place, direction 1..8) the first
    // circle that owns the link's solid end (-1: no link) with its momentum
    // exchange F_x, F_y, torque
    int *bl_list, *bl_pos, *lc;
    double* lt;
    unsigned* done;           // [0] blocks of k2_force that have finished, [1] length of bl_list
    int *rf_count, *rf_list;  // nodes to refill: count, list of RF_CAP
    GsBuf ga, gb;             // the two averages
};

__device__ __forceinline__ int IX(const D2& d, int i, int j) { return (i + 2) + d.X * (j + 2); }
__device__ __forceinline__ double& F(const D2& d, int a, int i, int j) { return d.f[a * d.C + IX(d, i, j)]; }
__device__ __forceinline__ double& FP(const D2& d, int a, int i, int j) { return d.fp[a * d.C + IX(d, i, j)]; }
__device__ __forceinline__ double sq(double x) { return x * x; }

// ((x - xc)^2 + (y - yc)^2) <= R^2 (particle_bounceback.F90:50-52)
__device__ __forceinline__ bool inside(const D2& d, const double* cen, int c, double x, double y) {
    const double r = d.p.radius;
    return sq(x - cen[3 * c]) + sq(y - cen[3 * c + 1]) <= sq(r);
}

// par: the buffer that holds the mask the state is frozen with (before the
// circles move, this step's; in the refill, the new one)
__device__ void fail(const D2& d, int code, int c, int par) {
    if (atomicCAS(d.status, 0, code) == 0) {
        d.status[1] = c;
        d.status[2] = par;
    }
}

// Has a step failed?  One answer for the whole block, so that it leaves together:
// other blocks of the same launch may be setting the status, and warps that read it
// late would leave the others to barriers and shared values that they never wrote.
// (Counters that such a block does not advance are reset by p2d_initial; until then
// the state is frozen.)
__device__ __forceinline__ bool stopped(const D2& d) { return __syncthreads_or(d.status[0]); }

// x index of a population read: case1 is periodic in x (its MPI exchange
// fills the ghost columns with the periodic partner's values); case4 reads
// its own ghost columns
__device__ __forceinline__ int wxi(const D2& d, int i) {
    if (d.p.variant != P2_SHEAR) return i;
    return i < 1 ? i + d.p.nx : (i > d.p.nx ? i - d.p.nx : i);
}

// ------------------------------------------------------------------ fluid --
// rho, u, v of a fluid node are the previous macro's (or the initial fields)
template <bool GROUPED>
__device__ __forceinline__ void collide_node(const D2& d, int c) {
    double f[9], fp[9];
#pragma unroll
    for (int a = 0; a < 9; a++) f[a] = d.f[a * d.C + c];
    double r = d.rho[c], u = d.u[c], v = d.v[c];
    d2q9_collide<GROUPED, false>(f, r, u, v, d.p.snu, d.p.sq, fp);
#pragma unroll
    for (int a = 0; a < 9; a++) d.fp[a * d.C + c] = fp[a];
}
// refilling: nodes that left a circle in the last step (solid in the mask that
// on still holds) are being refilled beside this kernel, and collided there
template <bool GROUPED>
__global__ void __launch_bounds__(128) k2_collide(D2 d, bool refilling) {
    after_previous();
    const int i = 1 + blockIdx.x * blockDim.x + threadIdx.x, j = 1 + blockIdx.y;
    if (i > d.p.nx || d.status[0]) return;
    const int c = IX(d, i, j);
    if (d.ob[c] != 0 || (refilling && d.on[c] != 0)) return;
    collide_node<GROUPED>(d, c);
}

constexpr int e2x(int a) { return a == 1 || a == 5 || a == 8 ? 1 : (a == 3 || a == 6 || a == 7 ? -1 : 0); }
constexpr int e2y(int a) { return a == 2 || a == 5 || a == 6 ? 1 : (a == 4 || a == 7 || a == 8 ? -1 : 0); }
constexpr int r2(int a) { return a == 0 ? 0 : (a <= 4 ? (a + 1) % 4 + 1 : (a - 3) % 4 + 5); }

// Pull from fluid sources (every interior node, fluid or solid, receives; case1
// wraps the source column, fluid.F90:105-110); a population that would come
// from beyond a wall is the node's own reflected one (the four walls of case4,
// :115-161, where a corner gets the same value from both of its walls; the two
// moving walls of case1, :127-169).  A fluid node with no solid neighbour then
// takes its macro from the nine values in registers; one with a solid neighbour
// is listed for k2_boundary.  Bound by the loads and stores of the two
// population sets and by macro's FP64 quotients; fusing the three sweeps saves
// reading the populations again (400x800: 26 + 8 + 40 us as three kernels).
template <bool SHEAR>
__global__ void __launch_bounds__(128) k2_stream(D2 d) {
    after_previous();
    const int i = 1 + blockIdx.x * blockDim.x + threadIdx.x, j = 1 + blockIdx.y;
    if (i > d.p.nx || d.status[0]) return;
    const int nx = d.p.nx, ny = d.p.ny, c = IX(d, i, j);
    // the next step's mask, cleared with the ghosts that k2_mark may set
    d.on[c] = 0;
    if (i == 1 || i == nx || j == 1 || j == ny) {
        const int gi = i == 1 ? 0 : nx + 1, gj = j == 1 ? 0 : ny + 1;
        if (i == 1 || i == nx) d.on[IX(d, gi, j)] = 0;
        if (j == 1 || j == ny) d.on[IX(d, i, gj)] = 0;
        if ((i == 1 || i == nx) && (j == 1 || j == ny)) d.on[IX(d, gi, gj)] = 0;
    }
    double g[9];
    bool near = false;
#pragma unroll
    for (int a = 0; a < 9; a++) {
        int ip = i - e2x(a);
        const int jp = j - e2y(a);
        bool wall = jp < 1 || jp > ny;
        if (SHEAR) ip = wxi(d, ip);
        else wall = wall || ip < 1 || ip > nx;
        const int src = IX(d, ip, jp);
        const bool solid = d.ob[src] != 0;
        near = near || solid;
        // case1's links look at the ghost column itself, which the source wraps
        if (SHEAR && ip != i - e2x(a)) near = near || d.ob[IX(d, i - e2x(a), jp)] != 0;
        if (wall) {
            double val = FP(d, r2(a), i, j);
            if (SHEAR && e2x(a) != 0) {
                const double uw = d.p.uwall, u0 = d.p.u0;
                if (e2y(a) > 0) {  // bottom wall, moving at -uwall
                    const double t = (d.p.moving_frame ? -uw - u0 : -uw) / 6.0;
                    val = a == 5 ? val + t : val - t;
                } else {
                    const double t = (d.p.moving_frame ? uw - u0 : uw) / 6.0;
                    val = a == 7 ? val - t : val + t;
                }
            }
            g[a] = val;
            d.f[a * d.C + c] = val;
        } else if (!solid) {
            g[a] = d.fp[a * d.C + src];
            d.f[a * d.C + c] = g[a];
        } else {
            g[a] = 0.0;  // not used: near
        }
    }
    if (d.ob[c] != 0 || !near) d.bl_pos[c] = -1;
    if (d.ob[c] != 0) return;
    if (near) {
        const int pos = (int)atomicAdd(d.done + 1, 1u);
        d.bl_list[pos] = (j - 1) * nx + (i - 1);
        d.bl_pos[c] = pos;
        return;
    }
    double r, u, v;
    d2q9_macro(g, r, u, v);
    d.rho[c] = r;
    d.u[c] = u;
    d.v[c] = v;
}

// Sequential FP64 sums computed in parallel, bit for bit.  While the running
// sum s stays inside one binade [2^E, 2^(E+1)) and the addends are finite and
// non-negative, s is an integer S times u = 2^(E-52) with S in [2^52, 2^53),
// and RN(s + x) = (S + k) u where k is x/u rounded to an integer: down below
// one half, up above it, and on an exact half to the k that makes S + k even
// (ties to even).  Only the tie case reads the running sum, and only its
// parity, so an addend is a map from the incoming parity to (increment,
// outgoing parity); maps compose associatively, and an ordered tree reduction
// of a chunk's maps gives the chunk's sum.  A chunk that may leave the binade
// (or holds a negative or non-finite addend) is added one element at a time.
struct GridSeg {
    long long i0, i1;  // increment in units of u for incoming parity 0 / 1
    int o0, o1;        // outgoing parity for incoming parity 0 / 1
};

__device__ __forceinline__ GridSeg seg_identity() { return GridSeg{0, 0, 0, 1}; }

// a followed by b
__device__ __forceinline__ GridSeg seg_cat(const GridSeg& a, const GridSeg& b) {
    GridSeg r;
    r.i0 = a.i0 + (a.o0 ? b.i1 : b.i0);
    r.o0 = a.o0 ? b.o1 : b.o0;
    r.i1 = a.i1 + (a.o1 ? b.i1 : b.i0);
    r.o1 = a.o1 ? b.o1 : b.o0;
    return r;
}

__device__ __forceinline__ GridSeg seg_shfl_down(const GridSeg& g, int off) {
    GridSeg r;
    r.i0 = __shfl_down_sync(0xffffffffu, g.i0, off);
    r.i1 = __shfl_down_sync(0xffffffffu, g.i1, off);
    r.o0 = __shfl_down_sync(0xffffffffu, g.o0, off);
    r.o1 = __shfl_down_sync(0xffffffffu, g.o1, off);
    return r;
}

// ordered reduction over a warp: lane 0 ends with lane 0's map, then lane 1's, ...
__device__ __forceinline__ GridSeg seg_warp_reduce(GridSeg g) {
    for (int off = 1; off < 32; off <<= 1) {
        const GridSeg o = seg_shfl_down(g, off);
        if ((threadIdx.x & 31) + off < 32 && ((threadIdx.x & 31) & (2 * off - 1)) == 0)
            g = seg_cat(g, o);
    }
    return g;
}

constexpr long long MANT52 = (1LL << 52) - 1;
constexpr int NO_BINADE = 100000;

// the map of addend x (bits xb) on the grid of binade e (u = 2^(e-52)), from
// the bit pattern with integer operations only; false when x must be added the
// plain way (sign bit set, infinite or NaN, or x >= 2^(e+1)).  ub is an upper
// bound of the increment.
__device__ __forceinline__ bool seg_of(long long xb, int e, GridSeg& g, long long& ub) {
    if (xb < 0) return false;
    const int ex = (int)(xb >> 52);
    if (ex == 2047) return false;
    const long long M = (xb & MANT52) | (ex ? (1LL << 52) : 0);  // x = M 2^(max(ex,1)-1075)
    const int sh = max(ex, 1) - 1023 - e;                         // x / u = M 2^sh
    if (sh > 0) return false;
    long long m;
    int cls = 0;  // fraction of x / u: 0 below one half, 1 above, 2 exactly one half
    if (sh == 0) {
        m = M;
    } else if (sh >= -62) {
        const int k = -sh;
        m = M >> k;
        const long long rem = M & ((1LL << k) - 1), half = 1LL << (k - 1);
        cls = rem > half ? 1 : (rem == half ? 2 : 0);
    } else {
        m = 0;  // x < u / 2
    }
    if (cls == 2) {
        g.i0 = m + (m & 1);
        g.i1 = m + ((m + 1) & 1);
        g.o0 = g.o1 = 0;
        ub = m + 1;
    } else {
        const long long v = m + cls;
        g.i0 = g.i1 = v;
        g.o0 = (int)(v & 1);
        g.o1 = (int)((v + 1) & 1);
        ub = v;
    }
    return true;
}

// binade of a positive normal running sum, NO_BINADE when the grid path is off
// (integer tests only: one FP64 compare holds a warp for 64 cycles here)
__device__ __forceinline__ int binade_of(double acc) {
    const long long b = __double_as_longlong(acc);
    const int e = (int)((b >> 52) & 0x7ff) - 1023;
    return (b > 0 && e >= -900 && e <= 1000) ? e : NO_BINADE;
}

// acc + (the addends whose composed map is h and increment bound hb) on binade
// e; false when the sum may leave the binade
__device__ __forceinline__ bool grid_apply(double& acc, int e, const GridSeg& h, long long hb) {
    const long long S = (__double_as_longlong(acc) & MANT52) | (1LL << 52);
    if (!(hb < (1LL << 53) - S)) return false;
    const long long S1 = S + ((S & 1) ? h.i1 : h.i0);
    acc = __longlong_as_double(((long long)(e + 1023) << 52) | (S1 & MANT52));
    return true;
}

__device__ __forceinline__ long long warp_incl_scan(long long x) {
    const int lane = threadIdx.x & 31;
    for (int off = 1; off < 32; off <<= 1) {
        const long long y = __shfl_up_sync(0xffffffffu, x, off);
        if (lane >= off) x += y;
    }
    return x;
}

__device__ __forceinline__ GridSeg seg_select(bool keep, const GridSeg& g) {
    return keep ? g : seg_identity();
}

// Warp 0 adds the addends [lo, hi) of sr (where sm is set) to acc (held by
// lane 0) in order, 32 at a time: the lanes up to the first addend that cannot
// take the grid path of the current binade (it is not finite and non-negative,
// or the sum may leave the binade) are added as one map, that addend the plain
// way, and the rest start over on the new binade.
__device__ void warp_sum_pieces(const double* sr, const unsigned char* sm, int lo, int hi,
                                double& acc) {
    const int lane = threadIdx.x & 31;
    for (int p = lo; p < hi; p += 32) {
        int lstart = 0;
        while (lstart < 32) {
            const double a0 = __shfl_sync(0xffffffffu, acc, 0);
            const int ep = binade_of(a0);
            const long long S = ep == NO_BINADE ? 0 : (__double_as_longlong(a0) & MANT52) | (1LL << 52);
            const int q = p + lane;
            const bool valid = lane >= lstart && q < hi && sm[q];
            GridSeg g = seg_identity();
            long long ub = 0;
            bool bad = false;
            if (valid) bad = ep == NO_BINADE || !seg_of(__double_as_longlong(sr[q]), ep, g, ub);
            const long long incl = warp_incl_scan(ub);
            const bool ok = !bad && (ep == NO_BINADE || incl < (1LL << 53) - S);
            const unsigned nb = __ballot_sync(0xffffffffu, !ok);
            const int lstar = nb ? __ffs(nb) - 1 : 32;
            const GridSeg h = seg_warp_reduce(seg_select(lane < lstar, g));
            const long long hb = __shfl_sync(0xffffffffu, incl, lstar > 0 ? lstar - 1 : 0);
            if (lane == 0) {
                if (ep != NO_BINADE && lstar > 0) grid_apply(acc, ep, h, hb);
                if (lstar < 32) acc = acc + sr[p + lstar];
            }
            lstart = lstar + 1;
        }
    }
}

// The sequential sum x_0 + x_1 + ... over the addends t = 0..total-1 that a
// fetch functor keeps (fetch(t, keep, x)), with the rounding of that order,
// in chunks of CH addends (EPT consecutive addends per thread of an SB-thread
// block):
//   k_gs_part  (one block per chunk) plain partial sums (any order) and counts;
//   k_gs_map   (one block per chunk) from the sum of the partial sums before
//              it, an estimate of the running sum at each addend (in fixed
//              point: integer adds are cheap here, FP64 ones are not): an
//              addend where the estimate enters a new binade, or that cannot
//              take the grid path, ends a piece of the chunk.  A piece is the
//              composed grid map of the addends before that one, with its
//              increment bound, and the addend itself, to be added the plain
//              way; a segmented scan composes all pieces of a warp at once.
//              The last block to finish then walks the pieces in order
//              (gs_walk): a piece whose binade is the exact running sum's and
//              whose bound keeps the sum in it is added as its map; a chunk
//              with any other piece, or with more than GS_PIECES of them, is
//              added by chunk_split.  Estimates decide only how fast it is.
// The pieces matter because the sum of n densities near 1 enters about log2 n
// binades: re-adding the eight chunks of 400x800 that hold one (and the twelve
// in the first chunk) with chunk_split took 121 of an average's 140 us; the
// average takes 39 now.
// chunk_split adds one chunk with the whole block: the warps up to the first
// one holding an addend that cannot take the grid path of the current binade
// are added as one map, that warp's addends by warp 0 (warp_sum_pieces), and
// the rest start over on the new binade.
constexpr int SB = 1024;  // threads of the ordered sweeps (one block)
constexpr int EPT = 4;    // addends per thread and chunk
constexpr int CH = SB * EPT;
constexpr long long UB_CAP = 1LL << 61;  // saturation of chunk increment bounds

struct SumShared {
    double sr[CH];
    unsigned char sm[CH];  // 1 = kept
    GridSeg wseg[SB / 32];
    long long wub[SB / 32];
    int wbad[SB / 32];
    double acc;  // the running sum
    int next;
};

constexpr int GS_PIECES = 16;  // pieces of one chunk that are kept
constexpr int GS_GROUP = 256;  // chunks walked from shared memory at a time, at most
constexpr int GS_WALK = 512;   // and pieces of them
constexpr int RF_CAP = 4096;   // nodes that the refill sorts in shared memory

struct GsPiece {
    GridSeg m;     // the map of the addends before x, on binade e
    long long ub;  // bound of its increment
    double x;      // the addend that ends the piece
    int e;         // binade of m; NO_BINADE when there is no addend before x
    int has;       // x is there (in the walk: bit 1, first of its chunk; chunk << 2)
};

union GsShared {
    SumShared sum;
    GsPiece walk[GS_WALK];
    struct {
        GridSeg seg[GS_PIECES][SB / 32];
        long long ub[GS_PIECES][SB / 32];
    } map;
    int keys[RF_CAP];  // the refill's sorted list
};

// adds the chunk at base (this thread's addends fc/xc) to sh.acc; all threads
// call it; it ends with a barrier
__device__ void chunk_split(int base, int total, const bool (&fc)[EPT], const double (&xc)[EPT],
                            SumShared& sh) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int u = 0; u < EPT; u++) {
        sh.sm[threadIdx.x * EPT + u] = fc[u];
        sh.sr[threadIdx.x * EPT + u] = xc[u];
    }
    int startw = 0;
    for (;;) {
        const int e = binade_of(sh.acc);
        GridSeg g = seg_identity();
        long long ub = 0;  // at most 128 bounds below 2^53 per warp: no overflow
        bool bad = false;
        if (w >= startw) {
#pragma unroll
            for (int u = 0; u < EPT; u++) {
                if (!fc[u] || bad) continue;
                GridSeg gu;
                long long bu;
                if (e != NO_BINADE && seg_of(__double_as_longlong(xc[u]), e, gu, bu)) {
                    g = seg_cat(g, gu);
                    ub += bu;
                } else {
                    bad = true;
                }
            }
        }
        g = seg_warp_reduce(g);
        for (int off = 16; off > 0; off >>= 1) ub += __shfl_down_sync(0xffffffffu, ub, off);
        const int wb = __any_sync(0xffffffffu, bad);
        if (lane == 0) {
            sh.wseg[w] = g;
            sh.wub[w] = ub;
            sh.wbad[w] = wb;
        }
        __syncthreads();
        if (w == 0) {
            double acc = sh.acc;
            const long long S = e == NO_BINADE ? 0 : (__double_as_longlong(acc) & MANT52) | (1LL << 52);
            // the prefix grows by at most 2^60 a lane, so it cannot wrap before
            // the first lane past the bound, and only lanes before that are used
            const long long incl = warp_incl_scan(sh.wub[lane]);
            const bool ok = lane < startw ||
                            (!sh.wbad[lane] && e != NO_BINADE && incl < (1LL << 53) - S);
            const unsigned nb = __ballot_sync(0xffffffffu, !ok);
            const int wstar = nb ? __ffs(nb) - 1 : 32;
            const GridSeg h = seg_warp_reduce(seg_select(lane < wstar, sh.wseg[lane]));
            const long long hb = __shfl_sync(0xffffffffu, incl, wstar > 0 ? wstar - 1 : 0);
            if (lane == 0 && e != NO_BINADE && wstar > startw) grid_apply(acc, e, h, hb);
            if (wstar < 32) {
                const int lo = wstar * 32 * EPT;
                warp_sum_pieces(sh.sr, sh.sm, lo, min(lo + 32 * EPT, total - base), acc);
            }
            if (lane == 0) {
                sh.acc = acc;
                sh.next = wstar >= 31 ? 32 : wstar + 1;
            }
        }
        __syncthreads();
        startw = sh.next;
        if (startw >= 32) break;
    }
}

template <class Fetch>
__global__ void __launch_bounds__(SB) k_gs_part(Fetch fetch, int total, GsBuf b) {
    after_previous();
    __shared__ double ws[SB / 32];
    __shared__ int wc[SB / 32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, c = blockIdx.x;
    double v = 0.0;
    int n = 0;
#pragma unroll
    for (int u = 0; u < EPT; u++) {
        bool fl;
        double x;
        const int t = c * CH + threadIdx.x * EPT + u;
        fetch(t, fl, x);
        fetch.visit(t, fl);
        if (fl) {
            v += x;
            n++;
        }
    }
    for (int off = 16; off > 0; off >>= 1) {
        v += __shfl_down_sync(0xffffffffu, v, off);
        n += __shfl_down_sync(0xffffffffu, n, off);
    }
    if (lane == 0) {
        ws[w] = v;
        wc[w] = n;
    }
    __syncthreads();
    if (w == 0) {
        v = ws[lane];
        n = wc[lane];
        for (int off = 16; off > 0; off >>= 1) {
            v += __shfl_down_sync(0xffffffffu, v, off);
            n += __shfl_down_sync(0xffffffffu, n, off);
        }
        if (lane == 0) {
            b.part[c] = v;
            b.cnt[c] = n;
        }
    }
}

// The ordered walk, by one whole block: the sum (returned to every thread) and
// the number of kept addends.  One warp walks; its chain per piece is a few
// integer operations on the running sum's significand S (the loads of the next
// piece run ahead), and a plain FP64 add where a piece ends in one.
template <class Fetch>
__device__ double gs_walk(const Fetch& fetch, int total, int nch, const GsBuf& b, GsShared& sh,
                          long long& count) {
    __shared__ long long wn[SB / 32];
    __shared__ int s_off[GS_GROUP / 32];
    __shared__ double s_acc;
    __shared__ int s_next, s_fail, s_lim, s_np;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    long long n = 0;
    for (int c = threadIdx.x; c < nch; c += SB) n += __ldcg(b.cnt + c);
    for (int off = 16; off > 0; off >>= 1) n += __shfl_down_sync(0xffffffffu, n, off);
    if (lane == 0) wn[w] = n;
    if (threadIdx.x == 0) {
        s_acc = 0.0;
        s_next = 0;
    }
    __syncthreads();
    for (;;) {
        const int g0 = s_next;  // chunks before g0 are in s_acc
        if (g0 >= nch) break;
        // the pieces of the next chunks, one thread per chunk, packed in order;
        // a chunk without pieces gets one that the walk refuses
        const int c = g0 + (int)threadIdx.x;
        const bool mine = threadIdx.x < GS_GROUP && c < nch;
        const int np = mine ? __ldcg(b.np + c) : 0;
        const int room = mine ? max(np, 1) : 0;
        int incl = room;
        if (threadIdx.x < GS_GROUP) {
            for (int off = 1; off < 32; off <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, incl, off);
                if (lane >= off) incl += y;
            }
            if (lane == 31) s_off[w] = incl;
        }
        if (threadIdx.x == 0) s_lim = s_np = 0;
        __syncthreads();
        if (threadIdx.x < GS_GROUP) {
            for (int q = 0; q < w; q++) incl += s_off[q];
            if (mine && incl <= GS_WALK) {  // a prefix of the chunks
                atomicMax(&s_lim, (int)threadIdx.x + 1);
                atomicMax(&s_np, incl);
                GsPiece* dst = sh.walk + (incl - room);
                for (int q = 0; q < np; q++) {
                    const long long* from = (const long long*)(b.piece + (size_t)c * GS_PIECES + q);
                    long long* to = (long long*)(dst + q);
#pragma unroll
                    for (int k = 0; k < (int)(sizeof(GsPiece) / 8); k++) to[k] = __ldcg(from + k);
                    dst[q].has |= (q == 0 ? 2 : 0) | ((int)threadIdx.x << 2);
                }
                if (np == 0) {
                    dst->e = -NO_BINADE;
                    dst->has = 2 | ((int)threadIdx.x << 2);
                }
            }
        }
        __syncthreads();
        const int lim = s_lim;
        if (w == 0) {  // every lane walks the same sums
            double acc = s_acc;
            long long S = (__double_as_longlong(acc) & MANT52) | (1LL << 52);
            int e = binade_of(acc), fail = lim;
            long long S0 = S;  // the running sum at the start of the piece's chunk
            int e0 = e;
            double acc0 = acc;
            bool plain = true;  // acc holds the sum (S, e otherwise)
            GsPiece nx = sh.walk[0];
            const int all = s_np;
            for (int q = 0; q < all; q++) {
                const GsPiece pc = nx;
                nx = sh.walk[min(q + 1, GS_WALK - 1)];
                if (pc.has & 2) {
                    S0 = S;
                    e0 = e;
                    if (plain) acc0 = acc;
                }
                if (pc.e != NO_BINADE) {
                    if (pc.e != e || !(pc.ub < (1LL << 53) - S)) {
                        fail = pc.has >> 2;
                        break;
                    }
                    S += (S & 1) ? pc.m.i1 : pc.m.i0;
                    plain = false;
                }
                if (pc.has & 1) {
                    if (!plain)
                        acc = __longlong_as_double(((long long)(e + 1023) << 52) | (S & MANT52));
                    acc = acc + pc.x;
                    S = (__double_as_longlong(acc) & MANT52) | (1LL << 52);
                    e = binade_of(acc);
                    // outside the grid's binades only acc tells the sum
                    plain = e == NO_BINADE;
                }
            }
            if (fail < lim) {
                S = S0;
                e = e0;
                acc = acc0;
            }
            if (e != NO_BINADE) acc = __longlong_as_double(((long long)(e + 1023) << 52) | (S & MANT52));
            if (lane == 0) {
                s_acc = acc;
                s_fail = fail;
            }
        }
        __syncthreads();
        const int fc = g0 + s_fail;
        if (s_fail < lim) {
            bool f4[EPT];
            double x4[EPT];
#pragma unroll
            for (int u = 0; u < EPT; u++) fetch(fc * CH + threadIdx.x * EPT + u, f4[u], x4[u]);
            if (threadIdx.x == 0) sh.sum.acc = s_acc;
            __syncthreads();
            chunk_split(fc * CH, total, f4, x4, sh.sum);
            if (threadIdx.x == 0) {
                s_acc = sh.sum.acc;
                s_next = fc + 1;
            }
        } else if (threadIdx.x == 0) {
            s_next = g0 + lim;
        }
        __syncthreads();
    }
    long long cnt = 0;
    for (int q = 0; q < SB / 32; q++) cnt += wn[q];
    count = cnt;
    return s_acc;
}

// x in units of 2^(E - 44) (an estimate: rounded down), 0 for a negative or
// non-finite x; the sum of all addends lies in binade E
__device__ __forceinline__ long long gs_fixed(double x, int E) {
    const long long xb = __double_as_longlong(x);
    const int ex = (int)(xb >> 52);  // negative with the sign bit
    if (xb < 0 || ex == 2047 || ex == 0) return 0;
    const long long M = (xb & MANT52) | (1LL << 52);
    const int s = ex - 1031 - E;
    return s > -63 ? (s <= 0 ? M >> -s : (s <= 8 ? M << s : 0)) : 0;
}
__device__ __forceinline__ int gs_binade(long long v, int E) {
    return v > 0 ? 63 - __clzll(v) + E - 44 : NO_BINADE;
}

// pieces of this block's chunk; the last block walks them all and hands the
// sum to fetch.finish (with every thread of the block)
template <class Fetch>
__global__ void __launch_bounds__(SB) k_gs_map(Fetch fetch, int total, int nch, GsBuf b) {
    after_previous();
    if (__syncthreads_or(fetch.stop())) return;
    __shared__ GsShared sh;
    __shared__ double ws[SB / 32], wall[SB / 32], s_x[GS_PIECES];
    __shared__ long long wt[SB / 32];
    __shared__ int wr[SB / 32], s_e[GS_PIECES];
    __shared__ int s_last, s_E;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, c = blockIdx.x;
    // estimate of the running sum at the chunk's start, and of the whole sum
    if (w < min(SB / 32, (nch + 31) / 32)) {
        double v = 0.0, a = 0.0;
        for (int t = threadIdx.x; t < nch; t += SB) {
            const double y = b.part[t];
            a += y;
            if (t < c) v += y;
        }
        for (int off = 16; off > 0; off >>= 1) {
            v += __shfl_down_sync(0xffffffffu, v, off);
            a += __shfl_down_sync(0xffffffffu, a, off);
        }
        if (lane == 0) {
            ws[w] = v;
            wall[w] = a;
        }
    } else if (lane == 0) {
        ws[w] = wall[w] = 0.0;
    }
    bool fl[EPT];
    double x[EPT];
#pragma unroll
    for (int u = 0; u < EPT; u++) fetch(c * CH + threadIdx.x * EPT + u, fl[u], x[u]);
    if (threadIdx.x < GS_PIECES) s_e[threadIdx.x] = NO_BINADE;
    __syncthreads();
    if (w == 0) {
        double v = ws[lane], a = wall[lane];
        for (int off = 16; off > 0; off >>= 1) {
            v += __shfl_down_sync(0xffffffffu, v, off);
            a += __shfl_down_sync(0xffffffffu, a, off);
        }
        if (lane == 0) {
            ws[0] = v;
            s_E = binade_of(a);
        }
    }
    __syncthreads();
    const int E = s_E;
    long long own = 0;
#pragma unroll
    for (int u = 0; u < EPT; u++)
        if (fl[u]) own += gs_fixed(x[u], E);
    long long incl = warp_incl_scan(own);
    if (lane == 31) wt[w] = incl;
    __syncthreads();
    long long p = gs_fixed(ws[0], E) + (incl - own);
    for (int q = 0; q < w; q++) p += wt[q];
    // addends that end a piece, and the number of them before this thread's
    int nend = 0;
    bool end[EPT];
    int eb[EPT];
#pragma unroll
    for (int u = 0; u < EPT; u++) {
        end[u] = false;
        eb[u] = gs_binade(p, E);
        if (fl[u]) {
            p += gs_fixed(x[u], E);
            GridSeg g;
            long long ub;
            end[u] = eb[u] == NO_BINADE || gs_binade(p, E) != eb[u] ||
                     !seg_of(__double_as_longlong(x[u]), eb[u], g, ub);
        }
        nend += end[u];
    }
    int rank = nend;
    for (int off = 1; off < 32; off <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, rank, off);
        if (lane >= off) rank += y;
    }
    if (lane == 31) wr[w] = rank;
    __syncthreads();
    rank -= nend;
    int all = 0;
    for (int q = 0; q < SB / 32; q++) {
        if (q < w) rank += wr[q];
        all += wr[q];
    }
    const bool many = all > GS_PIECES - 1 || E == NO_BINADE;
    if (!many) {
        for (int k = w; k <= all; k += SB / 32) {  // pieces that a warp does not meet
            sh.map.seg[k][lane] = seg_identity();
            sh.map.ub[k][lane] = 0;
        }
        // the binade of a piece: the estimate's at one of its kept addends (the
        // same for all of them, or some do not fit it and the walk refuses it)
        int k = rank;
#pragma unroll
        for (int u = 0; u < EPT; u++) {
            if (!fl[u]) continue;
            if (end[u]) s_x[k++] = x[u];
            else s_e[k] = eb[u];
        }
        __syncthreads();
        // this thread's addends before its first end, and after its last;
        // pieces in between are whole
        GridSeg head = seg_identity(), run = seg_identity();
        long long hub = 0, rub = 0;
        k = rank;
#pragma unroll
        for (int u = 0; u < EPT; u++) {
            if (!fl[u]) continue;
            if (end[u]) {
                if (k == rank) {
                    head = run;
                    hub = rub;
                } else {
                    sh.map.seg[k][w] = run;
                    sh.map.ub[k][w] = rub;
                }
                k++;
                run = seg_identity();
                rub = 0;
                continue;
            }
            GridSeg gu;
            long long bu;
            if (seg_of(__double_as_longlong(x[u]), s_e[k], gu, bu)) {
                run = seg_cat(run, gu);
                rub += bu;
            } else {
                rub += 1LL << 54;  // more than any binade holds: the walk refuses it
            }
        }
        // segmented scan: the map since the last end before or in each lane
        // (128 bounds of at most 2^54 a warp: no overflow)
        int flag = nend > 0;
        GridSeg sc = run;
        long long su = rub;
        for (int off = 1; off < 32; off <<= 1) {
            GridSeg o;
            o.i0 = __shfl_up_sync(0xffffffffu, sc.i0, off);
            o.i1 = __shfl_up_sync(0xffffffffu, sc.i1, off);
            o.o0 = __shfl_up_sync(0xffffffffu, sc.o0, off);
            o.o1 = __shfl_up_sync(0xffffffffu, sc.o1, off);
            const long long ou = __shfl_up_sync(0xffffffffu, su, off);
            const int of = __shfl_up_sync(0xffffffffu, flag, off);
            if (lane >= off && !flag) {
                sc = seg_cat(o, sc);
                su += ou;
                flag = of;
            }
        }
        GridSeg before;
        before.i0 = __shfl_up_sync(0xffffffffu, sc.i0, 1);
        before.i1 = __shfl_up_sync(0xffffffffu, sc.i1, 1);
        before.o0 = __shfl_up_sync(0xffffffffu, sc.o0, 1);
        before.o1 = __shfl_up_sync(0xffffffffu, sc.o1, 1);
        long long bu = __shfl_up_sync(0xffffffffu, su, 1);
        if (lane == 0) {
            before = seg_identity();
            bu = 0;
        }
        if (nend > 0) {
            sh.map.seg[rank][w] = seg_cat(before, head);
            sh.map.ub[rank][w] = bu + hub;
        }
        if (lane == 31) {
            sh.map.seg[rank + nend][w] = sc;
            sh.map.ub[rank + nend][w] = su;
        }
        __syncthreads();
        for (int kk = w; kk <= all; kk += SB / 32) {
            const GridSeg h = seg_warp_reduce(sh.map.seg[kk][lane]);
            long long hb = min(sh.map.ub[kk][lane], UB_CAP);
            for (int off = 16; off > 0; off >>= 1)
                hb = min(hb + __shfl_down_sync(0xffffffffu, hb, off), UB_CAP);  // both <= 2^61
            if (lane == 0) {
                GsPiece pc;
                pc.m = h;
                pc.ub = hb;
                pc.has = kk < all;
                pc.x = kk < all ? s_x[kk] : 0.0;
                pc.e = s_e[kk];
                b.piece[(size_t)c * GS_PIECES + kk] = pc;
            }
        }
    }
    if (threadIdx.x == 0) b.np[c] = many ? 0 : all + 1;
    // the last block to get here sees every chunk's pieces
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) s_last = atomicAdd(b.done, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    if (threadIdx.x == 0) *b.done = 0;
    long long count;
    const double sum = gs_walk(fetch, total, nch, b, sh, count);
    __syncthreads();
    fetch.finish(sum, count, sh);
}

__device__ void refill(const D2& d, double ra, bool collide, int* keys);

// the fluid densities of a mask in the reference's loop order (j outer).
// NEW: over the new mask; the first kernel lists the nodes that left a circle
// (solid before, fluid now), and the last block refills them with the average.
// collide: the next step's collision leaves those nodes to that block.
template <bool NEW>
struct RhoFetch {
    D2 d;
    bool collide;
    __device__ void operator()(int t, bool& fl, double& x) const {
        fl = false;
        x = 0.0;
        const int nx = d.p.nx;
        if (t < nx * d.p.ny) {
            const int j = 1 + t / nx, i = 1 + t % nx;
            fl = (NEW ? d.on : d.ob)[IX(d, i, j)] == 0;
            x = d.rho[IX(d, i, j)];
        }
    }
    __device__ void visit(int t, bool fl) const;
    __device__ bool stop() const { return d.status[0] != 0; }
    __device__ void finish(double sum, long long count, GsShared& sh) const {
        const double avg = sum / (double)count;
        if (threadIdx.x == 0) d.ravg[NEW ? 1 : 0] = avg;
        if (NEW) refill(d, avg, collide, sh.keys);
    }
};

struct ArrayFetch {
    const double* x;
    const int* keep;
    int total;
    double* out;  // sum, count
    __device__ void operator()(int t, bool& fl, double& v) const {
        fl = t < total && keep[t] != 0;
        v = t < total ? x[t] : 0.0;
    }
    __device__ void visit(int, bool) const {}
    __device__ bool stop() const { return false; }
    __device__ void finish(double sum, long long count, GsShared&) const {
        if (threadIdx.x == 0) {
            out[0] = sum;
            out[1] = (double)count;
        }
    }
};

int gs_chunks(long long total) { return (int)((total + CH - 1) / CH) > 0 ? (int)((total + CH - 1) / CH) : 1; }

template <class Fetch>
void gs_launch(const Fetch& f, int total, const GsBuf& b, cudaStream_t s) {
    const int nch = gs_chunks(total);
    launch_next(k_gs_part<Fetch>, nch, SB, 0, s, f, total, b);
    launch_next(k_gs_map<Fetch>, nch, SB, 0, s, f, total, nch, b);
}

// calQ / calQ2 from node (x, y) along direction a towards circle c
__device__ bool calq(const D2& d, int c, double x, double y, int a, double& x0, double& y0,
                     double& q) {
    const double xc = d.xc[3 * c], yc = d.xc[3 * c + 1], R = d.p.radius;
    if (!d.p.q_bisection) {
        const double ea = c_ex[a], eb = c_ey[a], ec = 0.0;
        const double ca = ea * ea + eb * eb + ec * ec;
        const double cb = 2.0 * (ea * (x - xc) + eb * (y - yc) + 0.0);
        const double cc = (x - xc) * (x - xc) + (y - yc) * (y - yc) + 0.0 - R * R;
        const double delta = cb * cb - 4.0 * ca * cc;
        if (delta < 0) return false;
        q = (-cb - sqrt(delta)) / (2.0 * ca);
        x0 = x + q * ea;
        y0 = y + q * eb;
    } else {
        const double epsR = (double)1e-9f;  // default-real literal 1e-9 (:106)
        double qq = 0.5, qt = 0.5;
        double px = x + qt * (double)c_ex[a], py = y + qt * (double)c_ey[a];
        auto dist = [&]() { return sqrt((px - xc) * (px - xc) + (py - yc) * (py - yc) + 0.0); };
        int guard = 0;
        while (fabs(dist() - R) >= epsR) {
            if (++guard > 200) return false;
            if (dist() > R) {
                qt = qt / 2.0;
                px = px + qt * (double)c_ex[a];
                py = py + qt * (double)c_ey[a];
                qq = qq + qt;
            } else if (dist() < R) {
                qt = qt / 2.0;
                px = px - qt * (double)c_ex[a];
                py = py - qt * (double)c_ey[a];
                qq = qq - qt;
            } else {
                return false;
            }
        }
        q = qq;
        x0 = px;
        y0 = py;
    }
    return !(q > 1.0 || q < 0.0);
}

// calq by one warp (same arguments in every lane, same result).  calQ bisects
// [0, 1]: its k-th trial is the middle of the dyadic interval of length 2^-k
// that holds the root, the step to the next one is decided by the sign of
// |x - X| - R, and it stops at the first trial within epsR of the circle.  With
// the root known to rounding (calQ2's formula), lane k writes down trial k and
// evaluates it with calQ's own operations; trial coordinates are exact, so
// they are calQ's bit for bit as long as each trial before the one that stops
// decides for the next lane's, which is checked; otherwise calq bisects.  One
// pass replaces a chain of some thirty dependent square roots.
__device__ bool calq_warp(const D2& d, int c, int i, int j, int a, double& x0, double& y0,
                          double& q) {
    const double x = (double)i, y = (double)j;
    const double xc = d.xc[3 * c], yc = d.xc[3 * c + 1], R = d.p.radius;
    const int ex = c_ex[a], ey = c_ey[a], lane = threadIdx.x & 31;
    if (d.p.q_bisection && i < (1 << 20) && j < (1 << 20)) {
        const double epsR = (double)1e-9f;
        const double ox = x - xc, oy = y - yc, ca = ex != 0 && ey != 0 ? 2.0 : 1.0;
        const double hb = (double)ex * ox + (double)ey * oy;  // cb / 2
        const double delta = hb * hb - ca * (ox * ox + oy * oy - R * R);
        if (delta >= 0.0) {
            const double root = (-hb - sqrt(delta)) * (ca == 1.0 ? 1.0 : 0.5);
            const double two_k = __longlong_as_double((long long)(1023 + lane) << 52);
            const double inv2k1 = __longlong_as_double((long long)(1023 - lane - 1) << 52);
            const double lo = fmin(fmax(floor(root * two_k), 0.0), two_k - 1.0);
            const double ql = (2.0 * lo + 1.0) * inv2k1;
            const double px = x + ql * (double)ex, py = y + ql * (double)ey;
            const double dist = sqrt((px - xc) * (px - xc) + (py - yc) * (py - yc) + 0.0);
            const unsigned stop = __ballot_sync(0xffffffffu, fabs(dist - R) < epsR);
            const double qn = __shfl_down_sync(0xffffffffu, ql, 1);
            const unsigned wrong = __ballot_sync(0xffffffffu, (dist > R) != (qn > ql));
            const int k = __ffs(stop) - 1;
            if (k >= 0 && (wrong & ((1u << k) - 1u)) == 0) {
                q = __shfl_sync(0xffffffffu, ql, k);
                x0 = __shfl_sync(0xffffffffu, px, k);
                y0 = __shfl_sync(0xffffffffu, py, k);
                return !(q > 1.0 || q < 0.0);
            }
        }
    }
    return calq(d, c, x, y, a, x0, y0, q);
}

// the interpolated bounce-back of the link (i, j) -> a with fraction q
// (particle_bounceback.F90:37-97)
__device__ __forceinline__ void ibb_link(const D2& d, int i, int j, int a, int c, double x0,
                                         double y0, double q, double ravg) {
    const double Om = d.om[3 * c + 2];
    const double rot0 = -(y0 - d.xc[3 * c + 1]) * Om, rot1 = (x0 - d.xc[3 * c]) * Om;
    const int ra = c_r[a];
    const double eu = c_ex[ra] * (d.uc[3 * c] + rot0) + c_ey[ra] * (d.uc[3 * c + 1] + rot1);
    const int ex = c_ex[a], ey = c_ey[a];
    const int i1 = wxi(d, i - ex), i2 = wxi(d, i - 2 * ex);
    if (d.p.linear) {  // case1 particle_bounceback.F90:66-76
        if (q < 0.5) {
            F(d, ra, i, j) = 2.0 * q * FP(d, a, i, j) + (1.0 - 2.0 * q) * FP(d, a, i1, j - ey) +
                             6.0 * c_w[a] * ravg * eu;
        } else {
            F(d, ra, i, j) = 0.5 / q * FP(d, a, i, j) + (1.0 - 0.50 / q) * FP(d, ra, i, j) +
                             3.0 * c_w[a] * ravg / q * eu;
        }
    } else if (q < 0.5) {
        F(d, ra, i, j) = q * (1.0 + 2.0 * q) * FP(d, a, i, j) +
                         (1.0 - 4.0 * q * q) * FP(d, a, i1, j - ey) -
                         q * (1.0 - 2.0 * q) * FP(d, a, i2, j - 2 * ey) +
                         6.0 * c_w[a] * ravg * eu;
    } else {
        F(d, ra, i, j) = FP(d, a, i, j) / q / (1.0 + 2.0 * q) +
                         FP(d, ra, i, j) * (2.0 * q - 1.0) / q -
                         FP(d, ra, i1, j - ey) * (2.0 * q - 1.0) / (2.0 * q + 1.0) +
                         6.0 * c_w[a] * ravg / q / (1.0 + 2.0 * q) * eu;
    }
}

// momentum exchange of the link (i, j) -> a of circle c, whose wall point is
// x0, y0 (particle_force.F90:59-66)
__device__ __forceinline__ void link_force(const D2& d, int i, int j, int a, int c, double x0,
                                           double y0, double& Fx, double& Fy, double& T) {
    const double xcc = d.xc[3 * c], ycc = d.xc[3 * c + 1];
    const double Om = d.om[3 * c + 2], U0 = d.uc[3 * c], U1 = d.uc[3 * c + 1];
    const double rot0 = -(y0 - ycc) * Om, rot1 = (x0 - xcc) * Om;
    const int ra = c_r[a];
    Fx = (c_ex[a] - U0 - rot0) * FP(d, a, i, j) - (c_ex[ra] - U0 - rot0) * F(d, ra, i, j);
    Fy = (c_ey[a] - U1 - rot1) * FP(d, a, i, j) - (c_ey[ra] - U1 - rot1) * F(d, ra, i, j);
    const double rx = x0 - xcc, ry = y0 - ycc;
    T = rx * Fy - ry * Fx;
}

// The listed fluid nodes (a solid neighbour), one block of eight warps each:
// warp w finds calQ of direction w + 1, then eight lanes bounce back their
// links and take their momentum exchange, and the node takes its macro.  What
// counts is the chain of FP64 instructions of one node; as a thread per node
// with bisections one after another the bounce-back took 187 us and a second
// evaluation for the forces 169 (400x800, three circles of radius 10).
__global__ void __launch_bounds__(256) k2_boundary(D2 d) {
    after_previous();
    if (stopped(d)) return;
    // per direction: the first circle that owns the solid end, for the forces,
    // and the last one, whose bounce-back stands (they differ only where
    // circles overlap)
    __shared__ double s_x0[2][8], s_y0[2][8], s_q[8];
    __shared__ int s_c[2][8];
    const int n = (int)d.done[1], lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (int pos = blockIdx.x; pos < n; pos += gridDim.x) {
        const int t = d.bl_list[pos];
        const int j = 1 + t / d.p.nx, i = 1 + t % d.p.nx;
        int first = -1, last = -1;
        {
            const int a = w + 1, ip = i + c_ex[a], jp = j + c_ey[a];
            if (d.ob[IX(d, ip, jp)] == 1) {
                bool ok = true;
                for (int c = 0; c < d.p.np; c++) {
                    if (!inside(d, d.xc, c, (double)ip, (double)jp)) continue;
                    double x0, y0, q;
                    if (!calq_warp(d, c, i, j, a, x0, y0, q)) {
                        if (lane == 0) fail(d, S_Q, c, d.par);
                        ok = false;
                        break;
                    }
                    if (lane == 0) {
                        if (first < 0) {
                            s_x0[0][w] = x0;
                            s_y0[0][w] = y0;
                        }
                        s_x0[1][w] = x0;
                        s_y0[1][w] = y0;
                        s_q[w] = q;
                    }
                    if (first < 0) first = c;
                    last = c;
                }
                if (first < 0 && ok && lane == 0) fail(d, S_NO_OWNER, -1, d.par);
            }
            if (lane == 0) {
                s_c[0][w] = first;
                s_c[1][w] = last;
            }
        }
        __syncthreads();
        if (w == 0) {
            const int a = 1 + (lane & 7), b = lane & 7, ra = c_r[a];
            const bool act = lane < 8;
            double ga = F(d, a, i, j);
            const double g0 = F(d, 0, i, j);
            const int c1 = s_c[1][b];
            double fra = 0.0;
            if (act) {
                const int c0 = s_c[0][b];
                if (c1 >= 0) {
                    ibb_link(d, i, j, a, c1, s_x0[1][b], s_y0[1][b], s_q[b], d.ravg[0]);
                    fra = F(d, ra, i, j);
                    double Fx, Fy, T;
                    link_force(d, i, j, a, c0, s_x0[0][b], s_y0[0][b], Fx, Fy, T);
                    double* o = d.lt + LINK_TERMS * (NODE_LINKS * (size_t)pos + b);
                    o[0] = Fx;
                    o[1] = Fy;
                    o[2] = T;
                }
                d.lc[8 * (size_t)pos + b] = c0;
            }
            // the population that came back along a is the opposite lane's
            const double back = __shfl_sync(0xffffffffu, fra, ra - 1);
            const int cb = __shfl_sync(0xffffffffu, c1, ra - 1);
            if (cb >= 0) ga = back;
            double g[9];
            g[0] = g0;
#pragma unroll
            for (int q = 1; q < 9; q++) g[q] = __shfl_sync(0xffffffffu, ga, q - 1);
            double r, u, v;
            d2q9_macro(g, r, u, v);
            if (lane == 0) {
                const int c = IX(d, i, j);
                d.rho[c] = r;
                d.u[c] = u;
                d.v[c] = v;
            }
        }
        __syncthreads();
    }
}

// particle_update.F90:26-50: U += F/M, Omega += T/I, x += U_old + a/2
__device__ void move_circle(const D2& d, int c) {
    const P2Params& p = d.p;
    double force[2], torque;
    force[0] = __ldcg(d.force + 3 * c);
    force[1] = __ldcg(d.force + 3 * c + 1);
    torque = __ldcg(d.torque + 3 * c + 2);
    for (int q = 0; q < 3; q++) {
        d.xco[3 * c + q] = d.xc[3 * c + q];
        d.uco[3 * c + q] = d.uc[3 * c + q];
        d.omo[3 * c + q] = d.om[3 * c + q];
    }
    if (p.variant == P2_SHEAR) {  // case1 particle_update.F90:21-35: prescribed motion
        d.uc[3 * c] = p.moving_frame ? 0.0 : p.u0;
        d.uc[3 * c + 1] = 0.0;
        d.om[3 * c + 2] = 0.0;
        d.xc[3 * c] = d.xco[3 * c] + d.uco[3 * c];
        d.xc[3 * c + 1] = d.xco[3 * c + 1] + d.uco[3 * c + 1];
        return;
    }
    const double PI = p.pi, R0 = p.radius, r = p.radius;
    const double ax = force[0] / PI / (R0 * R0) / p.rho_solid;
    const double ay = force[1] / PI / (R0 * R0) / p.rho_solid;
    const double aom = torque / (0.5 * p.rho_solid * PI * (r * r * r * r));
    d.uc[3 * c] = d.uco[3 * c] + ax;
    d.uc[3 * c + 1] = d.uco[3 * c + 1] + ay;
    d.om[3 * c + 2] = d.omo[3 * c + 2] + aom;
    d.xc[3 * c] = d.xco[3 * c] + d.uco[3 * c] + 0.5 * ax;
    d.xc[3 * c + 1] = d.xco[3 * c + 1] + d.uco[3 * c + 1] + 0.5 * ay;
}

// springs and gravity of circle c (particle_force.F90:86-190), one thread: the
// terms that follow the link sums in the totals; 0, or the status of a circle
// that overlaps another or a wall
struct Extra {
    double fij0, fij1, fw0, fw1, grav;
};
__device__ int extra_force(const D2& d, int c, Extra& x) {
    const P2Params& p = d.p;
    const double PI = p.pi, R0 = p.radius, ravg = d.ravg[0];
    const double gmag = fabs(-p.gravity);
    double fij[3] = {0.0, 0.0, 0.0}, fw[3] = {0.0, 0.0, 0.0};
    const double Rc = R0;
    // particle-particle springs (:100-125)
    const double scale_p = PI * (Rc * Rc) * (p.rho_solid - ravg) * gmag / p.stiff_particle;
    for (int c2 = 0; c2 < p.np; c2++) {
        if (c2 == c) continue;
        const double d0 = d.xc[3 * c] - d.xc[3 * c2];
        const double d1 = d.xc[3 * c + 1] - d.xc[3 * c2 + 1];
        const double d2 = 0.0;
        const double dij = sqrt(d0 * d0 + d1 * d1 + d2 * d2);
        const double R2 = R0, thr = p.threshold_particle;
        if (dij >= Rc + R2 + thr) {
        } else if (dij < Rc + R2 + thr && dij >= Rc + R2) {
            const double t = (dij - Rc - R2 - thr) / thr;
            fij[0] = fij[0] + scale_p * (t * t) * d0 / dij;
            fij[1] = fij[1] + scale_p * (t * t) * d1 / dij;
            fij[2] = fij[2] + scale_p * (t * t) * d2 / dij;
        } else {
            return S_OVERLAP;
        }
    }
    // particle-wall springs (:128-178): left, right, bottom (no top spring)
    const double scale_w = PI * (Rc * Rc) * (p.rho_solid - p.rho0) * gmag / p.stiff_wall;
    const double thw = p.threshold_wall;
    for (int ax = 0; ax < 2; ax++) {
        const int n_ax = ax == 0 ? p.nx : p.ny;
        const bool high = ax == 0;
        const double cpos = d.xc[3 * c + ax];
        double dw = cpos - Rc - 1.0;
        if (dw < 0) return S_WALL;
        if (dw < thw) fw[ax] = fw[ax] + scale_w * ((dw - thw) / thw) * ((dw - thw) / thw);
        if (high) {
            dw = (double)n_ax - cpos - Rc;
            if (dw < 0) return S_WALL;
            if (dw < thw) fw[ax] = fw[ax] - scale_w * ((dw - thw) / thw) * ((dw - thw) / thw);
        }
    }
    x.fij0 = fij[0];
    x.fij1 = fij[1];
    x.fw0 = fw[0];
    x.fw1 = fw[1];
    x.grav = (p.rho_solid - ravg) * PI * (R0 * R0) * gmag;
    return 0;
}

// first and last node of a circle's box along one axis, clipped to [lo, hi];
// empty for a centre that is not finite
__device__ __forceinline__ int box_lo(double x, double r, int margin, int lo, int hi) {
    const double v = floor(x - r) - margin;
    return v > lo ? (v <= hi ? (int)v : hi + 1) : (v == v ? lo : hi + 1);
}
__device__ __forceinline__ int box_hi(double x, double r, int margin, int lo, int hi) {
    const double v = ceil(x + r) + margin;
    return v < hi ? (v >= lo ? (int)v : lo - 1) : (v == v ? hi : lo - 1);
}

// calForce (particle_force.F90:35-190) and updateCenter: one block per circle.
// One thread per node of the circle's box looks up the links that k2_boundary
// left (integers only); they are listed in the reference's loop order (j outer,
// i, direction inner), their terms are fetched together, and three threads add
// them one after another, so the sums are the sequential ones.  What is left is
// the chain of FP64 adds (a few hundred); a warp that evaluated 32 candidate
// links at a time needed 170 rounds (203 us at R = 10).  A link whose solid end
// a circle before this one owns too (overlapping circles) is evaluated here.
// The last block to finish moves every circle.
constexpr int FB = 1024, FT = 512;
__global__ void __launch_bounds__(FB) k2_force(D2 d) {
    after_previous();
    if (stopped(d)) return;
    __shared__ int list[8 * FB];  // place * 8 + direction - 1; negative (~): evaluate
    __shared__ double term[3][FT];
    __shared__ int wcount[FB / 32];
    __shared__ int s_last, s_bad, s_extra;
    __shared__ Extra s_x;
    const int c = blockIdx.x, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const P2Params& p = d.p;
    const double R0 = p.radius, xcc = d.xc[3 * c], ycc = d.xc[3 * c + 1];
    const int i0 = box_lo(xcc, R0, 2, 1, p.nx), i1 = box_hi(xcc, R0, 2, 1, p.nx);
    const int j0 = box_lo(ycc, R0, 2, 1, p.ny), j1 = box_hi(ycc, R0, 2, 1, p.ny);
    const int ni = max(0, i1 - i0 + 1), nj = max(0, j1 - j0 + 1);
    const long long nbox = (long long)ni * nj;
    if (threadIdx.x == 0) s_bad = 0;
    __syncthreads();
    // the last warp's first thread takes the springs meanwhile
    if (threadIdx.x == FB - 32) s_extra = p.variant == P2_SHEAR ? 0 : extra_force(d, c, s_x);
    double sum = 0.0;  // threads 0, 1, 2: F_x, F_y, torque
    for (long long base = 0; base < nbox; base += FB) {
        const long long t = base + threadIdx.x;
        int pos = -1, mask = 0, own = 0;
        if (t < nbox) {
            const int i = i0 + (int)(t % ni), j = j0 + (int)(t / ni);
            pos = d.bl_pos[IX(d, i, j)];
            if (pos >= 0) {
                const int4 lo = *(const int4*)(d.lc + 8 * (size_t)pos);
                const int4 hi = *(const int4*)(d.lc + 8 * (size_t)pos + 4);
                const int o[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
#pragma unroll
                for (int b = 0; b < 8; b++) {
                    if (o[b] == c) {
                        own |= 1 << b;
                        mask |= 1 << b;
                    } else if (o[b] >= 0 &&
                               inside(d, d.xc, c, (double)(i + c_ex[b + 1]), (double)(j + c_ey[b + 1]))) {
                        mask |= 1 << b;
                    }
                }
            }
        }
        int incl = __popc(mask);
        for (int off = 1; off < 32; off <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, incl, off);
            if (lane >= off) incl += y;
        }
        if (lane == 31) wcount[w] = incl;
        __syncthreads();
        int at = incl - __popc(mask), all = 0;
        for (int q = 0; q < FB / 32; q++) {
            if (q < w) at += wcount[q];
            all += wcount[q];
        }
        for (int m = mask; m; m &= m - 1) {
            const int b = __ffs(m) - 1;
            list[at++] = (own >> b) & 1 ? 8 * pos + b : ~(8 * pos + b);
        }
        __syncthreads();
        for (int k0 = 0; k0 < all; k0 += FT) {
            const int k1 = min(FT, all - k0);
            if (threadIdx.x < k1) {
                const int e = list[k0 + threadIdx.x];
                double Fx = 0.0, Fy = 0.0, T = 0.0;
                if (e >= 0) {
                    const double* o = d.lt + LINK_TERMS * (size_t)e;
                    Fx = o[0];
                    Fy = o[1];
                    T = o[2];
                } else {
                    const int slot = ~e, node = d.bl_list[slot >> 3], a = 1 + (slot & 7);
                    const int j = 1 + node / p.nx, i = 1 + node % p.nx;
                    double x0, y0, q;
                    if (calq(d, c, (double)i, (double)j, a, x0, y0, q))
                        link_force(d, i, j, a, c, x0, y0, Fx, Fy, T);
                    else s_bad = 1;
                }
                term[0][threadIdx.x] = Fx;
                term[1][threadIdx.x] = Fy;
                term[2][threadIdx.x] = T;
            }
            __syncthreads();
            if (threadIdx.x < 3) {
#pragma unroll 8
                for (int q = 0; q < k1; q++) sum = sum + term[threadIdx.x][q];
            }
            __syncthreads();
        }
    }
    __syncthreads();  // s_extra, also for an empty box
    // case1 has the momentum exchange only (particle_force.F90:86-92)
    if (w == 0) {
        const double fs0 = __shfl_sync(0xffffffffu, sum, 0), fs1 = __shfl_sync(0xffffffffu, sum, 1),
                     ts = __shfl_sync(0xffffffffu, sum, 2);
        if (lane == 0) {
            if (s_bad || s_extra) {
                fail(d, s_bad ? S_Q : s_extra, c, d.par);
            } else {
                const bool shear = p.variant == P2_SHEAR;  // totals (:184-190)
                d.force[3 * c] = shear ? fs0 : fs0 + s_x.fij0 + s_x.fw0;
                d.force[3 * c + 1] = shear ? fs1 : fs1 - s_x.grav + s_x.fij1 + s_x.fw1;
                d.force[3 * c + 2] = 0.0;
                d.torque[3 * c] = 0.0;
                d.torque[3 * c + 1] = 0.0;
                d.torque[3 * c + 2] = ts;
            }
            __threadfence();
            s_last = atomicAdd(d.done, 1u) == gridDim.x - 1;
        }
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    if (threadIdx.x == 0) {
        d.done[0] = 0;
        d.done[1] = 0;  // the next step's list of boundary nodes
    }
    if (__ldcg(d.status)) return;
    for (int q = threadIdx.x; q < p.np; q += FB) move_circle(d, q);
}

// obst from the centres over 0..nx+1 x 0..ny+1 (particle_update.F90:80-93) into
// a cleared mask, a block per circle and its box; interior solid nodes get
// rho_s and u = 0 (:94-102)
__global__ void __launch_bounds__(256) k2_mark(D2 d, int* mask, bool set_macro) {
    after_previous();
    if (d.status[0]) return;
    const int c = blockIdx.x;
    const double R0 = d.p.radius, xcc = d.xc[3 * c], ycc = d.xc[3 * c + 1];
    const int i0 = box_lo(xcc, R0, 1, 0, d.p.nx + 1), i1 = box_hi(xcc, R0, 1, 0, d.p.nx + 1);
    const int j0 = box_lo(ycc, R0, 1, 0, d.p.ny + 1), j1 = box_hi(ycc, R0, 1, 0, d.p.ny + 1);
    const int ni = max(0, i1 - i0 + 1), nj = max(0, j1 - j0 + 1);
    const long long n = (long long)ni * nj;
    for (long long t = threadIdx.x; t < n; t += blockDim.x) {
        const int i = i0 + (int)(t % ni), j = j0 + (int)(t / ni);
        if (!inside(d, d.xc, c, (double)i, (double)j)) continue;
        mask[IX(d, i, j)] = 1;
        if (set_macro && i >= 1 && i <= d.p.nx && j >= 1 && j <= d.p.ny) {
            d.rho[IX(d, i, j)] = d.p.rho_solid;
            d.u[IX(d, i, j)] = 0.0;
            d.v[IX(d, i, j)] = 0.0;
        }
    }
}

// refill of nodes that left a circle (particle_update.F90:122-193) for one
// node; false when it failed (status set)
__device__ bool refill_node(const D2& d, int i, int j, double ra) {
    const P2Params& p = d.p;
    bool found = false;
    for (int c = 0; c < p.np; c++) {
        if (!inside(d, d.xco, c, (double)i, (double)j)) continue;
        found = true;
        const double xc = d.xc[3 * c], yc = d.xc[3 * c + 1];
        double out = 0.0;
        int ec = 0;
        for (int a = 1; a < 9; a++) {
            const double t = ((i - xc) * c_ex[a] + (j - yc) * c_ey[a]) /
                             sqrt((i - xc) * (i - xc) + (j - yc) * (j - yc));
            if (t > out) {
                out = t;
                ec = a;
            }
        }
        if (ec == 0) {
            fail(d, S_NO_DIR, c, d.par ^ 1);
            return false;
        }
        const int e0 = c_ex[ec], e1 = c_ey[ec];
        const int i1 = wxi(d, i + e0), i2 = wxi(d, i + 2 * e0), i3 = wxi(d, i + 3 * e0);
        for (int a = 0; a < 9; a++) {
            if (p.linear)  // case1 particle_update.F90:115-119
                F(d, a, i, j) = 2.0 * F(d, a, i1, j + e1) - F(d, a, i2, j + 2 * e1);
            else
                F(d, a, i, j) = 3.0 * F(d, a, i1, j + e1) - 3.0 * F(d, a, i2, j + 2 * e1) +
                                F(d, a, i3, j + 3 * e1);
        }
        double G[9], m[9];
        for (int a = 0; a < 9; a++) G[a] = F(d, a, i, j);
        m[0] = G[0] + G[1] + G[2] + G[3] + G[4] + G[5] + G[6] + G[7] + G[8];
        m[1] = -4.0 * G[0] - G[1] - G[2] - G[3] - G[4] + 2.0 * G[5] + 2.0 * G[6] + 2.0 * G[7] + 2.0 * G[8];
        m[2] = 4.0 * G[0] - 2.0 * G[1] - 2.0 * G[2] - 2.0 * G[3] - 2.0 * G[4] + G[5] + G[6] + G[7] + G[8];
        if (p.variant == P2_SHEAR) {  // case1 :130,132: the first circle's (Uc, Vc)
            m[3] = ra * d.uc[0];
            m[5] = ra * d.uc[1];
        } else {
            m[3] = ra * (d.uc[3 * c] - (j - yc) * d.om[3 * c + 2]);
            m[5] = ra * (d.uc[3 * c + 1] + (i - xc) * d.om[3 * c + 2]);
        }
        m[4] = -2.0 * G[1] + 2.0 * G[3] + G[5] - G[6] - G[7] + G[8];
        m[6] = -2.0 * G[2] + 2.0 * G[4] + G[5] + G[6] - G[7] - G[8];
        m[7] = G[1] - G[2] + G[3] - G[4];
        m[8] = G[5] - G[6] + G[7] - G[8];
        G[0] = (m[0] - m[1] + m[2]) / 9.0;
        G[1] = m[0] / 9.0 - m[1] / 36.0 - m[2] / 18.0 + m[3] / 6.0 - m[4] / 6.0 + m[7] * 0.25;
        G[2] = m[0] / 9.0 - m[1] / 36.0 - m[2] / 18.0 + m[5] / 6.0 - m[6] / 6.0 - m[7] * 0.25;
        G[3] = m[0] / 9.0 - m[1] / 36.0 - m[2] / 18.0 - m[3] / 6.0 + m[4] / 6.0 + m[7] * 0.25;
        G[4] = m[0] / 9.0 - m[1] / 36.0 - m[2] / 18.0 - m[5] / 6.0 + m[6] / 6.0 - m[7] * 0.25;
        G[5] = m[0] / 9.0 + m[1] / 18.0 + m[2] / 36.0 + m[3] / 6.0 + m[4] / 12.0 + m[5] / 6.0 +
               m[6] / 12.0 + m[8] * 0.25;
        G[6] = m[0] / 9.0 + m[1] / 18.0 + m[2] / 36.0 - m[3] / 6.0 - m[4] / 12.0 + m[5] / 6.0 +
               m[6] / 12.0 - m[8] * 0.25;
        G[7] = m[0] / 9.0 + m[1] / 18.0 + m[2] / 36.0 - m[3] / 6.0 - m[4] / 12.0 - m[5] / 6.0 -
               m[6] / 12.0 + m[8] * 0.25;
        G[8] = m[0] / 9.0 + m[1] / 18.0 + m[2] / 36.0 + m[3] / 6.0 + m[4] / 12.0 - m[5] / 6.0 -
               m[6] / 12.0 - m[8] * 0.25;
        for (int a = 0; a < 9; a++) F(d, a, i, j) = G[a];
        const double r = G[0] + G[1] + G[2] + G[3] + G[4] + G[5] + G[6] + G[7] + G[8];
        d.rho[IX(d, i, j)] = r;
        d.u[IX(d, i, j)] = (G[1] - G[3] + G[5] - G[6] - G[7] + G[8]) / r;
        d.v[IX(d, i, j)] = (G[2] - G[4] + G[5] + G[6] - G[7] - G[8]) / r;
    }
    if (!found) {
        fail(d, S_NO_OWNER, -1, d.par ^ 1);
        return false;
    }
    return true;
}

// The refill sweep in the reference's order: each refill may read an earlier
// one, so one thread refills.  The nodes to refill (left a circle: solid
// before, fluid now) are listed by the average's first kernel in any order;
// refill sorts the list by node index and refills in that order.  A list
// longer than RF_CAP is replaced by refill_scan, which finds the nodes chunk by
// chunk with an ordered block compaction.
template <bool NEW>
__device__ void RhoFetch<NEW>::visit(int t, bool fl) const {
    if (!NEW || !fl || d.status[0]) return;
    const int nx = d.p.nx, j = 1 + t / nx, i = 1 + t % nx;
    if (d.ob[IX(d, i, j)] != 1) return;
    const int pos = atomicAdd(d.rf_count, 1);
    if (pos < RF_CAP) d.rf_list[pos] = t;
}

__device__ void refill_scan(const D2& d, double ra, int* list) {
    __shared__ int wcount[SB / 32];
    __shared__ int nlist, stop;
    const int nx = d.p.nx;
    const long long total = (long long)nx * d.p.ny;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (threadIdx.x == 0) stop = 0;
    auto left = [&](long long t) {  // solid before, fluid now
        if (t >= total) return false;
        const int j = 1 + (int)(t / nx), i = 1 + (int)(t % nx);
        return d.ob[IX(d, i, j)] == 1 && d.on[IX(d, i, j)] == 0;
    };
    // chunks of EPT sub-chunks of SB nodes; flags of the next chunk are read ahead
    bool fnext[EPT];
#pragma unroll
    for (int u = 0; u < EPT; u++) fnext[u] = left((long long)u * SB + threadIdx.x);
    for (long long cbase = 0; cbase < total; cbase += CH) {
        bool fcur[EPT];
        bool any = false;
#pragma unroll
        for (int u = 0; u < EPT; u++) {
            fcur[u] = fnext[u];
            any = any || fcur[u];
            fnext[u] = left(cbase + CH + (long long)u * SB + threadIdx.x);
        }
        if (!__syncthreads_or(any)) continue;  // most chunks have none
        for (int u = 0; u < EPT; u++) {
            const long long t = cbase + (long long)u * SB + threadIdx.x;
            const bool flag = fcur[u];
            if (!__syncthreads_or(flag)) continue;
            const unsigned bal = __ballot_sync(0xffffffffu, flag);
            if (lane == 0) wcount[w] = __popc(bal);
            __syncthreads();
            if (threadIdx.x == 0) {
                int acc = 0;
                for (int q = 0; q < SB / 32; q++) {
                    const int c = wcount[q];
                    wcount[q] = acc;
                    acc += c;
                }
                nlist = acc;
            }
            __syncthreads();
            if (flag) list[wcount[w] + __popc(bal & ((1u << lane) - 1u))] = (int)t;
            __syncthreads();
            if (threadIdx.x == 0) {
                for (int q = 0; q < nlist; q++) {
                    const int node = list[q];
                    if (!refill_node(d, 1 + node % nx, 1 + node / nx, ra)) {
                        stop = 1;
                        break;
                    }
                }
            }
            __syncthreads();
            if (stop) return;
        }
    }
}

// by every thread of one SB-thread block
__device__ void refill(const D2& d, double ra, bool collide, int* keys) {
    const int cnt = __ldcg(d.rf_count);
    if (cnt > RF_CAP) {
        refill_scan(d, ra, keys);
    } else if (cnt > 0) {
        int n2 = 1;
        while (n2 < cnt) n2 <<= 1;
        for (int q = threadIdx.x; q < n2; q += SB) keys[q] = q < cnt ? d.rf_list[q] : 0x7fffffff;
        __syncthreads();
        for (int k = 2; k <= n2; k <<= 1)  // bitonic sort, ascending
            for (int jj = k >> 1; jj > 0; jj >>= 1) {
                for (int q = threadIdx.x; q < n2; q += SB) {
                    const int r = q ^ jj;
                    if (r > q) {
                        const int a = keys[q], b = keys[r];
                        if ((a > b) == ((q & k) == 0)) {
                            keys[q] = b;
                            keys[r] = a;
                        }
                    }
                }
                __syncthreads();
            }
        if (threadIdx.x == 0) {
            const int nx = d.p.nx;
            for (int q = 0; q < cnt; q++)
                if (!refill_node(d, 1 + keys[q] % nx, 1 + keys[q] / nx, ra)) break;
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) d.rf_count[0] = 0;
    if (!collide || cnt == 0 || __ldcg(d.status)) return;
    const int nx = d.p.nx;
    if (cnt <= RF_CAP) {
        for (int q = threadIdx.x; q < cnt; q += SB) {
            const int c = IX(d, 1 + keys[q] % nx, 1 + keys[q] / nx);
            if (d.p.variant == P2_SHEAR) collide_node<true>(d, c);
            else collide_node<false>(d, c);
        }
    } else {
        for (long long t = threadIdx.x; t < (long long)nx * d.p.ny; t += SB) {
            const int c = IX(d, 1 + (int)(t % nx), 1 + (int)(t / nx));
            if (d.ob[c] != 1 || d.on[c] != 0) continue;
            if (d.p.variant == P2_SHEAR) collide_node<true>(d, c);
            else collide_node<false>(d, c);
        }
    }
}

// initial.F90:103-188 with the centres given by the caller: mask, rho = rho_s
// (solid) or rho0, u = 0, f = omega on fluid nodes, ghosts omega*rho0
__global__ void k2_init_fields(D2 d) {
    const int i = -2 + (int)(blockIdx.x * blockDim.x + threadIdx.x), j = -2 + (int)blockIdx.y;
    if (i > d.p.nx + 3) return;
    const int nx = d.p.nx, ny = d.p.ny;
    const bool interior = i >= 1 && i <= nx && j >= 1 && j <= ny;
    const bool ghost = !interior && i >= -1 && i <= nx + 2 && j >= -1 && j <= ny + 2;
    if (interior) {
        const bool solid = d.ob[IX(d, i, j)] == 1;
        d.rho[IX(d, i, j)] = solid ? d.p.rho_solid : d.p.rho0;
        double uu = 0.0;
        if (d.p.variant == P2_SHEAR) {  // case1 initial.F90:96-127
            const bool mf = d.p.moving_frame;
            uu = mf ? 0.0 : d.p.u0;
            if (j == 1) uu = mf ? -d.p.uwall - d.p.u0 : -d.p.uwall;
            if (j == ny) uu = mf ? d.p.uwall - d.p.u0 : d.p.uwall;
        }
        d.u[IX(d, i, j)] = uu;
        d.v[IX(d, i, j)] = 0.0;
        if (!solid) {
            const double vv = 0.0, us2 = uu * uu + vv * vv;
            for (int a = 0; a < 9; a++) {
                const double un = uu * c_ex[a] + vv * c_ey[a];
                F(d, a, i, j) = c_w[a] * (1.0 + 3.0 * un + 4.5 * un * un - 1.5 * us2);
            }
        }
    } else if (ghost && d.p.variant != P2_SHEAR) {  // case1 ghosts stay 0 (initial.F90:140)
        for (int a = 0; a < 9; a++) {
            F(d, a, i, j) = c_w[a] * d.p.rho0;
            FP(d, a, i, j) = c_w[a] * d.p.rho0;
        }
    }
}

// owner index of every interior node (-1 fluid)
__global__ void k2_owner(D2 d, int* out) {
    const int i = 1 + blockIdx.x * blockDim.x + threadIdx.x, j = 1 + blockIdx.y;
    if (i > d.p.nx) return;
    int o = -1;
    if (d.ob[IX(d, i, j)] == 1)
        for (int c = 0; c < d.p.np && o < 0; c++)
            if (inside(d, d.xc, c, (double)i, (double)j)) o = c;
    out[(i - 1) + d.p.nx * (j - 1)] = o;
}

}  // namespace

struct P2Ctx {
    D2 d{};
    cudaStream_t s = nullptr;
    bool own_stream = false;
    std::vector<double> centers;  // np x 3
    long long itc = 0;
    long long bytes = 0;
    int* owner_tmp = nullptr;
    // the average over the current mask runs beside the collision
    cudaStream_t side = nullptr;
    cudaEvent_t fork = nullptr, join = nullptr;
};

namespace {

int ck(cudaError_t e, const char* what, std::string& err) {
    if (e == cudaSuccess) return MGLC_OK;
    err = std::string(what) + ": " + cudaGetErrorString(e);
    return MGLC_ERR_CUDA;
}

template <typename T>
int dal(P2Ctx* c, T** p, size_t n, std::string& err) {
    cudaError_t e = cudaMalloc((void**)p, n * sizeof(T));
    if (e != cudaSuccess) {
        err = std::string("device allocation: ") + cudaGetErrorString(e);
        return MGLC_ERR_NOMEM;
    }
    c->bytes += (long long)(n * sizeof(T));
    return cudaMemsetAsync(*p, 0, n * sizeof(T), c->s) == cudaSuccess ? MGLC_OK : MGLC_ERR_CUDA;
}

dim3 rows_grid(const D2& d) { return dim3((d.p.nx + 127) / 128, d.p.ny); }

}  // namespace

int p2d_create(const P2Params& p, const double* centers_xy, P2Ctx** out, std::string& err) {
    P2Ctx* c = new P2Ctx();
    *out = c;
    c->d.p = p;
    c->d.X = p.nx + 6;
    c->d.C = (size_t)(p.nx + 6) * (p.ny + 6);
    if (cudaStreamCreateWithFlags(&c->s, cudaStreamNonBlocking) != cudaSuccess) {
        err = "stream creation failed";
        return MGLC_ERR_CUDA;
    }
    c->own_stream = true;
    if (cudaStreamCreateWithFlags(&c->side, cudaStreamNonBlocking) != cudaSuccess ||
        cudaEventCreateWithFlags(&c->fork, cudaEventDisableTiming) != cudaSuccess ||
        cudaEventCreateWithFlags(&c->join, cudaEventDisableTiming) != cudaSuccess) {
        err = "stream creation failed";
        return MGLC_ERR_CUDA;
    }
    const size_t cells = (size_t)(p.nx + 6) * (p.ny + 6), np3 = 3 * (size_t)(p.np > 0 ? p.np : 1);
    D2& d = c->d;
    int rc = 0;
    if ((rc = dal(c, &d.f, 9 * cells, err)) || (rc = dal(c, &d.fp, 9 * cells, err)) ||
        (rc = dal(c, &d.rho, cells, err)) || (rc = dal(c, &d.u, cells, err)) ||
        (rc = dal(c, &d.v, cells, err)) || (rc = dal(c, &d.ob, cells, err)) ||
        (rc = dal(c, &d.on, cells, err)))
        return rc;
    double** pa[] = {&d.xc, &d.uc, &d.om, &d.xco, &d.uco, &d.omo, &d.force, &d.torque};
    for (double** a : pa)
        if ((rc = dal(c, a, np3, err))) return rc;
    const size_t nodes = (size_t)p.nx * p.ny;
    if ((rc = dal(c, &d.bl_list, nodes, err)) || (rc = dal(c, &d.bl_pos, cells, err)) ||
        (rc = dal(c, &d.lc, NODE_LINKS * nodes, err)) ||
        (rc = dal(c, &d.lt, NODE_TERMS * nodes, err)) ||
        (rc = dal(c, &d.done, 2, err)))
        return rc;
    const size_t nch = (size_t)gs_chunks((long long)p.nx * p.ny);
    for (GsBuf* b : {&d.ga, &d.gb})
        if ((rc = dal(c, &b->part, nch, err)) || (rc = dal(c, &b->cnt, nch, err)) ||
            (rc = dal(c, &b->piece, nch * GS_PIECES, err)) || (rc = dal(c, &b->np, nch, err)) ||
            (rc = dal(c, &b->done, 1, err)))
            return rc;
    if ((rc = dal(c, &d.rf_count, 1, err)) || (rc = dal(c, &d.rf_list, RF_CAP, err))) return rc;
    if ((rc = dal(c, &d.ravg, 2, err)) || (rc = dal(c, &d.status, 3, err)) ||
        (rc = dal(c, &c->owner_tmp, (size_t)p.nx * p.ny, err)))
        return rc;
    c->centers.assign(3 * (size_t)p.np, 0.0);
    for (int q = 0; q < p.np; q++) {
        c->centers[3 * q] = centers_xy[2 * q];
        c->centers[3 * q + 1] = centers_xy[2 * q + 1];
    }
    return ck(cudaStreamSynchronize(c->s), "create", err);
}

void p2d_destroy(P2Ctx* c) {
    if (!c) return;
    D2& d = c->d;
    void* ps[] = {d.f, d.fp, d.rho, d.u, d.v, d.ob, d.on, d.xc, d.uc, d.om, d.xco, d.uco, d.omo,
                  d.force, d.torque, d.ravg, d.status, d.bl_list, d.bl_pos, d.lc, d.lt, d.done,
                  c->owner_tmp, d.ga.part, d.ga.cnt, d.ga.piece, d.ga.np, d.ga.done, d.gb.part,
                  d.gb.cnt, d.gb.piece, d.gb.np, d.gb.done, d.rf_count, d.rf_list};
    if (c->side) cudaStreamSynchronize(c->side);
    if (c->s) cudaStreamSynchronize(c->s);
    for (void* p : ps)
        if (p) cudaFree(p);
    if (c->fork) cudaEventDestroy(c->fork);
    if (c->join) cudaEventDestroy(c->join);
    if (c->side) cudaStreamDestroy(c->side);
    if (c->own_stream && c->s) cudaStreamDestroy(c->s);
    delete c;
}

int p2d_set_stream(P2Ctx* c, cudaStream_t s) {
    if (c->own_stream && c->s) cudaStreamSynchronize(c->s);
    if (!s) return MGLC_OK;  // keep the current stream
    if (c->own_stream) cudaStreamDestroy(c->s);
    c->s = s;
    c->own_stream = false;
    return MGLC_OK;
}

int p2d_initial(P2Ctx* c, std::string& err) {
    D2& d = c->d;
    const size_t cells = (size_t)d.X * (d.p.ny + 6), np3 = 3 * (size_t)(d.p.np > 0 ? d.p.np : 1);
    int rc = 0;
    for (auto& pr : {std::make_pair((void*)d.f, 9 * cells * 8), std::make_pair((void*)d.fp, 9 * cells * 8),
                     std::make_pair((void*)d.ob, cells * 4), std::make_pair((void*)d.on, cells * 4),
                     std::make_pair((void*)d.uc, np3 * 8), std::make_pair((void*)d.om, np3 * 8),
                     std::make_pair((void*)d.force, np3 * 8), std::make_pair((void*)d.torque, np3 * 8),
                     std::make_pair((void*)d.status, (size_t)12),
                     std::make_pair((void*)d.done, (size_t)8),
                     std::make_pair((void*)d.ga.done, (size_t)4),
                     std::make_pair((void*)d.gb.done, (size_t)4),
                     std::make_pair((void*)d.rf_count, (size_t)4)})
        if ((rc = ck(cudaMemsetAsync(pr.first, 0, pr.second, c->s), "reset", err))) return rc;
    if (d.p.np > 0) {
        if ((rc = ck(cudaMemcpyAsync(d.xc, c->centers.data(), sizeof(double) * 3 * d.p.np,
                                     cudaMemcpyHostToDevice, c->s), "centres", err)))
            return rc;
        if ((rc = ck(cudaMemcpyAsync(d.xco, d.xc, sizeof(double) * 3 * d.p.np, cudaMemcpyDeviceToDevice,
                                     c->s), "centres", err)))
            return rc;
    }
    if (d.p.variant == P2_SHEAR && d.p.np > 0) {  // case1 initial.F90:61-70
        std::vector<double> uc(3 * (size_t)d.p.np, 0.0);
        for (int q = 0; q < d.p.np; q++) uc[3 * q] = d.p.moving_frame ? 0.0 : d.p.u0;
        if ((rc = ck(cudaMemcpyAsync(d.uc, uc.data(), sizeof(double) * uc.size(),
                                     cudaMemcpyHostToDevice, c->s), "velocities", err)))
            return rc;
        if ((rc = ck(cudaStreamSynchronize(c->s), "velocities", err))) return rc;
    }
    if (d.p.np > 0) launch_next(k2_mark, d.p.np, 256, 0, c->s, d, d.ob, false);
    k2_init_fields<<<dim3((d.p.nx + 6 + 127) / 128, d.p.ny + 6), 128, 0, c->s>>>(d);
    c->itc = 0;
    return ck(cudaStreamSynchronize(c->s), "initial", err);
}

int p2d_step(P2Ctx* c, int nsteps, std::string& err) {
    D2& d = c->d;
    const dim3 g = rows_grid(d);
    const bool shear = d.p.variant == P2_SHEAR;
    // a block per node around the circles (a longer list is walked in strides)
    const long long near = (long long)d.p.np * (8 * (long long)std::ceil(d.p.radius) + 32);
    const int bg = (int)std::min<long long>(std::max<long long>(near, 1), 152 * 16);
    const int total = d.p.nx * d.p.ny;
    int rc = MGLC_OK;
    D2 prev = d;  // the last step's masks
    for (int n = 0; n < nsteps; n++) {
        if ((rc = ck(cudaEventRecord(c->fork, c->s), "fork", err)) ||
            (rc = ck(cudaStreamWaitEvent(c->side, c->fork, 0), "fork", err)))
            return rc;
        if (n > 0) gs_launch(RhoFetch<true>{prev, true}, total, d.gb, c->side);
        gs_launch(RhoFetch<false>{d, false}, total, d.ga, c->side);
        if ((rc = ck(cudaEventRecord(c->join, c->side), "join", err))) return rc;
        if (shear) launch_next(k2_collide<true>, g, 128, 0, c->s, d, n > 0);
        else launch_next(k2_collide<false>, g, 128, 0, c->s, d, n > 0);
        if ((rc = ck(cudaStreamWaitEvent(c->s, c->join, 0), "join", err))) return rc;
        if (shear) launch_next(k2_stream<true>, g, 128, 0, c->s, d);
        else launch_next(k2_stream<false>, g, 128, 0, c->s, d);
        if (d.p.np > 0) {
            launch_next(k2_boundary, bg, 256, 0, c->s, d);
            launch_next(k2_force, d.p.np, FB, 0, c->s, d);
            launch_next(k2_mark, d.p.np, 256, 0, c->s, d, d.on, true);
        }
        prev = d;
        std::swap(d.ob, d.on);
        d.par ^= 1;
        c->itc++;
    }
    if (nsteps > 0) gs_launch(RhoFetch<true>{prev, false}, total, d.gb, c->s);
    int st[3] = {0, 0, 0};
    rc = ck(cudaGetLastError(), "particle step launch", err);
    if (!rc) rc = ck(cudaMemcpyAsync(st, d.status, sizeof st, cudaMemcpyDeviceToHost, c->s), "status", err);
    if (!rc) rc = ck(cudaStreamSynchronize(c->s), "particle step", err);
    if (rc) return rc;
    if (st[0]) {
        if (st[2] != d.par) {  // the mask the state is frozen with
            std::swap(d.ob, d.on);
            d.par ^= 1;
        }
        static const char* what[] = {"", "no circle owns a solid boundary node",
                                     "interpolation fraction q outside [0,1]",
                                     "particle-particle interpenetration",
                                     "particle penetrates a wall",
                                     "no refill direction for a node leaving a circle"};
        char buf[200];
        std::snprintf(buf, sizeof buf, "%s (circle %d); the state is frozen at that step",
                      what[st[0] < 6 ? st[0] : 0], st[1]);
        err = buf;
        return MGLC_ERR_PARTICLE;
    }
    return MGLC_OK;
}

namespace {
// interior of a padded device array, row by row (x fastest)
template <typename T>
int get_interior(P2Ctx* c, const T* dev, int per, T* host, std::string& err) {
    const D2& d = c->d;
    const size_t pitch = sizeof(T) * per * d.X;
    const T* first = dev + (size_t)per * (3 + (size_t)d.X * 3);  // node (1, 1)
    cudaError_t e = cudaMemcpy2DAsync(host, sizeof(T) * per * d.p.nx, first, pitch,
                                      sizeof(T) * per * d.p.nx, d.p.ny, cudaMemcpyDeviceToHost, c->s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(c->s);
    return ck(e, "copy to host", err);
}
}  // namespace

// the interior populations, population fastest, plane by plane through a
// device buffer of the host array's layout
__global__ void __launch_bounds__(128) k2_pack_f(D2 d, double* out) {
    const int i = 1 + blockIdx.x * blockDim.x + threadIdx.x, j = 1 + blockIdx.y;
    if (i > d.p.nx) return;
    double* o = out + 9 * ((size_t)(i - 1) + (size_t)d.p.nx * (j - 1));
#pragma unroll
    for (int a = 0; a < 9; a++) o[a] = d.f[a * d.C + IX(d, i, j)];
}

int p2d_get_f(P2Ctx* c, double* f, std::string& err) {
    const D2& d = c->d;
    static_assert(NODE_TERMS >= 9, "lt takes the populations");  // it holds nothing between steps
    k2_pack_f<<<rows_grid(d), 128, 0, c->s>>>(d, d.lt);
    int rc = ck(cudaGetLastError(), "copy to host", err);
    if (rc) return rc;
    cudaError_t e = cudaMemcpyAsync(f, d.lt, sizeof(double) * 9 * d.p.nx * d.p.ny,
                                    cudaMemcpyDeviceToHost, c->s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(c->s);
    return ck(e, "copy to host", err);
}

int p2d_get_macros(P2Ctx* c, double* rho, double* u, double* v, double* w, std::string& err) {
    int rc = 0;
    if (rho && (rc = get_interior(c, c->d.rho, 1, rho, err))) return rc;
    if (u && (rc = get_interior(c, c->d.u, 1, u, err))) return rc;
    if (v && (rc = get_interior(c, c->d.v, 1, v, err))) return rc;
    if (w) std::memset(w, 0, sizeof(double) * (size_t)c->d.p.nx * c->d.p.ny);
    return MGLC_OK;
}

int p2d_state(P2Ctx* c, double* xc, double* uc, double* omega, double* force, double* torque,
              std::string& err) {
    const D2& d = c->d;
    const size_t b = sizeof(double) * 3 * d.p.np;
    const double* src[] = {d.xc, d.uc, d.om, d.force, d.torque};
    double* dst[] = {xc, uc, omega, force, torque};
    for (int q = 0; q < 5; q++)
        if (dst[q] && b) {
            int rc = ck(cudaMemcpyAsync(dst[q], src[q], b, cudaMemcpyDeviceToHost, c->s), "state", err);
            if (rc) return rc;
        }
    return ck(cudaStreamSynchronize(c->s), "state", err);
}

int p2d_mask(P2Ctx* c, int* owner, std::string& err) {
    const D2& d = c->d;
    k2_owner<<<rows_grid(d), 128, 0, c->s>>>(d, c->owner_tmp);
    cudaError_t e = cudaMemcpyAsync(owner, c->owner_tmp, sizeof(int) * (size_t)d.p.nx * d.p.ny,
                                    cudaMemcpyDeviceToHost, c->s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(c->s);
    return ck(e, "mask", err);
}

long long p2d_itc(const P2Ctx* c) { return c->itc; }
long long p2d_device_bytes(const P2Ctx* c) { return c->bytes; }

double p2d_rho_avg(P2Ctx* c) {
    double r = 0.0;
    cudaMemcpyAsync(&r, c->d.ravg + 1, sizeof r, cudaMemcpyDeviceToHost, c->s);
    cudaStreamSynchronize(c->s);
    return r;
}

}  // namespace mglc

extern "C" int mglc_sequential_sum(const double* x, const int* keep, int n, double* sum,
                                   long long* count) {
    if (n < 0 || !x || !keep || !sum || !count) return MGLC_ERR_INVALID;
    const size_t m = n > 0 ? (size_t)n : 1, nch = (size_t)mglc::gs_chunks(n);
    double *dx = nullptr, *dout = nullptr;
    int* dk = nullptr;
    mglc::GsBuf b{};
    cudaError_t e = cudaMalloc(&dx, m * sizeof(double));
    if (e == cudaSuccess) e = cudaMalloc(&dk, m * sizeof(int));
    if (e == cudaSuccess) e = cudaMalloc(&dout, 2 * sizeof(double));
    if (e == cudaSuccess) e = cudaMalloc(&b.part, nch * sizeof(double));
    if (e == cudaSuccess) e = cudaMalloc(&b.cnt, nch * sizeof(int));
    if (e == cudaSuccess) e = cudaMalloc(&b.piece, nch * mglc::GS_PIECES * sizeof(mglc::GsPiece));
    if (e == cudaSuccess) e = cudaMalloc(&b.np, nch * sizeof(int));
    if (e == cudaSuccess) e = cudaMalloc(&b.done, sizeof(unsigned));
    if (e == cudaSuccess) e = cudaMemset(b.done, 0, sizeof(unsigned));
    if (e == cudaSuccess && n > 0) e = cudaMemcpy(dx, x, (size_t)n * sizeof(double), cudaMemcpyHostToDevice);
    if (e == cudaSuccess && n > 0) e = cudaMemcpy(dk, keep, (size_t)n * sizeof(int), cudaMemcpyHostToDevice);
    double out[2] = {0.0, 0.0};
    if (e == cudaSuccess) {
        mglc::gs_launch(mglc::ArrayFetch{dx, dk, n, dout}, n, b, 0);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpy(out, dout, sizeof out, cudaMemcpyDeviceToHost);
    void* ps[] = {dx, dk, dout, b.part, b.cnt, b.piece, b.np, b.done};
    for (void* p : ps)
        if (p) cudaFree(p);
    if (e != cudaSuccess) return MGLC_ERR_CUDA;
    *sum = out[0];
    *count = (long long)out[1];
    return MGLC_OK;
}
