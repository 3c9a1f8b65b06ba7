// cell_map.cuh -- which cell a thread of a cavity step kernel works on.
//
// CellMap: thread t takes cell t of the linear order, so no lane is idle whatever
// nx is; its coordinates come from two divisions by multiplication.
// RowMap: a block takes a segment of a row of x, j and k are the block's.
// linear_cells picks the first where rows would leave lanes or blocks part empty
// (24% of the lanes at nx = 97) and 32-bit indices serve: us a step, rows against
// linear, FP32 lid 97^3 31.3 / 28.2, in place 23.7 / 21.5, heated 81^3 24.8 / 23.2,
// FP64 lid 33^3 10.5 / 8.5, 48^3 14.5 / 12.5, heated 65^3 53.5 / 40.9.  Full rows cost
// less to index: FP64 lid 32^3 8.2 / 9.3, heated 128^3 240 / 245, FP32 lid 128^3
// 56.4 / 56.9.  Blocks of 32 or 64 threads instead of 128 changed nothing.
#pragma once
#include <cuda_runtime.h>

#include "kernels.cuh"

namespace mglc {

// n / d for 0 <= n < 2^31, d >= 2: with 2^(l-1) < d <= 2^l and
// m = floor(2^(31+l) / d) + 1, the error e = m d - 2^(31+l) is at most 2^l, so
// floor(n m / 2^(31+l)) is the quotient (Granlund and Montgomery, "Division by
// invariant integers using multiplication", PLDI 1994, theorem 4.2).
struct DivBy {
    unsigned m;
    int s;  // l - 1
    __host__ __device__ __forceinline__ unsigned operator()(unsigned n) const {
#ifdef __CUDA_ARCH__
        return __umulhi(n, m) >> s;
#else
        return (unsigned)((unsigned long long)n * m >> 32) >> s;
#endif
    }
};
inline DivBy make_div(int d) {
    int l = 1;
    while ((1ll << l) < d) l++;
    return {(unsigned)((1ull << (31 + l)) / (unsigned)d + 1), l - 1};
}

struct CellMap {
    DivBy x, y;
    explicit CellMap(const Geom& g) : x(make_div(g.nx)), y(make_div(g.ny)) {}
    // coordinates of this thread's cell; false: it has none
    template <typename IDX>
    __device__ __forceinline__ bool at(int nx, int ny, IDX P, int& i, int& j, int& k) const {
        const unsigned c = blockIdx.x * blockDim.x + threadIdx.x;
        if (c >= (unsigned)P) return false;
        const unsigned r = x(c);
        i = (int)(c - r * (unsigned)nx);
        k = (int)y(r);
        j = (int)(r - (unsigned)k * (unsigned)ny);
        return true;
    }
};
struct RowMap {
    explicit RowMap(const Geom&) {}
    template <typename IDX>
    __device__ __forceinline__ bool at(int nx, int, IDX, int& i, int& j, int& k) const {
        i = blockIdx.x * blockDim.x + threadIdx.x;
        j = blockIdx.y;
        k = blockIdx.z;
        return i < nx;
    }
};

// 32-bit population indices?
inline bool index32(const Geom& g) { return 19 * g.plane < (1ll << 31); }

inline bool linear_cells(const Geom& g) {
    return index32(g) && (g.nx % 32 != 0 || (g.nx > 128 && g.nx % 128 != 0));
}

// launch shape of either mapping
struct CellLaunch {
    dim3 grid, block;
    explicit CellLaunch(const Geom& g) {
        if (linear_cells(g)) {
            block = dim3(128);
            grid = dim3((unsigned)((g.plane + 127) / 128));
        } else {
            int bx = ((g.nx + 31) / 32) * 32;
            if (bx > 128) bx = 128;
            block = dim3(bx);
            grid = dim3((g.nx + bx - 1) / bx, g.ny, g.nz);
        }
    }
};

}  // namespace mglc
