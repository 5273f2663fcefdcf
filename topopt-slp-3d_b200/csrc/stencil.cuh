// A node's product with a node-major stencil by one warp, shared by the sweeps of
// the small levels and the persistent cycle.
//
// The node's 243 values (offset o, row, column) are one run: value 27 k + l goes
// to lane l < 27, so each of the nine loads is contiguous, and since 27 is three
// blocks of nine, a lane keeps its row and column and needs one accumulator; its
// offsets are 3 k + l / 9, that is (x, z) from k and y from the lane, and the
// lanes' values of x are neighbours as well.  A lane per offset, nine values each,
// takes the same loads with a stride of 72 bytes: 16 lines a load where three do.
#pragma once

#include "tosp_internal.h"

namespace tosp {

template <typename T>
__device__ __forceinline__ void stencil_load(const T *__restrict__ sv, int lane, T (&s)[9]) {
#pragma unroll
    for (int k = 0; k < 9; ++k) s[k] = lane < 27 ? __ldg(sv + 27 * k + lane) : T(0);
}
// (K x) at node I = (xx, yy, zz): row r of it in lane 3 r.  ldx(d): x at dof d.
template <typename T, typename L>
__device__ __forceinline__ T stencil_apply(const T (&s)[9], L ldx, int I, int xx, int yy, int zz, const Grid &g,
                                           int lane) {
    const int oy = lane / 9 - 1, col = lane % 3;
    const bool iny = lane < 27 && (unsigned)(yy + oy) < (unsigned)g.ny;
    const int d0 = 3 * (I + oy) + col, rowx = 3 * g.ny, rowz = rowx * g.nx;
    T x[9], acc[3] = {T(0), T(0), T(0)};
#pragma unroll
    for (int k = 0; k < 9; ++k) {
        const int ox = k % 3 - 1, oz = k / 3 - 1;
        const bool in = iny && (unsigned)(xx + ox) < (unsigned)g.nx && (unsigned)(zz + oz) < (unsigned)g.nz;
        x[k] = in ? ldx(d0 + oz * rowz + ox * rowx) : T(0);
    }
#pragma unroll
    for (int k = 0; k < 9; ++k) acc[k % 3] += s[k] * x[k];
    T a = (acc[0] + acc[1]) + acc[2];
    a = (a + __shfl_down_sync(0xffffffffu, a, 9)) + __shfl_down_sync(0xffffffffu, a, 18);
    return (a + __shfl_down_sync(0xffffffffu, a, 1)) + __shfl_down_sync(0xffffffffu, a, 2);
}

}  // namespace tosp
