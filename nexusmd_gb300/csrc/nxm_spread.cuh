// B-spline weights and the charge-grid word of PME, shared by the engine's
// kernels (k_pme.cu) and the no-allocation entry (k_pme_noalloc.cu).
#pragma once

#include <cuda_runtime.h>

namespace nxm {

// Order-5 weights and derivatives at fraction dr, in the operation order of
// computeBSplineParameters (NonbondedForce.cpp:144-182).
template <typename R>
__device__ __forceinline__ void bspline5(R dr, R *th, R *dth) {
    th[4] = 0;
    th[1] = dr;
    th[0] = 1 - dr;
#pragma unroll
    for (int k = 3; k < 5; k++) {
        R div = (R)1 / (R)(k - 1);
        th[k - 1] = div * dr * th[k - 2];
#pragma unroll
        for (int l = 1; l < (k - 1); l++)
            th[k - l - 1] = div * ((dr + l) * th[k - l - 2] + ((R)(k - l) - dr) * th[k - l - 1]);
        th[0] = div * (1 - dr) * th[0];
    }
    dth[0] = -th[0];
#pragma unroll
    for (int k = 1; k < 5; k++) dth[k] = th[k - 1] - th[k];
    R div = (R)0.25;
    th[4] = div * dr * th[3];
#pragma unroll
    for (int l = 1; l < 4; l++) th[4 - l] = div * ((dr + l) * th[3 - l] + ((R)(5 - l) - dr) * th[4 - l]);
    th[0] = div * (1 - dr) * th[0];
}

// Mixed-mode grid word: int32 fixed point in units of 2^-24 e, for |Q| <
// 128 e per point.  A point holds q wx wy wz summed over the atoms whose
// 5-point stencils cover it, each weight at most 115/192 per axis (< 0.22 per
// atom), so physical charge densities stay two orders of magnitude inside the
// range.  Half the bytes of an int64 word per atomic: the spread's L2 atomic
// traffic is its bound (38 -> 33 us at 94,100 atoms on a 100^3 grid).
__device__ __forceinline__ int to_grid_fixed(float v) { return __float2int_rn(v * 16777216.0f); }
// One warp spreads one atom's 125 points, 32 consecutive ones per
// instruction: w holds wx[5] wy[5] wz[5] q, i0 the first grid index per axis.
// Consecutive points share grid rows (5 contiguous words per row), so one
// atomic instruction touches ~13 memory sectors instead of the 32 of one atom
// per lane.  Each value is ((q wx) wy) wz.
__device__ __forceinline__ void spread_points(const float *w, const int *i0, int K0, int K1, int K2, int *g,
                                              int lane) {
    const unsigned full = 0xffffffffu;
    // lane r < 25: grid row (ix, iy) = (r / 5, r % 5) of the atom, its
    // offset and its weight (q wx) wy
    long long row_off = 0;
    float row_w = 0.f;
    if (lane < 25) {
        const int ix = lane / 5, iy = lane - 5 * ix;
        int xi = i0[0] + ix, yi = i0[1] + iy;
        xi -= xi >= K0 ? K0 : 0;
        yi -= yi >= K1 ? K1 : 0;
        row_off = ((long long)xi * K1 + yi) * K2;
        row_w = w[15] * w[ix] * w[5 + iy];
    }
    const int z0 = i0[2];
    // point p = 5 row + iz
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const int p = lane + 32 * k;
        const int row = min(p / 5, 24), iz = min(p - 5 * row, 4);  // (clamped past point 124)
        const long long off = __shfl_sync(full, row_off, row);
        const float rw = __shfl_sync(full, row_w, row);
        int zi = z0 + iz;
        zi -= zi >= K2 ? K2 : 0;
        if (p < 125) atomicAdd(g + off + zi, to_grid_fixed(rw * w[10 + iz]));
    }
}

}  // namespace nxm
