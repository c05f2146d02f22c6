// What the dense passes share: the D2Q9 tile's shape and the halo's source cells.
#pragma once
#include "ffs_common.cuh"
#include "ffs_math.cuh"
#include "ffs_outlet.cuh"

namespace fflbm {

struct D2 {
    static constexpr int kTX = 32, kTY = 8, kThreads = kTX * kTY;
    static constexpr int kHX = kTX + 2, kHY = kTY + 2, kHalo = kHX * kHY;
};

// Source index of a halo cell, as the reference's shared-memory fill computes
// it (FsiCoupling2D.cu:104-105, FsiCoupling3D.cu:106-108):
// min(n - 1, max(0, (sm - 1) + blockDim * blockIdx)).  blockDim * blockIdx is
// unsigned, so below the grid the sum wraps to a huge unsigned value and the
// index comes out as n - 1; above it the min clamps to n - 1.  The halo
// therefore wraps at the low face and clamps at the high face of every axis.
// A periodic axis wraps at both.  v >= -1 always; v may exceed n by a tile
// width.
__device__ __forceinline__ int halo_index(int v, int n, bool wrap)
{
    if (!wrap) return (v < 0 || v >= n) ? n - 1 : v;
    if (v < 0) v += n;
    if (v >= n) v -= n;
    if (v >= n) v %= n;
    return v;
}

// The step of grids with the reference's own 2D options (ffs_ref2d.cu).
template <typename T> cudaError_t launch_ref2d(const GridArgs<T> &g, cudaStream_t s);

} // namespace fflbm
