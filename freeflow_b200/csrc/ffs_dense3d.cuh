#pragma once
#include "ffs_common.cuh"

namespace fflbm {

// Tile geometry of the z-marching D3Q27 kernel (ffs_dense3d.cu).
struct D3 {
    static constexpr int kTX = 32, kTY = 8, kTile = kTX * kTY;
    static constexpr int kHX = kTX + 2, kHY = kTY + 2, kHalo = kHX * kHY;
    static constexpr int kRing = kHalo - kTile;               // halo cells around the tile
    static constexpr int kPlaneFloats = 27 * kHalo;           // all populations of one halo plane
    static constexpr size_t kSmemBytes = 2 * (size_t)kPlaneFloats * sizeof(float); // double buffer
};

// The fused D3Q27 pass over a grid.
template <typename T> cudaError_t launch_dense3d(const GridArgs<T> &g, cudaStream_t s);

} // namespace fflbm
