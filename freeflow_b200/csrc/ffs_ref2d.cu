// D2Q9 dense pass for grids with options of the reference's own 2D kernel: the
// binary16 tile (ref_half_populations) and walls that stream
// (ref_2d_wall_stream); also grids whose moment indices do not fit in 32 bits.
//
// Reference: mrDeformableSolver2DKernel_Shrd (src/core/FsiCoupling2D.cu:82-255)
// followed by mrApplyOutlet2DKernel (:257-316).
//
// One CTA = one 32 x 8 tile, its populations plus a one-cell halo in shared
// memory, a thread per cell.
#include "ffs_dense2d.cuh"

namespace fflbm {

template <typename T, bool HALF> __global__ void __launch_bounds__(D2::kThreads) ref2d_kernel(GridArgs<T> g)
{
    using L = Lattice<2>;
    __shared__ float sp[9][D2::kHY][D2::kHX];
    const int tid = threadIdx.x, x0 = blockIdx.x * D2::kTX, y0 = blockIdx.y * D2::kTY;
    const bool wx = g.periodic & 1, wy = g.periodic & 2;
    constexpr int kPer = (D2::kHalo + D2::kThreads - 1) / D2::kThreads;
    T raw[kPer][6];
#pragma unroll
    for (int r = 0; r < kPer; ++r) {
        const int c = tid + r * D2::kThreads;
        if (c < D2::kHalo) {
            const int hx = c % D2::kHX, hy = c / D2::kHX;
            const uint32_t idx = (uint32_t)(halo_index(y0 + hy - 1, g.ny, wy) * g.nx + halo_index(x0 + hx - 1, g.nx, wx));
#pragma unroll
            for (int k = 0; k < 6; ++k) raw[r][k] = g.src[(size_t)k * g.ncell + idx];
        }
    }
#pragma unroll
    for (int r = 0; r < kPer; ++r) {
        const int c = tid + r * D2::kThreads;
        if (c < D2::kHalo) {
            const int hx = c % D2::kHX, hy = c / D2::kHX;
            float m[6], f[9];
#pragma unroll
            for (int k = 0; k < 6; ++k) m[k] = from_storage<2, T>(k, raw[r][k]);
            decode_moments<2, T>(m, g.codec);
            Coef<2> cf;
            cf.make(m);
            cf.populations(f);
#pragma unroll
            for (int i = 0; i < 9; ++i) sp[i][hy][hx] = HALF ? round_half(f[i]) : f[i];
        }
    }
    __syncthreads();

    const int tx = tid % D2::kTX, ty = tid / D2::kTX, x = x0 + tx, y = y0 + ty;
    if (x >= g.nx || y >= g.ny) return;
    const uint32_t idx = (uint32_t)(y * g.nx + x);
    const uint32_t f8 = g.flags[idx];
    if (!is_updated(f8 & kTypeMask) || (f8 & kBitLink)) return;
    float pop[9];
#pragma unroll
    for (int i = 0; i < 9; ++i) pop[i] = sp[i][ty + 1 - L::cy(i)][tx + 1 - L::cx(i)];
    const uint32_t wm = (f8 & (kBitNearWall | kBitOutletSrc)) ? g.wallmask[idx] : 0u;
    if ((f8 & kBitNearWall) && !g.wall_stream) {
        // bounce-back: f_i(x) = f_inv(i)^rec(x) when x - c_i is a wall (with
        // wall_stream the reference's 2D kernel is followed instead: it
        // overwrites that value with the ordinary pull, FsiCoupling2D.cu:
        // 171-224, since is_blocked is set only on the moving-wall path)
#pragma unroll
        for (int i = 1; i < 9; ++i)
            if (wm & (1u << i)) pop[i] = sp[L::inv(i)][ty + 1][tx + 1];
    }
#pragma unroll
    for (int i = 0; i < 9; ++i) pop[i] = fmaxf(pop[i], 0.0f);
    float R[6], m[6];
    raw_moments2(pop, R);
    collide2(R, g.omega, m);
    encode_store_strided<2, T>(m, g.dst, idx, g.ncell, g.codec);
    if (bad_state<2>(m)) atomicOr(g.status, kStatusNonFinite);
    if (f8 & g.feed) {
        float ms[6];
        stored_values<2, T>(m, ms, idx, g.codec);
        feed_outlets<2, T>(g, idx, ms, wm);
    }
}

template <typename T> cudaError_t launch_ref2d(const GridArgs<T> &g, cudaStream_t s)
{
    const dim3 grid((g.nx + D2::kTX - 1) / D2::kTX, (g.ny + D2::kTY - 1) / D2::kTY);
    if (g.half_pops) ref2d_kernel<T, true><<<grid, D2::kThreads, 0, s>>>(g);
    else ref2d_kernel<T, false><<<grid, D2::kThreads, 0, s>>>(g);
    return cudaGetLastError();
}
template cudaError_t launch_ref2d<float>(const GridArgs<float> &, cudaStream_t);
template cudaError_t launch_ref2d<__half>(const GridArgs<__half> &, cudaStream_t);
template cudaError_t launch_ref2d<__nv_bfloat16>(const GridArgs<__nv_bfloat16> &, cudaStream_t);

} // namespace fflbm
