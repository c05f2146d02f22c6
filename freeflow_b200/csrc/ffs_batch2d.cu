// Batched D2Q9 kernels of the serving pool: every kernel covers all admitted
// episodes of the pool in one launch (the dense pass with link detection is in
// ffs_dense2d.cu).
//
// Work items are numbered across episodes through the prefix sums of the
// active table (march units, surface elements, surface vertices); an item
// finds its episode by a binary search over at most kPoolMaxSlots prefixes.
// The per-item bodies are the single-grid ones (march2::run,
// detect_elements2_warp, link_cell_update2), so a pool episode computes bit for
// bit what the same grid computes alone through ffs_lbm_step.  The grids are persistent
// (a fixed number of CTAs striding over a count read from device memory), so
// one captured CUDA graph serves every mix of episodes.
//
// Reference: one Simulator2D per environment process, each step through
// fsi_coupling::solveLbmAndFsiStep2D (src/core/FsiCoupling2D.cu:358-432);
// the environment loop is rl/env.py:163-217.
#include "ffs_links_dev.cuh"
#include "ffs_pool.cuh"

namespace fflbm {

// ------------------------------------------------------------ kinematics
// Vertex v of an episode's swimmer at a substep (entry p of the parameters).
__device__ __forceinline__ void move_vertex(const PoolEpisode &e, const PoolParams &p, uint32_t v, int substep)
{
    float x, y, vx, vy;
    swimmer_vertex(e.rest[2 * v], e.rest[2 * v + 1], e.amp[v], e.sin_kx[v], e.cos_kx[v], e.segment[v], p.actions,
                   p.sb[substep], p.cb[substep], e.wave_omega, x, y, vx, vy);
    e.V[2 * v] = x;
    e.V[2 * v + 1] = y;
    e.U[2 * v] = vx;
    e.U[2 * v + 1] = vy;
}

// The surfaces of a control step's first substep (pool_finalize_kernel moves
// them on from there).
__global__ void pool_kinematics_kernel(const PoolEpisode *eps, const PoolParams *prm, const PoolActive *act,
                                       uint32_t *unit_next)
{
    after_predecessor();
    if (blockIdx.x == 0 && threadIdx.x < 2) unit_next[threadIdx.x] = 0; // the next dense pass counts from them
    const int n = (int)act->n;
    if (n == 0) return;
    const uint32_t total = act->vert_prefix[n];
    for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < total; t += gridDim.x * blockDim.x) {
        const int a = owner_of(act->vert_prefix, n, t);
        move_vertex(eps[act->slot[a]], prm[a], t - act->vert_prefix[a], 0);
    }
}

// ------------------------------------------------------------ link cells
template <typename T>
__global__ void __launch_bounds__(256, 2) pool_link_cells_kernel(const PoolEpisode *eps, LinkTable lt,
                                                                 const uint32_t *owner, int parity)
{
    constexpr int Q = 9, G = kPoolLinkGroup, kPerWarp = 32 / G;
    const int lane = threadIdx.x & (G - 1);
    const uint32_t group = (threadIdx.x & 31) / G;
    const uint32_t nwarps = (gridDim.x * blockDim.x) >> 5;
    after_predecessor();
    const LinkItems items(lt);
    const uint32_t n = items.n;
    // consecutive cells go to different CTAs: a few cells spread over the SMs
    for (uint32_t w = ((threadIdx.x >> 5) * gridDim.x + blockIdx.x) * kPerWarp; w < n; w += nwarps * kPerWarp) {
        // eight cells per warp, possibly of different episodes; a group past the
        // end of the list rides along on the first group's cell
        const bool valid = w + group < n;
        const uint32_t slot = items.slot(lt, valid ? w + group : w);
        const PoolEpisode &e = eps[owner[slot]];
        const uint32_t cell = lt.keys[slot] - 1 - e.cell_base;
        const GridArgs<T> g = episode_args<T>(e, parity);
        const SurfaceArgs sa = episode_surface(e);
        const StepScalars sc{e.cl, e.ct, e.cf};
        link_cell_update2<T, false, G>(g, lt.links, slot, cell, e.acc, sa, sc, valid);
        for (int l = lane; valid && l < Q; l += G) lt.links[(size_t)slot * Q + l] = ~0ull;
        __syncwarp();
        if (valid && lane == 0) {
            lt.keys[slot] = 0;
            set_link_bit(reinterpret_cast<uint32_t *>(e.flags), cell, false);
        }
    }
}

// -------------------------------------------------------------- finalize
// One CTA per active episode: scales the fixed-point sums to forces, clears
// them, and reduces total force, torque and power in a fixed order (so the
// sums do not depend on the mix or on launch order).
// The CTA then moves the episode's surface to substep `next` (if not 0), which
// saves a launch per substep.
__global__ void __launch_bounds__(256) pool_finalize_kernel(const PoolEpisode *eps, const PoolParams *prm,
                                                            const PoolActive *act, LinkTable lt, uint32_t *unit_next,
                                                            int next)
{
    __shared__ double red[4][8];
    after_predecessor();
    if (blockIdx.x == 0 && threadIdx.x < 2) unit_next[threadIdx.x] = 0; // the next dense pass counts from them
    const int n = (int)act->n;
    if (blockIdx.x == 0) clear_counts(lt);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int a = blockIdx.x; a < n; a += gridDim.x) {
        const PoolEpisode &e = eps[act->slot[a]];
        double fx = 0.0, fy = 0.0, tq = 0.0, pw = 0.0;
        for (int v = threadIdx.x; v < e.nv; v += blockDim.x) {
            // the single-grid finalize's expression (finalize_forces_kernel)
            const double f0 = (double)e.acc[2 * v] * (1.0 / kForceScale) * e.cf;
            const double f1 = (double)e.acc[2 * v + 1] * (1.0 / kForceScale) * e.cf;
            e.acc[2 * v] = 0;
            e.acc[2 * v + 1] = 0;
            e.force[2 * v] = f0;
            e.force[2 * v + 1] = f1;
            const double rx = (double)e.V[2 * v] - (double)e.cx0, ry = (double)e.V[2 * v + 1] - (double)e.cy0;
            fx += f0;
            fy += f1;
            tq += rx * f1 - ry * f0;
            pw -= f0 * (double)e.U[2 * v] + f1 * (double)e.U[2 * v + 1];
            if (next) move_vertex(e, prm[a], (uint32_t)v, next); // this thread's vertex is done with
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            fx += __shfl_xor_sync(0xffffffffu, fx, o);
            fy += __shfl_xor_sync(0xffffffffu, fy, o);
            tq += __shfl_xor_sync(0xffffffffu, tq, o);
            pw += __shfl_xor_sync(0xffffffffu, pw, o);
        }
        if (lane == 0) {
            red[0][warp] = fx;
            red[1][warp] = fy;
            red[2][warp] = tq;
            red[3][warp] = pw;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            double s[4] = {0.0, 0.0, 0.0, 0.0};
            for (int w = 0; w < (int)(blockDim.x >> 5); ++w)
                for (int k = 0; k < 4; ++k) s[k] += red[k][w];
            // rl/env.py:172-175: energy += power * dt when the power is positive
            if (s[3] > 0.0) e.sums[0] += s[3] * (double)e.ct;
            e.sums[1] += s[0];
            e.sums[2] += s[1];
            e.sums[3] += s[2];
        }
        __syncthreads();
    }
}

// One thread per active episode: publish the control step's sums and the
// latched status, then clear them for the next control step.
__global__ void pool_outputs_kernel(const PoolEpisode *eps, const PoolActive *act, PoolOutput *out, int substeps)
{
    after_predecessor();
    const int n = (int)act->n;
    const double inv = 1.0 / (double)substeps;
    for (int a = blockIdx.x * blockDim.x + threadIdx.x; a < n; a += gridDim.x * blockDim.x) {
        const uint32_t s = act->slot[a];
        const PoolEpisode &e = eps[s];
        PoolOutput o;
        o.energy = e.sums[0];
        o.force[0] = e.sums[1] * inv;
        o.force[1] = e.sums[2] * inv;
        o.torque = e.sums[3] * inv;
        o.status = *e.status;
        o.pad = 0;
        out[s] = o;
        for (int k = 0; k < 4; ++k) e.sums[k] = 0.0;
        *e.status = 0;
    }
}

// -------------------------------------------------------------- launchers
cudaError_t launch_pool_kinematics(const PoolEpisode *eps, const PoolParams *prm, const PoolActive *act,
                                   uint32_t *unit_next, int grid, cudaStream_t st)
{
    return launch_chained(pool_kinematics_kernel, grid, 256, st, eps, prm, act, unit_next);
}

template <typename T> int pool_link_cells_blocks_per_sm()
{
    int blocks = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, pool_link_cells_kernel<T>, 256, 0) != cudaSuccess ||
        blocks < 1)
        blocks = 1;
    return blocks;
}

template <typename T>
cudaError_t launch_pool_link_cells(const PoolEpisode *eps, const LinkTable &lt, const uint32_t *owner, int parity,
                                   int grid, cudaStream_t st)
{
    return launch_chained(pool_link_cells_kernel<T>, grid, 256, st, eps, lt, owner, parity);
}

cudaError_t launch_pool_finalize(const PoolEpisode *eps, const PoolParams *prm, const PoolActive *act,
                                 const LinkTable &lt, uint32_t *unit_next, int next, int grid, cudaStream_t st)
{
    return launch_chained(pool_finalize_kernel, grid, 256, st, eps, prm, act, lt, unit_next, next);
}

cudaError_t launch_pool_outputs(const PoolEpisode *eps, const PoolActive *act, PoolOutput *out, int substeps,
                                cudaStream_t st)
{
    return launch_chained(pool_outputs_kernel, (kPoolMaxSlots + 127) / 128, 128, st, eps, act, out, substeps);
}

#define FFS_INST_POOL(T)                                                                                               \
    template int pool_link_cells_blocks_per_sm<T>();                                                                   \
    template cudaError_t launch_pool_link_cells<T>(const PoolEpisode *, const LinkTable &, const uint32_t *, int, int, \
                                                   cudaStream_t);
FFS_INST_POOL(float)
FFS_INST_POOL(__half)
FFS_INST_POOL(__nv_bfloat16)

} // namespace fflbm
