// Fused D2Q9 step for all cells without moving-boundary links.
//
// Reference: mrDeformableSolver2DKernel_Shrd (src/core/FsiCoupling2D.cu:82-255)
// followed by mrApplyOutlet2DKernel (:257-316).
//
// Grids take the row march of ffs_march2d.cuh, one warp per unit of 64 columns
// and a few rows.  Outlet writes are issued by the outlet's feeding cell
// (ffs_outlet.cuh), so the step is one launch.  D2Q9 grids of the sizes
// FreeFlow runs (<= 1200 x 400) are L2-resident on B200, and the rows per unit
// are chosen by how much work the chip has (march_rows).
//
// Two options of the reference's own 2D kernel need populations as such: the
// binary16 tile (ref_half_populations) and walls that stream
// (ref_2d_wall_stream).  They, and grids whose moment indices do not fit in 32
// bits, take the tile kernel: one CTA = one 32 x 8 tile, its populations plus
// a one-cell halo in shared memory.
#include <algorithm>
#include <cstdlib>

#include "ffs_links_dev.cuh"
#include "ffs_march2d.cuh"
#include "ffs_pool.cuh"

namespace fflbm {

// March warps (one-warp CTAs) per SM that the register budget is cut for: four
// per scheduler leave 128 registers, which the march fills without spills; five
// (96 registers) spilled and ran the pool's pass 3 % slower, three 10 %.
constexpr int kMarchWarps = 16;

template <typename T, bool HALF>
__global__ void __launch_bounds__(D2::kThreads) dense2d_kernel(GridArgs<T> g)
{
    __shared__ float sp[9][D2::kHY][D2::kHX];
    dense2d_tile<T, HALF>(g, blockIdx.x * D2::kTX, blockIdx.y * D2::kTY, sp);
}

// The first `ndetect` CTAs detect the surface's links (`lanes` lanes an
// element), the others march.  A launch of its own for detection, on a second
// stream with events around it, cost more than detection itself on grids of
// this size.  Which link cells the march skips (it reads their LINK bit while
// detection sets it) does not matter: the link-cell kernel rewrites every link
// cell afterwards and feeds the outlets (ffs_outlet.cuh).
template <typename T, bool VEC>
__global__ void __launch_bounds__(32, kMarchWarps) march2d_kernel(GridArgs<T> g, int rows, int ndetect, int lanes, DetectArgs d)
{
    __shared__ march2::Ends ends;
    after_predecessor();
    if ((int)blockIdx.x < ndetect) {
        uint32_t *queue = reinterpret_cast<uint32_t *>(&ends);
        static_assert(sizeof(ends) >= 64 * sizeof(uint32_t), "the exact test's queue fits");
        const int per = 32 / lanes, group = (int)threadIdx.x / lanes;
        for (long long e = (long long)blockIdx.x * per; e < d.s.ne; e += (long long)ndetect * per)
            detect_elements2_warp<T>(g, d.flag_words, d.lt, d.s, d.sc, e + group, e + group < d.s.ne, lanes, queue);
        return;
    }
    const int W = march2::windows(g.nx), u = (int)blockIdx.x - ndetect;
    const int C = march2::chunks(g.ny, rows), c0 = u / W, w = u - c0 * W;
    // the top rows start right after the bottom ones: both may feed outlets,
    // which takes a unit longer (0.5 us of a 22 us step on 1200 x 400)
    const int c = c0 == 1 ? C - 1 : c0 > 1 ? c0 - 1 : 0;
    march2::Gate gate{nullptr, 0u, false};
    march2::run<T, VEC>(g, w, c * rows, min((c + 1) * rows, g.ny), ends, gate);
}

// Rows per unit: a unit reconstructs rows + 2 rows, a row of one warp alone
// takes about kRowLatency cycles, and a scheduler spends about kRowIssue on
// it, so few rows spread a small grid over the chip and many rows save the
// two extra ones where the chip is full.
static int march_rows(int nx, int ny)
{
    constexpr double kRowLatency = 900.0, kRowIssue = 310.0;
    const double schedulers = 4.0 * device_sms();
    int best = 1;
    double best_t = 1e300;
    for (int rows = 1; rows <= march2::kMaxRows; ++rows) {
        const double units = (double)march2::windows(nx) * march2::chunks(ny, rows);
        const double t = (rows + 2) * std::max(kRowLatency, units * kRowIssue / schedulers);
        if (t < best_t) { best_t = t; best = rows; }
    }
    // FFS_MARCH_ROWS pins the rows (tests run several)
    if (const char *e = std::getenv("FFS_MARCH_ROWS")) best = std::max(1, std::min(march2::kMaxRows, std::atoi(e)));
    return best;
}

template <typename T> bool dense2d_detects(const GridArgs<T> &g)
{
    return !g.half_pops && !g.wall_stream && 6ull * g.ncell <= 0xFFFFFFFFull;
}

template <typename T> cudaError_t launch_dense2d(const GridArgs<T> &g, cudaStream_t s, const DetectArgs *detect)
{
    if (!dense2d_detects(g)) {
        dim3 grid((g.nx + D2::kTX - 1) / D2::kTX, (g.ny + D2::kTY - 1) / D2::kTY);
        if (g.half_pops)
            dense2d_kernel<T, true><<<grid, D2::kThreads, 0, s>>>(g);
        else
            dense2d_kernel<T, false><<<grid, D2::kThreads, 0, s>>>(g);
        return cudaGetLastError();
    }
    const int rows = march_rows(g.nx, g.ny);
    const int units = march2::windows(g.nx) * march2::chunks(g.ny, rows);
    const int lanes = detect ? detect_lanes2(detect->s.ne, device_sms()) : 32, per = 32 / lanes;
    const int nd = detect ? (int)std::min<long long>(((long long)detect->s.ne + per - 1) / per, (long long)device_sms() * 32) : 0;
    const DetectArgs d = detect ? *detect : DetectArgs{};
    if (g.nx % 2 == 0) march2d_kernel<T, true><<<units + nd, 32, 0, s>>>(g, rows, nd, lanes, d);
    else march2d_kernel<T, false><<<units + nd, 32, 0, s>>>(g, rows, nd, lanes, d);
    return cudaGetLastError();
}

// ------------------------------------------------------- the serving pool
// One-warp CTAs take units from a counter: first the link detection of four
// elements each (with `detect`; each group of eight lanes finds its element's
// episode), then the march units of all episodes.  A warp that met outlets or
// walls takes fewer (with fixed shares the slowest SM ran 35 % longer than the
// fastest), and detection, a chain of dependent atomics that left the chip
// idle in a launch of its own, runs beside the march.  The next unit is
// fetched while the current one runs.  Every unit, a CTA's first too, comes
// from the counter in order: when a march unit waits for detection
// (unit_next[1] counts the finished units), every detection unit is with a
// warp that is running and waits for nothing, so the wait ends, however few of
// the CTAs fit beside other work on the GPU.
// Without `detect` (timing a shape) the pass feeds no outlets and latches
// nothing: it leaves all that the next step reads as it is.  Episodes hold
// fewer than 2^22 cells, so every moment index fits in 32 bits.
template <typename T>
__global__ void __launch_bounds__(32, kMarchWarps)
    pool_dense_kernel(const PoolEpisode *eps, const PoolActive *act, LinkTable lt, uint32_t *owner, uint32_t *unit_next,
                      int detect, int parity, int rows)
{
    __shared__ march2::Ends ends;
    after_predecessor();
    auto take = [&] { return threadIdx.x == 0 ? atomicAdd(unit_next, 1u) : 0u; };
    const uint32_t initial = take();
    const int n = (int)act->n;
    if (n == 0) return;
    const uint32_t elements = act->elem_prefix[n], first = detect ? (elements + 3) / 4 : 0u;
    const uint32_t total = first + act->tile_prefix[n];
    uint32_t t = __shfl_sync(0xffffffffu, initial, 0);
    march2::Gate gate{unit_next + 1, first, !detect};
    while (t < total) {
        const uint32_t next = take();
        if (t < first) {
            const uint32_t mine = 4 * t + (threadIdx.x >> 3), ge = min(mine, elements - 1);
            const int a = owner_of(act->elem_prefix, n, ge);
            const uint32_t s = act->slot[a];
            const PoolEpisode &e = eps[s];
            detect_elements2_warp<T>(episode_args<T>(e, parity), reinterpret_cast<uint32_t *>(e.flags), lt,
                                     episode_surface(e), StepScalars{e.cl, e.ct, e.cf},
                                     (long long)(ge - act->elem_prefix[a]), mine < elements, 8,
                                     reinterpret_cast<uint32_t *>(&ends), e.cell_base, owner, s);
            __syncwarp();
            if (threadIdx.x == 0) {
                __threadfence();
                atomicAdd(unit_next + 1, 1u);
            }
        } else {
            const int a = owner_of(act->tile_prefix, n, t - first);
            const uint32_t u = t - first - act->tile_prefix[a], W = act->tiles_x[a];
            GridArgs<T> g = episode_args<T>(eps[act->slot[a]], parity);
            if (!detect) g.feed = 0;
            const int c = (int)(u / W), w = (int)(u - c * W);
            const int yb = c * rows, ye = min(yb + rows, g.ny);
            if (g.nx % 2 == 0) march2::run<T, true>(g, w, yb, ye, ends, gate);
            else march2::run<T, false>(g, w, yb, ye, ends, gate);
        }
        t = __shfl_sync(0xffffffffu, next, 0);
    }
}

template <typename T>
cudaError_t launch_pool_dense(const PoolEpisode *eps, const PoolActive *act, const LinkTable &lt, uint32_t *owner,
                              uint32_t *unit_next, bool detect, int parity, int shape, int grid, cudaStream_t st)
{
    return launch_chained(pool_dense_kernel<T>, grid, 32, st, eps, act, lt, owner, unit_next, detect ? 1 : 0, parity,
                          kPoolRows[shape]);
}

template <typename T> int pool_dense_blocks_per_sm()
{
    int blocks = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, pool_dense_kernel<T>, 32, 0) != cudaSuccess || blocks < 1)
        blocks = 1;
    return blocks;
}

#define FFS_INST_POOL_DENSE(T)                                                                                          \
    template cudaError_t launch_pool_dense<T>(const PoolEpisode *, const PoolActive *, const LinkTable &, uint32_t *,  \
                                              uint32_t *, bool, int, int, int, cudaStream_t);                          \
    template int pool_dense_blocks_per_sm<T>();
FFS_INST_POOL_DENSE(float)
FFS_INST_POOL_DENSE(__half)
FFS_INST_POOL_DENSE(__nv_bfloat16)

#define FFS_INST_DENSE2D(T)                                                                                             \
    template bool dense2d_detects<T>(const GridArgs<T> &);                                                             \
    template cudaError_t launch_dense2d<T>(const GridArgs<T> &, cudaStream_t, const DetectArgs *);
FFS_INST_DENSE2D(float)
FFS_INST_DENSE2D(__half)
FFS_INST_DENSE2D(__nv_bfloat16)

} // namespace fflbm
