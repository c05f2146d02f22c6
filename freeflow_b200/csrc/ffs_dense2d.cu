// Fused D2Q9 step for all cells without moving-boundary links.
//
// Reference: mrDeformableSolver2DKernel_Shrd (src/core/FsiCoupling2D.cu:82-255)
// followed by mrApplyOutlet2DKernel (:257-316).
//
// Two forms of one update, with the same bits.  A single grid of the sizes
// FreeFlow runs (<= 1200 x 400, L2-resident on B200) is bound by latency and
// takes tiles, a thread per cell; a million cells and more, and the serving
// pool with all its episodes, are bound by instructions and take the row march
// of ffs_march2d.cuh, one warp per unit of 64 columns and a few rows.
//
// Two options of the reference's own 2D kernel need populations as such: the
// binary16 tile (ref_half_populations) and walls that stream
// (ref_2d_wall_stream).  They, and grids whose moment indices do not fit in 32
// bits, take the kernel of ffs_ref2d.cu.
#include <algorithm>
#include <cstdlib>

#include "ffs_links_dev.cuh"
#include "ffs_march2d.cuh"
#include "ffs_pool.cuh"

namespace fflbm {

// March warps (one-warp CTAs) per SM that the register budget is cut for: four
// per scheduler leave 128 registers, which the march fills (the pool's FP32
// kernel spills 88 B, the 16-bit ones 4); five (96 registers) ran the pool's pass
// 3 % slower, three 10 %.
constexpr int kMarchWarps = 16;

// Tile form of the march: one CTA = one 32 x 8 tile, a thread per cell.  The
// deviations F' of the tile and the cells around it go through shared memory,
// and every operation on a cell is march2::run's, in its order, so both give the
// same bits (the pool marches, and its episodes equal grids stepped alone).  A
// march unit reconstructs two rows more than it updates and walks its rows one
// after the other, which a grid of few units waits for: 1200 x 400 in FP32
// without a surface takes 6.7 us in tiles and 8.4 marched, 512 x 256 3.2 and 4.9.
template <typename T>
__device__ __forceinline__ void update_tile(const GridArgs<T> &g, int x0, int y0, float (*sp)[D2::kHY][D2::kHX])
{
    using P = typename march2::Pair<T>::type;
    const int tid = threadIdx.x, tx = tid % D2::kTX, ty = tid / D2::kTX, x = x0 + tx, y = y0 + ty;
    const bool wx = g.periodic & 1, wy = g.periodic & 2;
    // two cells side by side a thread, as packed pairs (one cell a thread: 7.3 us
    // instead of 6.7 on 1200 x 400)
    constexpr int kPairs = D2::kHalo / 2, kRow = D2::kHX / 2;
    const int hx = 2 * (tid % kRow), hy = tid / kRow;
    P raw[6];
    if (tid < kPairs) {
        const uint32_t row = (uint32_t)halo_index(y0 + hy - 1, g.ny, wy) * (uint32_t)g.nx;
        const uint32_t i0 = row + (uint32_t)halo_index(x0 + hx - 1, g.nx, wx), i1 = row + (uint32_t)halo_index(x0 + hx, g.nx, wx);
#pragma unroll
        for (int k = 0; k < 6; ++k) raw[k] = march2::load_pair<T, false>(g.src + (size_t)((uint32_t)k * g.ncell), i0, i1);
    }
    const uint32_t idx = (uint32_t)(y * g.nx + x);
    const uint32_t f8 = x < g.nx && y < g.ny ? g.flags[idx] : 0u;
    const bool updated = is_updated(f8 & kTypeMask) && !(f8 & kBitLink);
    const uint32_t wm = updated && (f8 & (kBitNearWall | kBitOutletSrc)) ? g.wallmask[idx] : 0u;
    if (tid < kPairs) {
        f2 m[6], d, F[3];
        march2::decode<T>(raw, g.codec, m, d);
        const march2::Rows<f2> rows(m, d);
        auto put = [&](int ky) {
#pragma unroll
            for (int kx = 0; kx < 3; ++kx)
                *reinterpret_cast<unsigned long long *>(&sp[kx + 3 * ky][hy][hx]) = march2::clamp1(F[kx]).v;
        };
        rows.template row<0>(F);
        put(0);
        rows.template row<1>(F);
        put(1);
        rows.template row<2>(F);
        put(2);
    }
    __syncthreads();
    // the halo holds what a cell on a high face pulls (halo_index), too
    if (updated)
        march2::update_cell<T>(
            g, idx, f8, wm, [&](int kx, int ky) { return sp[kx + 3 * ky][ty + 2 - ky][tx + 2 - kx]; },
            [&](int kx, int ky) { return sp[kx + 3 * ky][ty + 1][tx + 1]; });
}

// The first `ndetect` CTAs detect the surface's links (`lanes` lanes an
// element), the others update tiles.  A launch of its own for detection, on a
// second stream with events around it, cost more than detection itself on grids
// of this size.  Which link cells the tiles skip (they read their LINK bit while
// detection sets it) does not matter: the link-cell kernel rewrites every link
// cell afterwards and feeds the outlets (ffs_outlet.cuh).
template <typename T>
__device__ __forceinline__ void detect_block(const GridArgs<T> &g, int ndetect, int lanes, const DetectArgs &d, uint32_t *queue)
{
    const int per = 32 / lanes, group = ((int)threadIdx.x & 31) / lanes, warps = (int)blockDim.x >> 5;
    const long long w = (long long)blockIdx.x * warps + (threadIdx.x >> 5);
    for (long long e = w * per; e < d.s.ne; e += (long long)ndetect * warps * per)
        detect_elements2_warp<T>(g, d.flag_words, d.lt, d.s, d.sc, e + group, e + group < d.s.ne, lanes, queue);
}
// Registers: detection takes 61, so its CTAs leave room for four; without it the
// FP32 tile fits eight (32 registers) without spills, and the 16-bit one runs
// best at five (39; 1200 x 400 8.7 us, at eight 9.0).
template <typename T, bool DETECT>
__global__ void __launch_bounds__(D2::kThreads, DETECT ? 4 : sizeof(T) == 4 ? 8 : 5)
    tile2d_kernel(GridArgs<T> g, int tiles_x, int ndetect, int lanes, DetectArgs d)
{
    __shared__ __align__(16) float sp[9][D2::kHY][D2::kHX];
    after_predecessor();
    if (DETECT && (int)blockIdx.x < ndetect) {
        static_assert(sizeof(sp) >= D2::kThreads / 32 * 64 * sizeof(uint32_t), "the exact test's queues fit");
        detect_block<T>(g, ndetect, lanes, d, reinterpret_cast<uint32_t *>(sp) + 64 * (threadIdx.x >> 5));
        return;
    }
    const int t = (int)blockIdx.x - ndetect;
    update_tile<T>(g, t % tiles_x * D2::kTX, t / tiles_x * D2::kTY, sp);
}

// The march, with detection in its first CTAs as above.
template <typename T, bool VEC>
__global__ void __launch_bounds__(32, kMarchWarps) march2d_kernel(GridArgs<T> g, int rows, int ndetect, int lanes, DetectArgs d)
{
    __shared__ march2::Ends ends;
    after_predecessor();
    if ((int)blockIdx.x < ndetect) {
        static_assert(sizeof(ends) >= 64 * sizeof(uint32_t), "the exact test's queue fits");
        detect_block<T>(g, ndetect, lanes, d, reinterpret_cast<uint32_t *>(&ends));
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

// Grids of at most this many cells take tiles with detection beside them; twice
// as many without (that kernel has more CTAs per SM).  Ten steps in a graph,
// FP32, outlets on four sides, tile and march, us a step: 1399 x 480 21.2 and
// 22.8, 1400 x 720 26.9 and 26.1, 1800 x 900 40.5 and 33.3; without a surface
// 1600 x 800 14.8 and 16.0, 2048 x 2048 (scalar tiles) 61.7 and 46.9.
constexpr uint32_t kTileCells = 1u << 20;
// Rows of a march unit of one grid: 4 to 8 differ by less than 5 % from 1 to 8
// million cells (2048 x 2048 FP32: 48.7, 46.9 and 47.6 us), 14 take 13 % more.
constexpr int kGridRows = 6;

template <typename T> bool dense2d_detects(const GridArgs<T> &g)
{
    return !g.half_pops && !g.wall_stream && 6ull * g.ncell <= 0xFFFFFFFFull;
}

template <typename T> cudaError_t launch_dense2d(const GridArgs<T> &g, cudaStream_t s, const DetectArgs *detect)
{
    if (!dense2d_detects(g)) return launch_ref2d<T>(g, s);
    const int sms = device_sms();
    const int lanes = detect ? detect_lanes2(detect->s.ne, sms) : 32;
    const long long detectors = detect ? std::min<long long>(((long long)detect->s.ne * lanes + 31) / 32, (long long)sms * 32) : 0; // warps
    const DetectArgs d = detect ? *detect : DetectArgs{};
    const char *pinned = std::getenv("FFS_MARCH_ROWS"); // tests run the march with several row counts
    if (!pinned && g.ncell <= (detect ? kTileCells : 2 * kTileCells)) {
        const int tiles_x = (g.nx + D2::kTX - 1) / D2::kTX, tiles = tiles_x * ((g.ny + D2::kTY - 1) / D2::kTY);
        const int nd = (int)((detectors + D2::kThreads / 32 - 1) / (D2::kThreads / 32));
        if (detect) tile2d_kernel<T, true><<<tiles + nd, D2::kThreads, 0, s>>>(g, tiles_x, nd, lanes, d);
        else tile2d_kernel<T, false><<<tiles, D2::kThreads, 0, s>>>(g, tiles_x, 0, lanes, d);
        return cudaGetLastError();
    }
    const int rows = pinned ? std::max(1, std::min(march2::kMaxRows, std::atoi(pinned))) : kGridRows;
    const int units = march2::windows(g.nx) * march2::chunks(g.ny, rows);
    const int nd = (int)detectors;
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
