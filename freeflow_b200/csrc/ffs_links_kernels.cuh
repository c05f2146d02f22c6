// Moving-boundary (interpolated moving-wall) bounce-back and surface forces.
//
// Reference: the occupancy kernels mrSolver2DComputeOccupancyFlagKernel_v3 /
// mrSolver3DComputeOccupancyFlagKernel_v3 (FsiCoupling2D.cu:31-80,
// FsiCoupling3D.cu:31-81) fill a dense hitIndex of Q u32 per cell, memset to
// 0xFF every step, and the fused kernels consume it (FsiCoupling2D.cu:183-216,
// FsiCoupling3D.cu:224-275) with FP32 atomicAdd force scatter
// (SolidGeometryProxy_Device.cuh:184-194, :401-421).
//
// Here the link set is sparse and O(surface):
//   detect      a warp tests the (cell, direction) pairs whose link can cross
//               its element (D2Q9: four elements) and inserts hits into
//               an open-addressing table keyed by cell; per (cell, direction)
//               atomicMin keeps the nearest (depth, element) key.  The owning
//               cell gets a LINK bit in its flag byte, so the dense kernels
//               skip it.  Nothing proportional to the grid is touched.
//   link cells  one warp per D3Q27 link-owning cell, lane i = direction i (half a
//               warp per D2Q9 cell, or four lanes in the serving pool): wall
//               bounce-back, moving-wall reconstruction with the momentum
//               exchange force, or the ordinary pull (reconstructing the
//               neighbour's population from its moments).  The warp reduces
//               the raw moments with shuffles and lane 0 collides and stores.
//   forces      each link's DIM vertex shares are summed as 64-bit fixed point
//               (2^-32 lattice units) with integer atomics: integer addition is
//               associative, so the per-vertex sums are bit-reproducible
//               whatever the launch order, and exact up to the 2^-24
//               rounding of each share.  The last CTA of the link cells, or a
//               final pass, scales by Cf and adds to the caller's force array
//               (+ optional FP64 copy).
#pragma once
#include <algorithm>

#include "ffs_links_dev.cuh"

namespace fflbm {

// ------------------------------------------------------------------ detect
static int sm_count() { return device_sms(); }

// CTAs of `threads` threads of KERNEL that are resident on the device at
// once (no dynamic shared memory); the occupancy is queried once per kernel.
template <auto KERNEL> static int resident_grid(int threads)
{
    static int per_sm = 0;
    if (!per_sm && (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, KERNEL, threads, 0) != cudaSuccess ||
                    per_sm < 1))
        per_sm = 1;
    return sm_count() * per_sm;
}

// D3Q27: one warp per triangle, one lane per link direction (lanes 0..25 for
// l = 1..26).  The triangle's own geometry is evaluated once (tri_pre).  A
// link segment x -> x - c lies on one of the lattice lines parallel to c, and
// such a line meets the triangle's plane in one point, so each lane looks only
// at the lines that can pass through the triangle, and on each at the one or
// two cells whose link reaches that point, instead of at every cell of the
// triangle's bounding box (62 cells for a triangle of config D; the lanes' lines
// number 0 to 8).  With k the first axis that c moves along, a line is named
// by the integers q_j = x_j - (c_j / c_k) x_k of the other two axes j; the
// lines that can pass are those of the triangle's own range of q, widened.
//
// The cells found that way go through a conservative prefilter: the pair
// stays unless the plane is clearly not reached (s1 = n.(p - v0) against
// [-margin, |a| + margin] with a = cl n.c and a margin of 2e-3 cells) or the
// plane point lies outside the triangle by more than 1 % in barycentric terms.
// Every remaining pair gets the exact, explicitly rounded test, so the link
// set does not depend on this enumeration (the table keeps the minimum key per
// cell and direction).  Both the lines' range and the barycentric test assume
// that the exact test's own rounding stays far below 1 %: the plane point
// carries an absolute error of a few float ulps of the coordinates (about
// 2.4e-7 x the largest grid extent in cells x cl), and a barycentric
// coordinate divides it by (shortest edge x sin^2 of the angle between the
// edges).  Triangles with a tiny edge or angle (slivers, nearly coincident
// vertices) have every cell of the bounding box tested instead.
// The surviving pairs are queued in shared memory (64 entries per warp) and the
// exact test runs on 32 of them at a time; boxes larger than 1024 x 1024 x 128
// cells skip the queue.
template <typename T>
__global__ void __launch_bounds__(256) detect_links3_kernel(GridArgs<T> g, uint32_t *flag_words, LinkTable lt,
                                                            SurfaceArgs s, StepScalars sc)
{
    constexpr int Q = 27;
    const int lane = threadIdx.x & 31;
    const long long nwarps = ((long long)gridDim.x * blockDim.x) >> 5;
    const float cl = sc.cl, inv_cl = __fdividef(1.0f, cl);
    const float margin = 2e-3f * cl;
    const bool act = lane < Q - 1;
    const int l = act ? lane + 1 : 1;
    int cx, cy, cz;
    dir_vec<3>(l, cx, cy, cz);
    const float ccx = (float)cx * cl, ccy = (float)cy * cl, ccz = (float)cz * cl;
    // the axis k of the lattice lines, and c_j / c_k of the other two (in order)
    const int ax = cx != 0 ? 0 : cy != 0 ? 1 : 2;
    const int ck = ax == 0 ? cx : ax == 1 ? cy : cz;
    const int r1 = (ax == 0 ? cy : cx) * ck, r2 = (ax == 2 ? cy : cz) * ck;
    auto along = [&](const float *v) { return ax == 0 ? v[0] : ax == 1 ? v[1] : v[2]; };
    auto first = [&](const float *v) { return ax == 0 ? v[1] : v[0]; };
    auto second = [&](const float *v) { return ax == 2 ? v[1] : v[2]; };
    __shared__ uint32_t queue[8][64]; // per warp: (cell, direction) pairs for the exact test
    uint32_t *wq = queue[threadIdx.x >> 5];
    const unsigned full = 0xffffffffu, below = (1u << lane) - 1u;
    for (long long e = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5; e < s.ne; e += nwarps) {
        const uint32_t ia = s.E[3 * e], ib = s.E[3 * e + 1], ic = s.E[3 * e + 2];
        if (ia >= (uint32_t)s.nv || ib >= (uint32_t)s.nv || ic >= (uint32_t)s.nv) {
            if (lane == 0) atomicOr(g.status, kStatusBadElement);
            continue;
        }
        const geom::TriPre tr = geom::tri_pre(s.V, ia, ib, ic);
        const float inv_den = __fdividef(1.0f, tr.den);
        const float coord_err = 2.4e-7f * (float)max(g.nx, max(g.ny, g.nz)) * cl;
        const bool sound =
            sqrtf(fminf(tr.d00, tr.d11)) * (tr.den / (tr.d00 * tr.d11)) > 400.0f * coord_err; // error < 0.0025
        float bmin[3] = {3.402823466e+38f, 3.402823466e+38f, 3.402823466e+38f};
        float bmax[3] = {1.175494351e-38f, 1.175494351e-38f, 1.175494351e-38f};
        const uint32_t vid[3] = {ia, ib, ic};
        float X[3][3]; // vertices in cells
#pragma unroll
        for (int j = 0; j < 3; ++j)
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                float c = s.V[(size_t)vid[j] * 3 + k];
                X[j][k] = c * inv_cl;
                if (c < bmin[k]) bmin[k] = c;
                if (bmax[k] < c) bmax[k] = c;
            }
        const int n3[3] = {g.nx, g.ny, g.nz};
        int lo[3], hi[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            lo[k] = max(__float2int_rz(geom::dvd(bmin[k], cl)) - 1, 0);
            hi[k] = min(__float2int_rz(geom::dvd(bmax[k], cl)) + 1, n3[k] - 1);
        }
        // this lane's direction against the triangle's plane
        const float a = cl * (tr.n[0] * cx + tr.n[1] * cy + tr.n[2] * cz);
        const float fa = fabsf(a);
        const bool reach = fa > margin;              // else: the link runs (nearly) parallel to the plane
        const float sg = a > 0.0f ? 1.0f : -1.0f;
        const float inv_a = reach ? __fdividef(1.0f, a) : 0.0f;
        // the exact test of cell (i, j, k3), direction ll, and the insertion on a hit
        auto exact = [&](int i, int j, int k3, int ll) {
            int dx, dy, dz;
            dir_vec<3>(ll, dx, dy, dz);
            float p1[3] = {geom::mul((float)i, cl), geom::mul((float)j, cl), geom::mul((float)k3, cl)};
            float p2[3] = {geom::mul(geom::sub((float)i, (float)dx), cl), geom::mul(geom::sub((float)j, (float)dy), cl),
                           geom::mul(geom::sub((float)k3, (float)dz), cl)};
            const geom::Hit h = geom::isect3_pre(tr, p1, p2);
            if (!h.hit) return;
            const uint32_t cell = (uint32_t)(((long long)k3 * g.ny + j) * g.nx + i);
            insert_link<3>(g, lt, flag_words, cell, ll, geom::link_key(h.depth, (uint32_t)e));
        };
        const bool queued = hi[0] - lo[0] < 1024 && hi[1] - lo[1] < 1024 && hi[2] - lo[2] < 128;
        int qn = 0;
        auto drain = [&](int upto) { // run the exact test on the first `upto` queued pairs
            __syncwarp();
            const uint32_t code = wq[lane];
            __syncwarp();
            if (lane < qn - upto) wq[lane] = wq[upto + lane];
            __syncwarp();
            if (lane < upto)
                exact(lo[0] + (int)(code & 1023u), lo[1] + (int)((code >> 10) & 1023u), lo[2] + (int)((code >> 20) & 127u),
                      (int)(code >> 27) + 1);
            qn -= upto;
        };
        // every lane of the warp comes here together, with a cell or without one
        auto offer = [&](bool cand, int i, int j, int k3) {
            if (!queued) {
                if (cand) exact(i, j, k3, l);
                return;
            }
            const unsigned m = __ballot_sync(full, cand);
            if (cand)
                wq[qn + __popc(m & below)] = (uint32_t)(i - lo[0]) | ((uint32_t)(j - lo[1]) << 10) |
                                             ((uint32_t)(k3 - lo[2]) << 20) | ((uint32_t)(l - 1) << 27);
            qn += __popc(m);
            if (qn >= 32) drain(32);
        };
        // the plane of cell (i, j, k3) is not clearly out of its link's reach
        auto reached = [&](float px, float py, float pz, float &s1) {
            s1 = fmaf(tr.n[0], px, tr.n[1] * py + tr.n[2] * pz);
            if (!reach) return !(fabsf(s1) > 2.0f * margin);
            const float sa = sg * s1;
            return !(sa < -margin || sa > fa + margin);
        };
        if (sound) {
            // the lane's lines: ranges of q over the vertices, 2 % and 0.02 cells wider
            float q1min = 3e38f, q1max = -3e38f, q2min = 3e38f, q2max = -3e38f;
#pragma unroll
            for (int j = 0; j < 3; ++j) {
                const float q1 = first(X[j]) - (float)r1 * along(X[j]), q2 = second(X[j]) - (float)r2 * along(X[j]);
                q1min = fminf(q1min, q1); q1max = fmaxf(q1max, q1);
                q2min = fminf(q2min, q2); q2max = fmaxf(q2max, q2);
            }
            const float w1 = 0.02f * (q1max - q1min) + 0.02f, w2 = 0.02f * (q2max - q2min) + 0.02f;
            // of those, the lines that pass through the box
            auto pick = [&](const int *v, int which) {
                return which == 0 ? (ax == 0 ? v[0] : ax == 1 ? v[1] : v[2])
                                  : which == 1 ? (ax == 0 ? v[1] : v[0]) : (ax == 2 ? v[1] : v[2]);
            };
            const int lk = pick(lo, 0), hk = pick(hi, 0);
            const int q1lo = max((int)ceilf(q1min - w1), pick(lo, 1) - (r1 > 0 ? hk : r1 < 0 ? -lk : 0));
            const int q1hi = min((int)floorf(q1max + w1), pick(hi, 1) - (r1 > 0 ? lk : r1 < 0 ? -hk : 0));
            const int q2lo = max((int)ceilf(q2min - w2), pick(lo, 2) - (r2 > 0 ? hk : r2 < 0 ? -lk : 0));
            const int q2hi = min((int)floorf(q2max + w2), pick(hi, 2) - (r2 > 0 ? lk : r2 < 0 ? -hk : 0));
            const float q10 = first(X[0]) - (float)r1 * along(X[0]), q20 = second(X[0]) - (float)r2 * along(X[0]);
            // the plane meets line (q1, q2) at x_k = s: s falls off linearly in q; the
            // cells whose link reaches it are x_k = s .. s + c_k, wider by the margin
            const float inv_s = reach ? (float)ck * cl * inv_a : 0.0f; // 1 / (c_k n.c)
            const float g1 = first(tr.n) * inv_s, g2 = second(tr.n) * inv_s, s0 = along(X[0]);
            const float slack = reach ? 3e-3f * fabsf(inv_s) + 2e-3f : 1e9f;
            const float from = (ck > 0 ? 0.0f : -1.0f) - slack, to = (ck > 0 ? 1.0f : 0.0f) + slack;
            const float klo = (float)lk, khi = (float)hk;
            int q1 = q1lo, q2 = q2lo;
            bool more = act && q1lo <= q1hi && q2lo <= q2hi;
            while (__any_sync(full, more)) {
                int k = 1, kend = 0;
                if (more) {
                    const float sk = s0 - (g1 * ((float)q1 - q10) + g2 * ((float)q2 - q20));
                    k = (int)ceilf(fmaxf(sk + from, klo));
                    kend = (int)floorf(fminf(sk + to, khi));
                }
                while (__any_sync(full, k <= kend)) {
                    bool cand = false;
                    int i = 0, j = 0, k3 = 0;
                    if (k <= kend) {
                        const int a1 = q1 + r1 * k, a2 = q2 + r2 * k;
                        i = ax == 0 ? k : a1;
                        j = ax == 0 ? a1 : ax == 1 ? k : a2;
                        k3 = ax == 2 ? k : a2;
                        if (i >= lo[0] && i <= hi[0] && j >= lo[1] && j <= hi[1] && k3 >= lo[2] && k3 <= hi[2]) {
                            const float px = (float)i * cl - tr.v0[0], py = (float)j * cl - tr.v0[1],
                                        pz = (float)k3 * cl - tr.v0[2];
                            float s1;
                            cand = reached(px, py, pz, s1);
                            if (cand && reach) {
                                // plane point relative to v0: p1 - t c cl - v0
                                const float t = s1 * inv_a;
                                const float wx = px - t * ccx, wy = py - t * ccy, wz = pz - t * ccz;
                                const float d20 = wx * tr.e1[0] + wy * tr.e1[1] + wz * tr.e1[2];
                                const float d21 = wx * tr.e2[0] + wy * tr.e2[1] + wz * tr.e2[2];
                                const float u = (tr.d11 * d20 - tr.d01 * d21) * inv_den;
                                const float v = (tr.d00 * d21 - tr.d01 * d20) * inv_den;
                                cand = !(u < -0.01f || v < -0.01f || u + v > 1.01f);
                            }
                        }
                    }
                    offer(cand, i, j, k3);
                    ++k;
                }
                if (more && ++q1 > q1hi) {
                    q1 = q1lo;
                    more = ++q2 <= q2hi;
                }
            }
        } else {
            for (int k3 = lo[2]; k3 <= hi[2]; ++k3)
                for (int j = lo[1]; j <= hi[1]; ++j)
                    for (int i = lo[0]; i <= hi[0]; ++i) {
                        float s1;
                        const bool cand = reached((float)i * cl - tr.v0[0], (float)j * cl - tr.v0[1],
                                                  (float)k3 * cl - tr.v0[2], s1);
                        offer(act && cand, i, j, k3);
                    }
        }
        if (queued && qn > 0) drain(qn);
        __syncwarp();
    }
}

// D2Q9: one warp per segment, or per four (detect_lanes2).
template <typename T>
__global__ void __launch_bounds__(32) detect_links2_kernel(GridArgs<T> g, uint32_t *flag_words, LinkTable lt,
                                                            SurfaceArgs s, StepScalars sc, int lanes)
{
    __shared__ uint32_t queue[64]; // (cell, direction) pairs for the exact test
    const int per = 32 / lanes, group = (int)threadIdx.x / lanes;
    for (long long e = (long long)blockIdx.x * per; e < s.ne; e += (long long)gridDim.x * per)
        detect_elements2_warp<T>(g, flag_words, lt, s, sc, e + group, e + group < s.ne, lanes, queue);
}

// -------------------------------------------------------------- link cells
// One fixed-point force sum -> physical force: added to the surface's force
// arrays, or, in the coupled step, written to the mapped volume vertex (whose
// force the gather zeroed), as scatterSurfaceForcesToVolume assigns it
// (src/fsi/FsiCouplingKernels.cu:59-90).
template <int DIM>
__device__ __forceinline__ void finalize_force(const SurfaceArgs &s, long long t, long long a, double cf)
{
    double f = (double)a * (1.0 / kForceScale) * cf;
    if (s.vforces) {
        const long long i = t / DIM;
        const uint32_t m = s.map[i];
        if (m < (uint32_t)s.nvol) s.vforces[(size_t)m * DIM + (t - i * DIM)] = (float)f;
    } else {
        if (s.forces) s.forces[t] += (float)f;
        if (s.forces64) s.forces64[t] += f;
    }
}

template <int DIM, typename T, bool HALF, bool FOLD>
__global__ void __launch_bounds__(256, DIM == 2 ? 2 : 5) link_cells_kernel(const __grid_constant__ GridArgs<T> g,
                                                         uint32_t *flag_words, LinkTable lt, SurfaceArgs s,
                                                         StepScalars sc)
{
    constexpr int Q = Lattice<DIM>::Q, G = kLinkGroup<DIM>, kPerWarp = 32 / G;
    const int lane = threadIdx.x & (G - 1);
    const uint32_t group = (threadIdx.x & 31) / G;
    const uint32_t nwarps = (gridDim.x * blockDim.x) >> 5;
    const uint32_t feeders = *g.feeders_n; // made when the node types were set, long before the dense pass
    after_predecessor();
    const LinkItems items(lt);
    const uint32_t n = items.n;
    // consecutive cells go to different CTAs: a few cells spread over the SMs
    for (uint32_t w = ((threadIdx.x >> 5) * gridDim.x + blockIdx.x) * kPerWarp; w < n; w += nwarps * kPerWarp) {
        // a group past the end of the list rides along on the first group's cell
        const bool valid = w + group < n;
        const uint32_t slot = items.slot(lt, valid ? w + group : w);
        const uint32_t cell = lt.keys[slot] - 1;
        if constexpr (DIM == 2) link_cell_update2<T, HALF, G>(g, lt.links, slot, cell, lt.acc, s, sc, valid);
        else link_cell_update3<T>(g, lt.links, slot, cell, lt.acc, s, sc, valid);
        // return the slot to the empty state and drop the cell's LINK bit
        for (int l = lane; valid && l < Q; l += G) lt.links[(size_t)slot * Q + l] = ~0ull;
        __syncwarp();
        if (valid && lane == 0) {
            lt.keys[slot] = 0;
            set_link_bit(flag_words, cell, false);
        }
    }
    // the outlets of all other feeders, by the warps without link cells first
    if (feeders) feed_pass<DIM, T>(g, feeders, flag_words, nwarps - 1 - ((threadIdx.x >> 5) * gridDim.x + blockIdx.x), nwarps);
    if constexpr (!FOLD) return;
    // The CTA that finishes last converts the force sums: every other CTA's
    // atomics are complete and fenced before its count.  No CTA waits for
    // another.  The counters are reset for the next step.
    __shared__ bool last_cta;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        last_cta = atomicAdd(lt.done, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last_cta) return;
    __threadfence();
    const long long nf = (long long)s.nv * DIM;
    for (long long t = threadIdx.x; t < nf; t += blockDim.x) {
        const long long a = __ldcg(lt.acc + t);
        if (a != 0) {
            finalize_force<DIM>(s, t, a, sc.cf);
            lt.acc[t] = 0;
        }
    }
    clear_counts(lt);
    if (threadIdx.x == 0) *lt.done = 0;
}

// Fixed-point sums -> physical forces: added to the surface's force arrays,
// or, in the coupled step, written to the mapped volume vertices (whose
// forces the gather zeroed), as scatterSurfaceForcesToVolume assigns them
// (src/fsi/FsiCouplingKernels.cu:59-90).
template <int DIM>
__global__ void finalize_forces_kernel(LinkTable lt, SurfaceArgs s, double cf)
{
    const long long n = (long long)s.nv * DIM;
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x) {
        long long a = lt.acc[t];
        if (a != 0) {
            finalize_force<DIM>(s, t, a, cf);
            lt.acc[t] = 0;
        }
    }
    if (blockIdx.x == 0) clear_counts(lt);
}

template <int DIM>
__global__ void reset_links_kernel(LinkTable lt, uint32_t *flag_words)
{
    constexpr int Q = Lattice<DIM>::Q;
    for (uint32_t slot = blockIdx.x * blockDim.x + threadIdx.x; slot < lt.cap; slot += gridDim.x * blockDim.x) {
        const uint32_t key = lt.keys[slot];
        if (!key) continue;
        for (int l = 0; l < Q; ++l) lt.links[(size_t)slot * Q + l] = ~0ull;
        lt.keys[slot] = 0;
        set_link_bit(flag_words, key - 1, false);
    }
    if (blockIdx.x == 0) clear_counts(lt);
}

// ---------------------------------------------------------------- launchers
template <int DIM, typename T>
cudaError_t launch_detect_links(const GridArgs<T> &g, uint32_t *flag_words, const LinkTable &lt, const SurfaceArgs &s,
                                const StepScalars &sc, cudaStream_t st)
{
    if (s.ne <= 0) return cudaSuccess;
    if constexpr (DIM == 3) {
        const int grid = (int)std::min<long long>(((long long)s.ne + 7) / 8, (long long)sm_count() * 16);
        detect_links3_kernel<T><<<grid, 256, 0, st>>>(g, flag_words, lt, s, sc);
    } else {
        // one-warp CTAs: a small surface spreads over the SMs
        const int lanes = detect_lanes2(s.ne, sm_count()), per = 32 / lanes;
        const int grid = (int)std::min<long long>((s.ne + per - 1) / per, (long long)sm_count() * 32);
        detect_links2_kernel<T><<<grid, 32, 0, st>>>(g, flag_words, lt, s, sc, lanes);
    }
    return cudaGetLastError();
}

template <int DIM, typename T, bool HALF, bool FOLD>
static cudaError_t launch_link_cells_as(const GridArgs<T> &g, uint32_t *flag_words, const LinkTable &lt, const SurfaceArgs &s,
                                        const StepScalars &sc, cudaStream_t st, bool chained)
{
    // persistent warps over the device-side count, one wave: as many CTAs of
    // 8 warps as are resident together (a CTA beyond that would run its fixed
    // share of the cells after the others finish)
    int grid = resident_grid<link_cells_kernel<DIM, T, HALF, FOLD>>(256);
    // A 2D surface rarely gives more than eight link cells a segment, and a CTA
    // takes 16 at a time: fewer CTAs then start, and count themselves done in
    // one counter, sooner (0.6 us of a 15 us step on 256 x 128, 0.9 us on
    // 1200 x 400 in FP32).  At least one per SM, for long segments.
    if (DIM == 2) grid = (int)std::min<long long>(grid, std::max<long long>(sm_count(), s.ne / 2));
    if (chained) return launch_chained(link_cells_kernel<DIM, T, HALF, FOLD>, grid, 256, st, g, flag_words, lt, s, sc);
    link_cells_kernel<DIM, T, HALF, FOLD><<<grid, 256, 0, st>>>(g, flag_words, lt, s, sc);
    return cudaGetLastError();
}

template <int DIM, typename T>
cudaError_t launch_link_cells(const GridArgs<T> &g, uint32_t *flag_words, const LinkTable &lt, const SurfaceArgs &s,
                              const StepScalars &sc, cudaStream_t st, bool fold_forces, bool chained)
{
    if (DIM == 2 && g.half_pops)
        return fold_forces ? launch_link_cells_as<DIM, T, DIM == 2, true>(g, flag_words, lt, s, sc, st, chained)
                           : launch_link_cells_as<DIM, T, DIM == 2, false>(g, flag_words, lt, s, sc, st, chained);
    return fold_forces ? launch_link_cells_as<DIM, T, false, true>(g, flag_words, lt, s, sc, st, chained)
                       : launch_link_cells_as<DIM, T, false, false>(g, flag_words, lt, s, sc, st, chained);
}

template <int DIM>
cudaError_t launch_finalize_forces(const LinkTable &lt, const SurfaceArgs &s, double cf, cudaStream_t st)
{
    long long n = (long long)s.nv * DIM;
    int grid = (int)std::min<long long>((n + 255) / 256, (long long)sm_count() * 8);
    if (grid < 1) grid = 1;
    finalize_forces_kernel<DIM><<<grid, 256, 0, st>>>(lt, s, cf);
    return cudaGetLastError();
}

template <int DIM>
cudaError_t launch_reset_links(const LinkTable &lt, uint32_t *flag_words, cudaStream_t st)
{
    reset_links_kernel<DIM><<<sm_count(), 256, 0, st>>>(lt, flag_words);
    return cudaGetLastError();
}

// The launchers of one lattice (ffs_links.cu, ffs_links3.cu)
#define FFS_INST_LINKS_T(DIM, T)                                                                                       \
    template cudaError_t launch_detect_links<DIM, T>(const GridArgs<T> &, uint32_t *, const LinkTable &,              \
                                                     const SurfaceArgs &, const StepScalars &, cudaStream_t);          \
    template cudaError_t launch_link_cells<DIM, T>(const GridArgs<T> &, uint32_t *, const LinkTable &,                \
                                                   const SurfaceArgs &, const StepScalars &, cudaStream_t, bool, bool);
#define FFS_INST_LINKS(DIM)                                                                                            \
    FFS_INST_LINKS_T(DIM, float)                                                                                       \
    FFS_INST_LINKS_T(DIM, __half)                                                                                      \
    FFS_INST_LINKS_T(DIM, __nv_bfloat16)                                                                               \
    template cudaError_t launch_finalize_forces<DIM>(const LinkTable &, const SurfaceArgs &, double, cudaStream_t);    \
    template cudaError_t launch_reset_links<DIM>(const LinkTable &, uint32_t *, cudaStream_t);

} // namespace fflbm
