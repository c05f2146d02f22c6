// Device bodies of the moving-boundary stages, shared by the single-grid
// kernels (ffs_links_kernels.cuh) and the batched many-grid kernels (ffs_batch2d.cu).
#pragma once
#include "ffs_geom.cuh"
#include "ffs_links.cuh"
#include "ffs_math.cuh"
#include "ffs_outlet.cuh"
#include "ffs_dense2d.cuh"

namespace fflbm {

__device__ __forceinline__ uint32_t hash_cell(uint32_t c)
{
    c ^= c >> 16; c *= 0x7feb352dU; c ^= c >> 15; c *= 0x846ca68bU; c ^= c >> 16;
    return c;
}

__device__ __forceinline__ void set_link_bit(uint32_t *flag_words, uint32_t cell, bool on)
{
    uint32_t bit = (uint32_t)kBitLink << (8 * (cell & 3));
    if (on) atomicOr(flag_words + (cell >> 2), bit);
    else atomicAnd(flag_words + (cell >> 2), ~bit);
}

// The occupied slots of a table, numbered across its segments: every lane of
// a warp holds the numbers at which two segments start.
struct LinkItems {
    uint32_t n, start0, start1;
    __device__ __forceinline__ explicit LinkItems(const LinkTable &lt)
    {
        const uint32_t lane = threadIdx.x & 31;
        if (lt.seg_shift == 31) {
            n = *lt.count;
            start0 = lane == 0 ? 0u : 0xffffffffu;
            start1 = 0xffffffffu;
            return;
        }
        const uint32_t a = lt.count[2 * lane * kCountStride], b = lt.count[(2 * lane + 1) * kCountStride];
        uint32_t upto = a + b;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t v = __shfl_up_sync(0xffffffffu, upto, o);
            if ((int)lane >= o) upto += v;
        }
        n = __shfl_sync(0xffffffffu, upto, 31);
        start0 = upto - a - b;
        start1 = upto - b;
    }
    // slot of item w < n (each lane its own; every lane of the warp calls)
    __device__ __forceinline__ uint32_t slot(const LinkTable &lt, uint32_t w) const
    {
        int from = 0; // the last lane whose start0 is not beyond w
#pragma unroll
        for (int step = 16; step > 0; step >>= 1) {
            const uint32_t v = __shfl_sync(0xffffffffu, start0, from + step);
            if (v <= w) from += step;
        }
        const uint32_t s0 = __shfl_sync(0xffffffffu, start0, from), s1 = __shfl_sync(0xffffffffu, start1, from);
        const bool second = s1 <= w;
        const uint32_t seg = 2 * (uint32_t)from + (second ? 1u : 0u);
        return lt.list[(seg << lt.seg_shift) + (w - (second ? s1 : s0))];
    }
};
// Empties the counters (called by one block of at least kSegments threads, or
// any number for one segment, once every reader is done).
__device__ __forceinline__ void clear_counts(const LinkTable &lt)
{
    if (lt.seg_shift == 31) {
        if (threadIdx.x == 0) *lt.count = 0;
    } else if (threadIdx.x < kSegments) {
        lt.count[threadIdx.x * kCountStride] = 0;
    }
}

// Finds or claims the cell's slot and keeps the smallest key of direction l.
// The table key is key_base + cell + 1: one table can serve many grids whose
// cells are numbered from distinct bases; the claiming thread tags the slot
// with owner_id in `owner` when that array is given.  A lane waits for one or
// two round trips to L2 here (the compare-and-swap, and the list position of a
// new slot), which is most of a small surface's detection time.
// The claiming thread also marks the outlet nodes the cell feeds, unless the
// dense pass sees to them (mark_outlets).
template <int DIM, typename T>
__device__ __forceinline__ void insert_link(const GridArgs<T> &g, const LinkTable &lt, uint32_t *flag_words, uint32_t cell,
                                            int l, unsigned long long key, uint32_t key_base = 0,
                                            uint32_t *owner = nullptr, uint32_t owner_id = 0)
{
    constexpr int Q = Lattice<DIM>::Q;
    const uint32_t tkey = key_base + cell + 1;
    uint32_t slot = hash_cell(tkey - 1) & (lt.cap - 1);
    // (fetched beside the compare-and-swap)
    const bool feeds = !g.feed && (reinterpret_cast<const uint8_t *>(flag_words)[cell] & kBitOutletSrc);
    for (uint32_t probe = 0; probe < lt.cap; ++probe) {
        const uint32_t old = atomicCAS(lt.keys + slot, 0u, tkey);
        if (old == 0u || old == tkey) {
            atomicMin(lt.links + (size_t)slot * Q + l, key);
            if (old == 0u) {
                const uint32_t seg = slot >> lt.seg_shift;
                const uint32_t pos = atomicAdd(lt.count + seg * kCountStride, 1u);
                if (owner) owner[slot] = owner_id;
                set_link_bit(flag_words, cell, true);
                lt.list[(seg << lt.seg_shift) + pos] = slot;
                if (feeds) mark_outlets<DIM>(flag_words, g.wallmask, g.nx, (long long)g.nx * g.ny, cell);
            }
            return;
        }
        slot = (slot + 1) & (lt.cap - 1);
    }
    atomicOr(g.status, kStatusLinkOverflow);
}

// D2Q9 link detection of segment e by one warp: every cell of the segment's
// bounding box grown by one cell (getBoundingBox: min from FLT_MAX, max from
// FLT_MIN (sic), then / dx) and every direction 1 <= l < 9 whose link segment
// x -> x - c_l crosses the element gets a (depth, element) key.  Items are
// numbered cell * 8 + (l - 1) with cells in row-major order; 32 items are four
// cells, so a lane keeps one direction and steps its cell by four, carrying
// the cell's coordinates forward instead of dividing them out.
//
// Most pairs cannot cross: a hit needs the element's line to separate the
// link's two end points (line_intersect's t1 = s2 / (s2 - s1) in (0, 1), with
// s1, s2 their signed distances).  A cheap prefilter drops a pair only when
// both end points lie on the same side by more than a hundredth of a cell
// (times the element's length); then t1 is at least about 7e-3 outside
// (0, 1), far beyond the exact test's rounding, so the link set is the
// exact test's.  The surviving pairs are queued in `wq` (64 entries of this
// warp's shared memory) and the exact, explicitly rounded test runs on 32 of
// them at a time, so that its lanes are not idle.  Boxes wider or taller than
// 16,383 cells skip the queue (the packed item holds 14-bit coordinates).
template <typename T>
__device__ __forceinline__ void detect_element2_warp(const GridArgs<T> &g, uint32_t *flag_words, const LinkTable &lt,
                                                     const SurfaceArgs &s, const StepScalars &sc, long long e,
                                                     uint32_t *wq, uint32_t key_base = 0, uint32_t *owner = nullptr,
                                                     uint32_t owner_id = 0)
{
    constexpr int Q = 9;
    const int lane = threadIdx.x & 31;
    const unsigned full = 0xffffffffu;
    const uint32_t va = s.E[2 * e], vb = s.E[2 * e + 1];
    if (va >= (uint32_t)s.nv || vb >= (uint32_t)s.nv) {
        if (lane == 0) atomicOr(g.status, kStatusBadElement);
        return;
    }
    float bmin[2] = {3.402823466e+38f, 3.402823466e+38f};
    float bmax[2] = {1.175494351e-38f, 1.175494351e-38f};
    const uint32_t vid[2] = {va, vb};
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const float c = s.V[(size_t)vid[j] * 2 + k];
            if (c < bmin[k]) bmin[k] = c;
            if (bmax[k] < c) bmax[k] = c;
        }
    const float cl = sc.cl;
    const int lo0 = max(__float2int_rz(geom::dvd(bmin[0], cl)) - 1, 0);
    const int hi0 = min(__float2int_rz(geom::dvd(bmax[0], cl)) + 1, g.nx - 1);
    const int lo1 = max(__float2int_rz(geom::dvd(bmin[1], cl)) - 1, 0);
    const int hi1 = min(__float2int_rz(geom::dvd(bmax[1], cl)) + 1, g.ny - 1);
    const int ext0 = hi0 - lo0 + 1, ext1 = hi1 - lo1 + 1;
    if (ext0 <= 0 || ext1 <= 0) return;
    const long long items = (long long)ext0 * ext1 * (Q - 1);
    const int l = (lane & 7) + 1;
    int cx, cy, cz;
    dir_vec<2>(l, cx, cy, cz);
    // the exact test of cell (i, j), direction ll, and the insertion on a hit
    auto exact = [&](int i, int j, int ll) {
        int dx, dy, dz;
        dir_vec<2>(ll, dx, dy, dz);
        const geom::Hit h = geom::isect2(s.V, va, vb, geom::mul((float)i, cl), geom::mul((float)j, cl),
                                         geom::mul(geom::sub((float)i, (float)dx), cl),
                                         geom::mul(geom::sub((float)j, (float)dy), cl));
        if (!h.hit) return;
        const uint32_t cell = (uint32_t)((long long)j * g.nx + i);
        insert_link<2>(g, lt, flag_words, cell, ll, geom::link_key(h.depth, (uint32_t)e), key_base, owner,
                       owner_id);
    };
    int ci = lane >> 3, cj = 0;
    while (ci >= ext0) { ci -= ext0; ++cj; }
    if (ext0 > 16383 || ext1 > 16383) {
        for (long long it = lane; it < items; it += 32) {
            if (it != lane) {
                ci += 4;
                while (ci >= ext0) { ci -= ext0; ++cj; }
            }
            exact(lo0 + ci, lo1 + cj, l);
        }
        return;
    }
    // the element's line: normal (y3 - y4, x4 - x3) through vertex 4; the
    // prefilter's own rounding is far below its margin
    const float x3 = s.V[2 * (size_t)va], y3 = s.V[2 * (size_t)va + 1];
    const float x4 = s.V[2 * (size_t)vb], y4 = s.V[2 * (size_t)vb + 1];
    const float en0 = y3 - y4, en1 = x4 - x3;
    const float margin = 1e-2f * cl * sqrtf(en0 * en0 + en1 * en1);
    const float dstep = cl * (en0 * (float)cx + en1 * (float)cy); // s1 - s2 of this lane's direction
    const unsigned below = (1u << lane) - 1u;
    int qn = 0;
    for (long long base = 0; base < items; base += 32) {
        if (base != 0) {
            ci += 4;
            while (ci >= ext0) { ci -= ext0; ++cj; }
        }
        bool cand = false;
        if (base + lane < items) {
            const float s1 = en0 * ((float)(lo0 + ci) * cl - x4) + en1 * ((float)(lo1 + cj) * cl - y4);
            const float s2 = s1 - dstep;
            cand = !(fabsf(s1) > margin && fabsf(s2) > margin && ((s1 > 0.0f) == (s2 > 0.0f)));
        }
        const unsigned m = __ballot_sync(full, cand);
        if (cand) wq[qn + __popc(m & below)] = ((uint32_t)cj << 17) | ((uint32_t)ci << 3) | (uint32_t)(l - 1);
        qn += __popc(m);
        if (qn >= 32) {
            __syncwarp();
            const uint32_t code = wq[lane];
            __syncwarp();
            if (lane < qn - 32) wq[lane] = wq[32 + lane];
            __syncwarp();
            qn -= 32;
            exact(lo0 + (int)((code >> 3) & 0x3fffu), lo1 + (int)(code >> 17), (int)(code & 7u) + 1);
        }
    }
    __syncwarp();
    if (lane < qn) {
        const uint32_t code = wq[lane];
        exact(lo0 + (int)((code >> 3) & 0x3fffu), lo1 + (int)(code >> 17), (int)(code & 7u) + 1);
    }
    __syncwarp();
}

// D2Q9 link detection of one or four segments by one warp, `lanes` = 32 or 8
// lanes each (the eight directions, and the lines of one direction dealt out
// to the lanes that share it): the lane group's element e (when `valid`), of a
// surface and a grid that may differ from group to group.
//
// A link segment x -> x - c lies on one of the lattice lines parallel to c,
// and such a line meets the element's line in one point, so a lane looks only
// at the lines that can pass through the element and on each at the one or two
// cells whose link reaches that point, instead of at every cell of the
// element's bounding box.  With k the first axis that c moves along and j the
// other one, a line is named by the integer q = x_j - (c_j / c_k) x_k; the
// lines that can pass are those of the element's own range of q, 2 % and 0.02
// cells wider.  What remains goes through detect_element2_warp's prefilter
// (both end points on one side by more than a hundredth of a cell times the
// element's length) and then the exact test, so the link set is the exact
// test's.
//
// The exact test takes a point of the element's line as on the element by its
// x alone (line_intersect), with an error of a few float ulps of the
// coordinates (2.4e-7 x the largest grid extent in cells x cl).  Elements whose
// x extent is not 100 times that (nearly vertical ones) have every cell of
// their bounding box tested (detect_element2_warp), and so have boxes beyond
// 16,383 cells.
template <typename T>
__device__ __forceinline__ void detect_elements2_warp(const GridArgs<T> &g, uint32_t *flag_words, const LinkTable &lt,
                                                      const SurfaceArgs &s, const StepScalars &sc, long long e, bool valid,
                                                      int lanes, uint32_t *wq, uint32_t key_base = 0,
                                                      uint32_t *owner = nullptr, uint32_t owner_id = 0)
{
    constexpr int Q = 9;
    const int lane = threadIdx.x & 31, first = lane & ~(lanes - 1);
    const unsigned full = 0xffffffffu;
    uint32_t va = 0, vb = 0;
    if (valid) {
        va = s.E[2 * e];
        vb = s.E[2 * e + 1];
        if (va >= (uint32_t)s.nv || vb >= (uint32_t)s.nv) {
            if (lane == first) atomicOr(g.status, kStatusBadElement);
            valid = false;
        }
    }
    bool plain = false; // take every cell of the box
    if (valid) {
        const float cl = sc.cl;
        const float x3 = s.V[2 * (size_t)va], y3 = s.V[2 * (size_t)va + 1];
        const float x4 = s.V[2 * (size_t)vb], y4 = s.V[2 * (size_t)vb + 1];
        float bmin[2] = {3.402823466e+38f, 3.402823466e+38f}, bmax[2] = {1.175494351e-38f, 1.175494351e-38f};
        const float c2[2][2] = {{x3, y3}, {x4, y4}};
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                if (c2[j][k] < bmin[k]) bmin[k] = c2[j][k];
                if (bmax[k] < c2[j][k]) bmax[k] = c2[j][k];
            }
        const int lo0 = max(__float2int_rz(geom::dvd(bmin[0], cl)) - 1, 0);
        const int hi0 = min(__float2int_rz(geom::dvd(bmax[0], cl)) + 1, g.nx - 1);
        const int lo1 = max(__float2int_rz(geom::dvd(bmin[1], cl)) - 1, 0);
        const int hi1 = min(__float2int_rz(geom::dvd(bmax[1], cl)) + 1, g.ny - 1);
        const float coord_err = 2.4e-7f * (float)max(g.nx, g.ny) * cl;
        plain = !(fabsf(x4 - x3) > 100.0f * coord_err) || hi0 - lo0 > 16382 || hi1 - lo1 > 16382;
        if (!plain) {
            const int l = (lane & 7) + 1;
            int cx, cy, cz;
            dir_vec<2>(l, cx, cy, cz);
            const float inv_cl = __fdividef(1.0f, cl);
            const bool alongx = cx != 0;
            const int ck = alongx ? cx : cy, r = alongx ? cy * cx : 0;
            // the element's line: normal (y3 - y4, x4 - x3) through vertex 4
            const float en0 = y3 - y4, en1 = x4 - x3;
            const float margin = 1e-2f * cl * sqrtf(en0 * en0 + en1 * en1);
            const float dstep = cl * (en0 * (float)cx + en1 * (float)cy); // s1 - s2 of this lane's direction
            const float k3 = (alongx ? x3 : y3) * inv_cl, k4 = (alongx ? x4 : y4) * inv_cl;
            const float q3 = (alongx ? y3 : x3) * inv_cl - (float)r * k3, q4 = (alongx ? y4 : x4) * inv_cl - (float)r * k4;
            const float wide = 0.02f * fabsf(q4 - q3) + 0.02f;
            // of those, the lines that pass through the box
            const int lj = alongx ? lo1 : lo0, hj = alongx ? hi1 : hi0, lk = alongx ? lo0 : lo1, hk = alongx ? hi0 : hi1;
            int q = max((int)ceilf(fminf(q3, q4) - wide), lj - (r > 0 ? hk : r < 0 ? -lk : 0));
            const int qend = min((int)floorf(fmaxf(q3, q4) + wide), hj - (r > 0 ? lk : r < 0 ? -hk : 0));
            // the element's line meets line q at x_k = s; the cells whose link
            // reaches it are x_k = s .. s + c_k, wider by the margin.  A link nearly
            // parallel to the element takes the whole box along k.
            const bool reach = fabsf(dstep) > margin;
            const float inv = reach ? __fdividef((float)ck * cl, dstep) : 0.0f; // 1 / (c_k n.c), n not normalised
            const float gq = (alongx ? en1 : en0) * inv;
            const float slack = reach ? 1.2f * margin * fabsf(inv) * inv_cl + 2e-3f : 1e9f;
            const float from = (ck > 0 ? 0.0f : -1.0f) - slack, to = (ck > 0 ? 1.0f : 0.0f) + slack;
            const float klo = (float)lk, khi = (float)hk;
            for (q += (lane - first) >> 3; q <= qend; q += lanes >> 3) {
                const float sk = k4 - gq * ((float)q - q4);
                int k = (int)ceilf(fmaxf(sk + from, klo));
                const int kend = (int)floorf(fminf(sk + to, khi));
                for (; k <= kend; ++k) {
                    const int o = q + r * k;
                    const int i = alongx ? k : o, j = alongx ? o : k;
                    if (i < lo0 || i > hi0 || j < lo1 || j > hi1) continue;
                    const float s1 = en0 * ((float)i * cl - x4) + en1 * ((float)j * cl - y4);
                    const float s2 = s1 - dstep;
                    if (fabsf(s1) > margin && fabsf(s2) > margin && ((s1 > 0.0f) == (s2 > 0.0f))) continue;
                    const geom::Hit h = geom::isect2(s.V, va, vb, geom::mul((float)i, cl), geom::mul((float)j, cl),
                                                     geom::mul(geom::sub((float)i, (float)cx), cl),
                                                     geom::mul(geom::sub((float)j, (float)cy), cl));
                    if (!h.hit) continue;
                    const uint32_t cell = (uint32_t)((long long)j * g.nx + i);
                    insert_link<2>(g, lt, flag_words, cell, l, geom::link_key(h.depth, (uint32_t)e), key_base, owner,
                                   owner_id);
                }
            }
        }
    }
    // nearly vertical elements: the whole warp takes them one by one
    for (unsigned left = __ballot_sync(full, plain && lane == first); left; left &= left - 1) {
        const int from = __ffs(left) - 1;
        auto of = [&](auto v) {
            decltype(v) r;
            static_assert(sizeof(v) % 4 == 0, "whole words");
#pragma unroll
            for (int k = 0; k < (int)(sizeof(v) / 4); ++k)
                reinterpret_cast<uint32_t *>(&r)[k] = __shfl_sync(full, reinterpret_cast<const uint32_t *>(&v)[k], from);
            return r;
        };
        GridArgs<T> gf = g;
        gf.nx = of(g.nx);
        gf.ny = of(g.ny);
        gf.status = of(g.status);
        gf.wallmask = of(g.wallmask);
        SurfaceArgs sf = s;
        sf.V = of(s.V);
        sf.E = of(s.E);
        sf.nv = of(s.nv);
        const StepScalars scf{of(sc.cl), sc.ct, sc.cf};
        detect_element2_warp<T>(gf, of(flag_words), lt, sf, scf, of(e), wq, of(key_base), owner, of(owner_id));
    }
    __syncwarp();
}

// Per-vertex force shares of the links of one cell, added to the vertex
// accumulators in 2^-32 fixed point with 64-bit integer atomics, one per
// (link, vertex slot, component).  Integer sums are associative, so the
// per-vertex result does not depend on warp, lane or launch order.  Each
// share is first rounded to 2^-24 (as an int32) and then scaled by 2^8,
// which is exactly what summing the int32 shares of a cell's links to one
// element and scaling the sum would give; a share beyond +-127 lattice units
// is clamped and flagged.  (Summing the links of one element within the warp
// first, with __match_any_sync and __reduce_add_sync over partial masks, took
// about 120 instructions per cell, more than the atomics it saved.)
template <int DIM>
__device__ __forceinline__ void add_forces(long long *acc, const uint32_t *vert, const float (*share)[3], uint32_t *status)
{
#pragma unroll
    for (int j = 0; j < DIM; ++j)
#pragma unroll
        for (int k = 0; k < DIM; ++k) {
            float v = share[j][k];
            if (!(fabsf(v) < 127.0f)) {
                atomicOr(status, kStatusForceRange);
                v = isfinite(v) ? copysignf(127.0f, v) : 0.0f;
            }
            const int q = __float2int_rn(v * 16777216.0f); // 2^24
            if (q != 0)
                atomicAdd(reinterpret_cast<unsigned long long *>(acc + (size_t)vert[j] * DIM + k),
                          (unsigned long long)((long long)q * 256)); // 2^24 -> 2^32
        }
}

// Lanes per link cell.  A D3Q27 cell takes a whole warp, one lane per
// direction.  A D2Q9 cell takes 16 lanes of one direction each where a step
// has a few hundred link cells (one grid: its time is the chain of one cell's
// loads), and 4 lanes of up to three directions where it has tens of
// thousands (the serving pool: its time is the instructions, 390 per lane and
// cell, most of them the cell's own coefficients and idle lanes).  On one
// 1200 x 400 grid 4 lanes cost 2 us a step against 16; in the pool they take
// 5.9 M warp instructions a substep of 64 episodes, against 12.6 M.
template <int DIM> constexpr int kLinkGroup = DIM == 2 ? 16 : 32;
constexpr int kPoolLinkGroup = 4;

// Update of one link-owning D3Q27 cell by one warp (lane i = direction i;
// D2Q9: link_cell_update2): wall bounce-back, moving-wall
// reconstruction with its momentum-exchange force shares, or the ordinary
// pull; the raw moments are reduced across the group and its lane 0
// collides, stores and feeds outlets.  `links` holds the Q keys of the
// cell's table slot; the force shares go to `acc`.  Every lane of the warp
// calls this together (the force sums and the reduction are warp-wide); a
// group with valid = false has no cell in this iteration and only takes part in
// those, with arguments that still name a real cell.
template <typename T>
__device__ __forceinline__ void link_cell_update3(const GridArgs<T> &g, const unsigned long long *links,
                                                 uint32_t slot, uint32_t cell, long long *acc,
                                                 const SurfaceArgs &s, const StepScalars &sc, bool valid = true)
{
    constexpr int DIM = 3, Q = Lattice<DIM>::Q, NM = Lattice<DIM>::NM, G = kLinkGroup<DIM>;
    static_assert(Q <= G, "one lane per direction");
    const int lane = threadIdx.x & (G - 1);
    const unsigned full = 0xffffffffu;
    // cell indices are 32-bit (the link table keys them so), and so is every
    // index formed from them here
    const uint32_t nx = (uint32_t)g.nx, nxy = nx * (uint32_t)g.ny;
    const bool wx = g.periodic & 1, wy = g.periodic & 2, wz = g.periodic & 4;
    const uint32_t row = cell / nx;
    const int x = (int)(cell - row * nx);
    const uint32_t z32 = row / (uint32_t)g.ny;
    const int y = (int)(row - z32 * (uint32_t)g.ny);
    const int z = (int)z32;
    const uint8_t f8 = g.flags[cell];
    const bool upd = valid && is_updated(f8 & kTypeMask);
    float mc[NM];
    float pop = 0.0f;
    bool has_share = false;
    uint32_t vshare[3] = {0, 0, 0};
    float share[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}}; // [vertex][component]
    // Every load the update may need goes out before any of them is tested:
    // the cell's own moments and, per lane, the node type of the wrapped
    // neighbour, the link key and the moments of the cell an ordinary pull
    // reads (a lane that takes the bounce-back or a moving-wall link discards
    // its pull).  The update then waits for one round of loads where testing
    // the node type and the key first would make it wait for three.
    load_moments<DIM, T>(mc, g.src, g.ncell, cell, g.codec);
    if (upd) {
        Coef<DIM> own;
        own.make(mc);
        if (lane < Q) {
            const int i = lane;
            int cx, cy, cz;
            dir_vec<DIM>(i, cx, cy, cz);
            const int x1 = x - cx, y1 = y - cy, z1 = z - cz;
            const bool notCross = x1 >= 0 && x1 < g.nx && y1 >= 0 && y1 < g.ny && z1 >= 0 && z1 < g.nz;
            // the wrapped neighbour (x1, y1, z1 are within one cell of the grid)
            auto wrap1 = [](int v, int n) { return v < 0 ? v + n : (v >= n ? v - n : v); };
            const uint32_t ib = (uint32_t)wrap1(z1, g.nz) * nxy + (uint32_t)wrap1(y1, g.ny) * nx + (uint32_t)wrap1(x1, g.nx);
            // the ordinary pull's source: the upstream halo cell (halo_index)
            const int sx = halo_index(x1, g.nx, wx), sy = halo_index(y1, g.ny, wy), sz = halo_index(z1, g.nz, wz);
            const uint32_t sidx = (uint32_t)sz * nxy + (uint32_t)sy * nx + (uint32_t)sx;
            const uint8_t fb = g.flags[ib];
            const unsigned long long key = notCross ? links[(size_t)slot * Q + i] : ~0ull;
            float pulled;
            {
                float mn[NM];
                load_moments<DIM, T>(mn, g.src, g.ncell, sidx, g.codec);
                Coef<DIM> nc;
                nc.make(mn);
                float v = nc.population(cx, cy, cz);
                pulled = fmaxf(v, 0.0f);
            }
            bool done = false;
            // a wall neighbour: bounce-back, no link
            const bool bb = is_bounce_back<DIM>(fb & kTypeMask);
            if (bb) {
                float v = own.population(-cx, -cy, -cz);
                pop = fmaxf(v, 0.0f);
                done = true;
            } else if (notCross) {
                if (key != ~0ull) {
                    const uint32_t e = (uint32_t)(key & 0xffffffffull);
                    const float cl = sc.cl;
                    geom::Hit h;
                    uint32_t vv[3] = {s.E[DIM * (size_t)e], s.E[DIM * (size_t)e + 1], s.E[DIM * (size_t)e + 2]};
                    {
                        float p1[3] = {geom::mul((float)x, cl), geom::mul((float)y, cl), geom::mul((float)z, cl)};
                        float p2[3] = {geom::mul((float)x1, cl), geom::mul((float)y1, cl), geom::mul((float)z1, cl)};
                        h = geom::isect3(s.V, vv[0], vv[1], vv[2], p1, p2);
                    }
                    if (h.hit) {
                        // wall velocity at the hit point, in lattice units
                        float uw[3] = {0.0f, 0.0f, 0.0f};
#pragma unroll
                        for (int k = 0; k < DIM; ++k) {
                            float a = s.U[(size_t)vv[0] * DIM + k] * h.b[0] + s.U[(size_t)vv[1] * DIM + k] * h.b[1];
                            a += s.U[(size_t)vv[2] * DIM + k] * h.b[2];
                            uw[k] = (a * sc.ct) / sc.cl;
                        }
                        // moving-wall population: Hermite expansion with the cell's
                        // density, the wall velocity and pi' = pi + uw uw - u u
                        float mw[NM];
                        mw[0] = mc[0];
#pragma unroll
                        for (int k = 0; k < DIM; ++k) mw[1 + k] = uw[k];
#pragma unroll
                        for (int k = DIM + 1; k < NM; ++k) {
                            const int a = MomentLayout<DIM>::pa(k), b = MomentLayout<DIM>::pb(k);
                            mw[k] = mc[k] + uw[a] * uw[b] - mc[1 + a] * mc[1 + b];
                        }
                        Coef<DIM> wc;
                        wc.make(mw);
                        const float fout = wc.population(cx, cy, cz);
                        float fin = own.population(-cx, -cy, -cz);
                        fin = fmaxf(fin, 0.0f);
                        pop = fout;
                        done = true;
                        // momentum exchange, lattice units: fin (-c - uw) - fout (c - uw)
                        const float c3[3] = {(float)cx, (float)cy, (float)cz};
                        float F[3];
#pragma unroll
                        for (int k = 0; k < DIM; ++k) F[k] = fin * (-c3[k] - uw[k]) - fout * (c3[k] - uw[k]);
                        has_share = true;
#pragma unroll
                        for (int j = 0; j < DIM; ++j) {
                            vshare[j] = vv[j];
#pragma unroll
                            for (int k = 0; k < DIM; ++k) share[j][k] = F[k] * h.b[j];
                        }
                    }
                }
            }
            if (!done) pop = pulled;
        }
    }
    // forces: one share per (link, element vertex), summed per element
    if (has_share) add_forces<DIM>(acc, vshare, share, g.status);
    // raw moments by reduction within the group (lanes Q.. add exact zeros,
    // so the sums equal those of a whole-warp reduction)
    int cx = 0, cy = 0, cz = 0;
    if (lane < Q) dir_vec<DIM>(lane, cx, cy, cz);
    const float fx = (float)cx, fy = (float)cy, fz = (float)cz;
    float R[NM];
    R[0] = pop; R[1] = pop * fx; R[2] = pop * fy; R[3] = pop * fz;
    R[4] = pop * fx * fx; R[5] = pop * fy * fy; R[6] = pop * fz * fz;
    R[7] = pop * fx * fy; R[8] = pop * fy * fz; R[9] = pop * fx * fz;
#pragma unroll
    for (int k = 0; k < NM; ++k)
#pragma unroll
        for (int o = G / 2; o > 0; o >>= 1) R[k] += __shfl_xor_sync(full, R[k], o);
    if (upd) {
        if (lane == 0) {
            float m[NM];
            collide3(R, g.omega, m);
            T *planes[NM];
#pragma unroll
            for (int k = 0; k < NM; ++k) planes[k] = g.dst + (size_t)k * g.ncell;
            encode_store<DIM, T>(m, planes, cell, g.codec);
            if (bad_state<DIM>(m)) atomicOr(g.status, kStatusNonFinite);
            if (f8 & kBitOutletSrc) {
                float ms[NM];
                stored_values<DIM, T>(m, ms, cell, g.codec);
                feed_outlets<DIM, T>(g, cell, ms, g.wallmask[cell]);
            }
        }
    }
}

// Update of one link-owning D2Q9 cell by G lanes: lane q of the group takes
// directions q, q + G, ...  As link_cell_update3, with every load of a lane's
// directions issued before any is tested.  The raw moments are summed in the
// same order for G = 4 and 16: (q, q + 8), then q + 4, then across lanes by 2
// and by 1; every multiply-add here and in what it calls is explicit, or the
// compiler would choose them for each G and the pool and a grid round apart.
template <typename T, bool HALF, int G>
__device__ __forceinline__ void link_cell_update2(const GridArgs<T> &g, const unsigned long long *links, uint32_t slot,
                                                  uint32_t cell, long long *acc, const SurfaceArgs &s,
                                                  const StepScalars &sc, bool valid)
{
    static_assert(G == 4 || G == 16, "the order of the sums above");
    constexpr int N = G == 4 ? 3 : 1; // directions per lane
    const int q = threadIdx.x & (G - 1);
    const unsigned full = 0xffffffffu;
    const uint32_t nx = (uint32_t)g.nx;
    const bool wx = g.periodic & 1, wy = g.periodic & 2;
    const int y = (int)(cell / nx), x = (int)(cell - (uint32_t)y * nx);
    const uint8_t f8 = g.flags[cell];
    const bool upd = valid && is_updated(f8 & kTypeMask);
    float pop[N] = {};
    if (upd) {
        float mc[6], mn[N][6];
        unsigned long long key[N];
        uint8_t fb[N];
        load_moments<2, T>(mc, g.src, g.ncell, cell, g.codec);
        auto wrap1 = [](int v, int n) { return v < 0 ? v + n : (v >= n ? v - n : v); };
#pragma unroll
        for (int t = 0; t < N; ++t) {
            const int i = q + G * t;
            if (i >= 9) continue;
            int cx, cy, cz;
            dir_vec<2>(i, cx, cy, cz);
            const int x1 = x - cx, y1 = y - cy;
            const bool not_cross = x1 >= 0 && x1 < g.nx && y1 >= 0 && y1 < g.ny;
            fb[t] = g.flags[(uint32_t)wrap1(y1, g.ny) * nx + (uint32_t)wrap1(x1, g.nx)];
            key[t] = not_cross ? links[(size_t)slot * 9 + i] : ~0ull;
            load_moments<2, T>(mn[t], g.src, g.ncell, (uint32_t)halo_index(y1, g.ny, wy) * nx + (uint32_t)halo_index(x1, g.nx, wx),
                               g.codec);
        }
        Coef<2> own;
        own.make(mc);
#pragma unroll
        for (int t = 0; t < N; ++t) {
            const int i = q + G * t;
            if (i >= 9) continue;
            int cx, cy, cz;
            dir_vec<2>(i, cx, cy, cz);
            // a wall neighbour: bounce-back, no link (with wall_stream, the
            // reference's 2D kernel: the ordinary pull, no link either)
            const bool bb = is_bounce_back<2>(fb[t] & kTypeMask);
            const float back = own.population(-cx, -cy, 0);
            Coef<2> nc;
            nc.make(mn[t]);
            float v = bb && !g.wall_stream ? back : nc.population(cx, cy, 0);
            if (HALF) v = round_half(v);
            pop[t] = fmaxf(v, 0.0f);
            if (bb || key[t] == ~0ull) continue;
            const uint32_t e = (uint32_t)(key[t] & 0xffffffffull);
            const float cl = sc.cl;
            const uint32_t va = s.E[2 * (size_t)e], vb = s.E[2 * (size_t)e + 1];
            const geom::Hit h = geom::isect2(s.V, va, vb, geom::mul((float)x, cl), geom::mul((float)y, cl),
                                             geom::mul((float)(x - cx), cl), geom::mul((float)(y - cy), cl));
            if (!h.hit) continue;
            // wall velocity at the hit point, in lattice units
            float uw[2], a[2];
            const float scale = sc.ct / sc.cl;
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                a[k] = fmaf(s.U[(size_t)va * 2 + k], h.b[0], s.U[(size_t)vb * 2 + k] * h.b[1]);
                uw[k] = __fmul_rn(a[k], scale);
            }
            // moving-wall population: Hermite expansion with the cell's density,
            // the wall velocity and pi' = pi + uw uw - u u
            const float mw[6] = {mc[0], uw[0], uw[1], fmaf(-mc[1], mc[1], fmaf(uw[0], uw[0], mc[3])),
                                 fmaf(-mc[2], mc[2], fmaf(uw[1], uw[1], mc[4])), fmaf(-mc[1], mc[2], fmaf(uw[0], uw[1], mc[5]))};
            Coef<2> wc;
            wc.make(mw);
            const float fout = wc.population(cx, cy, 0);
            float fin = back;
            if (HALF) fin = round_half(fin);
            fin = fmaxf(fin, 0.0f);
            pop[t] = fout;
            // momentum exchange, lattice units: fin (-c - uw) - fout (c - uw)
            const float Fx = fmaf(fin, fmaf(-a[0], scale, -(float)cx), -(fout * fmaf(-a[0], scale, (float)cx)));
            const float Fy = fmaf(fin, fmaf(-a[1], scale, -(float)cy), -(fout * fmaf(-a[1], scale, (float)cy)));
            const uint32_t vert[3] = {va, vb, 0u};
            const float share[3][3] = {{Fx * h.b[0], Fy * h.b[0], 0.0f}, {Fx * h.b[1], Fy * h.b[1], 0.0f}, {0.0f, 0.0f, 0.0f}};
            add_forces<2>(acc, vert, share, g.status);
        }
    }
    float R[6] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
    for (int o = 0; o < N; ++o) {
        const int t = o == 0 ? 0 : N - o, i = q + G * t; // 0, 2, 1
        int cx = 0, cy = 0, cz = 0;
        if (i < 9) dir_vec<2>(i, cx, cy, cz);
        const float fx = (float)cx, fy = (float)cy, p = pop[t];
        R[0] += p; R[1] += p * fx; R[2] += p * fy;
        R[3] += p * fx * fx; R[4] += p * fy * fy; R[5] += p * fx * fy;
    }
#pragma unroll
    for (int k = 0; k < 6; ++k)
#pragma unroll
        for (int o = G / 2; o > 0; o >>= 1) R[k] += __shfl_xor_sync(full, R[k], o);
    if (upd && q == 0) {
        float m[6];
        collide2(R, g.omega, m);
        T *planes[6];
#pragma unroll
        for (int k = 0; k < 6; ++k) planes[k] = g.dst + (size_t)k * g.ncell;
        encode_store<2, T>(m, planes, cell, g.codec);
        if (bad_state<2>(m)) atomicOr(g.status, kStatusNonFinite);
        if (f8 & kBitOutletSrc) {
            float ms[6];
            stored_values<2, T>(m, ms, cell, g.codec);
            feed_outlets<2, T>(g, cell, ms, g.wallmask[cell]);
        }
    }
}

} // namespace fflbm
