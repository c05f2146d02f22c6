// Row-marching body of the fused D2Q9 update, one warp per unit, for the serving
// pool and large single grids, and the cell update it shares with the tiles of
// small ones (ffs_dense2d.cu).
//
// Reference: mrDeformableSolver2DKernel_Shrd (src/core/FsiCoupling2D.cu:82-255).
//
// A unit is 64 columns and up to 14 rows of one grid.  The warp walks up its
// rows; each lane owns two adjacent columns as packed FP32 pairs.  A row's cells
// are reconstructed once, and nothing leaves the registers: the rows y-1, y,
// y+1 that feed row y meet in three partial sums per c_x as they pass, and the
// columns x-1 and x+1 meet in six shuffles of completed sums per pair.  There
// is no shared memory and no barrier, so warps only wait for their own loads,
// which go out two rows ahead.  What the columns at either end of the unit
// feed into it is worked out first, one row a lane (ends), and handed round
// by the same shuffles.
//
// What bounds it: instruction issue, then HBM.  The tile-and-strip kernels it
// replaced in the pool staged populations in shared memory and spent about 347
// thread instructions per cell; the packed march takes 191 (FP16 serving mix,
// 14 rows, with detection).
//
// Bounce-back: a wall or solid cell is reconstructed from a zero state, so
// whatever a neighbour pulls from it adds nothing, and a cell next to a wall
// adds its own reflected populations max(0, f_inv(i)(x)) to its raw moments
// (FsiCoupling2D.cu:171-181).  A cell on the high face of a non-periodic axis
// pulls from a clamped halo while its wall test wraps (halo_index); such
// cells (Fluid cells there are unusual: the faces hold walls, inlets or
// outlets) are updated one by one after the march (edge_cell).
#pragma once
#include <type_traits>

#include "ffs_dense2d.cuh"

namespace fflbm {
namespace march2 {

constexpr int kWindow = 64;   // columns of a unit
constexpr int kMaxRows = 14;  // rows of a unit at most: with the two around them a half warp's lanes

__host__ __device__ constexpr int windows(int nx) { return (nx + kWindow - 1) / kWindow; }
__host__ __device__ constexpr int chunks(int ny, int rows) { return (ny + rows - 1) / rows; }

// One stored moment of two adjacent columns.
template <typename T> struct Pair {
    using type = uint32_t;
};
template <> struct Pair<float> {
    using type = unsigned long long;
};

// VEC: the two cells sit side by side on a boundary of the pair's size;
// otherwise they are fetched one by one (odd widths).
template <typename T, bool VEC>
__device__ __forceinline__ typename Pair<T>::type load_pair(const T *plane, uint32_t i0, uint32_t i1)
{
    using P = typename Pair<T>::type;
    if constexpr (VEC) return *reinterpret_cast<const P *>(plane + i0);
    if constexpr (sizeof(T) == 4) {
        return f2make(plane[i0], plane[i1]).v;
    } else {
        const unsigned short *u = reinterpret_cast<const unsigned short *>(plane);
        return (uint32_t)u[i0] | ((uint32_t)u[i1] << 16);
    }
}

__device__ __forceinline__ f2 halves(uint32_t u)
{
    const float2 v = __half22float2(*reinterpret_cast<const __half2 *>(&u));
    return f2make(v.x, v.y);
}
__device__ __forceinline__ f2 unpack(float, int, unsigned long long v) { return f2{v}; }
__device__ __forceinline__ f2 unpack(__half, int, uint32_t u) { return halves(u); }
__device__ __forceinline__ f2 unpack(__nv_bfloat16, int k, uint32_t u)
{
    if (k == 1 || k == 2) return halves(u); // velocities are binary16 (StorageTraits)
    return f2make(__uint_as_float(u << 16), __uint_as_float(u & 0xffff0000u));
}

// Stored moments of one or two cells, decoded (decode_moments); d = rho - 1,
// exact for both kinds of storage.
template <typename T, typename V> __device__ __forceinline__ void decode_values(const Codec &c, V *m, V &d)
{
    if constexpr (StorageTraits<T>::kEncoded) {
        const V isp = vconst<V>(c.inv_sp), isu = vconst<V>(c.inv_su);
        d = m[0];
        m[0] = vconst<V>(1.0f) + d;
        m[1] = m[1] * isu;
        m[2] = m[2] * isu;
        m[3] = vfma(m[3], isp, m[1] * m[1]);
        m[4] = vfma(m[4], isp, m[2] * m[2]);
        m[5] = vfma(m[5], isp, m[1] * m[2]);
    } else {
        d = m[0] - vconst<V>(1.0f);
    }
}
template <typename T> __device__ __forceinline__ void decode(const typename Pair<T>::type *raw, const Codec &c, f2 *m, f2 &d)
{
#pragma unroll
    for (int k = 0; k < 6; ++k) m[k] = unpack(T(), k, raw[k]);
    decode_values<T>(c, m, d);
}

// Populations are kept as deviations F' = F - 1 of their Hermite sums from the
// rest state's (all ones without the lattice weights), so that the sums below
// are of the size of the flow's own terms and round accordingly; F itself would
// bring the rounding of terms near 1 into the momentum.  A population is
// clamped at 0, so F' at -1; a bounce-back cell sends F = 0.
__device__ __forceinline__ f2 clamp1(f2 a)
{
    float lo, hi;
    f2split(a, lo, hi);
    return f2make(fmaxf(lo, -1.0f), fmaxf(hi, -1.0f));
}

// Reconstruction and collision are written so that no product feeds a plain
// sum: the assembler contracts packed multiplies into packed adds as it sees
// fit (-fmad does not reach them), copy by copy of the loop, and the bits of a
// row would then depend on where its unit starts.  Products by powers of two
// are exact and may stand anywhere.
//
// Hermite sums of a pair (Coef<2>), y level: the coefficients of {1, c_x,
// g(c_x)} for c_y = ky - 1 (the reference's D2Q9 expansion omits rho on the pi
// terms of its third order, LbmUtilsFunc.cu:488-490).
template <typename V> struct Rows {
    V r3, h3, pxx, C0[3], C1[3], q;
    static __device__ __forceinline__ V k(float a) { return vconst<V>(a); }
    __device__ __forceinline__ Rows(const V *m, V d)
    {
        const V r = m[0], ux = m[1], uy = m[2], pyy = m[4], pxy = m[5];
        pxx = m[3];
        r3 = k(3.0f) * r;
        h3 = k(-0.5f) * r3;
        const V n3 = k(-1.0f) * r3, r9 = k(3.0f) * r3, n9 = k(-3.0f) * r3;
        // Q_aab = 9 (pi_aa u_b + 2 u_a (pi_ab - rho u_a u_b))
        const V t18 = k(18.0f) * vfma(k(-1.0f) * (r * ux), uy, pxy), nine = k(9.0f);
        q = vfma(nine * pxx, uy, t18 * ux);                  // Q_xxy
        const V qyyx = vfma(nine * pyy, ux, t18 * uy);
        const V t0 = vfma(r3, pyy, d);
        C0[0] = vfma(n3, uy, t0);
        C0[1] = vfma(h3, pyy, d);
        C0[2] = vfma(r3, uy, t0);
        const V t1 = vfma(r3, ux, qyyx);
        C1[0] = vfma(n9, pxy, t1);
        C1[1] = vfma(k(-0.5f), qyyx, r3 * ux);
        C1[2] = vfma(r9, pxy, t1);
    }
    // the unweighted, unclamped populations with c_y = KY - 1, less 1: F'[kx]
    template <int KY> __device__ __forceinline__ void row(V *F) const
    {
        V t;
        if constexpr (KY == 1) {
            t = vfma(r3, pxx, C0[1]);
            F[1] = vfma(h3, pxx, C0[1]);
        } else {
            // C2 = 3 rho pi_xx + c_y Q_xxy, g(c_x) = 1 or -1/2
            const V c2 = vfma(KY == 2 ? r3 : k(-1.0f) * r3, pxx, q); // c_y C2
            t = KY == 2 ? C0[KY] + c2 : C0[KY] - c2;
            F[1] = vfma(k(KY == 2 ? -0.5f : 0.5f), c2, C0[KY]);
        }
        F[0] = t - C1[KY];
        F[2] = t + C1[KY];
    }
};

// collide2 from the sums S of F', of one cell or a pair: the raw moments are
// {1 + W0 S0, W0/4 S1, W0/4 S2, 1/3 + W0/4 S3, 1/3 + W0/4 S4, W0/16 S5} with
// W0 = 4/9 (the lattice weights are W0 times powers of 1/4).  The velocity
// comes out in its stored scale, u * su (su a power of two, isu2 = su^-2).
// d receives rho - 1.
constexpr float kW0 = wgt2(1, 1);
__device__ __forceinline__ float vrecip(float r) { return recip(r); }
__device__ __forceinline__ f2 vrecip(f2 r)
{
    float r0, r1;
    f2split(r, r0, r1);
    return f2make(recip(r0), recip(r1));
}
template <typename V> __device__ __forceinline__ void collide(const V *S, float omega, float su, float isu2, V *m, V &d)
{
    auto k = [](float a) { return vconst<V>(a); };
    const V r = vfma(k(kW0), S[0], k(1.0f));
    d = k(kW0) * S[0];
    const V wr = k(0.25f * kW0) * vrecip(r); // W0 / (4 rho)
    const V wu = wr * k(su);
    const V ux = S[1] * wu, uy = S[2] * wu; // u * su
    const V kr = wr * k(0.5f * (1.0f - omega));
    const V ux2 = ux * ux;
    const V sum = vfma(uy, uy, ux2), dif = vfma(k(-1.0f) * uy, uy, ux2);
    // half the difference of the normal stresses, relaxed
    const V n = vfma(S[3] - S[4], kr, k(0.5f * omega * isu2) * dif);
    const V half_u2 = k(0.5f * isu2) * sum;
    m[0] = r;
    m[1] = ux;
    m[2] = uy;
    m[3] = half_u2 + n;
    m[4] = half_u2 - n;
    m[5] = vfma(S[5], k(0.5f) * kr, k(omega * isu2) * (ux * uy));
}

// Stored form of a pair (encode_values of both cells; d = rho - 1, hash the
// first cell's number times the golden ratio, as in vel_dither)
template <typename T>
__device__ __forceinline__ void encode(const f2 *m, f2 d, uint32_t hash, const Codec &c, typename Pair<T>::type *out)
{
    if constexpr (!StorageTraits<T>::kEncoded) {
#pragma unroll
        for (int k = 0; k < 6; ++k) out[k] = m[k].v;
    } else {
        auto pack = [](f2 a) {
            float lo, hi;
            f2split(a, lo, hi);
            if constexpr (std::is_same<T, __half>::value) {
                const __half2 h = __floats2half2_rn(lo, hi);
                return *reinterpret_cast<const uint32_t *>(&h);
            } else {
                const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
                return *reinterpret_cast<const uint32_t *>(&h);
            }
        };
        float r0, r1, a0, a1;
        f2split(m[0], r0, r1);
        const uint32_t h0 = mix32(hash ^ __float_as_uint(r0)), h1 = mix32((hash + kGolden) ^ __float_as_uint(r1));
        const f2 sp = f2splat(c.sp);
        const f2 isu2 = f2splat(-(c.inv_su * c.inv_su)); // a power of two: u u from the stored u * su is exact scaling
        out[0] = pack(d);
        f2split(m[1], a0, a1);
        out[1] = half2_sr(a0, a1, __byte_perm(h0, h1, 0x5410));
        f2split(m[2], a0, a1);
        out[2] = half2_sr(a0, a1, __byte_perm(h0, h1, 0x7632));
        const f2 sx = halves(out[1]), sy = halves(out[2]);
        const f2 nx = isu2 * sx, ny = isu2 * sy;
        out[3] = pack(vfma(nx, sx, m[3]) * sp);
        out[4] = pack(vfma(ny, sy, m[4]) * sp);
        out[5] = pack(vfma(nx, sy, m[5]) * sp);
    }
}

// The same of one cell.
template <typename T>
__device__ __forceinline__ void encode(const float *m, float d, uint32_t hash, const Codec &c, T *out)
{
    if constexpr (!StorageTraits<T>::kEncoded) {
#pragma unroll
        for (int k = 0; k < 6; ++k) out[k] = m[k];
    } else {
        using Tr = StorageTraits<T>;
        const uint32_t u = half2_sr(m[1], m[2], mix32(hash ^ __float_as_uint(m[0])));
        float sx, sy;
        f2split(halves(u), sx, sy);
        const float isu2 = -(c.inv_su * c.inv_su), nx = isu2 * sx, ny = isu2 * sy;
        out[0] = Tr::to(d);
        out[1] = Tr::to_vel(sx); // binary16 values: exact
        out[2] = Tr::to_vel(sy);
        out[3] = Tr::to(fmaf(nx, sx, m[3]) * c.sp);
        out[4] = Tr::to(fmaf(ny, sy, m[4]) * c.sp);
        out[5] = Tr::to(fmaf(nx, sy, m[5]) * c.sp);
    }
}

// Update of one cell from populations F' given one by one: pull(kx, ky) of the
// cell that c = (kx - 1, ky - 1) comes from, own(kx, ky) of the cell itself (kx
// and ky as Rows).  A direction whose wall bit is set sends F = 0 and the cell
// adds its own reflected population.  wm: the mask word of a cell near walls or
// feeding outlets.  The operations and their order are run's.
template <typename T, typename Pull, typename Own>
__device__ __forceinline__ void update_cell(const GridArgs<T> &g, uint32_t idx, uint32_t f8, uint32_t wm, Pull &&pull, Own &&own)
{
    const uint32_t walls = f8 & kBitNearWall ? wm & wall_bits_mask<2>() : 0u;
    float p[3][3];
#pragma unroll
    for (int ky = 0; ky < 3; ++ky)
#pragma unroll
        for (int kx = 0; kx < 3; ++kx) p[ky][kx] = pull(kx, ky);
    if (walls) {
#pragma unroll
        for (int ky = 0; ky < 3; ++ky)
#pragma unroll
            for (int kx = 0; kx < 3; ++kx)
                if (walls >> dir_index<2>(kx, ky, 1) & 1u) p[ky][kx] = -1.0f;
    }
    float Y0[3], Y1[3], Y2[3], S[6];
#pragma unroll
    for (int kx = 0; kx < 3; ++kx) {
        const float A = p[2][kx], C = p[0][kx];
        Y0[kx] = fmaf(0.25f, C, fmaf(0.25f, A, p[1][kx]));
        Y1[kx] = A - C;
        Y2[kx] = A + C;
    }
    S[3] = Y0[2] + Y0[0];
    S[0] = fmaf(0.25f, S[3], Y0[1]);
    S[1] = Y0[2] - Y0[0];
    S[2] = fmaf(0.25f, Y1[2] + Y1[0], Y1[1]);
    S[4] = fmaf(0.25f, Y2[2] + Y2[0], Y2[1]);
    S[5] = Y1[2] - Y1[0];
    if (walls) {
#pragma unroll
        for (int ky = 0; ky < 3; ++ky)
#pragma unroll
            for (int kx = 0; kx < 3; ++kx) {
                if (kx == 1 && ky == 1) continue;
                const int cx = 1 - kx, cy = 1 - ky;
                const float w = (cx != 0 && cy != 0) ? 0.0625f : 0.25f; // the weight over W0
                const float t = walls >> dir_index<2>(2 - kx, 2 - ky, 1) & 1u ? 1.0f + own(kx, ky) : 0.0f;
                const float t4 = 4.0f * w * t, t16 = 16.0f * w * t;
                S[0] = fmaf(w, t, S[0]);
                if (cx) S[1] = cx > 0 ? S[1] + t4 : S[1] - t4;
                if (cy) S[2] = cy > 0 ? S[2] + t4 : S[2] - t4;
                if (cx) S[3] = S[3] + t4;
                if (cy) S[4] = S[4] + t4;
                if (cx && cy) S[5] = cx * cy > 0 ? S[5] + t16 : S[5] - t16;
            }
    }
    float m[6], d;
    T e[6];
    constexpr bool enc = StorageTraits<T>::kEncoded;
    collide<float>(S, g.omega, enc ? g.codec.su : 1.0f, enc ? g.codec.inv_su * g.codec.inv_su : 1.0f, m, d);
    encode<T>(m, d, idx * kGolden, g.codec, e);
#pragma unroll
    for (int k = 0; k < 6; ++k) g.dst[idx + (uint32_t)k * g.ncell] = e[k];
    if (bad_state<2>(m)) atomicOr(g.status, kStatusNonFinite);
    if (f8 & g.feed) {
        float ms[6] = {};
#pragma unroll
        for (int k = 1; k < 3; ++k) ms[k] = StorageTraits<T>::from_vel(e[k]) * (enc ? g.codec.inv_su : 1.0f);
        feed_outlets<2, T>(g, idx, ms, wm);
    }
}

// F' of one cell with c = (kx - 1, ky - 1)
template <typename T> __device__ __forceinline__ float population(const GridArgs<T> &g, uint32_t cell, int kx, int ky)
{
    float m[6], d, F[3];
#pragma unroll
    for (int k = 0; k < 6; ++k) m[k] = from_storage<2, T>(k, g.src[cell + (uint32_t)k * g.ncell]);
    decode_values<T>(g.codec, m, d);
    const Rows<float> rows(m, d);
    if (ky == 0) rows.template row<0>(F);
    else if (ky == 1) rows.template row<1>(F);
    else rows.template row<2>(F);
    return fmaxf(F[kx], -1.0f);
}

// Update of a Fluid cell on the high face of a non-periodic axis, gathering
// each of its populations from its halo source.
template <typename T> __device__ __noinline__ void edge_cell(const GridArgs<T> g, int x, int y)
{
    const uint32_t idx = (uint32_t)(y * g.nx + x);
    const uint32_t f8 = __ldcg(reinterpret_cast<const unsigned char *>(g.flags) + idx);
    if (!is_updated(f8 & kTypeMask) || (f8 & kBitLink)) return;
    const bool wx = g.periodic & 1, wy = g.periodic & 2;
    update_cell<T>(
        g, idx, f8, g.wallmask[idx],
        [&](int kx, int ky) {
            return population(g, (uint32_t)(halo_index(y + 1 - ky, g.ny, wy) * g.nx + halo_index(x + 1 - kx, g.nx, wx)), kx, ky);
        },
        [&](int kx, int ky) { return population(g, idx, kx, ky); });
}

// What a unit waits for before it feeds outlets or latches a bad state, both of
// which must not come from a cell whose links are not known yet: `*done` to
// reach `want` (the pool's detection units).  Polled by each lane for itself.
// The wait ends well within a launch (pool_dense_kernel); past its limit
// (seconds) the status says that the step is invalid.  A warp keeps its gate
// from unit to unit, open once it was seen open: a look at the counter in every
// unit with outlets took 4 % of the pool's step.
// dry: nothing is fed or latched.
struct Gate {
    const uint32_t *done;
    uint32_t want;
    bool dry;
    __device__ __forceinline__ void wait(uint32_t *status)
    {
        if (want == 0) return;
        poll(done, want, status);
        want = 0;
    }
    static __device__ __noinline__ void poll(const uint32_t *done, uint32_t want, uint32_t *status)
    {
        for (uint32_t k = 0; k < (1u << 24); ++k) {
            uint32_t v;
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(done) : "memory");
            if (v >= want) return;
            __nanosleep(100);
        }
        atomicOr(status, kStatusWaitTimeout);
    }
};
template <typename T> __device__ __forceinline__ bool is_link(const GridArgs<T> &g, uint32_t cell)
{
    return __ldcg(reinterpret_cast<const unsigned char *>(g.flags) + cell) & kBitLink;
}

template <typename T> __device__ __noinline__ void feed_outlet_of(const GridArgs<T> g, uint32_t p) { feed_cell<2, T>(g, p, g.wallmask[p], nullptr); }

// Shared memory of a unit's warp: per end, row (yb - 1 + index) and power of
// c_y, the completed sums that the end column sends in.
struct Ends {
    float y[3][2][16];
};

// Updates columns 64 w .. 64 w + 63 of rows yb .. ye - 1 (at most kMaxRows).  Every moment
// index k ncell + cell fits in 32 bits (the caller guarantees it).
template <typename T, bool VEC>
__device__ __forceinline__ void run(const GridArgs<T> &g, int w, int yb, int ye, Ends &ends, Gate &gate)
{
    using P = typename Pair<T>::type;
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const bool wx = g.periodic & 1, wy = g.periodic & 2;
    const int x = kWindow * w + 2 * lane; // the lane's columns x and x + 1
    // source columns (halo_index; columns at n and beyond feed only high-face
    // cells unless the axis wraps)
    const uint32_t c0 = (uint32_t)(x < g.nx ? x : wx ? x % g.nx : VEC ? g.nx - 2 : g.nx - 1);
    const uint32_t c1 = VEC ? c0 + 1 : (uint32_t)(x + 1 < g.nx ? x + 1 : wx ? (x + 1) % g.nx : g.nx - 1);
    const bool out0 = x < g.nx, out1 = x + 1 < g.nx;
    const bool edge0 = !wx && x == g.nx - 1, edge1 = !wx && x + 1 == g.nx - 1;
    bool edges = false;                 // a Fluid cell on a high face was met
    uint32_t bad = 0;                   // rows whose cells came out in a bad state: bits 0.. and 16..
    uint32_t feeders0 = 0, feeders1 = 0; // rows (from yb) whose cell feeds an outlet
    const uint32_t fastflags = out0 && out1 && !edge0 && !edge1 ? 0x0101u : 0x10000u; // two plain Fluid cells

    // every access forms its address from a cell number and a plane's base
    const T *sp[6];
    T *dp[6];
#pragma unroll
    for (int k = 0; k < 6; ++k) {
        sp[k] = g.src + (size_t)((uint32_t)k * g.ncell);
        dp[k] = g.dst + (size_t)((uint32_t)k * g.ncell);
    }
    P raw[2][6];
    uint32_t fl[2];    // flag bytes of the two source cells
    uint32_t wm[2][2]; // mask words of the near-wall cells of the last two rows
    auto load = [&](int r, P (&v)[6], uint32_t &f) {
        const uint32_t row = (uint32_t)halo_index(r, g.ny, wy) * (uint32_t)g.nx;
        const uint32_t i0 = row + c0, i1 = row + c1;
#pragma unroll
        for (int k = 0; k < 6; ++k) v[k] = load_pair<T, VEC>(sp[k], i0, i1);
        if constexpr (VEC) f = *reinterpret_cast<const unsigned short *>(g.flags + i0);
        else f = (uint32_t)g.flags[i0] | ((uint32_t)g.flags[i1] << 8);
    };

    // per c_x (kx = c_x + 1): P2 holds the c_y = +1 populations of row r - 1
    // (for row r); Q2, Q0 the sums of row r - 1 without its c_y = -1 part
    f2 P2[3], Q2[3], Q0[3];
    uint32_t fo = 0; // flags of row r - 1
    const f2 quarter = f2splat(0.25f);
    uint32_t idx = (uint32_t)yb * (uint32_t)g.nx + (uint32_t)x; // the lane's first cell of the row being finished
    uint32_t hash = idx * kGolden;
    const uint32_t hash_row = (uint32_t)g.nx * kGolden;

    // the end column's sums of the row being finished: what lane 31 passes round
    // to lane 0 (the left end's), and lane 0 to lane 31
    const char *end_at = reinterpret_cast<const char *>(&ends.y[0][lane == 31 ? 0 : 1][1]);
    // reconstruct row r from its moments (prefetched in v) and fetch row r + 2
    // (wb: mask words of its near-wall cells, wanted when row r + 1 has come)
    auto recon = [&](int r, P (&v)[6], uint32_t &f, uint32_t &fr, uint32_t (&wb)[2]) {
        f2 m[6], d;
        decode<T>(v, g.codec, m, d);
        fr = f;
        wb[0] = wb[1] = 0;
        if (r + 2 <= ye) load(r + 2, v, f);
        constexpr uint32_t kLook = (kTypeMask | kBitNearWall) * 0x0101u;
        if (__any_sync(full, (fr & kLook) != 0x0101u)) { // not plain Fluid cells away from walls
            const uint32_t at = (uint32_t)r * (uint32_t)g.nx + (uint32_t)x;
            if (out0 && r >= yb && r < ye && (fr & kBitNearWall)) wb[0] = g.wallmask[at];
            if (out1 && r >= yb && r < ye && (fr & (kBitNearWall << 8))) wb[1] = g.wallmask[at + 1];
            // bounce-back cells: a zero state has zero populations (F' = -1)
            const bool z0 = is_bounce_back<2>(fr & kTypeMask), z1 = is_bounce_back<2>((fr >> 8) & kTypeMask);
            if (__any_sync(full, z0 || z1)) {
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    float a, b;
                    f2split(m[k], a, b);
                    m[k] = f2make(z0 ? 0.0f : a, z1 ? 0.0f : b);
                }
                float a, b;
                f2split(d, a, b);
                d = f2make(z0 ? -1.0f : a, z1 ? -1.0f : b);
            }
        }
        return Rows<f2>(m, d);
    };
    // row r's own part of rows r and r + 1: c_y = 0 and c_y = +1
    auto feed = [&](const Rows<f2> &rows) {
        f2 F[3];
        rows.template row<1>(F);
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            Q0[k] = vfma(quarter, P2[k], clamp1(F[k]));
            Q2[k] = P2[k];
        }
        rows.template row<2>(F);
#pragma unroll
        for (int k = 0; k < 3; ++k) P2[k] = clamp1(F[k]);
    };

    auto step = [&](int r, P (&v)[6], uint32_t &f, const uint32_t (&wa)[2], uint32_t (&wb)[2]) {
        uint32_t fr;
        const Rows<f2> rows = recon(r, v, f, fr, wb);
        const int o = r - 1; // c_y = -1 completes row o
        f2 S[6];
        {
            f2 F[3];
            rows.template row<0>(F);
            f2 Y0[3], Y1[3], Y2[3];
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                const f2 C = clamp1(F[k]);
                Y2[k] = Q2[k] + C;
                Y1[k] = Q2[k] - C;
                Y0[k] = vfma(quarter, C, Q0[k]);
            }
            // column exchange: the c_x = +1 sums (kx = 2) come from the left
            // column, the c_x = -1 sums (kx = 0) from the right one; sum and
            // difference of the two, per column
            auto meet = [&](int k, f2 plus, f2 minus, f2 &sum, f2 &dif) {
                float pl, ph, ml, mh;
                f2split(plus, pl, ph);
                f2split(minus, ml, mh);
                // round the ends of the warp go the end columns' sums
                const float end = *reinterpret_cast<const float *>(end_at + k * (int)sizeof(ends.y[0]));
                ph = lane == 31 ? end : ph;
                ml = lane == 0 ? end : ml;
                const float left = __shfl_sync(full, ph, (lane + 31) & 31), right = __shfl_sync(full, ml, (lane + 1) & 31);
                sum = f2make(left + mh, pl + right);
                dif = f2make(left - mh, pl - right);
            };
            f2 s0, s1, s2, unused;
            meet(0, Y0[2], Y0[0], s0, S[1]);
            meet(1, Y1[2], Y1[0], s1, S[5]);
            meet(2, Y2[2], Y2[0], s2, unused);
            S[0] = vfma(quarter, s0, Y0[1]);
            S[2] = vfma(quarter, s1, Y1[1]);
            S[3] = s0;
            S[4] = vfma(quarter, s2, Y2[1]);
        }
        feed(rows);
        const bool fast = fo == fastflags && (wy || o != g.ny - 1);
        const bool special = __any_sync(full, out0 && !fast); // some cell of the row is not plain Fluid
        bool st0 = false, st1 = false; // columns stored one by one
        if (special && out0 && !fast) {
            auto plain = [&](bool out, uint32_t f8) { return out && is_updated(f8 & kTypeMask) && !(f8 & kBitLink); };
            st0 = plain(out0, fo & 0xffu);
            st1 = plain(out1, fo >> 8);
            if (st0 && (edge0 || (!wy && o == g.ny - 1))) { edges = true; st0 = false; }
            if (st1 && (edge1 || (!wy && o == g.ny - 1))) { edges = true; st1 = false; }
            if (st0 && (fo & kBitOutletSrc)) feeders0 |= 1u << (o - yb);
            if (st1 && (fo & (kBitOutletSrc << 8))) feeders1 |= 1u << (o - yb);
            const uint32_t walls = wall_bits_mask<2>();
            const uint32_t w0 = st0 ? wa[0] & walls : 0u, w1 = st1 ? wa[1] & walls : 0u;
            if (w0 | w1) {
                // reflected populations of the cell itself, from its stored moments
                P own[6];
                f2 mo[6], d;
                const uint32_t row = (uint32_t)o * (uint32_t)g.nx;
#pragma unroll
                for (int k = 0; k < 6; ++k) own[k] = load_pair<T, VEC>(sp[k], row + c0, row + c1);
                decode<T>(own, g.codec, mo, d);
                const Rows<f2> ro(mo, d);
                auto reflect = [&](auto ky_, const f2 *G) {
                    constexpr int ky = decltype(ky_)::value;
#pragma unroll
                    for (int kx = 0; kx < 3; ++kx) {
                        if (kx == 1 && ky == 1) continue;
                        const int i = dir_index<2>(2 - kx, 2 - ky, 1); // the direction whose inverse is (kx, ky)
                        const int cx = 1 - kx, cy = 1 - ky;
                        const float w = (cx != 0 && cy != 0) ? 0.0625f : 0.25f; // the weight over W0
                        float a, b;
                        f2split(f2splat(1.0f) + clamp1(G[kx]), a, b);
                        const f2 t = f2make(w0 >> i & 1u ? a : 0.0f, w1 >> i & 1u ? b : 0.0f);
                        const f2 t4 = f2splat(4.0f * w) * t, t16 = f2splat(16.0f * w) * t;
                        S[0] = vfma(f2splat(w), t, S[0]);
                        if (cx) S[1] = cx > 0 ? S[1] + t4 : S[1] - t4;
                        if (cy) S[2] = cy > 0 ? S[2] + t4 : S[2] - t4;
                        if (cx) S[3] = S[3] + t4;
                        if (cy) S[4] = S[4] + t4;
                        if (cx && cy) S[5] = cx * cy > 0 ? S[5] + t16 : S[5] - t16;
                    }
                };
                f2 G[3];
                ro.template row<0>(G);
                reflect(std::integral_constant<int, 0>(), G);
                ro.template row<1>(G);
                reflect(std::integral_constant<int, 1>(), G);
                ro.template row<2>(G);
                reflect(std::integral_constant<int, 2>(), G);
            }
        }
        f2 n[6], d;
        P e[6];
        constexpr bool enc = StorageTraits<T>::kEncoded;
        collide(S, g.omega, enc ? g.codec.su : 1.0f, enc ? g.codec.inv_su * g.codec.inv_su : 1.0f, n, d);
        encode<T>(n, d, hash, g.codec, e);
        // a density that is not positive, or a sum that is not finite (bad_state)
        float ra, rb, sa, sb;
        f2split(n[0], ra, rb);
        f2split((n[0] + n[1]) + n[2], sa, sb);
        const float inf = __int_as_float(0x7f800000);
        if (!(fminf(ra, rb) > 0.0f && fabsf(sa + sb) < inf)) {
            const bool b0 = !(ra > 0.0f) || !isfinite(sa), b1 = !(rb > 0.0f) || !isfinite(sb);
            if (b0 && ((out0 && fast) || st0)) bad |= 1u << (o - yb);
            if (b1 && ((out1 && fast) || st1)) bad |= 0x10000u << (o - yb);
        }
        if (VEC && fast) {
#pragma unroll
            for (int k = 0; k < 6; ++k) *reinterpret_cast<P *>(dp[k] + idx) = e[k];
        }
        if (!VEC || special) {
            constexpr int kBits = 8 * (int)sizeof(T);
            using U = typename std::conditional<sizeof(T) == 4, uint32_t, unsigned short>::type;
            if (!VEC && fast) st0 = st1 = true;
#pragma unroll
            for (int k = 0; k < 6; ++k) {
                U *d = reinterpret_cast<U *>(dp[k]);
                if (st0) d[idx] = (U)e[k];
                if (st1) d[idx + 1] = (U)(e[k] >> kBits);
            }
        }
        fo = fr;
        idx += (uint32_t)g.nx;
        hash += hash_row;
        end_at += sizeof(float);
    };

    load(yb - 1, raw[0], fl[0]);
    load(yb, raw[1], fl[1]);
    // the end columns, one row a lane (lanes 0..15 the left end's, 16..31 the
    // right one's): the sums of step(), in its order
    {
        const int side = lane >> 4, row = lane & 15;
        float f[3] = {0.0f, 0.0f, 0.0f};
        if (row < ye - yb + 2) {
            const uint32_t at = (uint32_t)halo_index(yb - 1 + row, g.ny, wy) * (uint32_t)g.nx +
                                (uint32_t)halo_index(side ? kWindow * (w + 1) : kWindow * w - 1, g.nx, wx);
            float m[6], d, F[3];
#pragma unroll
            for (int k = 0; k < 6; ++k) m[k] = from_storage<2, T>(k, sp[k][at]);
            const bool zero = is_bounce_back<2>(g.flags[at] & kTypeMask);
            decode_values<T>(g.codec, m, d);
            if (zero) {
                m[0] = m[1] = m[2] = 0.0f;
                d = -1.0f;
            }
            const Rows<float> rows(m, d);
            rows.template row<0>(F);
            f[0] = fmaxf(side ? F[0] : F[2], -1.0f);
            rows.template row<1>(F);
            f[1] = fmaxf(side ? F[0] : F[2], -1.0f);
            rows.template row<2>(F);
            f[2] = fmaxf(side ? F[0] : F[2], -1.0f);
        }
        const float A = __shfl_up_sync(full, f[2], 1), C = __shfl_down_sync(full, f[0], 1);
        ends.y[0][side][row] = fmaf(0.25f, C, fmaf(0.25f, A, f[1]));
        ends.y[1][side][row] = A - C;
        ends.y[2][side][row] = A + C;
    }
    __syncwarp();
    {
        // rows yb - 1 and yb finish nothing
        uint32_t fr;
        f2 F[3];
        const Rows<f2> before = recon(yb - 1, raw[0], fl[0], fr, wm[0]);
        before.template row<2>(F);
#pragma unroll
        for (int k = 0; k < 3; ++k) P2[k] = clamp1(F[k]);
        feed(recon(yb, raw[1], fl[1], fo, wm[1]));
    }
    for (int r = yb + 1; r <= ye; r += 2) {
        step(r, raw[0], fl[0], wm[1], wm[0]);
        if (r + 1 > ye) break;
        step(r + 1, raw[1], fl[1], wm[0], wm[1]);
    }
    if (gate.dry) bad = 0, edges = false;
    if (!g.feed) feeders0 = feeders1 = 0;
    if (__any_sync(full, edges || (bad | feeders0 | feeders1) != 0)) gate.wait(g.status);
    for (; bad; bad &= bad - 1) {
        const int r = __ffs(bad) - 1;
        if (!is_link(g, (uint32_t)(yb + (r & 15)) * (uint32_t)g.nx + (uint32_t)(x + (r >> 4)))) {
            atomicOr(g.status, kStatusNonFinite);
            break;
        }
    }
    if (__any_sync(full, (feeders0 | feeders1) != 0)) {
        __syncwarp(); // the feeders' new moments, stored by other lanes
        // Each call is two round trips to L2, so a warp makes as few as it can:
        // a pair of columns with several feeding rows (outlets at the left or
        // right, at a corner too) takes one, its rows dealt out to the lanes,
        // unless many columns are like that (a grid of a few rows).
        unsigned tall = __ballot_sync(full, ((feeders0 & (feeders0 - 1)) | (feeders1 & (feeders1 - 1))) != 0);
        if (__popc(tall) > 8) tall = 0;
        const bool mine = tall >> lane & 1u;
        for (; tall; tall &= tall - 1) {
            const int from = __ffs(tall) - 1;
            const uint32_t f0 = __shfl_sync(full, feeders0, from), f1 = __shfl_sync(full, feeders1, from);
            const int r = lane & 15;
            if ((lane < 16 ? f0 : f1) >> r & 1u)
                feed_outlet_of<T>(g, (uint32_t)(yb + r) * (uint32_t)g.nx + (uint32_t)(kWindow * w + 2 * from + (lane >> 4)));
        }
        if (!mine) {
            for (uint32_t f = feeders0; f; f &= f - 1)
                feed_outlet_of<T>(g, (uint32_t)(yb + __ffs(f) - 1) * (uint32_t)g.nx + (uint32_t)x);
            for (uint32_t f = feeders1; f; f &= f - 1)
                feed_outlet_of<T>(g, (uint32_t)(yb + __ffs(f) - 1) * (uint32_t)g.nx + (uint32_t)x + 1);
        }
    }
    if (edges) {
        for (int y = yb; y < ye; ++y) {
            const bool top = !wy && y == g.ny - 1;
            if (out0 && (edge0 || top)) edge_cell<T>(g, x, y);
            if (out1 && (edge1 || top)) edge_cell<T>(g, x + 1, y);
        }
    }
    __syncwarp(); // the next unit's ends
}

} // namespace march2
} // namespace fflbm
