// Fused D3Q27 step for all cells without moving-boundary links.
//
// Reference: mrDeformableSolver3DKernel_ShrdM (src/core/FsiCoupling3D.cu:83-334)
// followed by mrApplyOutlet3DKernel (:336-420).
//
// B200 design.  The reference gives each 8x4x4 block a 10x6x6 halo and
// reconstructs all 27 populations of every halo cell (2.8x the interior),
// then pulls them back out of shared memory.  Here a CTA owns a 32 x 8 column
// of cells and marches up z through a chunk of planes:
//
//   * each plane is reconstructed once for its 34 x 10 xy halo: eight tile
//     warps reconstruct the tile's own cells; of the 84 cells around it only
//     the 9 populations that point into the tile are evaluated, in FP32 by two
//     ring warps while the tile warps still pull the plane before, in 16-bit
//     storage by the first 84 tile threads (kRingWarps);
//   * the populations of plane p go to one of two shared-memory buffers
//     (2 x 27 x 340 floats) and are consumed as soon as they exist: the
//     c_z = -1 slice completes the raw moments of the cell below (plane p-1),
//     the c_z = 0 slice feeds plane p, the c_z = +1 slice starts plane p+1.
//     Each thread keeps the partial raw moments of its column's next two
//     cells in registers, so there is one barrier per plane;
//   * bounce-back: a halo cell of a bounce-back type (wall, solid) gets zeros
//     in its 27 population slots instead of a reconstruction, so whatever a
//     fluid neighbour pulls from it adds nothing; each fluid cell next to a
//     wall then adds its own reflected populations max(0, f_inv(i)^rec(x))
//     once, while its own plane is in shared memory.  The result is the
//     reference's f_i(x) = max(0, f_inv(i)^rec(x)) for wall neighbours x - c_i
//     (FsiCoupling3D.cu:209-222), whose wall test looks at the wrapped index.
//     The halo index is the reference's too (halo_index: it wraps at the low
//     face and clamps at the high face of a non-periodic axis), so the halo
//     cell and the tested cell coincide everywhere except across a high face:
//     halo cells beyond a high face are always reconstructed, walls included
//     (the reference pulls them when the wrapped test says fluid), and a cell
//     whose wrapped neighbour across the face is a wall removes that pulled
//     value explicitly (wall_fix_part);
//   * moments are SoA planes in HBM (128 B coalesced per warp and moment);
//     moments, flag bytes and wall masks are prefetched a plane ahead;
//     outlets are fed by their inner neighbour in the same pass, and cells with
//     moving-boundary links are left to the sparse link kernel (ffs_links_kernels.cuh).
#include "ffs_dense2d.cuh"
#include "ffs_dense3d.cuh"

#include <algorithm>
#include <cstdlib>
#include <map>
#include <mutex>
#include <utility>

namespace fflbm {

namespace {
constexpr int kTX = D3::kTX, kTY = D3::kTY, kHX = D3::kHX, kHalo = D3::kHalo;
constexpr int kPlane = D3::kPlaneFloats;

// raw-moment slot: {rho, jx, jy, jz, Pxx, Pyy, Pzz, Pxy, Pyz, Pxz}
//
// Unweighted populations.  The kernel stores each population
// as its Hermite sum F_i without the lattice weight and applies the weights
// on the way into the raw moments.  The D3Q27 weights are one constant times
// powers of four, w_i = W0 4^-n(i) with W0 = wgt3(1,1,1) = 8/27 and n(i) the
// number of non-zero components of c_i (8/27, 2/27, 1/54, 1/216 exactly, as
// float constants too), and max(0, w F) = w max(0, F), so every weighted sum
// follows from the unweighted one by exact power-of-two scalings.  The kernel
// accumulates R''_k = R_k / (W0 s_k) with
//   s = {1/4, 1/16, 1/16, 1/4, 1/16, 1/16, 1/4, 1/64, 1/16, 1/16},
// chosen so that the c_z = +-1 slices add their sums as they are and the
// c_z = 0 slice adds 4 Y; a completed cell's sums are multiplied by W0 s_k.
// This replaces the 27 weight multiplications of every reconstruction (own
// cell and ring) by 10 per updated cell.  (W0 s_k are exact products.)
constexpr float kW0 = wgt3(1, 1, 1);
__device__ __forceinline__ void raw_from_scaled(const float *Rs, float *R)
{
    constexpr float s[10] = {0.25f, 0.0625f, 0.0625f, 0.25f, 0.0625f, 0.0625f, 0.25f, 0.015625f, 0.0625f, 0.0625f};
#pragma unroll
    for (int k = 0; k < 10; ++k) R[k] = Rs[k] * (kW0 * s[k]);
}

// The x/y sums of one c_z slice are
// Y = {Y00, Y01, Y02, Y10, Y11, Y20}; the weighted sums are
// W0 4^-|c_z| c_k Y_k with c = {1, 1/4, 1/4, 1/4, 1/16, 1/4}.
//
// add the slice with c_z = CZ to the scaled sums R''
template <int CZ> __device__ __forceinline__ void slice_add(float *R, const float *Y)
{
    if (CZ == 0) {
        R[0] = fmaf(4.0f, Y[0], R[0]); R[2] = fmaf(4.0f, Y[1], R[2]); R[5] = fmaf(4.0f, Y[2], R[5]);
        R[1] = fmaf(4.0f, Y[3], R[1]); R[7] = fmaf(4.0f, Y[4], R[7]); R[4] = fmaf(4.0f, Y[5], R[4]);
    } else {
        R[0] += Y[0]; R[2] += Y[1]; R[5] += Y[2]; R[1] += Y[3]; R[7] += Y[4]; R[4] += Y[5];
        R[3] += CZ * Y[0]; R[6] += Y[0]; R[8] += CZ * Y[1]; R[9] += CZ * Y[3];
    }
}
__device__ __forceinline__ void slice_init_plus(float *R, const float *Y)
{
    R[0] = Y[0]; R[2] = Y[1]; R[5] = Y[2]; R[1] = Y[3]; R[7] = Y[4]; R[4] = Y[5];
    R[3] = Y[0]; R[6] = Y[0]; R[8] = Y[1]; R[9] = Y[3];
}

// Paired layout.  For each (c_x, c_y) set and halo cell,
// the c_z = -1 and +1 populations sit side by side as one float2 (a plane of
// 9 x kHalo float2), and the c_z = 0 population in a plane of floats after
// it: the cells of a tile pull the three from the same neighbour, so one
// 64-bit and one 32-bit load replace three, the reconstruction stores them
// the same way, and the c_z = -1 / +1 pair is one 64-bit register pair for
// the packed f32x2 arithmetic below.  (One float plane per population took
// 7 % more time on 384 x 192 x 192.)
constexpr int kPairFloats = 9 * kHalo * 2;  // the float2 plane; the c_z = 0 plane follows
// float index of population (kx, ky, kz) (k = c + 1) of halo cell c
__device__ __forceinline__ int pop_index(int kx, int ky, int kz, int c)
{
    const int s9 = (kx + 3 * ky) * kHalo + c;
    return kz == 1 ? kPairFloats + s9 : 2 * s9 + (kz == 2);
}
__device__ __forceinline__ void store_pair(float *buf, int s9, f2 p, float mid)
{
    *reinterpret_cast<unsigned long long *>(buf + 2 * s9) = p.v;
    buf[kPairFloats + s9] = mid;
}
__device__ __forceinline__ void load_pair(const float *buf, int s9, float &lo, float &hi, float &mid)
{
    const float2 v = *reinterpret_cast<const float2 *>(buf + 2 * s9);
    lo = v.x;
    hi = v.y;
    mid = buf[kPairFloats + s9];
}

// slice_sums of the c_z = -1 and +1 slices (as the lo and hi halves of Sp)
// and of the c_z = 0 slice (Sm), from the paired layout
__device__ __forceinline__ void slice_sums_paired(const float *buf, int c_own, f2 *Sp, float *Sm)
{
    const f2 quarter = f2splat(0.25f);
    f2 X0p[3], X1p[3], X2p[3];
    float X0m[3], X1m[3], X2m[3];
#pragma unroll
    for (int ky = 0; ky < 3; ++ky) {
        const int crow = c_own - (ky - 1) * kHX;
        float4 a, b, d;   // x, y: c_z = -1, +1; z: c_z = 0
        load_pair(buf, (3 * ky) * kHalo + crow + 1, a.x, a.y, a.z);
        load_pair(buf, (1 + 3 * ky) * kHalo + crow, b.x, b.y, b.z);
        load_pair(buf, (2 + 3 * ky) * kHalo + crow - 1, d.x, d.y, d.z);
        const f2 fm = f2make(fmaxf(a.x, 0.0f), fmaxf(a.y, 0.0f));
        const f2 f0 = f2make(fmaxf(b.x, 0.0f), fmaxf(b.y, 0.0f));
        const f2 fp = f2make(fmaxf(d.x, 0.0f), fmaxf(d.y, 0.0f));
        const f2 sp = fp + fm;
        X1p[ky] = fp - fm;
        X0p[ky] = vfma(quarter, sp, f0);
        X2p[ky] = sp;
        const float gm = fmaxf(a.z, 0.0f), g0 = fmaxf(b.z, 0.0f), gp = fmaxf(d.z, 0.0f);
        const float sm = gp + gm;
        X1m[ky] = gp - gm;
        X0m[ky] = fmaf(0.25f, sm, g0);
        X2m[ky] = sm;
    }
    const f2 s0 = X0p[2] + X0p[0];
    Sp[0] = vfma(quarter, s0, X0p[1]);
    Sp[1] = X0p[2] - X0p[0];
    Sp[2] = s0;
    Sp[3] = vfma(quarter, X1p[2] + X1p[0], X1p[1]);
    Sp[4] = X1p[2] - X1p[0];
    Sp[5] = vfma(quarter, X2p[2] + X2p[0], X2p[1]);
    const float t0 = X0m[2] + X0m[0];
    Sm[0] = fmaf(0.25f, t0, X0m[1]);
    Sm[1] = X0m[2] - X0m[0];
    Sm[2] = t0;
    Sm[3] = fmaf(0.25f, X1m[2] + X1m[0], X1m[1]);
    Sm[4] = X1m[2] - X1m[0];
    Sm[5] = fmaf(0.25f, X2m[2] + X2m[0], X2m[1]);
}

// The z level of the expansion (the Hermite sums over c_z of the
// six coefficient groups), with the c_z = -1 / +1 entries as pairs (p) and
// the c_z = 0 entry apart (m): herm3v gives ((a0 + a2) - a1, fma(-1/2, a2,
// a0), (a0 + a2) + a1), herm2v (a0 - a1, a0, a0 + a1).
struct ZLevel {
    f2 p00, p10, p01, p20, p02, p11;
    float m00, m10, m01, m20, m02, m11;
    __device__ __forceinline__ explicit ZLevel(const Coef3V<float> &c)
    {
        auto h3 = [](float a0, float a1, float a2, f2 &p, float &m) {
            const float t = a0 + a2;
            p = f2make(t - a1, t + a1);
            m = fmaf(-0.5f, a2, a0);
        };
        auto h2 = [](float a0, float a1, f2 &p, float &m) {
            p = f2make(a0 - a1, a0 + a1);
            m = a0;
        };
        h3(c.rho, c.m1z, c.m2zz, p00, m00);
        h3(c.m1x, c.m2xz, c.qxzz, p10, m10);
        h3(c.m1y, c.m2yz, c.qyzz, p01, m01);
        h2(c.m2xx, c.qxxz, p20, m20);
        h2(c.m2yy, c.qyyz, p02, m02);
        h2(c.m2xy, c.qxyz, p11, m11);
    }
};

// All 27 unweighted populations of one cell into the paired layout: the y and
// x levels of the expansion, paired over c_z = -1 / +1.
__device__ __forceinline__ void store_populations_paired(const Coef3V<float> &c, float *buf, int cell)
{
    const ZLevel z(c);
    f2 C0p[3], C1p[3], C2p[3];
    float C0m[3], C1m[3], C2m[3];
    herm3v(z.p00, z.p01, z.p02, C0p);
    herm3v(z.p10, z.p11, f2splat(c.qxyy), C1p);
    herm2v(z.p20, f2splat(c.qxxy), C2p);
    herm3v(z.m00, z.m01, z.m02, C0m);
    herm3v(z.m10, z.m11, c.qxyy, C1m);
    herm2v(z.m20, c.qxxy, C2m);
#pragma unroll
    for (int ky = 0; ky < 3; ++ky) {
        f2 Fp[3];
        float Fm[3];
        herm3v(C0p[ky], C1p[ky], C2p[ky], Fp);
        herm3v(C0m[ky], C1m[ky], C2m[ky], Fm);
#pragma unroll
        for (int kx = 0; kx < 3; ++kx) store_pair(buf, (kx + 3 * ky) * kHalo + cell, Fp[kx], Fm[kx]);
    }
}

// The 9 populations with c_y = KY - 1 of a halo row cell
// into the paired layout.
template <int KY> __device__ __forceinline__ void store_row_paired(const Coef3V<float> &c, float *buf, int cell)
{
    const ZLevel z(c);
    auto h3p = [](f2 a0, f2 a1, f2 a2) {
        if constexpr (KY == 1) return vfma(f2splat(-0.5f), a2, a0);
        else if constexpr (KY == 0) return (a0 + a2) - a1;
        else return (a0 + a2) + a1;
    };
    auto h2p = [](f2 a0, f2 a1) {
        if constexpr (KY == 1) return a0;
        else if constexpr (KY == 0) return a0 - a1;
        else return a0 + a1;
    };
    auto h3m = [](float a0, float a1, float a2) {
        if constexpr (KY == 1) return fmaf(-0.5f, a2, a0);
        else if constexpr (KY == 0) return (a0 + a2) - a1;
        else return (a0 + a2) + a1;
    };
    auto h2m = [](float a0, float a1) {
        if constexpr (KY == 1) return a0;
        else if constexpr (KY == 0) return a0 - a1;
        else return a0 + a1;
    };
    f2 Fp[3];
    float Fm[3];
    herm3v(h3p(z.p00, z.p01, z.p02), h3p(z.p10, z.p11, f2splat(c.qxyy)), h2p(z.p20, f2splat(c.qxxy)), Fp);
    herm3v(h3m(z.m00, z.m01, z.m02), h3m(z.m10, z.m11, c.qxyy), h2m(z.m20, c.qxxy), Fm);
#pragma unroll
    for (int kx = 0; kx < 3; ++kx) store_pair(buf, (kx + 3 * KY) * kHalo + cell, Fp[kx], Fm[kx]);
}

// The 9 populations with c_x = sx of a halo column cell
// into the paired layout; kx = sx + 1.
__device__ __forceinline__ void store_col_paired(const Coef3V<float> &c, float sx, int kx, float *buf, int cell)
{
    const ZLevel z(c);
    f2 C0p[3], C1p[3], C2p[3];
    float C0m[3], C1m[3], C2m[3];
    herm3v(z.p00, z.p01, z.p02, C0p);
    herm3v(z.p10, z.p11, f2splat(c.qxyy), C1p);
    herm2v(z.p20, f2splat(c.qxxy), C2p);
    herm3v(z.m00, z.m01, z.m02, C0m);
    herm3v(z.m10, z.m11, c.qxyy, C1m);
    herm2v(z.m20, c.qxxy, C2m);
    const f2 sxp = f2splat(sx);
#pragma unroll
    for (int ky = 0; ky < 3; ++ky)
        store_pair(buf, (kx + 3 * ky) * kHalo + cell, vfma(sxp, C1p[ky], C0p[ky] + C2p[ky]),
                   fmaf(sx, C1m[ky], C0m[ky] + C2m[ky]));
}

// R'' += (basis(c) w F) / (W0 s) for one unweighted population F of
// direction c: the weight and the scales are powers of two
__device__ __forceinline__ void add_basis_scaled(float *R, int cx, int cy, int cz, float F)
{
    const int n = (cx != 0) + (cy != 0) + (cz != 0);
    const float t = F * (n == 0 ? 1.0f : n == 1 ? 0.25f : n == 2 ? 0.0625f : 0.015625f);
    const float fx = (float)cx, fy = (float)cy, fz = (float)cz;
    R[0] = fmaf(4.0f, t, R[0]);
    R[1] = fmaf(16.0f * fx, t, R[1]); R[2] = fmaf(16.0f * fy, t, R[2]); R[3] = fmaf(4.0f * fz, t, R[3]);
    R[4] = fmaf(16.0f * fx * fx, t, R[4]); R[5] = fmaf(16.0f * fy * fy, t, R[5]); R[6] = fmaf(4.0f * fz * fz, t, R[6]);
    R[7] = fmaf(64.0f * fx * fy, t, R[7]); R[8] = fmaf(16.0f * fy * fz, t, R[8]); R[9] = fmaf(16.0f * fx * fz, t, R[9]);
}

// Bounce-back corrections that the current plane (buf, plane p) allows:
//   cell p-1 (Rp, mask wp): remove the pulled c_z = -1 populations of wall
//                           directions (they came from plane p);
//   cell p   (Rc, mask wc): remove the pulled c_z = 0 ones, add the cell's own
//                           reflected populations f_inv(i)(x) (its plane is p);
//   cell p+1 (Rn, mask wn): remove the pulled c_z = +1 ones.
// Reference rule: FsiCoupling3D.cu:209-222, f_i(x) = max(0, f_inv(i)^rec(x)).
// Only the set bits are visited (a wall face sets nine of them).
// R'' += basis(c_i) w_i max(0, F_inv(i)(x)) (scaled as above) for every wall
// direction i in w, with the cell's own unweighted populations read from the
// current plane.
__device__ __forceinline__ void add_reflected(const float *buf, int c_own, uint32_t w, float (&R)[10])
{
#pragma unroll
    for (int kz = 0; kz < 3; ++kz)
#pragma unroll
        for (int ky = 0; ky < 3; ++ky)
#pragma unroll
            for (int kx = 0; kx < 3; ++kx) {
                const int i = dir_index<3>(kx, ky, kz);
                if (i == 0) continue;
                float f = fmaxf(buf[pop_index(2 - kx, 2 - ky, 2 - kz, c_own)], 0.0f);
                f = (w & (1u << i)) ? f : 0.0f;
                add_basis_scaled(R, kx - 1, ky - 1, kz - 1, f);
            }
}

// Removes from R'' the pulled populations of the wall directions in w whose
// c_z slice is kz_sel (their source is the current plane): across a high
// face the halo cell holds real populations, but the wrapped test found a
// wall, so the step takes the cell's reflected population instead
// (add_reflected).
__device__ __forceinline__ void wall_fix_part(const float *buf, int c_own, uint32_t w, int kz_sel, float (&R)[10])
{
    while (w) {
        const int i = __ffs(w) - 1;
        w &= w - 1;
        int cx, cy, cz;
        dir_vec<3>(i, cx, cy, cz);
        if (cz + 1 == kz_sel) {
            const float pulled = fmaxf(buf[pop_index(cx + 1, cy + 1, cz + 1, c_own - cx - cy * kHX)], 0.0f);
            add_basis_scaled(R, cx, cy, cz, -pulled);
        }
    }
}

// The planes of the ten moments, src + k ncell and dst + k ncell, as kernel
// parameters: they sit in the constant bank, so a moment access of the 32-bit
// index path forms its address from the cell index in one multiply-add
// instead of adding k ncell first.
template <typename T> struct MomentPlanes {
    const T *src[10];
    T *dst[10];
};

} // namespace

// Whether the 84 halo cells around the tile have two warps of their own.  They
// write plane p's halo populations while the tile warps still pull plane p - 1
// from the other buffer, so the ring (a third of a cell's reconstruction per
// tile cell) is off the tile's path between two barriers, and only they hold
// and load ring moments; with the ring on three of the tile's own warps the
// others wait for those at every barrier.  In FP32 that takes 128^3 from 78 to
// 69 us and 384 x 192 x 192 from 0.53 to 0.50 ms a step.  In 16-bit storage a
// cell's decoding makes the ring warp with two rows the slowest of the CTA: no
// gain on 384 x 192 x 192 and 96 against 86 us on 189 x 93 x 101 (with three
// ring warps only 80 registers are left a thread, and the pass spills), so
// there the first 84 tile threads take a ring cell each.
template <typename T> constexpr bool kRingWarps = !StorageTraits<T>::kEncoded;
template <typename T> constexpr int kThreads3 = D3::kTile + (kRingWarps<T> ? 64 : 0);

// The one barrier of a plane.  Tile and ring warps meet at it from different
// places of the source, which __syncthreads() does not allow for; every warp
// passes it ze - zb + 2 times.
template <typename T> __device__ __forceinline__ void plane_barrier()
{
    asm volatile("barrier.cta.sync.aligned 1, %0;" ::"n"(kThreads3<T>) : "memory");
}

// One CTA: 8 warps own the 32 x 8 tile's columns, and the ring warps, where
// there are any, the 84 halo cells around it.
// IDX32: every moment, flag and mask index (k * ncell + cell) fits in 32
// bits, as it does for grids of up to 429 M cells; each access then takes one
// 32-bit index and one widening multiply-add instead of 64-bit arithmetic.
// FEED: the pass feeds outlets itself (GridArgs::feed).
template <typename T, bool IDX32, bool FEED>
__global__ void __launch_bounds__(kThreads3<T>, 2) dense3d_kernel(GridArgs<T> g, const MomentPlanes<T> mp, int zchunk)
{
    extern __shared__ __align__(128) float smem[];
    const int tid = threadIdx.x;
    const int x0 = blockIdx.x * kTX, y0 = blockIdx.y * kTY;
    const int zb = blockIdx.z * zchunk;
    const int ze = min(zb + zchunk, g.nz);
    const long long nxy = (long long)g.nx * g.ny;
    const bool wx = g.periodic & 1, wy = g.periodic & 2, wz = g.periodic & 4;
    auto planar = [&](int c) {
        int hx = c % kHX, hy = c / kHX;
        return (uint32_t)(halo_index(y0 + hy - 1, g.ny, wy) * g.nx + halo_index(x0 + hx - 1, g.nx, wx));
    };
    // halo cells beyond a high face keep their real populations even when
    // they are walls (x and y per thread, z per plane)
    auto beyond_hi = [&](int c) {
        const int hx = x0 + c % kHX - 1, hy = y0 + c / kHX - 1;
        return (!wx && hx >= g.nx) || (!wy && hy >= g.ny);
    };
    // stored moments and node type of one halo cell in plane z
    auto load_cell = [&](int z, uint32_t off, T (&m)[10], uint32_t &h) {
        if constexpr (IDX32) {
            const uint32_t i = (uint32_t)halo_index(z, g.nz, wz) * (uint32_t)nxy + off;
#pragma unroll
            for (int k = 0; k < 10; ++k) m[k] = mp.src[k][i];
            h = g.flags[i] & kTypeMask;
        } else {
            const size_t i = (size_t)halo_index(z, g.nz, wz) * nxy + off;
#pragma unroll
            for (int k = 0; k < 10; ++k) m[k] = g.src[(size_t)k * g.ncell + i];
            h = g.flags[i] & kTypeMask;
        }
    };
    auto coefficients = [&](const T *raw) {
        float m[10];
#pragma unroll
        for (int k = 0; k < 10; ++k) m[k] = from_storage<3, T>(k, raw[k]);
        decode_moments<3, T>(m, g.codec);
        Coef3V<float> cf;
        cf.make(m);
        return cf;
    };

    if (kRingWarps<T> && tid >= D3::kTile) {
        // ---- ring warps.  A ring cell feeds the tile only the 9 populations
        // that point into it: the first warp evaluates c_y = +1 of the row
        // below and c_y = -1 of the row above, the second c_x = +-1 of the
        // columns (10 cells each).  No other slot of a ring cell is ever read.
        const int lane = tid & 31;
        auto zero_slot = [&](uint32_t h, bool hi, int p) { return is_bounce_back<3>(h) && !(hi || (!wz && p >= g.nz)); };
        const f2 z2 = f2make(0.0f, 0.0f);
        if (tid < D3::kTile + 32) {
            const int cb = lane + 1, ca = kHalo - kHX + lane + 1;
            const uint32_t ob = planar(cb), oa = planar(ca);
            const bool hib = beyond_hi(cb), hia = beyond_hi(ca);
            T rb[10], ra[10];
            uint32_t hb = 0, ha = 0;
            load_cell(zb - 1, ob, rb, hb);
            load_cell(zb - 1, oa, ra, ha);
            for (int p = zb - 1; p <= ze; ++p) {
                float *buf = smem + (p & 1) * kPlane;
                if (zero_slot(hb, hib, p)) {
#pragma unroll
                    for (int k = 0; k < 3; ++k) store_pair(buf, (k + 6) * kHalo + cb, z2, 0.0f);
                } else {
                    store_row_paired<2>(coefficients(rb), buf, cb);
                }
                if (p < ze) load_cell(p + 1, ob, rb, hb);
                if (zero_slot(ha, hia, p)) {
#pragma unroll
                    for (int k = 0; k < 3; ++k) store_pair(buf, k * kHalo + ca, z2, 0.0f);
                } else {
                    store_row_paired<0>(coefficients(ra), buf, ca);
                }
                if (p < ze) load_cell(p + 1, oa, ra, ha);
                plane_barrier<T>(); // plane p is in buf; the tile has left the other buffer
            }
        } else {
            const bool has = lane < 2 * D3::kHY, left = lane < D3::kHY;
            const int c = left ? lane * kHX : ((has ? lane : 2 * D3::kHY - 1) - D3::kHY) * kHX + kHX - 1;
            const uint32_t off = planar(c);
            const bool hi = beyond_hi(c);
            const float sx = left ? 1.0f : -1.0f; // c_x of the fed populations
            const int kx = left ? 2 : 0;          // and its index
            T raw[10];
            uint32_t h = 0;
            load_cell(zb - 1, off, raw, h);
            for (int p = zb - 1; p <= ze; ++p) {
                float *buf = smem + (p & 1) * kPlane;
                if (has) {
                    if (zero_slot(h, hi, p)) {
#pragma unroll
                        for (int k = 0; k < 3; ++k) store_pair(buf, (kx + 3 * k) * kHalo + c, z2, 0.0f);
                    } else {
                        store_col_paired(coefficients(raw), sx, kx, buf, c);
                    }
                }
                if (p < ze) load_cell(p + 1, off, raw, h);
                plane_barrier<T>();
            }
        }
        return;
    }

    // ---- tile warps
    const int tx = tid % kTX, ty = tid / kTX;
    const int x = x0 + tx, y = y0 + ty;
    const bool inside = x < g.nx && y < g.ny;
    const int c_own = (ty + 1) * kHX + (tx + 1);
    const uint32_t off_own = planar(c_own);
    const bool own_hi = beyond_hi(c_own);
    const uint32_t col = inside ? (uint32_t)(y * g.nx + x) : 0u;
    // directions whose pull crosses the high x or y face of a non-periodic
    // axis (only there can the halo cell and the wrapped test differ)
    uint32_t oor_xy = 0;
    if (inside && ((!wx && x == g.nx - 1) || (!wy && y == g.ny - 1))) {
#pragma unroll
        for (int i = 1; i < 27; ++i) {
            int cx, cy, cz;
            dir_vec<3>(i, cx, cy, cz);
            if ((!wx && x - cx >= g.nx) || (!wy && y - cy >= g.ny)) oor_xy |= 1u << i;
        }
    }
    uint32_t oor_zhi = 0; // directions pulling across z = nz-1 from above
    if (!wz) {
#pragma unroll
        for (int i = 1; i < 27; ++i) {
            int cx, cy, cz;
            dir_vec<3>(i, cx, cy, cz);
            if (cz == -1) oor_zhi |= 1u << i;
        }
    }
    // the column's halo cell of the next plane, converted when it is reconstructed
    T raw[10];
    uint32_t h = 0;
    // without ring warps: the thread's ring cell (the row below: warp 0, the
    // row above: warp 1, the columns: warp 2, so each warp runs one path)
    const bool has_ring = !kRingWarps<T> && tid < D3::kRing;
    const bool left = tid < 64 + D3::kHY;
    int c_ring = c_own;
    if (has_ring)
        c_ring = tid < 32   ? tid + 1
                 : tid < 64 ? kHalo - kHX + tid - 31
                 : left     ? (tid - 64) * kHX
                            : (tid - 64 - D3::kHY) * kHX + kHX - 1;
    const uint32_t off_ring = kRingWarps<T> ? 0u : planar(c_ring);
    const bool ring_hi = !kRingWarps<T> && beyond_hi(c_ring);
    T rawr[10];
    uint32_t hr = 0;
    auto load_own = [&](int z) {
        if constexpr (kRingWarps<T>) {
            load_cell(z, off_own, raw, h);
        } else {
            // the ring loads are predicated one by one, which overlaps them with
            // the own-cell loads: a branch around them measured 9 % slower on
            // 384 x 192 x 192
            const size_t zo = IDX32 ? (size_t)0 : (size_t)halo_index(z, g.nz, wz) * nxy;
            const uint32_t z32 = IDX32 ? (uint32_t)halo_index(z, g.nz, wz) * (uint32_t)nxy : 0u;
            const uint32_t io = z32 + off_own, ir = z32 + off_ring;
#pragma unroll
            for (int k = 0; k < 10; ++k) {
                const T *plane = IDX32 ? mp.src[k] : g.src + (size_t)k * g.ncell + zo;
                raw[k] = plane[io];
                if (has_ring) rawr[k] = plane[ir];
            }
            h = g.flags[zo + io] & kTypeMask;
            if (has_ring) hr = g.flags[zo + ir] & kTypeMask;
        }
    };
    auto store_ring = [&](float *buf, int p) {
        const int kx = left ? 2 : 0;
        const f2 z2 = f2make(0.0f, 0.0f);
        if (is_bounce_back<3>(hr) && !(ring_hi || (!wz && p >= g.nz))) {
#pragma unroll
            for (int k = 0; k < 3; ++k)
                store_pair(buf, (tid < 32 ? k + 6 : tid < 64 ? k : kx + 3 * k) * kHalo + c_ring, z2, 0.0f);
            return;
        }
        const Coef3V<float> cf = coefficients(rawr);
        if (tid < 32) store_row_paired<2>(cf, buf, c_ring);
        else if (tid < 64) store_row_paired<0>(cf, buf, c_ring);
        else store_col_paired(cf, left ? 1.0f : -1.0f, kx, buf, c_ring);
    };
    // index of the column's cell in plane z (32 or 64-bit, as above)
    auto cell_at = [&](int z) {
        if constexpr (IDX32) return (size_t)((uint32_t)z * (uint32_t)nxy + col);
        else return (size_t)z * nxy + col;
    };
    auto flag_at = [&](int z) -> uint32_t {
        return (inside && z >= zb && z < ze) ? (uint32_t)g.flags[cell_at(z)] : 0u;
    };

    // Two register sets hold the partial raw moments of the column's cells at
    // z = p-1 and z = p; their roles swap every plane (loop unrolled by two).
    float X[10], Y[10];
#pragma unroll
    for (int k = 0; k < 10; ++k) X[k] = Y[k] = 0.0f;
    // flag bytes of z = p-1, p, p+1 and wall masks of z = p-1, p
    uint32_t fp = 0, fc = 0, fn = flag_at(zb);
    uint32_t wp = 0, wc = 0;

    // one plane: Rp = sums of z = p-1 (completed here), Rc = sums of z = p,
    // Rn receives the new c_z = +1 slice (the cell at z = p+1)
    auto plane = [&](int p, float (&Rp)[10], float (&Rc)[10]) {
        float *buf = smem + (p & 1) * kPlane;
        // bounce-back cells get zero slots unless they lie beyond a high face
        if (is_bounce_back<3>(h) && !(own_hi || (!wz && p >= g.nz))) {
#pragma unroll
            for (int j = 0; j < 9; ++j) store_pair(buf, j * kHalo + c_own, f2make(0.0f, 0.0f), 0.0f);
        } else {
            store_populations_paired(coefficients(raw), buf, c_own);
        }
        if constexpr (!kRingWarps<T>) {
            if (has_ring) store_ring(buf, p);
        }
        if (p < ze) load_own(p + 1);
        const uint32_t fnn = flag_at(p + 2);
        // mask word (wall and outlet bits) of the cell at z = p+1; only cells
        // this pass updates use it (walls, inlets and outlets carry mask bits
        // of their own neighbours that must not trigger any work)
        const bool upd_n = is_updated(fn & kTypeMask) && !(fn & kBitLink);
        const uint32_t wn = (upd_n && (fn & (kBitNearWall | kBitOutletSrc))) ? g.wallmask[cell_at(p + 1)] : 0u;
        plane_barrier<T>();
        if (inside) {
            constexpr uint32_t kWall = wall_bits_mask<3>();
            // the cell at z = p - 1 is complete: collide, store, feed outlets
            auto finish = [&](const float (&R)[10]) {
                const int d = p - 1;
                if (d >= zb && is_updated(fp & kTypeMask) && !(fp & kBitLink)) {
                    const uint32_t idx = (uint32_t)(d * nxy + col);
                    float m[10];
                    collide3(R, g.omega, m);
                    if constexpr (IDX32) encode_store<3, T>(m, mp.dst, idx, g.codec);
                    else encode_store_strided<3, T>(m, g.dst, (size_t)idx, g.ncell, g.codec);
                    if (bad_state<3>(m)) atomicOr(g.status, kStatusNonFinite);
                    if (FEED && (fp & kBitOutletSrc)) {
                        float ms[10];
                        stored_values<3, T>(m, ms, idx, g.codec);
                        feed_outlets<3, T>(g, idx, ms, wp);
                    }
                }
            };
            // wall directions across a high face (their halo cell held real
            // populations): remove the pulled value, per destination cell
            // z = p-1 (c_z = -1 slice) and z = p (c_z = 0)
            const uint32_t oor_p = oor_xy | ((p - 1 == g.nz - 1) ? oor_zhi : 0u);
            f2 Sp[6];
            float Sm[6], lo[6], hi[6];
            slice_sums_paired(buf, c_own, Sp, Sm);
#pragma unroll
            for (int k = 0; k < 6; ++k) f2split(Sp[k], lo[k], hi[k]);
            slice_add<-1>(Rp, lo);
            slice_add<0>(Rc, Sm);
            if ((wc | wp) & kWall) { // near-wall cells only: one test on the common path
                if (wc & kWall) add_reflected(buf, c_own, wc & kWall, Rc);
                if (wp & kWall & oor_p) wall_fix_part(buf, c_own, wp & kWall & oor_p, 0, Rp);
                if (wc & kWall & oor_xy) wall_fix_part(buf, c_own, wc & kWall & oor_xy, 1, Rc);
            }
            float R[10];
            raw_from_scaled(Rp, R);
            // Rp is free: it becomes the cell at z = p + 1
            slice_init_plus(Rp, hi);
            if (wn & kWall & oor_xy) wall_fix_part(buf, c_own, wn & kWall & oor_xy, 2, Rp);
            finish(R);
        }
        fp = fc; fc = fn; fn = fnn;
        wp = wc; wc = wn;
    };

    load_own(zb - 1);
    int p = zb - 1;
    for (; p + 1 <= ze; p += 2) {
        plane(p, X, Y);     // completes X (z = p-1); X := z = p+1
        plane(p + 1, Y, X); // completes Y (z = p);   Y := z = p+2
    }
    if (p <= ze) plane(p, X, Y);
}

// CTAs of `kernel` resident on the current device at once (SMs x occupancy),
// with the kernel's dynamic shared-memory limit raised to `smem` first.
// Cached per (kernel, device ordinal): a process may step grids on several
// GPUs, and the first launch on each device configures the kernel there.
static cudaError_t resident_slots(const void *kernel, int threads, size_t smem, int &slots)
{
    static std::mutex mu;
    static std::map<std::pair<const void *, int>, int> cache;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    std::lock_guard<std::mutex> lock(mu);
    auto it = cache.find({kernel, dev});
    if (it != cache.end()) {
        slots = it->second;
        return cudaSuccess;
    }
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    int per_sm = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem);
    if (e != cudaSuccess) return e;
    slots = device_sms() * (per_sm > 0 ? per_sm : 1);
    cache[{kernel, dev}] = slots;
    return cudaSuccess;
}

// Number of z chunks that best fills the GPU: whole waves of CTAs, with the
// two extra planes each chunk reconstructs counted as overhead.
static int choose_zchunks(int tiles, int nz, int slots)
{
    // CTAs next to walls and outlets carry extra work; several waves of CTAs
    // let the scheduler even that out, so aim for three waves or more while
    // chunks keep at least 16 planes
    int nmin = 1;
    while ((long long)tiles * nmin < 3LL * slots && nz / (nmin + 1) >= 16) ++nmin;
    int best = nmin;
    double best_eff = 0.0;
    for (int n = nmin; n <= nmin + 8 && n <= nz; ++n) {
        int chunk = (nz + n - 1) / n;
        long long ctas = (long long)tiles * ((nz + chunk - 1) / chunk);
        long long waves = (ctas + slots - 1) / slots;
        double eff = (double)ctas / (double)(waves * slots) * (double)chunk / (double)(chunk + 2);
        if (eff > best_eff + 1e-9) { best_eff = eff; best = n; }
    }
    return best;
}

template <typename T, bool IDX32, bool FEED> static cudaError_t launch_as(const GridArgs<T> &g, cudaStream_t s)
{
    int slots = 0;
    const cudaError_t e =
        resident_slots(reinterpret_cast<const void *>(dense3d_kernel<T, IDX32, FEED>), kThreads3<T>, D3::kSmemBytes, slots);
    if (e != cudaSuccess) return e;
    int tx = (g.nx + kTX - 1) / kTX, ty = (g.ny + kTY - 1) / kTY;
    int nchunk = choose_zchunks(tx * ty, g.nz, slots);
    int zchunk = (g.nz + nchunk - 1) / nchunk;
    // FFS_DENSE3D_PLANES pins the planes per chunk (tests run several cuts)
    if (const char *planes = std::getenv("FFS_DENSE3D_PLANES")) zchunk = std::max(1, std::min(g.nz, std::atoi(planes)));
    dim3 grid(tx, ty, (g.nz + zchunk - 1) / zchunk);
    MomentPlanes<T> mp;
    for (int k = 0; k < 10; ++k) {
        mp.src[k] = g.src + (size_t)k * g.ncell;
        mp.dst[k] = g.dst + (size_t)k * g.ncell;
    }
    dense3d_kernel<T, IDX32, FEED><<<grid, kThreads3<T>, D3::kSmemBytes, s>>>(g, mp, zchunk);
    return cudaGetLastError();
}

// 32-bit indices whenever every moment index of the grid fits (FFS_DENSE3D_INDEX64
// forces 64-bit indices, so that tests reach that path on small grids)
template <typename T> cudaError_t launch_dense3d(const GridArgs<T> &g, cudaStream_t s)
{
    const char *force64 = std::getenv("FFS_DENSE3D_INDEX64");
    if (10ull * g.ncell <= 0xFFFFFFFFull && !(force64 && force64[0] == '1'))
        return g.feed ? launch_as<T, true, true>(g, s) : launch_as<T, true, false>(g, s);
    return g.feed ? launch_as<T, false, true>(g, s) : launch_as<T, false, false>(g, s);
}

template cudaError_t launch_dense3d<float>(const GridArgs<float> &, cudaStream_t);
template cudaError_t launch_dense3d<__half>(const GridArgs<__half> &, cudaStream_t);
template cudaError_t launch_dense3d<__nv_bfloat16>(const GridArgs<__nv_bfloat16> &, cudaStream_t);

} // namespace fflbm
