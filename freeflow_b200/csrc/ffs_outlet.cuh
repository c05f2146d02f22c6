// Zero-gradient outlets, fused into the fluid update.
//
// The reference runs a separate full-grid kernel after the buffer swap
// (mrApplyOutlet2DKernel, FsiCoupling2D.cu:257-316; mrApplyOutlet3DKernel,
// FsiCoupling3D.cu:336-420): an outlet node q copies the normal velocity of its
// inner neighbour p = q - n (a Fluid node) when that velocity points outward,
// and sets pi_nn = u_n(p)^2, in place on the freshly written buffer.  Each
// outlet has exactly one feeder p, so the same writes are issued here once p's
// new moments are final, straight into the buffer being written.  No other node
// reads q's entries of that buffer during the step, so the result is the
// reference's.
#pragma once
#include <type_traits>

#include "ffs_common.cuh"

namespace fflbm {

struct OutletRule {
    uint8_t type;   // outlet flag of the node q fed by this cell
    int comp;       // normal velocity component in the moment vector
    int pcomp;      // pi_nn index
    int sign;       // +1: copy when u_n > 0, -1: copy when u_n < 0
};

// q = p + offset(rule) for the six / four outlet types
template <int DIM> __device__ __forceinline__ long long outlet_offset(int r, int nx, long long nxy)
{
    if (DIM == 2) {
        switch (r) {
        case 0: return nx;   // OutletUp   : p = q - nx
        case 1: return -nx;  // OutletDown : p = q + nx
        case 2: return -1;   // OutletLeft : p = q + 1
        default: return 1;   // OutletRight: p = q - 1
        }
    } else {
        switch (r) {
        case 0: return nxy;  // OutletUp   (z)
        case 1: return -nxy; // OutletDown
        case 2: return -1;   // OutletLeft
        case 3: return 1;    // OutletRight
        case 4: return -nx;  // OutletFront: p = q + nx
        default: return nx;  // OutletBack : p = q - nx
        }
    }
}

template <int DIM> __device__ __forceinline__ OutletRule outlet_rule(int r)
{
    if (DIM == 2) {
        switch (r) {
        case 0: return {kOutletUp, 2, 4, 1};
        case 1: return {kOutletDown, 2, 4, -1};
        case 2: return {kOutletLeft, 1, 3, -1};
        default: return {kOutletRight, 1, 3, 1};
        }
    } else {
        switch (r) {
        case 0: return {kOutletUp, 3, 6, 1};
        case 1: return {kOutletDown, 3, 6, -1};
        case 2: return {kOutletLeft, 1, 4, -1};
        case 3: return {kOutletRight, 1, 4, 1};
        case 4: return {kOutletFront, 2, 5, -1};
        default: return {kOutletBack, 2, 5, 1};
        }
    }
}

template <int DIM> constexpr int kNumOutletRules = DIM == 2 ? 4 : 6;

// Outlet rules a cell feeds, kept in the spare bits of its wall-mask word
// (bit i < Q of that word is the bounce-back mask of direction i; bit 0 is
// never a wall because direction 0 does not move):
//   D2Q9 : rules 0..3 at bits 16..19;  D3Q27: rules 0..4 at bits 27..31, rule 5 at bit 0.
template <int DIM> __host__ __device__ constexpr uint32_t outlet_bit(int r)
{
    return DIM == 2 ? (1u << (16 + r)) : (r < 5 ? (1u << (27 + r)) : 1u);
}
template <int DIM> __host__ __device__ constexpr uint32_t outlet_bits_mask()
{
    return DIM == 2 ? 0xF0000u : 0xF8000001u;
}
template <int DIM> __host__ __device__ constexpr uint32_t wall_bits_mask()
{
    return DIM == 2 ? 0x1FEu : 0x07FFFFFEu;
}

// Who feeds.  Every outlet node has one feeder and is fed once a step, with the
// feeder's final moments: a feed keeps part of what the node holds, so a feed
// with a value that is replaced later could not be undone.  The dense pass
// updates cells beside link detection, and a cell whose links it does not
// know yet is rewritten by the link-cell kernel.  So:
//   * a step without a surface: the dense pass feeds (GridArgs::feed);
//   * a link cell feeds its own outlets (link_cell_update*);
//   * the other feeders of a step with a surface are fed for by warps of the
//     link-cell kernel (feed_pass); detection marks the outlet nodes of link
//     cells for it, because their LINK bits go while it runs (mark_outlets);
//   * the serving pool's march waits for detection before it feeds
//     (march2::Gate).
//
// Marks the outlet nodes that cell p feeds; p has just been found to have links.
template <int DIM>
__device__ __noinline__ void mark_outlets(uint32_t *flag_words, const uint32_t *wallmask, int nx, long long nxy, uint32_t p)
{
    const uint32_t word = wallmask[p];
    for (int r = 0; r < kNumOutletRules<DIM>; ++r) {
        if (!(word & outlet_bit<DIM>(r))) continue;
        const uint32_t q = (uint32_t)((long long)p + outlet_offset<DIM>(r, nx, nxy));
        atomicOr(flag_words + (q >> 2), (uint32_t)kBitOutletSrc << (8 * (q & 3)));
    }
}

// Outlets fed by cell p (mask word `word`), whose new moments are in g.dst, in
// one body for all rules: this code is met cold, and a copy per rule took longer
// to fetch than to run.  Link cells are left out: by their LINK bit, or with
// flag_words (bits are on their way out) by the marks of their outlet nodes,
// which are taken off.
template <int DIM, typename T>
__device__ __forceinline__ void feed_cell(const GridArgs<T> &g, uint32_t p, uint32_t word, uint32_t *flag_words)
{
    constexpr int NM = Lattice<DIM>::NM;
    const long long nxy = (long long)g.nx * g.ny;
    word &= outlet_bits_mask<DIM>();
    if (!flag_words && (__ldcg(reinterpret_cast<const unsigned char *>(g.flags) + p) & kBitLink)) return;
#pragma unroll 1
    for (; word; word &= word - 1) {
        const int b = __ffs(word) - 1, r = DIM == 2 ? b - 16 : b ? b - 27 : 5; // outlet_bit
        const uint32_t q = (uint32_t)((long long)p + outlet_offset<DIM>(r, g.nx, nxy));
        // all loads before any is tested
        const uint32_t fq = flag_words ? g.flags[q] : 0u;
        const OutletRule rule = outlet_rule<DIM>(r);
        float up = StorageTraits<T>::from_vel(g.dst[(size_t)rule.comp * g.ncell + p]);
        if constexpr (StorageTraits<T>::kEncoded) up *= g.codec.inv_su;
        float mq[NM];
        if constexpr (StorageTraits<T>::kEncoded) load_moments<DIM, T>(mq, g.dst, g.ncell, q, g.codec);
        if (fq & kBitOutletSrc) {
            atomicAnd(flag_words + (q >> 2), ~((uint32_t)kBitOutletSrc << (8 * (q & 3))));
            continue;
        }
        const bool outward = (rule.sign > 0 && up > 0.0f) || (rule.sign < 0 && up < 0.0f);
        if constexpr (!StorageTraits<T>::kEncoded) {
            if (outward) g.dst[(size_t)rule.comp * g.ncell + q] = up;
            g.dst[(size_t)rule.pcomp * g.ncell + q] = up * up;
        } else {
#pragma unroll
            for (int k = 1; k <= 2 * DIM; ++k) {
                if (k == rule.comp && outward) mq[k] = up;
                if (k == rule.pcomp) mq[k] = up * up;
            }
            encode_store_strided<DIM, T>(mq, g.dst, q, g.ncell, g.codec);
        }
    }
}

// feed_pass for grids with more feeders than their list holds: the feeders are
// found in the flag bytes, by warps `warp` of `nwarps`.
template <int DIM, typename T>
__device__ __noinline__ void feed_scan(const GridArgs<T> &g, uint32_t *flag_words, uint32_t warp, uint32_t nwarps)
{
    constexpr uint32_t kFeeder = 0x01010101u * (kBitOutletSrc | kFluid), kSeen = 0x01010101u * (kBitOutletSrc | kTypeMask);
    const uint32_t *words = reinterpret_cast<const uint32_t *>(g.flags); // the bytes up to a whole word are there, zero
    const uint32_t n = (g.ncell + 3) / 4;
    for (uint32_t i = warp * 32 + (threadIdx.x & 31); i < n; i += nwarps * 32)
        for (uint32_t f = __vcmpeq4(words[i] & kSeen, kFeeder) & 0x01010101u; f; f &= f - 1) {
            const uint32_t p = 4 * i + (uint32_t)(__ffs(f) - 1) / 8;
            feed_cell<DIM, T>(g, p, g.wallmask[p], flag_words);
        }
}

// Feeds the outlets of the grid's n = *g.feeders_n feeders but the link cells,
// by warps `warp` of `nwarps`.  The list of feeders was made when the node types
// were set; finding them in the flag bytes took 1 us of a 17 us step on
// 800 x 300.
template <int DIM, typename T>
__device__ __noinline__ void feed_pass(const GridArgs<T> &g, uint32_t n, uint32_t *flag_words, uint32_t warp, uint32_t nwarps)
{
    if (n > g.feeders_cap) {
        feed_scan<DIM, T>(g, flag_words, warp, nwarps);
        return;
    }
    for (uint32_t i = warp * 32 + (threadIdx.x & 31); i < n; i += nwarps * 32) {
        const uint2 f = g.feeders[i];
        feed_cell<DIM, T>(g, f.x, f.y, flag_words);
    }
}

// Called by the thread that has just stored cell p's new moments into g.dst.
// `ms` are the stored values as they read back (after storage rounding) and
// `word` the cell's mask word, whose outlet bits name the outlet neighbours
// q = p + offset(rule) to update.  No flag or moment of p is re-read.
template <int DIM, typename T>
__device__ __forceinline__ void feed_outlets(const GridArgs<T> &g, uint32_t p, const float *ms, uint32_t word)
{
    constexpr int NM = Lattice<DIM>::NM;
    const long long nxy = (long long)g.nx * g.ny;
#pragma unroll
    for (int r = 0; r < kNumOutletRules<DIM>; ++r) {
        if (!(word & outlet_bit<DIM>(r))) continue;
        const uint32_t q = (uint32_t)((long long)p + outlet_offset<DIM>(r, g.nx, nxy));
        const OutletRule rule = outlet_rule<DIM>(r);
        float up = 0.0f;
#pragma unroll
        for (int k = 0; k < NM; ++k)
            if (k == rule.comp) up = ms[k];
        const bool outward = (rule.sign > 0 && up > 0.0f) || (rule.sign < 0 && up < 0.0f);
        if constexpr (!StorageTraits<T>::kEncoded) {
            if (outward) g.dst[(size_t)rule.comp * g.ncell + q] = up;
            g.dst[(size_t)rule.pcomp * g.ncell + q] = up * up;
        } else {
            float mq[NM];
            load_moments<DIM, T>(mq, g.dst, g.ncell, q, g.codec);
#pragma unroll
            for (int k = 0; k < NM; ++k) {
                if (k == rule.comp && outward) mq[k] = up;
                if (k == rule.pcomp) mq[k] = up * up;
            }
            encode_store_strided<DIM, T>(mq, g.dst, q, g.ncell, g.codec);
        }
    }
}

} // namespace fflbm
