// Moving-boundary links: detection, the sparse update of cells that own
// links, and the per-vertex force reduction.
#pragma once
#include "ffs_common.cuh"

namespace fflbm {

// Sparse link table, rebuilt every step.  A cell that owns at least one link
// gets one open-addressing slot: keys[slot] = cell + 1 and links[slot * Q + l]
// = the smallest (depth, element) key of direction l (~0 if none).  `list`
// holds the occupied slots in claim order, one list per segment of the table
// (segment = slot >> seg_shift, its list at the segment's own first slot, its
// length in count[kCountStride * segment]).  Claims in one counter serialise:
// they took about 1 ns each, most of detection's time in a serving pool
// (50,000 claims a substep at 256 episodes), so a table counts in kSegments of
// them, each in a line of its own.  The sparse kernel returns every slot it
// visits to the empty state, so the table is clean again at the end of the
// step without touching unused slots.
constexpr uint32_t kSegments = 64, kCountStride = 32;
constexpr uint32_t kOneCounterCap = 1u << 15; // 2D tables of at most this many slots keep one counter
constexpr size_t kCountWords = (size_t)kSegments * kCountStride;
struct LinkTable {
    uint32_t cap = 0;                  // power of two (0: not allocated)
    uint32_t seg_shift = 31;           // log2(cap / kSegments), or 31: one segment
    uint32_t *keys = nullptr;          // [cap]
    unsigned long long *links = nullptr; // [cap * Q]
    uint32_t *list = nullptr;          // [cap]
    uint32_t *count = nullptr;         // [kCountWords], or [1] for one segment
    long long *acc = nullptr;          // [acc_cap * DIM] fixed-point force sums (2^-32 units)
    uint32_t acc_cap = 0;              // vertices
    uint32_t *done = nullptr;          // [1] CTAs of link_cells_kernel that finished (zero between steps)
};
inline uint32_t segment_shift(uint32_t cap)
{
    uint32_t s = 0;
    while ((cap >> s) > kSegments) ++s;
    return s;
}

// Surfaces of at most this many force components have their fixed-point
// sums converted by the last CTA of link_cells_kernel instead of a kernel of
// their own: one launch less per step where launches dominate (the 2D
// configurations), one CTA's work where that is cheap.
constexpr long long kFoldForcesMax = 2048;

struct SurfaceArgs {
    const float *V;
    const float *U;
    const uint32_t *E;
    int nv, ne;
    float *forces;
    double *forces64;
    // coupled step: the surface is the boundary of a volume mesh; the step's
    // forces are written to vforces[map[i]] (nvol volume vertices) instead
    const uint32_t *map = nullptr;
    float *vforces = nullptr;
    int nvol = 0;
};

struct StepScalars {
    float cl;       // lattice spacing (physical)
    float ct;       // time step (physical)
    double cf;      // force scale rho_f dx^DIM dx / dt^2
};

// fixed-point scale of the per-vertex force sums
constexpr double kForceScale = 4294967296.0; // 2^32

// The D2Q9 dense pass (ffs_dense2d.cu).  With `detect`, the same launch does
// launch_detect_links's work in blocks of its own; only grids for which
// dense2d_detects() says so can.
struct DetectArgs {
    uint32_t *flag_words;
    LinkTable lt;
    SurfaceArgs s;
    StepScalars sc;
};
template <typename T> bool dense2d_detects(const GridArgs<T> &g);

// Lanes per segment in the 2D detection of one surface.  Where every segment
// can have a warp that is resident at once, 32: a warp's time is then its
// chain of table insertions, which four lanes per direction share (a step on
// 300 x 181 with 198 segments: 16.0 us in FP32, against 17.3 with 8 lanes; on
// 160 x 96 the same).  Otherwise 8, which take a quarter of the instructions.
inline int detect_lanes2(long long segments, int sms) { return segments <= 16ll * sms ? 32 : 8; }
template <typename T> cudaError_t launch_dense2d(const GridArgs<T> &g, cudaStream_t s, const DetectArgs *detect = nullptr);

template <int DIM, typename T>
cudaError_t launch_detect_links(const GridArgs<T> &g, uint32_t *flag_words, const LinkTable &lt, const SurfaceArgs &s,
                                const StepScalars &sc, cudaStream_t st);
// With fold_forces, the last CTA also does launch_finalize_forces's work
// (the caller launches no finalize kernel); lt.done must be allocated.
// chained: the stream's last operation is the launch of the dense pass with
// detection in it, which lets this kernel in early (launch_chained).
template <int DIM, typename T>
cudaError_t launch_link_cells(const GridArgs<T> &g, uint32_t *flag_words, const LinkTable &lt, const SurfaceArgs &s,
                              const StepScalars &sc, cudaStream_t st, bool fold_forces = false, bool chained = false);
template <int DIM>
cudaError_t launch_finalize_forces(const LinkTable &lt, const SurfaceArgs &s, double cf, cudaStream_t st);
template <int DIM>
cudaError_t launch_reset_links(const LinkTable &lt, uint32_t *flag_words, cudaStream_t st);
// first stage of the coupled step: gathers the surface from the volume
// arrays through the map and zeroes the volume forces
cudaError_t launch_gather_surface(int dim, const float *vpos, const float *vvel, const uint32_t *map, int nv, int nvol,
                                  float *spos, float *svel, float *vforces, uint32_t *status, cudaStream_t st);

template <int DIM>
cudaError_t launch_prepare_flags(uint8_t *flags, uint32_t *wallmask, uint2 *feeders, uint32_t *feeders_n, uint32_t feeders_cap,
                                 int nx, int ny, int nz, cudaStream_t st);
template <int DIM, typename T>
cudaError_t launch_initialize(const GridArgs<T> &g, T *other, const float *bcvel, cudaStream_t st);
cudaError_t launch_fill_solid2(uint8_t *flags, int nx, int ny, float cl, const SurfaceArgs &s, cudaStream_t st);
// bits: ny * nz * ceil(nx / 32) words, zero on entry and on return
cudaError_t launch_fill_solid3(uint8_t *flags, uint32_t *bits, int nx, int ny, int nz, float cl, const SurfaceArgs &s,
                               cudaStream_t st);

template <int DIM, typename T>
cudaError_t launch_convert_in(const float *in, bool aos, T *out, uint32_t ncell, Codec c, cudaStream_t st);
template <int DIM, typename T>
cudaError_t launch_convert_out(const T *in, float *out, bool aos, uint32_t ncell, Codec c, cudaStream_t st);

} // namespace fflbm
