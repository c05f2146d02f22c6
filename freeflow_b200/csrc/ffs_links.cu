// Links of D2Q9 grids (ffs_links_kernels.cuh) and the coupled step's surface
// gather.  Compiled without implicit multiply-add contraction (build.py): a
// link cell takes 16 lanes here and 4 in the serving pool (ffs_batch2d.cu), and
// both must round alike.  The multiply-adds are explicit in the source.
#include "ffs_links_kernels.cuh"

namespace fflbm {

// First stage of the coupled step (updateSurfaceStatesFromVolume,
// src/fsi/FsiCouplingKernels.cu:14-57, plus the volume-force zeroing of the
// solid solver's applyForces, src/fem/VBDSolver.cpp:105,289).  Map entries
// out of range latch the element-index status bit and gather zeros.
template <int DIM>
__global__ void gather_surface_kernel(const float *vpos, const float *vvel, const uint32_t *map, int nv, int nvol,
                                      float *spos, float *svel, float *vforces, uint32_t *status)
{
    const long long ns = (long long)nv * DIM, nz = (long long)nvol * DIM;
    const long long n = ns > nz ? ns : nz;
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x) {
        if (t < nz) vforces[t] = 0.0f;
        if (t < ns) {
            const long long i = t / DIM;
            const uint32_t m = map[i];
            float p = 0.0f, u = 0.0f;
            if (m < (uint32_t)nvol) {
                p = vpos[(size_t)m * DIM + (t - i * DIM)];
                u = vvel[(size_t)m * DIM + (t - i * DIM)];
            } else {
                atomicOr(status, kStatusBadElement);
            }
            spos[t] = p;
            svel[t] = u;
        }
    }
}

cudaError_t launch_gather_surface(int dim, const float *vpos, const float *vvel, const uint32_t *map, int nv, int nvol,
                                  float *spos, float *svel, float *vforces, uint32_t *status, cudaStream_t st)
{
    const long long n = (long long)std::max(nv, nvol) * dim;
    if (n == 0) return cudaSuccess;
    const int grid = (int)std::max<long long>(1, std::min<long long>((n + 255) / 256, (long long)sm_count() * 8));
    if (dim == 2) gather_surface_kernel<2><<<grid, 256, 0, st>>>(vpos, vvel, map, nv, nvol, spos, svel, vforces, status);
    else gather_surface_kernel<3><<<grid, 256, 0, st>>>(vpos, vvel, map, nv, nvol, spos, svel, vforces, status);
    return cudaGetLastError();
}

FFS_INST_LINKS(2)

} // namespace fflbm
