// Links of D3Q27 grids (ffs_links_kernels.cuh).
#include "ffs_links_kernels.cuh"

namespace fflbm {

FFS_INST_LINKS(3)

} // namespace fflbm
