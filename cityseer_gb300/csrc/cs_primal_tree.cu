// cs_primal_tree.cu -- the tree (isochrone) and accessibility kernels (cs_primal.cuh).
#include "cs_primal.cuh"

namespace cs {

void launch_tree(const PrimalParams &p, int P, int minb, int blocks, cudaStream_t stream) {
    launch_per_warp<MODE_TREE>(p, P, minb, blocks, stream);
}

void launch_access(const PrimalParams &p, int P, int minb, int blocks, cudaStream_t stream) {
    launch_per_warp<MODE_ACCESS>(p, P, minb, blocks, stream);
}

}  // namespace cs
