// cs_primal_shortest.cu -- the shortest-path and origin-destination kernels (cs_primal.cuh).
#include "cs_primal.cuh"

namespace cs {

cudaError_t occupancy_primal(int P, int minb, int *blocks_per_sm) {
    if (P > 8)
        return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, primal_kernel<CS_MAX_DEGREE, 2, 0>, 256, 0);
    if (minb == 4) return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, primal_kernel<8, 4, 0>, 256, 0);
    if (minb == 3) return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, primal_kernel<8, 3, 0>, 256, 0);
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, primal_kernel<8, 2, 0>, 256, 0);
}

void launch_shortest(const PrimalParams &p, int P, int minb, int blocks, bool sync, cudaStream_t stream) {
    if (P > 8 || !sync) {
        launch_per_warp<MODE_SHORTEST>(p, P, minb, blocks, stream);
        return;
    }
    // whole 8-warp blocks in lockstep: on the 202,500-node lattice 12- and 24-warp blocks ran no
    // faster and 4-warp groups (named barriers) 3% slower
    if (P <= 4 && minb == 4) primal_sync_kernel<4, 4, 8, 8><<<blocks, 256, 0, stream>>>(p);
    else if (P <= 4 && minb == 3) primal_sync_kernel<4, 3, 8, 8><<<blocks, 256, 0, stream>>>(p);
    else if (minb == 4) primal_sync_kernel<8, 4, 8, 8><<<blocks, 256, 0, stream>>>(p);
    else if (minb == 3) primal_sync_kernel<8, 3, 8, 8><<<blocks, 256, 0, stream>>>(p);
    else primal_sync_kernel<8, 2, 8, 8><<<blocks, 256, 0, stream>>>(p);
}

void launch_od(const PrimalParams &p, int P, int minb, int blocks, cudaStream_t stream) {
    launch_per_warp<MODE_OD>(p, P, minb, blocks, stream);
}

void launch_seed_table_shortest(cudaStream_t stream) {
    seed_table_kernel<<<(SEED_TAB + 255) / 256, 256, 0, stream>>>();
}

}  // namespace cs
