// cs_primal_segment.cu -- the segment kernels (cs_primal.cuh).
#include "cs_primal.cuh"

namespace cs {

void launch_segment(const PrimalParams &p, int P, int minb, int blocks, bool sync, cudaStream_t stream) {
    if (P > 8 || !sync) launch_per_warp<MODE_SEGMENT>(p, P, minb, blocks, stream);
    else if (P <= 4 && minb == 4) segment_sync_kernel<4, 4><<<blocks, 256, 0, stream>>>(p);
    else if (P <= 4 && minb == 3) segment_sync_kernel<4, 3><<<blocks, 256, 0, stream>>>(p);
    else if (minb == 4) segment_sync_kernel<8, 4><<<blocks, 256, 0, stream>>>(p);
    else if (minb == 3) segment_sync_kernel<8, 3><<<blocks, 256, 0, stream>>>(p);
    else segment_sync_kernel<8, 2><<<blocks, 256, 0, stream>>>(p);
}

}  // namespace cs
