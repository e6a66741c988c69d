// cs_primal_batch.cu -- the batched kernels (cs_primal.cuh).
#include "cs_primal.cuh"

namespace cs {

namespace {
template <int MODE>
void launch_items(const PrimalParams &p, int minb, int blocks, const cs_batch_job *jobs, int n_jobs, long long lo,
                  long long hi, cudaStream_t stream) {
    if (p.P > 8) batch_kernel<CS_MAX_DEGREE, 2, MODE><<<blocks, 256, 0, stream>>>(p, jobs, n_jobs, lo, hi);
    else if (minb == 4) batch_kernel<8, 4, MODE><<<blocks, 256, 0, stream>>>(p, jobs, n_jobs, lo, hi);
    else if (minb == 3) batch_kernel<8, 3, MODE><<<blocks, 256, 0, stream>>>(p, jobs, n_jobs, lo, hi);
    else batch_kernel<8, 2, MODE><<<blocks, 256, 0, stream>>>(p, jobs, n_jobs, lo, hi);
}

template <int MODE>
void launch_sync(const PrimalParams &p, int minb, int blocks, const cs_batch_job *jobs, int n_jobs, long long lo,
                 long long hi, cudaStream_t stream) {
    if (p.P <= 4 && minb == 4) batch_sync_kernel<4, 4, MODE><<<blocks, 256, 0, stream>>>(p, jobs, n_jobs, lo, hi);
    else if (p.P <= 4 && minb == 3) batch_sync_kernel<4, 3, MODE><<<blocks, 256, 0, stream>>>(p, jobs, n_jobs, lo, hi);
    else if (minb == 4) batch_sync_kernel<8, 4, MODE><<<blocks, 256, 0, stream>>>(p, jobs, n_jobs, lo, hi);
    else if (minb == 3) batch_sync_kernel<8, 3, MODE><<<blocks, 256, 0, stream>>>(p, jobs, n_jobs, lo, hi);
    else batch_sync_kernel<8, 2, MODE><<<blocks, 256, 0, stream>>>(p, jobs, n_jobs, lo, hi);
}
}  // namespace

void launch_batch_items(const PrimalParams &p, int mode, int minb, int blocks, bool sync, const cs_batch_job *jobs,
                        int n_jobs, long long lo, long long hi, cudaStream_t stream) {
    const bool lock = sync && p.P <= 8 && !p.rerun;
    if (mode == MODE_SHORTEST && lock) launch_sync<MODE_SHORTEST>(p, minb, blocks, jobs, n_jobs, lo, hi, stream);
    else if (mode == MODE_SEGMENT && lock) launch_sync<MODE_SEGMENT>(p, minb, blocks, jobs, n_jobs, lo, hi, stream);
    else if (mode == MODE_SHORTEST) launch_items<MODE_SHORTEST>(p, minb, blocks, jobs, n_jobs, lo, hi, stream);
    else if (mode == MODE_SEGMENT) launch_items<MODE_SEGMENT>(p, minb, blocks, jobs, n_jobs, lo, hi, stream);
    else launch_items<-1>(p, minb, blocks, jobs, n_jobs, lo, hi, stream);
}

void launch_seed_table_batch(cudaStream_t stream) {
    seed_table_kernel<<<(SEED_TAB + 255) / 256, 256, 0, stream>>>();
}

}  // namespace cs
