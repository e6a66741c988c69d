// cs_tile.cuh -- host/device interface of the tile kernel (cs_tile.cu): 32 sources per thread block,
// one source per lane.
#pragma once
#include <cstddef>
#include <cstdint>
#include <cuda_runtime.h>

#include "cs_common.cuh"

namespace cs {
namespace tile {

constexpr int TPB = 512;        // threads per block
constexpr int NW = TPB / 32;    // warps per block
constexpr int BPSM = 2;         // resident blocks per SM
constexpr int PMAX = 8;         // out-edges per node (the graph's maximum out-degree)
constexpr int MMAX = 65536;     // nodes of one tile (dirty bits live in shared memory)
constexpr int SERVED_SLOT = 11; // header word: sources whose rows the tile kernel wrote itself

// Per-block scratch: offsets of its arrays, each indexed by the tile's node number.
struct Geometry {
    int32_t mcap;   // nodes per tile
    uint32_t tcap;  // dependency rows (32 lanes x 2 f64) per tile
    uint32_t icap;  // schedule items per tile
    uint32_t lcap;  // schedule levels per tile
    size_t o_rl, o_node, o_adj, o_link, o_dist, o_pm, o_masks, o_sig, o_items, o_lvl, o_dep, o_trip;
    size_t total;
};

struct Params {
    // graph (primal CSR, cs_primal_graph)
    int32_t n_bound;
    const int32_t *in_ptr, *in_nb;
    const float *in_w;
    const int32_t *out_ptr, *out_to;
    const float *out_w;
    const uint8_t *out_cnt;
    const float *node_w;
    // query
    int32_t k;
    float dk[MAXK];
    float beta[MAXK];
    float maxsec, speed, tol, delta;
    int32_t closeness, betweenness, track_reach;
    const int32_t *src_list;
    int64_t n_src;
    int32_t lanes;  // sources per tile, 1..32
    const float *src_wt;
    const uint8_t *eligible;
    const int32_t *od_ptr, *od_dst;
    const float *od_w;
    // outputs: rows [7][K][n_bound] (OD: [2][K][n_bound]), closeness bucket [3][K][n_bound]
    double *out, *bucket;
    uint32_t *reach;
    // workspace: the per-warp slots' clean dense arrays (block b uses slot b's) and their compact region
    WsHeader *hdr;
    int32_t *failed;  // item0 + the indices into src_list of the sources left to the per-warp kernel
    unsigned *n_failed;
    int32_t fail_cap;
    int64_t item0;
    char *dense;
    size_t dense_stride, aux_off;
    char *region;
    Geometry geo;
};

// The scratch layout for `region_bytes` per block (mcap 0: too small to be of use).
Geometry geometry(size_t region_bytes, int k, const float *dk, bool od);
// Launches `blocks` persistent blocks on `stream`; returns the launch error.
cudaError_t launch(const Params &p, bool od, int blocks, cudaStream_t stream);
// Launches `blocks` persistent blocks over a batch's shortest-path jobs [lo, hi), at most kmax thresholds
// each; p holds what the jobs share (scratch, header, lists).
cudaError_t launch_batch(const Params &p, const cs_batch_job *jobs_dev, int lo, int hi, int kmax, int blocks,
                         cudaStream_t stream);
// Tabulates the seed exponentials of this kernel (cs_seed.cuh) on `stream`.
cudaError_t launch_seed_table(cudaStream_t stream);

}  // namespace tile
}  // namespace cs
