// cs_primal.cu -- host side of the primal kernels (cs_primal.cuh): planning, workspaces, the C-ABI entry
// points for shortest paths, trips, segments, trees, accessibility and batches, and the small kernels
// around them.
#include <cstdio>
#include <cstring>
#include <string>
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <vector>

#include "cs_common.cuh"
#include "cs_cta.cuh"
#include "cs_primal.cuh"
#include "cs_tile.cuh"

namespace cs {

// Completes the bucketed closeness rows: out[m][k] += sum_{j<=k} bucket[m][j] for density,
// farness and harmonic (rows 0, 1, 3).
__global__ void bucket_prefix_kernel(const double *bucket, double *out, int K, int N) {
    const size_t KN = (size_t)K * N;
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < N; t += gridDim.x * blockDim.x) {
        const int rows[3] = {0, 1, 3};
        for (int m = 0; m < 3; m++) {
            double acc = 0.0;
            for (int k = 0; k < K; k++) {
                acc += bucket[(size_t)m * KN + (size_t)k * N + t];
                out[(size_t)rows[m] * KN + (size_t)k * N + t] += acc;
            }
        }
    }
}

// Batched form: the same prefix for every shortest-path job with closeness (blockIdx.y strides the
// jobs), and the bucket is zeroed as it is read, so that buckets are zero between runs.
__global__ void batch_prefix_kernel(const cs_batch_job *jobs, int n_jobs) {
    for (int j = blockIdx.y; j < n_jobs; j += gridDim.y) {
        const cs_batch_job &jb = jobs[j];
        if ((jb.mode != MODE_SHORTEST && jb.mode != MODE_BOTH) || !jb.compute_closeness || jb.n_sources <= 0)
            continue;
        const int K = jb.k, N = jb.g.n_bound;
        const size_t KN = (size_t)K * N;
        double *bucket = jb.bucket_dev;
        double *out = jb.out_dev;
        for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < N; t += gridDim.x * blockDim.x) {
            const int rows[3] = {0, 1, 3};
            for (int m = 0; m < 3; m++) {
                double acc = 0.0;
                for (int k = 0; k < K; k++) {
                    const size_t o = (size_t)m * KN + (size_t)k * N + t;
                    acc += bucket[o];
                    bucket[o] = 0.0;
                    out[(size_t)rows[m] * KN + (size_t)k * N + t] += acc;
                }
            }
        }
    }
}

// Source-indexed plan on the device (prepare_source_sampling with source_indices): src_wt = node
// weight and eligible = 1 at each listed source, 0 elsewhere.  Pass 0 clears, pass 1 scatters.
__global__ void source_weights_kernel(const int32_t *sources, long long n, const float *node_w, int n_bound,
                                      float *src_wt, uint8_t *eligible, int pass) {
    const long long stride = (long long)gridDim.x * blockDim.x;
    long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (pass == 0) {
        for (; t < n_bound; t += stride) {
            src_wt[t] = 0.0f;
            eligible[t] = 0u;
        }
    } else {
        for (; t < n; t += stride) {
            const int s = sources[t];
            if (s < 0 || s >= n_bound) continue;
            src_wt[s] = node_w[s];
            eligible[s] = 1u;
        }
    }
}

__global__ void fill_dense_kernel(char *dense, size_t dense_stride, int n_bound, const int32_t *slots, int n_list,
                                  int all_slots) {
    // Resets dist (=inf) and aux (=0) of the listed slots (or of slots [0, all_slots)).
    const int n_sl = slots ? n_list : all_slots;
    const size_t per = (size_t)n_bound;
    const size_t total = per * (size_t)n_sl;
    for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < total; t += (size_t)gridDim.x * blockDim.x) {
        const int si = (int)(t / per);
        const size_t j = t % per;
        const int slot = slots ? slots[si] : si;
        char *d = dense + dense_stride * (size_t)slot;
        ((float *)d)[j] = __int_as_float(INF_BITS);
        ((uint32_t *)(d + al256(per * 4)))[j] = 0u;
    }
}

}  // namespace cs


// ==========================================================================================
// Host side (C-ABI).
// ==========================================================================================
namespace cs_host {
thread_local std::string g_last_error;
thread_local long long g_counters[4] = {0, 0, 0, 0};
thread_local long long g_phase[16] = {};
}

extern "C" void cs_set_error_internal(const char *msg) { cs_host::g_last_error = msg ? msg : ""; }

namespace cs_host {
thread_local long long g_retries[2] = {0, 0};
}
extern "C" void cs_set_retries_internal(long long overflowed, long long inexact) {
    cs_host::g_retries[0] = overflowed;
    cs_host::g_retries[1] = inexact;
}
// Phase cycle sums and diagnostics of the last call (the header's pad[0..15]); the dual host code
// sets them too.
extern "C" void cs_set_phase_internal(const unsigned long long *pad) {
    for (int i = 0; i < 16; i++) cs_host::g_phase[i] = (long long)pad[i];
}
// Device counters of the last call (sources done, edges relaxed, states settled, launches).
extern "C" void cs_set_counters_internal(long long sources, long long relaxed, long long settled, long long launches) {
    cs_host::g_counters[0] = sources;
    cs_host::g_counters[1] = relaxed;
    cs_host::g_counters[2] = settled;
    cs_host::g_counters[3] = launches;
}
extern "C" cs_status cs_last_retries(int64_t *overflowed, int64_t *inexact) {
    if (overflowed) *overflowed = cs_host::g_retries[0];
    if (inexact) *inexact = cs_host::g_retries[1];
    return CS_OK;
}

namespace {
using cs_host::g_counters;
using cs_host::g_phase;

cs_status fail(cs_status code, const std::string &msg) {
    cs_host::g_last_error = msg;
    return code;
}
cs_status cuda_fail(cudaError_t e, const char *what) {
    return fail(CS_ERR_CUDA, std::string(what) + ": " + cudaGetErrorString(e));
}

int sm_count() {
    int dev = 0, n = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 0;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 0;
    return n;
}

struct Layout {
    size_t hdr_off, failed_off, failed2_off, bucket_off, dense_off, compact_off, compact_total, cta_off, total;
    size_t dense_stride;
    int fail_cap;
};

// sources that overflow their slot are listed for the in-call retry; beyond this many the call
// reports CS_ERR_CAPACITY (plan a larger cap)
int fail_capacity(int n_slots) { return std::max(n_slots, 1 << 18); }

// cta_blocks: blocks of the block-per-source kernel whose global scratch follows the per-warp regions.
Layout layout(int n_bound, int n_slots, int cap, int P, int L, int cta_blocks = 0) {
    Layout l;
    l.hdr_off = 0;
    l.failed_off = 256;
    l.fail_cap = fail_capacity(n_slots);
    l.failed2_off = cs::al256(l.failed_off + sizeof(int32_t) * (size_t)l.fail_cap);
    l.bucket_off = cs::al256(l.failed2_off + sizeof(int32_t) * (size_t)l.fail_cap);
    l.dense_off = cs::al256(l.bucket_off + sizeof(double) * 3 * (size_t)L * (size_t)n_bound);
    l.dense_stride = cs::al256((size_t)n_bound * 4) * 2;
    l.compact_off = l.dense_off + l.dense_stride * (size_t)n_slots;
    l.compact_total = cs::compact_bytes((size_t)cap, P, L) * (size_t)n_slots;
    // the in-call retry runs at cap = n_bound on the same compact region: keep room for one slot
    l.compact_total = std::max(l.compact_total, cs::compact_bytes((size_t)n_bound, P, L));
    l.cta_off = cs::al256(l.compact_off + l.compact_total);
    l.total = l.cta_off + cs::cta::scratch_bytes() * (size_t)std::max(0, cta_blocks);
    return l;
}

// Items that overflowed their slot's capacity run again at 4x the capacity (then 4x again, up to
// cap = full_n, where nothing can overflow), each level on as many slots as the compact region
// holds at that capacity; overflows of one level are listed for the next.  `run` launches one
// level: run(params, slots).  first_cap: the first level's capacity where the listed items have not run
// at the plan's.  Leaves the last header in h.
template <typename Launch>
cs_status retry_chain(const cs::PrimalParams &p, const cs_plan *plan, const Layout &lay, char *base, int full_n, int P,
                      cs::WsHeader &h, cudaStream_t stream, bool poll, Launch run, int first_cap = 0) {
    int32_t *listA = (int32_t *)(base + lay.failed_off);
    int32_t *listB = (int32_t *)(base + lay.failed2_off);
    const int32_t *list = listA;
    unsigned n_in = h.n_failed;
    int cap_l = first_cap > 0 ? std::min(full_n, first_cap)
                              : (int)std::min<long long>(full_n, 4ll * std::max(plan->cap, 8));
    while (n_in > 0u) {
        if (n_in > (unsigned)lay.fail_cap) return fail(CS_ERR_CAPACITY, "more overflowed sources than the list holds");
        int32_t *out_l = (list == listA) ? listB : listA;
        cs::PrimalParams p2 = p;
        p2.cap = cap_l;
        p2.rerun = 1;
        p2.remap = list;
        p2.n_src = (int64_t)n_in;
        p2.failed = out_l;
        cudaError_t e = cudaMemsetAsync(&p.hdr->work_next2, 0, sizeof(unsigned long long), stream);
        if (e == cudaSuccess) e = cudaMemsetAsync(&p.hdr->n_failed, 0, sizeof(unsigned), stream);
        if (e != cudaSuccess) return cuda_fail(e, "retry counter reset");
        const size_t per = cs::compact_bytes((size_t)cap_l, P, plan->lanes);
        int slots2 = (int)std::min<size_t>(lay.compact_total / per, (size_t)plan->n_slots);
        slots2 = std::max(1, std::min<int>(slots2, (int)n_in));
        cs_status st = run(p2, slots2);
        if (st != CS_OK) return st;
        e = cs::read_header(p.hdr, h, stream, poll);
        if (e != cudaSuccess) return cuda_fail(e, "retry kernel");
        if (h.err != 0u)
            return fail((cs_status)h.err, "device-side check failed in retry (code " + std::to_string(h.err) + ")");
        if (cap_l >= full_n && h.n_failed > 0u) return fail(CS_ERR_INTERNAL, "overflow at full capacity");
        n_in = h.n_failed;
        list = out_l;
        cap_l = (int)std::min<long long>(full_n, 4ll * cap_l);
    }
    return CS_OK;
}

int lanes_for(int mode, int k) {
    return (mode == cs::MODE_SHORTEST || mode == cs::MODE_BOTH || mode == cs::MODE_OD) ? 2 * k
                                                                                      : (mode == cs::MODE_SEGMENT ? k : 1);
}

cs_status validate_primal(const cs_primal_graph *g) {
    if (!g) return fail(CS_ERR_ARG, "graph is NULL");
    if (g->n_bound <= 0) return fail(CS_ERR_ARG, "NetworkStructure contains no nodes.");
    if (g->max_out_degree > CS_MAX_DEGREE)
        return fail(CS_ERR_ARG, "node out-degree " + std::to_string(g->max_out_degree) + " exceeds CS_MAX_DEGREE");
    return CS_OK;
}

// Register budget of the P <= 8 kernels: 4 resident 256-thread blocks per SM (64 registers), 3
// (80 registers) or 2 (128 registers).  A plan's variant field (2-4) or the environment variable
// CS_MIN_BLOCKS_PER_SM selects one for every launch.  Otherwise (variant 0) plans are sized for 4
// blocks, the most slots, and each launch picks by mode: 3 for shortest-path and OD centrality (on the
// 202,500-node lattice 4 blocks ran 395 ms per pass against 372 ms with 3, the spills of the
// dependency pass outweighing the extra warps), 4 for segments, trees and accessibility (segment
// centrality on the 250x250 curved lattice: 2.67M sources/s against 2.49M with 3).
int requested_variant(const cs_plan *plan) {
    const int v = plan ? plan->variant & 0xff : 0;
    if (v >= 2 && v <= 4) return v;
    const char *e = getenv("CS_MIN_BLOCKS_PER_SM");
    return (e && e[0] >= '2' && e[0] <= '4') ? e[0] - '0' : 0;
}
// the budget a plan's slot count is sized for
int resolve_variant(const cs_plan *plan) {
    const int v = requested_variant(plan);
    return v ? v : 4;
}
// the budget one launch of a mode runs with
int launch_variant(const cs_plan *plan, int mode) {
    const int v = requested_variant(plan);
    if (v) return v;
    return (mode == cs::MODE_SHORTEST || mode == cs::MODE_OD) ? 3 : 4;
}

// Block-synchronous phases for the shortest-path mode (CS_PHASE_SYNC=0 selects the per-warp form).
bool phase_sync() {
    const char *e = getenv("CS_PHASE_SYNC");
    return !(e && e[0] == '0');
}

// Block-per-source kernel for shortest-path and OD calls; CS_BLOCK_PER_SOURCE=0 in the environment
// leaves every source to the per-warp kernel (plans then hold no scratch for it).
bool block_kernel_enabled() {
    const char *e = getenv("CS_BLOCK_PER_SOURCE");
    return !(e && e[0] == '0');
}

// Schedule of one call: one block per source gives a source a whole SM (the lowest latency per
// source) and one warp per source keeps ~24 sources per SM in flight (the highest throughput).  Blocks
// take the sources in waves of one per SM; a warp's time for one source hides all of them, and grows
// faster with the reach than a block's.  So blocks pay for as many waves as the hops to the cutoff
// (seconds / median edge seconds, half a plan's band width) over 13, between 1 and 4 (a fifth wave at
// 5 km was 8% faster on one lattice, less than whole calls vary).
// Measured, blocks against warps (152 SMs, ms per call):
//    6 hops   152 sources 0.433 / 0.461, 304 0.496 / 0.462     25 hops  304 1.020 / 1.087, 456 1.246 / 1.070
//   12 hops   152 sources 0.510 / 0.592, 304 0.601 / 0.585     32 hops  304 1.129 / 1.445, 456 1.527 / 1.435
//   16 hops   152 sources 0.442 / 0.559, 608 0.924 / 0.569     40 hops  456 1.947 / 2.185, 608 2.410 / 2.309
//   62 hops   152 sources 1.442 / 4.643, 608 4.071 / 5.288, 700 4.874 / 5.315, 800 5.584 / 5.381
// CS_BLOCK_SOURCES_MAX sets the most sources of a call for blocks; CS_BLOCK_PER_SOURCE=1 forces them.
bool block_schedule(long long n_src, float maxsec, float delta) {
    const char *e = getenv("CS_BLOCK_PER_SOURCE");
    if (e && e[0] == '0') return false;
    if (e && e[0] == '1') return true;
    const char *m = getenv("CS_BLOCK_SOURCES_MAX");
    if (m) return n_src <= atoll(m);
    const double waves = delta > 0.0f ? std::min(4.0, std::max(1.0, 2.0 * maxsec / delta / 13.0)) : 4.0;
    return (double)n_src <= waves * std::max(1, sm_count());
}

// Tile kernel (cs_tile.cu): 32 nearby sources per block, one per lane.  A tile does its sources' common
// work once, over the union of their reaches, so it pays where the reach is much wider than the tile and
// there is a tile for every resident block:
//  - the caller vouches for the sources' order (CS_PLAN_NEAR_SOURCES, CS_BATCH_NEAR_SOURCES);
//  - 32 sources for each of the 2 blocks per SM (9,728 on 152 SMs), and CS_TILE_SOURCES_MIN;
//  - the reach's radius, in hops (seconds / median edge seconds, half a plan's band width; at most half
//    the side of a square of all nodes), over the tile's, sqrt(16 N / sources) hops, is at least
//    (4 + 1.5 rows) (1 + 0.3 blocks / tiles), with rows = the sum over thresholds of (d / d_max)^2, the
//    dependency rows that a node of the union needs; three quarters of that beyond 4 out-edges, where the
//    per-warp kernel loses more to absent edges than the tiles.
// Measured, tiles against one warp per source (152 SMs, ms per call, by radius over radius; one threshold |
// 1/4, 1/2, 1 of the farthest | 0.4, 0.6, 0.8, 1 of it; lines at 5.5 | 6 | 7.2 before the tiles' share):
//  90,000 nodes, all       5.0 13.6/13.1  16.7/14.4  20.7/16.2     6.2 17.9/20.1  21.5/21.9  26.6/24.5
//                          7.5 22.7/28.6  26.9/31.0  33.1/34.6    11.0 38.3/60.7  44.6/65.3  54.8/72.6
//    half of them          5.3 14.4/14.6  17.5/15.8  22.0/17.7     6.4 18.0/20.9  21.7/22.5  26.7/25.2
//    a quarter             4.5 12.9/11.0  16.0/11.8  21.4/13.1     5.5 16.0/16.2  19.8/17.4  24.2/19.2
//  19,881 nodes, all       6.2 4.21/4.27  5.15/4.71  6.32/5.22     7.5 5.15/5.95  6.17/6.46  7.62/7.18
//  10,000 nodes, all       6.2 2.51/2.33  3.05/2.59  3.69/2.90     7.5 2.99/3.21  3.57/3.48  4.42/3.92
//  40,000, diagonals, all  5.0 6.40/7.04  7.79/7.70  9.66/8.57     6.2 8.29/10.6  9.97/11.5  12.3/12.7
//  7 towns, 81,000, batch  5.0 12.0/11.4  14.8/12.8  18.3/14.6     6.2 15.5/17.1  18.9/18.9  23.3/21.6
//  4 towns, 13,600, batch  7.5 3.87/3.72  4.68/4.09  5.76/4.68    11.0 5.39/6.29  6.71/6.99  7.93/8.03
// By the sources' order, tiles against warps, every node: 202,500 nodes to 5 km along a curve 169 ms against
// 297, in rows 255 against 301, at random 359 against 345; 19,881 nodes to 3.2 km 8.9 against 11.1, 14.7
// against 11.0 and 13.9 against 13.2.
// Trips (3 to 9 per origin, two thresholds, by radius over radius): 10,000 nodes 10.0 4.6 ms against 5.4;
// 14,641 nodes 8.0 6.0 against 6.2; 90,000 nodes 10.0 34.8 against 51.3, 7.1 22.3 against 26.1, 5.0 16.5
// against 14.7; 40,000 nodes 7.1 11.3 against 12.8, 5.0 8.3 against 7.1.
// CS_TILE=0 leaves every source to the other kernels, CS_TILE=1 takes every call the kernel can serve.
long long tile_call() {
    return std::max<long long>(CS_TILE_SOURCES_MIN, 32ll * cs::tile::BPSM * std::max(1, sm_count()));
}
// The radius over the tile's, by the rows: 1 where tiles and warps are level in a large call.
double tile_margin(long long n_src, int n_bound, int k, const uint32_t *distances, const uint32_t *seconds, float delta) {
    if (!(delta > 0.0f) || n_src <= 0 || k <= 0) return 0.0;
    const uint32_t maxs = *std::max_element(seconds, seconds + k), maxd = *std::max_element(distances, distances + k);
    double rows = 0.0;
    for (int i = 0; i < k; i++) {
        const double r = maxd > 0 ? (double)distances[i] / maxd : 1.0;
        rows += r * r;
    }
    const double hops = std::min(2.0 * maxs / delta, 0.5 * std::sqrt((double)n_bound));
    return hops / std::sqrt(16.0 * n_bound / (double)n_src) / (4.0 + 1.5 * rows);
}
bool tile_pays(double margin, long long n_src, int P) {
    const double share = 32.0 * cs::tile::BPSM * std::max(1, sm_count()) / (double)n_src;  // blocks / tiles
    return margin >= (1.0 + 0.3 * share) * (P > 4 ? 0.75 : 1.0);
}
// Returns the sources per tile, 0: not this kernel.
int tile_lanes(const cs_query &q, int blocks, int n_bound, int P, float delta, bool near) {
    const char *e = getenv("CS_TILE");
    if (e && e[0] == '0') return 0;
    if (e && e[0] == '1') return (int)std::max(1ll, std::min(32ll, ((long long)q.n_sources + blocks - 1) / blocks));
    return near && q.n_sources >= tile_call() &&
                   tile_pays(tile_margin(q.n_sources, n_bound, q.k, q.distances, q.seconds, delta), q.n_sources, P)
               ? 32 : 0;
}

// The shortest-path jobs of a batch that go to the tile kernel: the rule's reach for each job by itself, its
// sources for all of them together (one launch serves them), where the caller vouches for the sources' order
// (near: a tile of sources from all over a graph holds their whole reaches one by one).  They have to be
// one run of consecutive jobs [lo, hi), each small enough for the list of sources left to the per-warp kernel
// (a launch takes as many of them as the list holds; with a larger job the whole batch runs one warp per
// source, as does a batch whose jobs of wide reach are not consecutive: cs_tile_margin sorts them).
// Measured on nine lattices of 2,500 to 22,200 nodes at 1.6 or 3.2 km, three with segments too: 52.5 ms a
// replay against 57.4 (six of the nine jobs tiled); 32 lattices of 2,000 to 150,000 nodes at up to 4.8 km, each
// with segments: 776 ms against 908.
void tile_jobs(const cs_batch_job *jobs, int n_jobs, int P, bool near, long long list, int &lo, int &hi) {
    lo = hi = 0;
    const char *e = getenv("CS_TILE");
    const bool all = e && e[0] == '1';
    if ((e && e[0] == '0') || (!near && !all)) return;
    long long shortest = 0, total = 0;
    for (int j = 0; j < n_jobs; j++)
        if (jobs[j].mode == cs::MODE_SHORTEST) shortest += std::max(0, jobs[j].n_sources);
    for (int j = 0; j < n_jobs; j++) {
        const cs_batch_job &b = jobs[j];
        if (b.mode != cs::MODE_SHORTEST || b.n_sources <= 0 || !(b.delta_seconds > 0.0f)) continue;
        if (!all && !tile_pays(cs_tile_margin(&b), shortest, P)) continue;
        if (total == 0) lo = hi = j;
        if (hi != j || b.n_sources > list) {
            hi = lo;
            return;
        }
        hi = j + 1;
        total += b.n_sources;
    }
    if (!all && total < tile_call()) hi = lo;
}

// Settle-order sort: distance buckets by default, CS_SORT=radix selects the LSD radix sort.
int radix_sort_choice() {
    const char *e = getenv("CS_SORT");
    return (e && strcmp(e, "radix") == 0) ? 1 : 0;
}

cs_status launch_primal(cs::PrimalParams &p, const cs_plan *plan, int n_slots, cudaStream_t stream) {
    const int tpb = 256;
    const int wpb = tpb / 32;
    const int minb = launch_variant(plan, p.mode);
    int blocks = (n_slots + wpb - 1) / wpb;
    if (p.P <= 8 && minb < resolve_variant(plan)) {
        // a tighter launch than the plan's slots were sized for: the blocks that are resident at once
        blocks = std::max(1, std::min(blocks, std::max(1, sm_count()) * minb));
        n_slots = std::min(n_slots, blocks * wpb);
    }
    p.n_slots = n_slots;
    if (p.mode == cs::MODE_SHORTEST) cs::launch_shortest(p, p.P, minb, blocks, phase_sync(), stream);
    else if (p.mode == cs::MODE_SEGMENT) cs::launch_segment(p, p.P, minb, blocks, phase_sync(), stream);
    else if (p.mode == cs::MODE_OD) cs::launch_od(p, p.P, minb, blocks, stream);
    else if (p.mode == cs::MODE_ACCESS) cs::launch_access(p, p.P, minb, blocks, stream);
    else cs::launch_tree(p, p.P, minb, blocks, stream);
    g_counters[3]++;
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return cuda_fail(e, "primal_kernel launch");
    return CS_OK;
}

// mode: the jobs' common mode (0 or 1) for a mode-specialised kernel, else -1
cs_status launch_batch(cs::PrimalParams &p, const cs_plan *plan, const cs_batch_job *jobs_dev, int n_jobs,
                       long long item_lo, long long item_hi, int n_slots, int mode, cudaStream_t stream) {
    // mixed-mode launches (and reruns) take the shortest-path budget
    const int minb = launch_variant(plan, mode == cs::MODE_SEGMENT ? cs::MODE_SEGMENT : cs::MODE_SHORTEST);
    int blocks = (n_slots + 7) / 8;
    if (p.P <= 8 && minb < resolve_variant(plan)) {
        blocks = std::max(1, std::min(blocks, std::max(1, sm_count()) * minb));
        n_slots = std::min(n_slots, blocks * 8);
    }
    p.n_slots = n_slots;
    cs::launch_batch_items(p, mode, minb, blocks, phase_sync(), jobs_dev, n_jobs, item_lo, item_hi, stream);
    g_counters[3]++;
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return cuda_fail(e, "batch_kernel launch");
    return CS_OK;
}

// Tabulates exp(-j / 256) for the beta-weighted seeds (cs_seed.cuh) on the call's stream.
cs_status launch_seed_table(cudaStream_t stream, void (*launch)(cudaStream_t)) {
    launch(stream);
    g_counters[3]++;
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? CS_OK : cuda_fail(e, "seed_table_kernel launch");
}

cs_status reset_dense(char *dense, size_t stride, int n_bound, int n_slots, cudaStream_t stream) {
    const size_t total = (size_t)n_bound * (size_t)n_slots;
    int blocks = (int)std::min<size_t>((total + 255) / 256, (size_t)sm_count() * 16);
    if (blocks < 1) blocks = 1;
    cs::fill_dense_kernel<<<blocks, 256, 0, stream>>>(dense, stride, n_bound, nullptr, 0, n_slots);
    g_counters[3]++;
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return cuda_fail(e, "fill_dense_kernel launch");
    return CS_OK;
}

constexpr int TILE_LEFT_SLOT = 10;  // header word: items that a batch's tiles left to the per-warp kernel

// The tile kernel's view of a call.
cs::tile::Params tile_params(const cs::PrimalParams &p, const Layout &lay, const cs::tile::Geometry &geo, int lanes) {
    cs::tile::Params c;
    memset(&c, 0, sizeof(c));
    const bool od = p.mode == cs::MODE_OD;
    c.n_bound = p.g.n_bound;
    c.in_ptr = p.g.in_ptr_dev;
    c.in_nb = p.g.in_nb_dev;
    c.in_w = p.g.in_w_dev;
    c.out_ptr = p.g.out_ptr_dev;
    c.out_to = p.g.out_to_dev;
    c.out_w = p.g.out_w_dev;
    c.out_cnt = p.g.out_cnt_dev;
    c.node_w = p.g.node_w_dev;
    c.k = p.k;
    for (int i = 0; i < p.k; i++) {
        c.dk[i] = p.dk[i];
        c.beta[i] = p.beta[i];
    }
    c.maxsec = p.maxsec;
    c.speed = p.speed;
    c.tol = p.tol;
    c.delta = p.delta;
    c.closeness = p.closeness;
    c.betweenness = p.betweenness;
    c.track_reach = p.track_reach;
    c.src_list = p.src_list;
    c.n_src = p.n_src;
    c.lanes = lanes;
    c.src_wt = p.src_wt;
    c.eligible = od ? nullptr : p.eligible;  // trips carry their own weights
    c.od_ptr = p.od_ptr;
    c.od_dst = p.od_dst;
    c.od_w = p.od_w;
    c.out = p.out;
    c.bucket = p.bucket;
    c.reach = p.reach;
    c.hdr = p.hdr;
    c.failed = p.failed;
    c.n_failed = &p.hdr->n_failed;
    c.fail_cap = p.fail_cap;
    c.dense = p.dense;
    c.dense_stride = p.dense_stride;
    c.aux_off = lay.dense_stride / 2;
    c.region = p.compact;
    c.geo = geo;
    return c;
}

// Completes a call's rows after its kernels and records its counters (h: the last header read).
cs_status finish_primal(const cs::PrimalParams &p, const cs::WsHeader &h, bool bucketed, long long n_over,
                        cudaStream_t stream) {
    if (bucketed) {
        const int blocks = std::max(1, std::min((p.g.n_bound + 255) / 256, sm_count() * 8));
        cs::bucket_prefix_kernel<<<blocks, 256, 0, stream>>>(p.bucket, p.out, p.k, p.g.n_bound);
        g_counters[3]++;
        const cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return cuda_fail(e, "bucket_prefix_kernel launch");
    }
    g_counters[0] = (long long)h.sources_done;
    g_counters[1] = (long long)h.edges_relaxed;
    g_counters[2] = (long long)h.nodes_settled;
    for (int i = 0; i < 16; i++) cs_host::g_phase[i] = (long long)h.pad[i];
    cs_set_retries_internal(n_over, 0);
    return CS_OK;
}

cs_status run_primal(const cs_primal_graph *g, const cs_query *q, const cs_plan *plan, void *ws, size_t ws_bytes,
                     cs_outputs out, void *stream_v, int mode, int32_t row_cap, int32_t *t_count, int32_t *t_node,
                     float *t_agg, int32_t *t_pred, const int32_t *tree_src, int32_t n_tree, uint32_t tree_maxsec,
                     float tree_speed, bool poll = false, const int32_t *od_ptr = nullptr,
                     const int32_t *od_dst = nullptr, const float *od_w = nullptr) {
    cs_status st = validate_primal(g);
    if (st != CS_OK) return st;
    if (!plan || !ws) return fail(CS_ERR_ARG, "plan/workspace is NULL");
    const int P = std::max(1, g->max_out_degree);
    const int K = (mode == cs::MODE_TREE) ? 1 : q->k;
    if (K < 1 || K > CS_MAX_THRESHOLDS) return fail(CS_ERR_ARG, "threshold count out of range");
    const int L = lanes_for(mode, K);
    if (plan->lanes < L) return fail(CS_ERR_ARG, "plan was made for fewer thresholds");
    if (plan->n_bound > 0 && plan->n_bound != g->n_bound)
        return fail(CS_ERR_ARG, "plan was made for a graph of another node bound");
    Layout lay = layout(g->n_bound, plan->n_slots, plan->cap, P, plan->lanes, plan->cta_blocks);
    if (ws_bytes < lay.total) return fail(CS_ERR_ARG, "workspace too small for this plan");
    cudaStream_t stream = (cudaStream_t)stream_v;
    char *base = (char *)ws;
    cs::PrimalParams p;
    memset(&p, 0, sizeof(p));
    p.radix_sort = radix_sort_choice();
    p.g = *g;
    p.k = K;
    uint32_t maxs = 0;
    if (mode == cs::MODE_TREE) {
        maxs = tree_maxsec;
        p.speed = tree_speed;
        p.tol = cs::TIE_EPSILON;
        p.src_list = tree_src;
        p.n_src = n_tree;
    } else {
        if (!q) return fail(CS_ERR_ARG, "query is NULL");
        for (int i = 0; i < K; i++) {
            p.dk[i] = (float)q->distances[i];
            p.beta[i] = q->betas[i];
            p.inb[i] = 1.0f / -p.beta[i];
            maxs = std::max(maxs, q->seconds[i]);
        }
        p.speed = q->speed_m_s;
        p.tol = q->tolerance;
        p.closeness = q->compute_closeness;
        p.betweenness = q->compute_betweenness;
        p.track_reach = q->track_reach;
        p.src_list = q->sources_dev;
        p.n_src = q->n_sources;
        p.src_wt = q->src_wt_dev;
        p.eligible = q->eligible_dev;
        if (mode == cs::MODE_OD) {
            if (p.n_src > 0 && (!od_ptr || !od_dst || !od_w))
                return fail(CS_ERR_ARG, "origin-destination rows are NULL");
            p.closeness = 0;
            p.betweenness = 1;
            p.track_reach = 0;
            p.od_ptr = od_ptr;
            p.od_dst = od_dst;
            p.od_w = od_w;
        }
        if (p.track_reach && !out.reach_dev) return fail(CS_ERR_ARG, "reach_dev required when track_reach");
        if (!out.out_dev) return fail(CS_ERR_ARG, "out_dev is NULL");
    }
    if (!(p.speed > 0.0f) || !std::isfinite(p.speed)) return fail(CS_ERR_ARG, "speed_m_s must be finite and positive");
    p.maxsec = (float)maxs;
    p.delta = plan->delta_seconds > 0.0f ? plan->delta_seconds : std::max(1.0f, p.maxsec / 48.0f);
    const bool block = (mode == cs::MODE_SHORTEST || mode == cs::MODE_OD) && plan->cta_blocks > 0 &&
                       cs::cta::supported(P, K) && q && block_schedule(q->n_sources, p.maxsec, plan->delta_seconds);
    p.out = out.out_dev;
    p.bucket = (double *)(base + lay.bucket_off);
    p.reach = out.reach_dev;
    p.hdr = (cs::WsHeader *)(base + lay.hdr_off);
    p.failed = (int32_t *)(base + lay.failed_off);
    p.fail_cap = lay.fail_cap;
    p.dense = base + lay.dense_off;
    p.dense_stride = lay.dense_stride;
    p.compact = base + lay.compact_off;
    p.cap = plan->cap;
    p.P = P;
    p.L = plan->lanes;
    p.mode = mode;
    p.row_cap = row_cap;
    p.t_count = t_count;
    p.t_node = t_node;
    p.t_agg = t_agg;
    p.t_pred = t_pred;
    g_counters[0] = g_counters[1] = g_counters[2] = g_counters[3] = 0;
    if (p.n_src <= 0) return CS_OK;
    cudaError_t e = cudaMemsetAsync(p.hdr, 0, sizeof(cs::WsHeader), stream);
    if (e != cudaSuccess) return cuda_fail(e, "workspace header reset");
    const bool bucketed = (mode == cs::MODE_SHORTEST) && p.closeness;
    if (bucketed) {
        e = cudaMemsetAsync(p.bucket, 0, sizeof(double) * 3 * (size_t)K * (size_t)g->n_bound, stream);
        if (e != cudaSuccess) return cuda_fail(e, "bucket reset");
    }
    if (p.betweenness && (mode == cs::MODE_SHORTEST || mode == cs::MODE_OD)) {
        st = launch_seed_table(stream, cs::launch_seed_table_shortest);
        if (st != CS_OK) return st;
    }
    cs::tile::Geometry geo{};
    int tile_blocks = 0, lanes = 0;
    if ((mode == cs::MODE_SHORTEST || mode == cs::MODE_OD) && P <= cs::tile::PMAX) {
        tile_blocks = std::max(1, std::min(sm_count() * cs::tile::BPSM, plan->n_slots));
        lanes = tile_lanes(*q, tile_blocks, g->n_bound, P, plan->delta_seconds,
                           (plan->variant & CS_PLAN_NEAR_SOURCES) != 0);
        if (lanes > 0) {
            tile_blocks = (int)std::min<long long>(tile_blocks, (p.n_src + lanes - 1) / lanes);
            geo = cs::tile::geometry((lay.compact_total / tile_blocks) & ~size_t(255), K, p.dk, mode == cs::MODE_OD);
        }
    }
    if (geo.mcap >= plan->cap) {
        // the list of sources left to the per-warp kernel holds fail_cap: more sources run in shares
        const int64_t n_all = p.n_src;
        const int32_t *all = p.src_list;
        long long n_left = 0;
        cs::WsHeader h;
        e = cs::tile::launch_seed_table(stream);
        if (e != cudaSuccess) return cuda_fail(e, "seed table launch");
        for (int64_t lo = 0; lo < n_all; lo += lay.fail_cap) {
            p.src_list = all + lo;
            p.n_src = std::min<int64_t>(n_all - lo, lay.fail_cap);
            if (lo > 0) {
                e = cudaMemsetAsync(&p.hdr->work_next, 0, sizeof(unsigned long long), stream);
                if (e == cudaSuccess) e = cudaMemsetAsync(&p.hdr->n_failed, 0, sizeof(unsigned), stream);
                if (e != cudaSuccess) return cuda_fail(e, "tile counter reset");
            }
            e = cs::tile::launch(tile_params(p, lay, geo, lanes), mode == cs::MODE_OD, tile_blocks, stream);
            g_counters[3] += 2;
            if (e != cudaSuccess) return cuda_fail(e, "tile_kernel launch");
            e = cs::read_header(p.hdr, h, stream, poll);
            if (e != cudaSuccess) return cuda_fail(e, "tile kernel");
            if (h.err != 0u)
                return fail((cs_status)h.err, "device-side check failed (code " + std::to_string(h.err) + " at " +
                                                  std::to_string(h.err_where) + ")");
            n_left += h.n_failed;
            if (h.n_failed > 0u) {
                st = retry_chain(p, plan, lay, base, g->n_bound, P, h, stream, poll,
                                 [&](cs::PrimalParams &p2, int slots2) { return launch_primal(p2, plan, slots2, stream); },
                                 plan->cap);
                if (st != CS_OK) return st;
            }
        }
        return finish_primal(p, h, bucketed, n_left, stream);
    }
    if (block) {
        // one block per source with its state on chip; the sources it lists (reach or queues beyond
        // its capacity) run through the per-warp kernel's capacity chain below
        e = cs::cta::launch_seed_table(stream);
        if (e != cudaSuccess) return cuda_fail(e, "seed table launch");
        cs::cta::Params c;
        memset(&c, 0, sizeof(c));
        c.n_bound = g->n_bound;
        c.in_ptr = g->in_ptr_dev;
        c.in_nb = g->in_nb_dev;
        c.in_w = g->in_w_dev;
        c.out_ptr = g->out_ptr_dev;
        c.out_to = g->out_to_dev;
        c.out_w = g->out_w_dev;
        c.out_cnt = g->out_cnt_dev;
        c.node_w = g->node_w_dev;
        c.k = K;
        for (int i = 0; i < K; i++) {
            c.dk[i] = p.dk[i];
            c.beta[i] = p.beta[i];
        }
        c.maxsec = p.maxsec;
        c.speed = p.speed;
        c.tol = p.tol;
        // the block kernel's rounds are paced by barriers: wider bands (fewer rounds, more
        // re-relaxations) suit it; CS_BLOCK_DELTA_SCALE overrides the width factor
        {
            const char *ev = getenv("CS_BLOCK_DELTA_SCALE");
            const float scale = ev ? (float)atof(ev) : 4.0f;
            c.delta = (scale > 0.0f) ? p.delta * scale : p.delta;
        }
        c.closeness = p.closeness;
        c.betweenness = p.betweenness;
        c.track_reach = p.track_reach;
        c.od = (mode == cs::MODE_OD) ? 1 : 0;
        c.src_list = p.src_list;
        c.n_src = p.n_src;
        c.src_wt = p.src_wt;
        c.eligible = p.eligible;
        c.od_ptr = p.od_ptr;
        c.od_dst = p.od_dst;
        c.od_w = p.od_w;
        c.out = p.out;
        c.bucket = p.bucket;
        c.reach = p.reach;
        c.hdr = p.hdr;
        c.failed = p.failed;
        c.fail_cap = p.fail_cap;
        c.scratch = base + lay.cta_off;
        c.scratch_stride = cs::cta::scratch_bytes();
        e = cs::cta::launch(c, plan->cta_blocks, stream);
        g_counters[3] += 2;
        if (e != cudaSuccess) return cuda_fail(e, "source_block_kernel launch");
    } else {
        st = launch_primal(p, plan, plan->n_slots, stream);
        if (st != CS_OK) return st;
    }
    cs::WsHeader h;
    e = cs::read_header(p.hdr, h, stream, poll);
    if (e != cudaSuccess) return cuda_fail(e, "centrality kernel");
    if (h.err != 0u)
        return fail((cs_status)h.err, "device-side check failed (code " + std::to_string(h.err) + " at " +
                                          std::to_string(h.err_where) + ")");
    const long long n_over = h.n_failed;
    if (h.n_failed > 0u) {
        // Sources whose reach overflowed `cap` (their slots already reset themselves)
        st = retry_chain(p, plan, lay, base, g->n_bound, P, h, stream, poll,
                         [&](cs::PrimalParams &p2, int slots2) { return launch_primal(p2, plan, slots2, stream); });
        if (st != CS_OK) return st;
    }
    return finish_primal(p, h, bucketed, n_over, stream);
}

cs_status plan_common(int n_bound, int P, int L, int cap, int max_slots, int64_t budget, cs_plan *plan,
                      bool block_kernel = false) {
    const int variant = resolve_variant(plan);
    if (!plan) return fail(CS_ERR_ARG, "plan is NULL");
    int sms = sm_count();
    if (sms <= 0) return fail(CS_ERR_CUDA, "no CUDA device");
    int bpsm = 0;
    cudaError_t e = cs::occupancy_primal(P, variant, &bpsm);
    if (e != cudaSuccess) return cuda_fail(e, "occupancy query");
    if (bpsm < 1) bpsm = 1;
    int slots = sms * bpsm * 8;
    if (max_slots > 0) slots = std::min(slots, max_slots);
    if (cap <= 0) cap = std::min(n_bound, 16384);
    cap = std::max(32, std::min(cap, n_bound));
    const int cta_blocks = block_kernel ? sms : 0;
    auto total_for = [&](int ns) { return layout(n_bound, ns, cap, P, L, cta_blocks).total; };
    if (budget > 0) {
        while (slots > 8 && (int64_t)total_for(slots) > budget) slots = (slots * 7) / 8;
    }
    slots = std::max(1, slots);
    plan->n_slots = slots;
    plan->cap = cap;
    plan->threads_per_block = 256;
    plan->blocks = (slots + 7) / 8;
    if (plan->delta_seconds != plan->delta_seconds) plan->delta_seconds = 0.0f;
    plan->lanes = L;
    plan->variant = requested_variant(plan);  // 0: each launch picks its budget by mode
    plan->max_degree = P;
    plan->n_bound = n_bound;
    plan->cta_blocks = cta_blocks;
    plan->workspace_bytes = total_for(slots);
    return CS_OK;
}

}  // namespace

extern "C" {

size_t cs_last_error(char *buf, size_t len) {
    const std::string &m = cs_host::g_last_error;
    const size_t n = m.size();
    if (buf && len) {
        const size_t c = std::min(n, len - 1);
        memcpy(buf, m.data(), c);
        buf[c] = 0;
    }
    return n;
}

int32_t cs_device_sm_count(void) { return sm_count(); }

cs_status cs_last_phase_cycles(int64_t *cycles, int32_t n) {
    if (!cycles || n < 0) return fail(CS_ERR_ARG, "cycles is NULL");
    for (int i = 0; i < n && i < 16; i++) cycles[i] = cs_host::g_phase[i];
    return CS_OK;
}

cs_status cs_last_counters(int64_t *sources, int64_t *edges_relaxed, int64_t *nodes_settled, int64_t *launches) {
    if (sources) *sources = g_counters[0];
    if (edges_relaxed) *edges_relaxed = g_counters[1];
    if (nodes_settled) *nodes_settled = g_counters[2];
    if (launches) *launches = g_counters[3];
    return CS_OK;
}

cs_status cs_plan_primal(const cs_primal_graph *g, int32_t mode, int32_t k, int32_t cap, int32_t max_slots,
                         int64_t mem_budget_bytes, cs_plan *plan) {
    cs_status st = validate_primal(g);
    if (st != CS_OK) return st;
    if (mode < 0 || mode > 2) return fail(CS_ERR_ARG, "unknown mode");
    if (mode != cs::MODE_TREE && (k < 1 || k > CS_MAX_THRESHOLDS)) return fail(CS_ERR_ARG, "threshold count out of range");
    const int P = std::max(1, g->max_out_degree);
    const float keep_delta = plan ? plan->delta_seconds : 0.0f;
    if (plan) plan->delta_seconds = keep_delta;
    const bool block = mode == cs::MODE_SHORTEST && block_kernel_enabled() && cs::cta::supported(P, k);
    return plan_common(g->n_bound, P, lanes_for(mode, mode == cs::MODE_TREE ? 1 : k), cap, max_slots,
                       mem_budget_bytes, plan, block);
}

cs_status cs_workspace_init(const cs_plan *plan, int32_t n_bound, void *workspace_dev, size_t workspace_bytes,
                            void *stream) {
    if (!plan || !workspace_dev) return fail(CS_ERR_ARG, "plan/workspace is NULL");
    if (workspace_bytes < plan->workspace_bytes) return fail(CS_ERR_ARG, "workspace smaller than plan");
    if (plan->lanes < 1) return fail(CS_ERR_ARG, "plan has no lanes");
    // the dense region's offset depends only on (n_bound, n_slots, lanes): same as every call
    Layout lay = layout(n_bound, plan->n_slots, plan->cap, 1, plan->lanes);
    cudaStream_t s = (cudaStream_t)stream;
    cudaError_t e = cudaMemsetAsync(workspace_dev, 0, 256, s);
    if (e != cudaSuccess) return cuda_fail(e, "workspace init");
    return reset_dense((char *)workspace_dev + lay.dense_off, lay.dense_stride, n_bound, plan->n_slots, s);
}

cs_status cs_centrality_shortest(const cs_primal_graph *g, const cs_query *q, const cs_plan *plan,
                                 void *workspace_dev, size_t workspace_bytes, cs_outputs out, void *stream) {
    return run_primal(g, q, plan, workspace_dev, workspace_bytes, out, stream, cs::MODE_SHORTEST, 0, nullptr, nullptr,
                      nullptr, nullptr, nullptr, 0, 0, 0.0f, true);
}

cs_status cs_betweenness_od_shortest(const cs_primal_graph *g, const cs_query *q, const int32_t *od_ptr_dev,
                                     const int32_t *od_dst_dev, const float *od_w_dev, const cs_plan *plan,
                                     void *workspace_dev, size_t workspace_bytes, cs_outputs out, void *stream) {
    return run_primal(g, q, plan, workspace_dev, workspace_bytes, out, stream, cs::MODE_OD, 0, nullptr, nullptr,
                      nullptr, nullptr, nullptr, 0, 0, 0.0f, true, od_ptr_dev, od_dst_dev, od_w_dev);
}

cs_status cs_segment_centrality(const cs_primal_graph *g, const cs_query *q, const cs_plan *plan,
                                void *workspace_dev, size_t workspace_bytes, cs_outputs out, void *stream) {
    return run_primal(g, q, plan, workspace_dev, workspace_bytes, out, stream, cs::MODE_SEGMENT, 0, nullptr, nullptr,
                      nullptr, nullptr, nullptr, 0, 0, 0.0f, true);
}

cs_status cs_tree_shortest(const cs_primal_graph *g, int32_t n_queries, const int32_t *src_dev, uint32_t max_seconds,
                           float speed_m_s, const cs_plan *plan, void *workspace_dev, size_t workspace_bytes,
                           int32_t row_cap, int32_t *count_dev, int32_t *node_dev, float *agg_seconds_dev,
                           int32_t *pred_dev, void *stream) {
    if (!count_dev || !node_dev || !agg_seconds_dev || !pred_dev || row_cap <= 0)
        return fail(CS_ERR_ARG, "tree outputs missing");
    cs_outputs o{nullptr, nullptr};
    return run_primal(g, nullptr, plan, workspace_dev, workspace_bytes, o, stream, cs::MODE_TREE, row_cap, count_dev,
                      node_dev, agg_seconds_dev, pred_dev, src_dev, n_queries, max_seconds, speed_m_s, true);
}

cs_status cs_accessibility(const cs_primal_graph *g, const cs_data_map *dm, const cs_query *q,
                           const float *max_curve_wts, int32_t n_classes, const cs_plan *plan, void *workspace_dev,
                           size_t workspace_bytes, double *unweighted_dev, double *weighted_dev,
                           uint32_t *nearest_dev, void *stream) {
    cs_status st = validate_primal(g);
    if (st != CS_OK) return st;
    if (!dm || !q || !max_curve_wts || !plan || !workspace_dev) return fail(CS_ERR_ARG, "accessibility: NULL argument");
    if (q->k < 1 || q->k > CS_MAX_THRESHOLDS) return fail(CS_ERR_ARG, "threshold count out of range");
    if (n_classes < 0) return fail(CS_ERR_ARG, "accessibility: negative class count");
    if (q->n_sources > 0 && (!dm->node_ptr_dev || !dm->assign_entry_dev || !dm->assign_dist_dev ||
                             !dm->assign_node_dev || !dm->assign_rank_dev || !dm->entry_group_dev ||
                             !dm->entry_class_dev || !dm->group_ptr_dev || !dm->group_assign_dev))
        return fail(CS_ERR_ARG, "accessibility: data map array is NULL");
    if (n_classes > 0 && q->n_sources > 0 && (!unweighted_dev || !weighted_dev || !nearest_dev))
        return fail(CS_ERR_ARG, "accessibility: output is NULL");
    for (int i = 0; i < q->k; i++)
        if (!(max_curve_wts[i] > 0.0f && max_curve_wts[i] <= 1.0f))
            return fail(CS_ERR_ARG, "Max curve weight must be in the range [0, 1].");
    const int P = std::max(1, g->max_out_degree);
    Layout lay = layout(g->n_bound, plan->n_slots, plan->cap, P, plan->lanes, plan->cta_blocks);
    if (workspace_bytes < lay.total) return fail(CS_ERR_ARG, "workspace too small for this plan");
    if (plan->n_bound > 0 && plan->n_bound != g->n_bound)
        return fail(CS_ERR_ARG, "plan was made for a graph of another node bound");
    cudaStream_t stream_c = (cudaStream_t)stream;
    char *base = (char *)workspace_dev;
    cs::PrimalParams p;
    memset(&p, 0, sizeof(p));
    p.g = *g;
    p.k = q->k;
    uint32_t maxs = 0, maxd = 0;
    for (int i = 0; i < q->k; i++) {
        p.dk[i] = (float)q->distances[i];
        p.beta[i] = q->betas[i];
        p.mcw[i] = max_curve_wts[i];
        maxs = std::max(maxs, q->seconds[i]);
        maxd = std::max(maxd, q->distances[i]);
    }
    p.max_dist = (float)maxd;
    p.speed = q->speed_m_s;
    if (!(p.speed > 0.0f) || !std::isfinite(p.speed)) return fail(CS_ERR_ARG, "speed_m_s must be finite and positive");
    p.tol = cs::TIE_EPSILON;
    p.maxsec = (float)maxs;
    p.delta = plan->delta_seconds > 0.0f ? plan->delta_seconds : std::max(1.0f, p.maxsec / 48.0f);
    p.src_list = q->sources_dev;
    p.n_src = q->n_sources;
    p.dm = *dm;
    p.acc_unw = unweighted_dev;
    p.acc_wt = weighted_dev;
    p.acc_near = nearest_dev;
    p.hdr = (cs::WsHeader *)(base + lay.hdr_off);
    p.failed = (int32_t *)(base + lay.failed_off);
    p.fail_cap = lay.fail_cap;
    p.dense = base + lay.dense_off;
    p.dense_stride = lay.dense_stride;
    p.compact = base + lay.compact_off;
    p.cap = plan->cap;
    p.P = P;
    p.L = plan->lanes;
    p.mode = cs::MODE_ACCESS;
    p.radix_sort = radix_sort_choice();
    g_counters[0] = g_counters[1] = g_counters[2] = g_counters[3] = 0;
    if (p.n_src <= 0 || n_classes == 0) return CS_OK;
    cudaError_t e = cudaMemsetAsync(p.hdr, 0, sizeof(cs::WsHeader), stream_c);
    if (e != cudaSuccess) return cuda_fail(e, "workspace header reset");
    st = launch_primal(p, plan, plan->n_slots, stream_c);
    if (st != CS_OK) return st;
    cs::WsHeader h;
    e = cs::read_header(p.hdr, h, stream_c, true);
    if (e != cudaSuccess) return cuda_fail(e, "accessibility kernel");
    if (h.err != 0u) return fail((cs_status)h.err, "device-side check failed (code " + std::to_string(h.err) + ")");
    if (h.n_failed > 0u) {
        st = retry_chain(p, plan, lay, base, g->n_bound, P, h, stream_c, true,
                         [&](cs::PrimalParams &p2, int slots2) { return launch_primal(p2, plan, slots2, stream_c); });
        if (st != CS_OK) return st;
    }
    g_counters[0] = (long long)h.sources_done;
    g_counters[1] = (long long)h.edges_relaxed;
    g_counters[2] = (long long)h.nodes_settled;
    return CS_OK;
}

}  // extern "C"

// ==========================================================================================
// Allocation-free entry point (cs_centrality_shortest_noalloc).
//
// Some callers cannot allocate device memory at the time they want centralities: code running
// inside a host application that owns every device allocation through its own pool, plugins whose
// memory budget is fixed when the process starts, or code paths where an allocation could fail or
// block.  For them this entry point draws its scratch from one static device array that the CUDA
// module reserves when it is loaded, so the call itself allocates nothing.
//
// Limits and rules:
//  - The array holds 64 MiB; every GPU that loads this library keeps it until the process exits.
//  - One search needs 8 bytes per node of dense state plus its per-node arrays for the whole
//    graph (the capacity is node_bound, so no search can overflow).  Graphs whose single search
//    does not fit are rejected with CS_ERR_ARG and a message naming the sizes.
//  - All calls share the array and it keeps the previous call's contents; each call therefore
//    re-initialises the state that must start clean.  Calls that overlap on the GPU (two streams,
//    two host threads) race on the array: issue them one after another.
//  - Every call looks up the array's device address with cudaGetSymbolAddress while the
//    caller's device and context are current, so the address always belongs to the context the
//    call runs in (a context the host application created itself, or one re-created after
//    cudaDeviceReset).  The lookup allocates nothing.
//  - With lazy module loading (the CUDA default since 12.2) this file's device code, and with it
//    the 64 MiB array, is loaded on the first use of any of its kernels or of the array on a
//    device, and the code of the kernels that this call launches (cs_primal_shortest.cu) on their own
//    first use: measured, 2 MiB inside the first call where only trees, accessibility or source
//    weights ran before, nothing after a shortest-path or segment call.  Callers that must not see it
//    make one call of this entry point while setting up, before the device's memory is handed to their
//    pool and before any stream capture.
// ==========================================================================================
namespace {
constexpr size_t kNoAllocScratchBytes = size_t(64) << 20;
}  // namespace

static __device__ __align__(256) unsigned char cs_noalloc_scratch[kNoAllocScratchBytes];

namespace {
cs_status noalloc_scratch_address(void **out) {
    void *p = nullptr;
    const cudaError_t e = cudaGetSymbolAddress(&p, cs_noalloc_scratch);
    if (e != cudaSuccess) return cuda_fail(e, "cudaGetSymbolAddress(static scratch)");
    if (!p) return fail(CS_ERR_CUDA, "static scratch has no device address");
    *out = p;
    return CS_OK;
}
}  // namespace

extern "C" cs_status cs_centrality_shortest_noalloc(const cs_primal_graph *g, const cs_query *q, cs_outputs out,
                                                    void *stream) {
    cs_status st = validate_primal(g);
    if (st != CS_OK) return st;
    if (!q) return fail(CS_ERR_ARG, "query is NULL");
    if (q->k < 1 || q->k > CS_MAX_THRESHOLDS) return fail(CS_ERR_ARG, "threshold count out of range");
    const int P = std::max(1, g->max_out_degree);
    const int L = lanes_for(cs::MODE_SHORTEST, q->k);
    const int cap = g->n_bound;  // a search can never overflow: no retry pass is needed
    const size_t one = layout(g->n_bound, 1, cap, P, L).total;
    if (one > kNoAllocScratchBytes)
        return fail(CS_ERR_ARG, "graph too large for the allocation-free path: one search needs " +
                                    std::to_string(one) + " bytes of scratch, the static array holds " +
                                    std::to_string(kNoAllocScratchBytes) + " bytes");
    int sms = sm_count();
    if (sms <= 0) return fail(CS_ERR_CUDA, "no CUDA device");
    int bpsm = 0;
    cudaError_t e = cs::occupancy_primal(P, launch_variant(nullptr, cs::MODE_SHORTEST), &bpsm);
    if (e != cudaSuccess) return cuda_fail(e, "occupancy query");
    int slots = std::max(1, sms * std::max(1, bpsm) * 8);
    while (slots > 1 && layout(g->n_bound, slots, cap, P, L).total > kNoAllocScratchBytes) {
        const int next = (slots * 7) / 8;
        slots = next < slots ? next : slots - 1;
    }
    void *ws = nullptr;
    st = noalloc_scratch_address(&ws);
    if (st != CS_OK) return st;
    cs_plan plan;
    memset(&plan, 0, sizeof(plan));
    plan.n_slots = slots;
    plan.cap = cap;
    plan.threads_per_block = 256;
    plan.blocks = (slots + 7) / 8;
    plan.delta_seconds = 0.0f;
    plan.lanes = L;
    plan.variant = launch_variant(nullptr, cs::MODE_SHORTEST);
    plan.max_degree = P;
    const Layout lay = layout(g->n_bound, slots, cap, P, L);
    plan.workspace_bytes = lay.total;
    cudaStream_t s = (cudaStream_t)stream;
    // The array keeps whatever the previous call left there (another graph's dense state or
    // compact scratch, or the remains of a call that failed midway), and this call's regions sit
    // at offsets set by its own node bound and threshold count.  Put every region that must start
    // clean into its clean state: the header, the dense per-slot state and the [3][K][n_bound]
    // closeness bucket.  The compact per-source arrays are written before they are read.
    e = cudaMemsetAsync(ws, 0, 256, s);
    if (e != cudaSuccess) return cuda_fail(e, "static scratch header reset");
    e = cudaMemsetAsync((char *)ws + lay.bucket_off, 0, sizeof(double) * 3 * (size_t)q->k * (size_t)g->n_bound, s);
    if (e != cudaSuccess) return cuda_fail(e, "static scratch bucket reset");
    st = reset_dense((char *)ws + lay.dense_off, lay.dense_stride, g->n_bound, slots, s);
    if (st != CS_OK) return st;
    return run_primal(g, q, &plan, ws, kNoAllocScratchBytes, out, stream, cs::MODE_SHORTEST, 0, nullptr, nullptr,
                      nullptr, nullptr, nullptr, 0, 0, 0.0f);
}

// ==========================================================================================
// Batched persistent form (cs_batch_*).
// ==========================================================================================
namespace {
struct BatchShape {
    int max_n, P, L;
};

cs_status batch_shape(const cs_batch_job *jobs, int n_jobs, BatchShape &b) {
    if (!jobs || n_jobs <= 0) return fail(CS_ERR_ARG, "empty batch");
    b.max_n = 1;
    b.P = 1;
    b.L = 1;
    for (int j = 0; j < n_jobs; j++) {
        cs_status st = validate_primal(&jobs[j].g);
        if (st != CS_OK) return st;
        if (jobs[j].mode != cs::MODE_SHORTEST && jobs[j].mode != cs::MODE_SEGMENT && jobs[j].mode != cs::MODE_BOTH)
            return fail(CS_ERR_ARG, "batch job mode must be 0 (shortest), 1 (segment) or 3 (both)");
        if (jobs[j].mode == cs::MODE_BOTH && !jobs[j].out2_dev) return fail(CS_ERR_ARG, "mode 3 job without out2_dev");
        if (jobs[j].k < 1 || jobs[j].k > CS_MAX_THRESHOLDS) return fail(CS_ERR_ARG, "threshold count out of range");
        if (!(jobs[j].speed_m_s > 0.0f)) return fail(CS_ERR_ARG, "speed_m_s must be finite and positive");
        if (!jobs[j].out_dev) return fail(CS_ERR_ARG, "job without out_dev");
        if ((jobs[j].mode == cs::MODE_SHORTEST || jobs[j].mode == cs::MODE_BOTH) && jobs[j].compute_closeness &&
            !jobs[j].bucket_dev)
            return fail(CS_ERR_ARG, "shortest job with closeness needs bucket_dev");
        b.max_n = std::max(b.max_n, jobs[j].g.n_bound);
        b.P = std::max(b.P, jobs[j].g.max_out_degree);
        b.L = std::max(b.L, lanes_for(jobs[j].mode, jobs[j].k));
    }
    return CS_OK;
}
}  // namespace

extern "C" {

float cs_tile_margin(const cs_batch_job *job) {
    if (!job || job->k < 1 || job->k > CS_MAX_THRESHOLDS) return 0.0f;
    return (float)tile_margin(job->n_sources, job->g.n_bound, job->k, job->distances, job->seconds, job->delta_seconds);
}

cs_status cs_batch_prepare(cs_batch_job *jobs_host, int32_t n_jobs, int64_t *n_items) {
    if (!jobs_host || n_jobs <= 0 || !n_items) return fail(CS_ERR_ARG, "empty batch");
    int64_t acc = 0;
    for (int j = 0; j < n_jobs; j++) {
        jobs_host[j].item_begin = acc;
        acc += std::max(0, jobs_host[j].n_sources);
    }
    *n_items = acc;
    return CS_OK;
}

cs_status cs_batch_plan(const cs_batch_job *jobs_host, int32_t n_jobs, int32_t cap, int32_t max_slots,
                        int64_t mem_budget_bytes, cs_plan *plan) {
    BatchShape b;
    cs_status st = batch_shape(jobs_host, n_jobs, b);
    if (st != CS_OK) return st;
    return plan_common(b.max_n, b.P, b.L, cap, max_slots, mem_budget_bytes, plan);
}

cs_status cs_batch_run(const cs_batch_job *jobs_host, const cs_batch_job *jobs_dev, int32_t n_jobs, const cs_plan *plan,
                       void *ws, size_t ws_bytes, int32_t flags, void *stream_v) {
    BatchShape b;
    cs_status st = batch_shape(jobs_host, n_jobs, b);
    if (st != CS_OK) return st;
    if (!plan || !ws || !jobs_dev) return fail(CS_ERR_ARG, "plan/workspace/jobs_dev is NULL");
    if (plan->lanes < b.L) return fail(CS_ERR_ARG, "plan was made for fewer lanes");
    const int P = std::max(1, plan->max_degree);
    if (P < b.P) return fail(CS_ERR_ARG, "plan was made for a smaller degree");
    // slot geometry is the plan's, so one workspace serves batches of any graphs up to its size
    const int geo_n = plan->n_bound > 0 ? plan->n_bound : b.max_n;
    if (geo_n < b.max_n) return fail(CS_ERR_ARG, "plan was made for a smaller graph");
    const Layout lay = layout(geo_n, plan->n_slots, plan->cap, P, plan->lanes);
    if (ws_bytes < lay.total) return fail(CS_ERR_ARG, "workspace too small for this plan");
    long long n_items = 0;
    for (int j = 0; j < n_jobs; j++) {
        if (jobs_host[j].item_begin != n_items) return fail(CS_ERR_ARG, "jobs not prepared (cs_batch_prepare)");
        n_items += std::max(0, jobs_host[j].n_sources);
    }
    cudaStream_t stream = (cudaStream_t)stream_v;
    char *base = (char *)ws;
    cs::PrimalParams p;
    memset(&p, 0, sizeof(p));
    p.radix_sort = radix_sort_choice();
    p.g.n_bound = geo_n;  // slot geometry only; each job brings its own graph
    p.hdr = (cs::WsHeader *)(base + lay.hdr_off);
    p.failed = (int32_t *)(base + lay.failed_off);
    p.fail_cap = lay.fail_cap;
    p.dense = base + lay.dense_off;
    p.dense_stride = lay.dense_stride;
    p.compact = base + lay.compact_off;
    p.cap = plan->cap;
    p.P = P;
    p.L = plan->lanes;
    g_counters[0] = g_counters[1] = g_counters[2] = g_counters[3] = 0;
    cudaError_t e = cudaMemsetAsync(p.hdr, 0, sizeof(cs::WsHeader), stream);
    if (e != cudaSuccess) return cuda_fail(e, "batch reset");
    if (n_items == 0) return CS_OK;
    // jobs for the tile kernel
    int t_lo = 0, t_hi = 0, t_k = 1;
    cs::tile::Geometry geo{};
    const int tile_blocks = std::max(1, std::min(sm_count() * cs::tile::BPSM, plan->n_slots));
    if (P <= cs::tile::PMAX)
        tile_jobs(jobs_host, n_jobs, P, (flags & CS_BATCH_NEAR_SOURCES) != 0, lay.fail_cap, t_lo, t_hi);
    for (int j = t_lo; j < t_hi; j++) {  // the layout that suits the job with the most dependency rows per node
        float dk[cs::MAXK];
        for (int i = 0; i < jobs_host[j].k; i++) dk[i] = (float)jobs_host[j].distances[i];
        const cs::tile::Geometry g =
            cs::tile::geometry((lay.compact_total / tile_blocks) & ~size_t(255), jobs_host[j].k, dk, false);
        if (j == t_lo || g.mcap < geo.mcap) geo = g;
        t_k = std::max(t_k, jobs_host[j].k);
    }
    if (geo.mcap < plan->cap) t_hi = t_lo;
    // consecutive jobs of one mode run as one launch of that mode's kernel (a smaller instruction
    // footprint than the all-mode kernel); more than four such runs use the all-mode kernel once
    struct Run {
        long long lo, hi;
        int mode;
    };
    std::vector<Run> runs;
    for (bool again = true; again;) {
        again = false;
        runs.clear();
        for (int j = 0; j < n_jobs; j++) {
            if (j >= t_lo && j < t_hi) continue;
            const int m = (jobs_host[j].mode == cs::MODE_SHORTEST || jobs_host[j].mode == cs::MODE_SEGMENT)
                              ? jobs_host[j].mode : -1;
            const long long lo = jobs_host[j].item_begin, hi = lo + std::max(0, jobs_host[j].n_sources);
            if (!runs.empty() && runs.back().mode == m && runs.back().hi == lo) runs.back().hi = hi;
            else runs.push_back({lo, hi, m});
        }
        if (runs.size() > 4 && t_hi > t_lo) {
            t_hi = t_lo;  // then without the tile kernel
            again = true;
        }
    }
    if (runs.size() > 4) runs.assign(1, Run{0, n_items, -1});
    st = launch_seed_table(stream, cs::launch_seed_table_batch);
    if (st != CS_OK) return st;
    for (int lo = t_lo, hi = t_lo; lo < t_hi; lo = hi) {
        // The tile kernel, then the per-warp kernel over the items that it lists.  How many there are stays on
        // the device, so that a captured batch needs no host in between; what overflows there is listed as
        // ever, in the other list.
        long long n = 0;
        while (hi < t_hi && n + jobs_host[hi].n_sources <= lay.fail_cap) n += jobs_host[hi++].n_sources;
        cs::tile::Params c = tile_params(p, lay, geo, 32);
        c.failed = (int32_t *)(base + lay.failed2_off);
        c.n_failed = (unsigned *)&p.hdr->pad[TILE_LEFT_SLOT];
        if (lo == t_lo) {
            e = cs::tile::launch_seed_table(stream);
            g_counters[3]++;
        } else {
            e = cudaMemsetAsync(&p.hdr->work_next, 0, 2 * sizeof(unsigned long long), stream);  // and work_next2
            if (e == cudaSuccess) e = cudaMemsetAsync(c.n_failed, 0, sizeof(unsigned), stream);
        }
        if (e == cudaSuccess) e = cs::tile::launch_batch(c, jobs_dev, lo, hi, t_k, tile_blocks, stream);
        if (e != cudaSuccess) return cuda_fail(e, "tile_batch_kernel launch");
        g_counters[3]++;
        cs::PrimalParams p2 = p;
        p2.rerun = 1;
        p2.remap = c.failed;
        p2.n_remap = c.n_failed;
        st = launch_batch(p2, plan, jobs_dev, n_jobs, 0, n_items, plan->n_slots, cs::MODE_SHORTEST, stream);
        if (st != CS_OK) return st;
    }
    for (const Run &r : runs) {
        if (r.hi <= r.lo) continue;
        e = cudaMemsetAsync(&p.hdr->work_next, 0, sizeof(unsigned long long), stream);
        if (e != cudaSuccess) return cuda_fail(e, "batch counter reset");
        st = launch_batch(p, plan, jobs_dev, n_jobs, r.lo, r.hi, plan->n_slots, r.mode, stream);
        if (st != CS_OK) return st;
    }
    if (!(flags & CS_BATCH_ASYNC)) {
        cs::WsHeader h;
        e = cs::read_header(p.hdr, h, stream, true);
        if (e != cudaSuccess) return cuda_fail(e, "batch kernel");
        if (h.err != 0u) return fail((cs_status)h.err, "device-side check failed (code " + std::to_string(h.err) + ")");
        const long long n_over = h.n_failed;
        if (h.n_failed > 0u) {
            st = retry_chain(p, plan, lay, base, b.max_n, P, h, stream, true, [&](cs::PrimalParams &p2, int slots2) {
                return launch_batch(p2, plan, jobs_dev, n_jobs, 0, n_items, slots2, -1, stream);
            });
            if (st != CS_OK) return st;
        }
        cs_set_retries_internal(n_over, 0);
        g_counters[0] = (long long)h.sources_done;
        g_counters[1] = (long long)h.edges_relaxed;
        g_counters[2] = (long long)h.nodes_settled;
        for (int i = 0; i < 16; i++) g_phase[i] = (long long)h.pad[i];
    }
    int max_n = 0, n_pref = 0;
    for (int j = 0; j < n_jobs; j++) {
        const cs_batch_job &jb = jobs_host[j];
        if ((jb.mode == cs::MODE_SHORTEST || jb.mode == cs::MODE_BOTH) && jb.compute_closeness && jb.n_sources > 0) {
            max_n = std::max(max_n, jb.g.n_bound);
            n_pref++;
        }
    }
    if (n_pref > 0) {
        const int sms = std::max(1, sm_count());
        const int gy = std::min(n_pref, 65535);
        const int gx = std::max(1, std::min((max_n + 255) / 256, std::max(1, sms * 8 / gy)));
        cs::batch_prefix_kernel<<<dim3(gx, gy), 256, 0, stream>>>(jobs_dev, n_jobs);
        g_counters[3]++;
        e = cudaGetLastError();
        if (e != cudaSuccess) return cuda_fail(e, "batch_prefix_kernel launch");
    }
    return CS_OK;
}

cs_status cs_batch_status(void *ws, int64_t *n_overflowed, int64_t *sources_done, void *stream) {
    if (!ws) return fail(CS_ERR_ARG, "workspace is NULL");
    cs::WsHeader h;
    cudaError_t e = cs::read_header((const cs::WsHeader *)ws, h, (cudaStream_t)stream, true);
    if (e != cudaSuccess) return cuda_fail(e, "batch status");
    if (n_overflowed) *n_overflowed = (int64_t)h.n_failed;
    if (sources_done) *sources_done = (int64_t)h.sources_done;
    g_counters[0] = (long long)h.sources_done;
    g_counters[1] = (long long)h.edges_relaxed;
    g_counters[2] = (long long)h.nodes_settled;
    if (h.err != 0u) return fail((cs_status)h.err, "device-side check failed (code " + std::to_string(h.err) + ")");
    return CS_OK;
}

cs_status cs_batch_failed(void *ws, const cs_plan *plan, int32_t *items_host, int32_t max_items, int64_t *n_failed,
                          void *stream) {
    if (!ws || !plan || !n_failed) return fail(CS_ERR_ARG, "workspace/plan/n_failed is NULL");
    cs::WsHeader h;
    cudaStream_t st = (cudaStream_t)stream;
    cudaError_t e = cs::read_header((const cs::WsHeader *)ws, h, st, true);
    if (e != cudaSuccess) return cuda_fail(e, "batch failed list");
    const Layout lay = layout(std::max(1, plan->n_bound), plan->n_slots, plan->cap, 1, plan->lanes);
    const int64_t nf = (int64_t)h.n_failed;
    *n_failed = nf;
    if (nf > (int64_t)lay.fail_cap) return fail(CS_ERR_CAPACITY, "more overflowed items than the failed list holds");
    const int64_t c = std::min<int64_t>(nf, std::max(0, max_items));
    if (c > 0 && items_host) {
        e = cudaMemcpyAsync(items_host, (char *)ws + lay.failed_off, sizeof(int32_t) * (size_t)c, cudaMemcpyDeviceToHost,
                            st);
        if (e == cudaSuccess) e = cudaStreamSynchronize(st);
        if (e != cudaSuccess) return cuda_fail(e, "batch failed list");
    }
    return CS_OK;
}

}  // extern "C"

extern "C" cs_status cs_source_weights(const int32_t *sources_dev, int64_t n_sources, const float *node_w_dev,
                                        int32_t n_bound, float *src_wt_dev, uint8_t *eligible_dev, void *stream) {
    if (n_bound <= 0 || !node_w_dev || !src_wt_dev || !eligible_dev || (n_sources > 0 && !sources_dev))
        return fail(CS_ERR_ARG, "source weights: bad arguments");
    cudaStream_t st = (cudaStream_t)stream;
    const int sms = std::max(1, sm_count());
    const int b0 = std::max(1, std::min((n_bound + 255) / 256, sms * 4));
    cs::source_weights_kernel<<<b0, 256, 0, st>>>(sources_dev, n_sources, node_w_dev, n_bound, src_wt_dev, eligible_dev,
                                                  0);
    if (n_sources > 0) {
        const int b1 = (int)std::max<long long>(1, std::min<long long>((n_sources + 255) / 256, sms * 4));
        cs::source_weights_kernel<<<b1, 256, 0, st>>>(sources_dev, n_sources, node_w_dev, n_bound, src_wt_dev,
                                                      eligible_dev, 1);
    }
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? CS_OK : cuda_fail(e, "source_weights_kernel launch");
}

namespace cs {
__global__ void seed_check_kernel(const float *w, const float *beta, const float *cost, double *out, long long n) {
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x)
        out[t] = seed_exp(w[t], beta[t], cost[t]);
}
}  // namespace cs

namespace {
void seed_table_here(cudaStream_t s) { cs::seed_table_kernel<<<(cs::SEED_TAB + 255) / 256, 256, 0, s>>>(); }
}  // namespace

extern "C" cs_status cs_debug_seed_exp(const float *w_dev, const float *beta_dev, const float *cost_dev,
                                       double *out_dev, int64_t n, void *stream) {
    if (n < 0 || (n > 0 && (!w_dev || !beta_dev || !cost_dev || !out_dev))) return fail(CS_ERR_ARG, "seed check: bad arguments");
    cudaStream_t st = (cudaStream_t)stream;
    cs_status rc = launch_seed_table(st, seed_table_here);
    if (rc != CS_OK) return rc;
    if (n == 0) return CS_OK;
    const int blocks = (int)std::min<long long>((n + 255) / 256, 4096);
    cs::seed_check_kernel<<<blocks, 256, 0, st>>>(w_dev, beta_dev, cost_dev, out_dev, n);
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? CS_OK : cuda_fail(e, "seed_check_kernel launch");
}

// Live progress: the completed-source count the kernels keep in the workspace header, copied on a
// stream of its own (so it does not wait for the call's kernels) into pinned memory of this thread.
extern "C" cs_status cs_workspace_progress(const void *workspace_dev, int64_t *sources_done) {
    if (!workspace_dev || !sources_done) return fail(CS_ERR_ARG, "workspace/sources_done is NULL");
    thread_local unsigned long long *pinned = nullptr;
    thread_local cudaStream_t side = nullptr;
    cudaError_t e = cudaSuccess;
    if (!pinned) e = cudaHostAlloc((void **)&pinned, sizeof(unsigned long long), cudaHostAllocDefault);
    if (e == cudaSuccess && !side) e = cudaStreamCreateWithFlags(&side, cudaStreamNonBlocking);
    if (e != cudaSuccess) return cuda_fail(e, "progress buffer");
    const cs::WsHeader *h = (const cs::WsHeader *)workspace_dev;
    e = cudaMemcpyAsync(pinned, &h->pad[cs::PROGRESS_SLOT], sizeof(unsigned long long), cudaMemcpyDeviceToHost, side);
    if (e == cudaSuccess) e = cudaStreamSynchronize(side);
    if (e != cudaSuccess) return cuda_fail(e, "progress read");
    *sources_done = (int64_t)*pinned;
    return CS_OK;
}

extern "C" cs_status cs_abi_sizes(int32_t *out, int32_t n) {
    // sizes of the public structs, for bindings to check their layouts against
    const int32_t v[7] = {(int32_t)sizeof(cs_primal_graph), (int32_t)sizeof(cs_dual_graph), (int32_t)sizeof(cs_query),
                          (int32_t)sizeof(cs_plan),         (int32_t)sizeof(cs_outputs),    (int32_t)sizeof(cs_batch_job),
                          (int32_t)sizeof(cs_dual_batch_job)};
    if (!out) return fail(CS_ERR_ARG, "out is NULL");
    for (int i = 0; i < n && i < 7; i++) out[i] = v[i];
    return CS_OK;
}
