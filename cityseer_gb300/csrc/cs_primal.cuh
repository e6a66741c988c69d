// cs_primal.cuh -- GB300 kernels for shortest-path node centrality, OD-weighted betweenness, segment
// centrality and shortest-path trees (isochrones) on the primal graph.
//
// Reference behaviour (cityseer-api v4.24.0):
//   centrality_shortest        rust/src/centrality.rs:1624-1874
//   dijkstra_brandes_shortest  rust/src/centrality.rs:1344-1494
//   circuit_ranks_from_traversal rust/src/centrality.rs:470-526
//   brandes_backprop_with_beta rust/src/centrality.rs:823-873
//   betweenness_od_shortest    rust/src/centrality.rs:2419-2540
//   segment_centrality         rust/src/centrality.rs:2134-2407
//   dijkstra_tree_segment      rust/src/centrality.rs:1524-1611
//   dijkstra_tree_shortest_inner rust/src/centrality.rs:1141-1200
//
// Design (one warp per source; persistent warps pull sources from a work counter, and in the
// block-synchronous form the warps of a block run each phase together):
//  1. Bounded label-correcting search ("near-far" banded Bellman-Ford) from the source over
//     reversed edges.  Every relaxation is fl(d[u] + w) with w >= 0, so the least fixpoint is
//     unique and bit-identical to the reference's heap Dijkstra whatever the relaxation order.
//  2. Warp sort of the reached set by distance (cs_sort.cuh: distance buckets, or LSD radix): the
//     reference's settle order.
//  3. Replay, per reached node and in parallel, of the exact sequence of candidate offers the
//     heap Dijkstra would make to it (offering neighbours in settle order), through the
//     reference's Phase-1 tie rules (and Phase 2 when tolerance > 1e-4).  This reproduces its
//     multi-predecessor lists; sigma follows chunk by chunk in settle order in the same pass.
//  4. Closeness into target rows and circuit ranks; one backward Brandes sweep carrying all K
//     thresholds (a state beyond threshold k contributes nothing to lane k, so one sweep equals
//     the reference's K sweeps).
// Per-slot scratch: dense dist/aux arrays over node_bound (reset touched entries only) plus
// compact per-reached-node arrays of capacity `cap`; sources that overflow `cap` are redone inside
// the same API call at 4x the capacity, then 4x again, up to cap = node_bound.
//
// The kernels are templates, instantiated per mode in cs_primal_shortest.cu, cs_primal_segment.cu,
// cs_primal_tree.cu and cs_primal_batch.cu (compiled in parallel); cs_primal.cu holds the host side.
#pragma once
#include "cs_common.cuh"
#include "cs_seed.cuh"
#include "cs_sort.cuh"

namespace cs {

struct SlotPtrs {
    float *dist;
    uint32_t *aux;
    int32_t *rl;
    uint2 *qa, *qb, *qf;  // (node, dist bits) entries, capacity 2 * cap
    uint32_t *kb;
    int32_t *vb;
    int32_t *ord;
    float *sd;
    double *sig;
    uint8_t *np;
    int32_t *pr;
    double *dl;
    float *fa, *fb;
    int32_t *eb;
};

__host__ __device__ inline size_t al256(size_t x) { return (x + 255) & ~size_t(255); }

__host__ __device__ inline size_t compact_bytes(size_t cap, int P, int L) {
    size_t b = 0;
    b += 4 * al256(cap * 4);      // rl kb vb ord
    b += 3 * al256(cap * 16);     // qa qb qf: 2 * cap entries of 8 bytes
    b += al256(cap * 4);          // sd
    b += al256(cap * 8);          // sig
    b += al256(cap);              // np
    b += al256(cap * 4 * (size_t)P);  // pr
    b += al256(cap * 8 * (size_t)L);  // dl
    b += 3 * al256(cap * 4);      // fa fb eb
    return b;
}

__host__ __device__ inline SlotPtrs slot_ptrs(char *dense, size_t dense_stride, char *compact, size_t cap, int P,
                                              int L, int slot, int n_bound) {
    SlotPtrs s;
    char *d = dense + dense_stride * (size_t)slot;
    s.dist = (float *)d;
    s.aux = (uint32_t *)(d + al256((size_t)n_bound * 4));
    char *c = compact + compact_bytes(cap, P, L) * (size_t)slot;
    size_t o = 0;
    s.rl = (int32_t *)(c + o); o += al256(cap * 4);
    s.qa = (uint2 *)(c + o); o += al256(cap * 16);
    s.qb = (uint2 *)(c + o); o += al256(cap * 16);
    s.qf = (uint2 *)(c + o); o += al256(cap * 16);
    s.kb = (uint32_t *)(c + o); o += al256(cap * 4);
    s.vb = (int32_t *)(c + o); o += al256(cap * 4);
    s.ord = (int32_t *)(c + o); o += al256(cap * 4);
    s.sd = (float *)(c + o); o += al256(cap * 4);
    s.sig = (double *)(c + o); o += al256(cap * 8);
    s.np = (uint8_t *)(c + o); o += al256(cap);
    s.pr = (int32_t *)(c + o); o += al256(cap * 4 * (size_t)P);
    s.dl = (double *)(c + o); o += al256(cap * 8 * (size_t)L);
    s.fa = (float *)(c + o); o += al256(cap * 4);
    s.fb = (float *)(c + o); o += al256(cap * 4);
    s.eb = (int32_t *)(c + o); o += al256(cap * 4);
    return s;
}

// BOTH: batched jobs only.  OD: betweenness seeded by an origin-destination matrix.
// ACCESS: accessibility sums over data assigned to the reached nodes.
enum Mode { MODE_SHORTEST = 0, MODE_SEGMENT = 1, MODE_TREE = 2, MODE_BOTH = 3, MODE_OD = 4, MODE_ACCESS = 5 };

struct PrimalParams {
    cs_primal_graph g;
    int32_t k;
    float dk[MAXK];
    float beta[MAXK];
    float inb[MAXK];  // 1 / -beta
    float maxsec;
    float speed;
    float tol;
    float delta;
    int32_t closeness, betweenness, track_reach;
    const int32_t *src_list;
    int64_t n_src;
    const float *src_wt;
    const uint8_t *eligible;
    double *out;
    double *bucket;  // [3][K][N] threshold-bucketed closeness terms (density, farness, harmonic)
    double *out2;    // MODE_BOTH: segment rows [4][K][N] (out holds the shortest rows)
    uint32_t *reach;
    WsHeader *hdr;
    int32_t *failed;  // [fail_cap] indices (into src_list) of sources that overflowed
    int32_t fail_cap;
    char *dense;
    size_t dense_stride;
    char *compact;
    int32_t cap, P, L;
    int32_t n_slots;
    int32_t rerun;
    const int32_t *remap;  // rerun: indices into src_list of the sources to redo
    const unsigned *n_remap;  // batched rerun: how many there are, where the host has not read it (else n_src)
    int32_t mode;
    int32_t row_cap;
    int32_t *t_count, *t_node, *t_pred;
    float *t_agg;
    // MODE_OD: per origin node, its row [od_ptr[o], od_ptr[o+1]) of destinations (ascending) and weights
    const int32_t *od_ptr, *od_dst;
    const float *od_w;
    int32_t radix_sort;  // settle-order sort: 0 distance buckets, 1 LSD radix
    // MODE_ACCESS: the data map (cs_data_map) and the per-class rows
    cs_data_map dm;
    float mcw[MAXK];   // max curve weights (clip_wts_curve)
    float max_dist;    // the largest distance threshold (metres)
    double *acc_unw, *acc_wt;  // [n_classes][K][n_bound]
    uint32_t *acc_near;        // [n_classes][n_bound] f32 bits of the nearest distance
};

// ------------------------------------------------------------------------------------------
// 1. Banded label-correcting search.  Returns R (reached count incl. source) or -1 on overflow.
//    Queues hold (node, distance-at-push) entries with lazy deletion: an entry is live only while
//    its distance still equals the node's, so no flag atomics are needed to de-duplicate.
// ------------------------------------------------------------------------------------------
// Edges per node loaded together for a kernel's largest out-degree PM; higher degrees loop.
__host__ __device__ constexpr int deg_fast(int pm) { return pm < 8 ? pm : 8; }
// Backward sweep: predecessors per lane kept in shared memory (row and f64 factor); a node's
// further predecessors (high-degree graphs) are read from the per-source scratch.
constexpr int BW_COLS = 8;
__host__ __device__ constexpr int bw_cols(int pm) { return pm < BW_COLS ? pm : BW_COLS; }

__device__ __forceinline__ void push_entries(bool first, int route, int v, float c, int &R, int &nnext, int &nfar,
                                             int cap, int qcap, const SlotPtrs &s, uint2 *nxt, unsigned lt) {
    const unsigned mf = __ballot_sync(FULL, first);
    const unsigned mn = __ballot_sync(FULL, route == 1);
    const unsigned mr = __ballot_sync(FULL, route == 2);
    if (first) {
        const int q = R + __popc(mf & lt);
        if (q < cap) s.rl[q] = v;
    }
    if (route == 1) {
        const int q = nnext + __popc(mn & lt);
        if (q < qcap) nxt[q] = make_uint2((unsigned)v, __float_as_uint(c));
    }
    if (route == 2) {
        const int q = nfar + __popc(mr & lt);
        if (q < qcap) s.qf[q] = make_uint2((unsigned)v, __float_as_uint(c));
    }
    R += __popc(mf);
    nnext += __popc(mn);
    nfar += __popc(mr);
}

#ifndef CS_PHASE_INLINE
#define CS_PHASE_INLINE
#endif

// dmax: an upper bound of every reached distance (the last band's end, at most the cutoff).
template <int DEG_FAST>
CS_PHASE_INLINE __device__ int warp_search(const PrimalParams &p, const SlotPtrs &s, int src, long long &relaxed,
                                           float &dmax) {
    const int lane = lane_id();
    const unsigned lt = lanemask_lt();
    const int cap = p.cap;
    const int qcap = 2 * cap;
    const int32_t *__restrict__ in_ptr = p.g.in_ptr_dev;
    const int32_t *__restrict__ in_nb = p.g.in_nb_dev;
    const float *__restrict__ in_w = p.g.in_w_dev;
    const float maxsec = p.maxsec, delta = p.delta;  // in registers (p may live in shared memory)
    float *dist = s.dist;
    if (lane == 0) {
        dist[src] = 0.0f;
        s.rl[0] = src;
        s.qa[0] = make_uint2((unsigned)src, 0u);
    }
    __syncwarp();
    int R = 1, nnear = 1, nfar = 0;
    uint2 *cur = s.qa, *nxt = s.qb;
    float T = delta;
    float fmn = __int_as_float(INF_BITS);  // this lane's smallest distance queued far since the last split
    bool overflow = false;
    while (true) {
        while (nnear > 0) {
            int nnext = 0;
            for (int base = 0; base < nnear; base += 32) {
                const int i = base + lane;
                uint2 ent = make_uint2(0u, 0u);
                if (i < nnear) ent = cur[i];
                const int u = (int)ent.x;
                const float du = (i < nnear) ? __ldcg(&dist[u]) : 0.0f;
                const bool live = (i < nnear) && (__float_as_uint(du) == ent.y);
                const int beg = live ? __ldg(&in_ptr[u]) : 0;
                const int deg = live ? __ldg(&in_ptr[u + 1]) - beg : 0;
                relaxed += deg;
                // load this node's first DEG_FAST edges together, then issue their atomics together
                int vv[DEG_FAST];
                float cc[DEG_FAST];
                int old[DEG_FAST];
#pragma unroll
                for (int j = 0; j < DEG_FAST; j++) {
                    vv[j] = u;
                    cc[j] = 0.0f;
                    if (j < deg) {
                        vv[j] = __ldg(&in_nb[beg + j]);
                        cc[j] = fadd(du, __ldg(&in_w[beg + j]));
                    }
                }
#pragma unroll
                for (int j = 0; j < DEG_FAST; j++) {
                    old[j] = 0;
                    if (j < deg && vv[j] != u && cc[j] <= maxsec)
                        old[j] = atomicMin((int *)&dist[vv[j]], __float_as_int(cc[j]));
                }
                const int maxdeg = warp_max_i(deg);
#pragma unroll
                for (int j = 0; j < DEG_FAST; j++) {
                    if (j >= maxdeg) break;
                    const bool imp = (j < deg) && vv[j] != u && cc[j] <= maxsec && __float_as_int(cc[j]) < old[j];
                    const int route = imp ? (cc[j] < T ? 1 : 2) : 0;
                    if (route == 2) fmn = fminf(fmn, cc[j]);
                    push_entries(imp && old[j] == INF_BITS, route, vv[j], cc[j], R, nnext, nfar, cap, qcap, s, nxt,
                                 lt);
                }
                // rare high-degree nodes: remaining edges one at a time
                for (int j = DEG_FAST; j < maxdeg; j++) {
                    int v = u;
                    float c = 0.0f;
                    bool imp = false, first = false;
                    if (j < deg) {
                        v = __ldg(&in_nb[beg + j]);
                        c = fadd(du, __ldg(&in_w[beg + j]));
                        if (v != u && c <= maxsec) {
                            const int o = atomicMin((int *)&dist[v], __float_as_int(c));
                            imp = __float_as_int(c) < o;
                            first = imp && o == INF_BITS;
                        }
                    }
                    const int route = imp ? (c < T ? 1 : 2) : 0;
                    if (route == 2) fmn = fminf(fmn, c);
                    push_entries(first, route, v, c, R, nnext, nfar, cap, qcap, s, nxt, lt);
                }
            }
            __syncwarp();
            if (R > cap || nnext > qcap || nfar > qcap) { overflow = true; break; }
            uint2 *t = cur; cur = nxt; nxt = t;
            nnear = nnext;
        }
        if (overflow) break;
        if (nfar == 0) break;
        // Next band: [mn, mn + delta) from the smallest queued far distance (the lanes' minima over
        // the pushes and over the entries the last split kept), strictly above mn even when delta is
        // below mn's ulp.  One streaming pass over the far queue, by the queued distances: entries
        // that died since they were queued are dropped when their band runs.
        const float mn = warp_min_f(fmn);
        T = fmaxf(fadd(mn, delta), __int_as_float(__float_as_int(mn) + 1));
        fmn = __int_as_float(INF_BITS);
        int nn = 0, nf2 = 0;
        for (int base = 0; base < nfar; base += 32) {
            const int i = base + lane;
            const bool act = i < nfar;
            const uint2 ent = act ? s.qf[i] : make_uint2(0u, 0u);
            const float d = __uint_as_float(ent.y);
            const bool tonear = act && d < T;
            const bool keep = act && !tonear;
            if (keep) fmn = fminf(fmn, d);
            const unsigned mt = __ballot_sync(FULL, tonear);
            const unsigned mk = __ballot_sync(FULL, keep);
            __syncwarp();
            if (tonear) cur[nn + __popc(mt & lt)] = ent;
            if (keep) s.qf[nf2 + __popc(mk & lt)] = ent;
            nn += __popc(mt);
            nf2 += __popc(mk);
            __syncwarp();
        }
        nnear = nn;
        nfar = nf2;
    }
    __syncwarp();
    dmax = fminf(T, maxsec);
    if (overflow) return -1;  // the slot's dense state is dirty: the caller resets it
    return R;
}

// ------------------------------------------------------------------------------------------
// 2. Warp LSD radix sort of the reached set by distance (cs_sort.cuh): the settle order.
// ------------------------------------------------------------------------------------------
// The distance-bucket sort (3 passes) unless p.radix_sort selects the 4-pass LSD radix sort; both
// give the same order (ascending distance, ties in reached-list order).
__device__ __forceinline__ void warp_sort(const PrimalParams &p, const SlotPtrs &s, int R, float dmax, uint32_t *hist) {
    const float *dist = s.dist;
    auto key_of = [dist](int v) { return (uint32_t)__float_as_int(__ldcg(&dist[v])); };
    if (p.radix_sort) warp_radix_sort(R, s.rl, key_of, s.kb, s.vb, (uint32_t *)s.sd, s.ord, hist);
    else warp_bucket_sort(R, dmax, s.rl, key_of, s.kb, s.vb, (uint32_t *)s.sd, s.ord, hist);
}

// ------------------------------------------------------------------------------------------
// 3. Offer replay for the node at sorted position i.  Everything per node stays in registers:
//    the kernel is instantiated for a maximum out-degree PM (8 for street graphs, 32 otherwise)
//    and all per-edge arrays are fixed-size and fully unrolled.
// ------------------------------------------------------------------------------------------
__device__ __forceinline__ float route_cost(float secs, float speed) { return fmul(secs, speed); }

// Reached out-neighbours of v: slot j holds out-CSR edge beg + j (pos -1: unreached or self loop).
template <int PM>
struct Nb {
    int pos[PM];
    float d[PM];
    int beg, deg;
};

template <int PM>
__device__ __forceinline__ void load_nb(const PrimalParams &p, const SlotPtrs &s, int v, int R, Nb<PM> &nb,
                                        bool &bad) {
    nb.beg = __ldg(&p.g.out_ptr_dev[v]);
    nb.deg = min(__ldg(&p.g.out_ptr_dev[v + 1]) - nb.beg, PM);
    int uu[PM];
    uint32_t aa[PM];
#pragma unroll
    for (int j = 0; j < PM; j++) uu[j] = (j < nb.deg) ? __ldg(&p.g.out_to_dev[nb.beg + j]) : v;
#pragma unroll
    for (int j = 0; j < PM; j++) aa[j] = (uu[j] != v) ? s.aux[uu[j]] : 0u;
#pragma unroll
    for (int j = 0; j < PM; j++) {
        const bool ok = aa[j] != 0u && aa[j] <= (uint32_t)R;
        if (aa[j] > (uint32_t)R) bad = true;  // scratch not clean: refuse to index
        nb.pos[j] = ok ? (int)aa[j] - 1 : -1;
        nb.d[j] = ok ? s.sd[aa[j] - 1] : 0.0f;
    }
}

// Offers to the node at position i are the reached neighbours settled before it, taken in order of
// the offering node's position (parallel edges keep list order).  Candidate seconds per slot:
template <int PM>
__device__ __forceinline__ unsigned offer_cands(const PrimalParams &p, const Nb<PM> &nb, int i, float *c) {
    unsigned todo = 0;
#pragma unroll
    for (int j = 0; j < PM; j++) {
        const bool off = nb.pos[j] >= 0 && nb.pos[j] < i;
        c[j] = off ? fadd(nb.d[j], __ldg(&p.g.out_w_dev[nb.beg + j])) : 0.0f;
        if (off) todo |= 1u << j;
    }
    return todo;
}

// next offer in settle order: lowest position, then lowest slot
template <int PM>
__device__ __forceinline__ int next_offer(const Nb<PM> &nb, unsigned todo, const float *c, int &bp, float &bc) {
    int best = -1;
    bp = 0x7fffffff;
    bc = 0.0f;
#pragma unroll
    for (int j = 0; j < PM; j++) {
        if (((todo >> j) & 1u) && nb.pos[j] < bp) {
            bp = nb.pos[j];
            best = j;
            bc = c[j];
        }
    }
    return best;
}

template <int PM>
__device__ __forceinline__ bool pos_in(const Nb<PM> &nb, unsigned mask, int pos) {
    bool has = false;
#pragma unroll
    for (int j = 0; j < PM; j++) has |= ((mask >> j) & 1u) && nb.pos[j] == pos;
    return has;
}

// Phase-1 (+ Phase-2) predecessor replay, rust/src/centrality.rs:1413-1437 and 1444-1483.
// Returns the predecessor slots as a bit mask; ok = false if the replayed distance does not
// reproduce the searched one (internal inconsistency).
template <int PM>
__device__ __forceinline__ unsigned replay_brandes(const PrimalParams &p, const Nb<PM> &nb, int i, float dv,
                                                   bool &ok) {
    const float one_plus = 1.0f + TIE_EPSILON;
    const float one_minus = 1.0f - TIE_EPSILON;
    float c[PM];
    const unsigned todo = offer_cands<PM>(p, nb, i, c);
    unsigned t = todo, pm = 0u;
    float cur = __int_as_float(INF_BITS);
    while (t) {
        int bp;
        float bc;
        const int best = next_offer<PM>(nb, t, c, bp, bc);
        t &= ~(1u << best);
        if (bc > p.maxsec) continue;
        const bool improved = bc < cur;
        const bool tied = bc <= fmul(cur, one_plus);
        if (improved) {
            if (bc < fmul(cur, one_minus)) pm = 0u;
            pm |= 1u << best;
            cur = bc;
        } else if (tied && !pos_in<PM>(nb, pm, bp)) {
            pm |= 1u << best;
        }
    }
    ok = __float_as_int(cur) == __float_as_int(dv);
    if (p.tol > TIE_EPSILON) {
        const float lim = fmul(dv, 1.0f + p.tol);
        pm = 0u;
        t = todo;
        while (t) {
            int bp;
            float bc;
            const int best = next_offer<PM>(nb, t, c, bp, bc);
            t &= ~(1u << best);
            if (bc <= lim && !pos_in<PM>(nb, pm, bp)) pm |= 1u << best;
        }
    }
    return pm;
}

// Strict-< single predecessor (dijkstra_tree_* / dijkstra_tree_segment): the first offer in settle
// order that reaches the final distance.  Returns its slot or -1; ok as above.
template <int PM>
__device__ __forceinline__ int replay_first_min(const PrimalParams &p, const Nb<PM> &nb, int i, float dv, bool &ok) {
    float c[PM];
    unsigned t = offer_cands<PM>(p, nb, i, c);
    float cur = __int_as_float(INF_BITS);
    int pick = -1;
    while (t) {
        int bp;
        float bc;
        const int best = next_offer<PM>(nb, t, c, bp, bc);
        t &= ~(1u << best);
        if (bc > p.maxsec) continue;
        if (bc < cur) {
            cur = bc;
            pick = best;
        }
    }
    ok = __float_as_int(cur) == __float_as_int(dv);
    return pick;
}

// ------------------------------------------------------------------------------------------
// 4a. Shortest-path centrality for one source (after search and sort).
// ------------------------------------------------------------------------------------------
// Per-phase cycle counters live in the warp's shared-memory row (lane 0 adds), not in registers.
__device__ __forceinline__ void phase_mark(long long *ph, int idx, long long &t) {
    const long long now = clock64();
    if (lane_id() == 0) ph[idx] += now - t;
    t = now;
}

// first threshold index k with c <= dk[k] (thresholds strictly increasing), K if none
__device__ __forceinline__ int first_k(const PrimalParams &p, float c) {
    int k = 0;
    while (k < p.k && !(c <= p.dk[k])) k++;
    return k;
}

// Dependency lanes of the backward sweep: the node at settle position i holds the lanes of the
// thresholds it lies within (k >= k0(i)), plain and beta-weighted interleaved, packed in settle
// order.  Positions are sorted by cost, so k0 steps up at the boundaries nk[k] (positions with cost
// <= d_k) and the offsets follow from them: lane (i, k, b) sits at lane_index(i) + 2 k + b.
// nk[] and cum[] (cum[k] = lanes held by the positions below nk[k - 1]) are the warp's shared rows.
__device__ __forceinline__ int lane_index(int i, int K, const int *nk, const int *cum) {
    int k0 = 0;
    while (k0 < K && i >= nk[k0]) k0++;
    const int lo = k0 ? nk[k0 - 1] : 0;
    return 2 * (cum[k0] + (i - lo) * (K - k0)) - 2 * k0;
}

// predecessor positions of the node at position i, in registers
template <int PM>
__device__ __forceinline__ int load_preds(const SlotPtrs &s, int i, int P, int *pl) {
    const int np = s.np[i];
#pragma unroll
    for (int r = 0; r < PM; r++) pl[r] = (r < np) ? s.pr[(size_t)i * P + r] : 0;
    return np;
}

// Sources a block of nw warps claims at a time: a whole round of its warps, or fewer when the launch has
// fewer sources than warps, so that they spread over all blocks (and SMs) instead of filling the first.
__device__ __forceinline__ int block_claim(int nw, long long n) {
    return max(0, min(nw, (int)min((n + gridDim.x - 1) / (long long)gridDim.x, 32ll)));
}

// Phase barrier of the block-synchronous forms: GW warps (a whole 8-warp block: __syncthreads;
// 4: a named barrier per half block) meet at the end of each phase.  GW = 0: no barrier.
template <int GW>
__device__ __forceinline__ void phase_barrier() {
    if constexpr (GW == 8) {
        __syncthreads();
    } else if constexpr (GW > 0) {
        asm volatile("bar.sync %0, %1;" ::"r"(1 + (int)(threadIdx.x >> 5) / GW), "r"(GW * 32) : "memory");
    }
}

// With SYNC, every warp of the block runs each phase together (a block barrier ends each phase,
// and a warp without a source runs the phases with R = 0), so at any time a block's warps fetch one
// phase's code; there is no early return in that form.
// Trip weight of the pair (src, v) in the origin-destination rows, 0 when the pair has none.
__device__ __forceinline__ float od_weight(const PrimalParams &p, int src, int v) {
    int lo = __ldg(&p.od_ptr[src]);
    const int end = __ldg(&p.od_ptr[src + 1]);
    int hi = end;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (__ldg(&p.od_dst[mid]) < v) lo = mid + 1;
        else hi = mid;
    }
    return (lo < end && __ldg(&p.od_dst[lo]) == v) ? __ldg(&p.od_w[lo]) : 0.0f;
}

// OD: betweenness only, seeded per pair by the origin-destination weights instead of the 0.5 / 1.0
// pair counts (rust/src/centrality.rs:2495-2507), source weight 1, written to rows 0 and 1.
template <int PM, int SYNC, bool OD = false>
CS_PHASE_INLINE __device__ void shortest_accumulate(const PrimalParams &p, const SlotPtrs &s, int src, int R, long long *ph,
                                    int *cnt, int *bw_pl, double *bw_fr) {
    const int lane = lane_id();
    bool failed = false;
    long long tph = clock64();
    const int K = p.k;
    const int P = p.P;
    const int N = p.g.n_bound;
    const float wt = OD ? 1.0f : __ldg(&p.src_wt[src]);
    const float cycles_wt = OD ? 0.0f : wt / __ldg(&p.g.node_w_dev[src]);
    const bool closeness = !OD && p.closeness;
    // cnt[0..K): nodes whose first qualifying threshold is k; cnt[MAXK..MAXK+K): same for edges;
    // cnt[2 MAXK..): nk, the positions with cost <= d_k; cnt[3 MAXK..): cum, lanes below nk[k - 1]
    for (int q = lane; q < 2 * MAXK; q += 32) cnt[q] = 0;
    int *nk = cnt + 2 * MAXK, *cum = cnt + 3 * MAXK;
    if (lane < K) {
        int lo = 0, hi = R;  // first position whose cost exceeds d_k
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (route_cost(s.sd[mid], p.speed) <= p.dk[lane]) lo = mid + 1;
            else hi = mid;
        }
        nk[lane] = lo;
    }
    __syncwarp();
    if (lane == 0) {
        int acc = 0, prev = 0;
        for (int k = 0; k < K; k++) {
            cum[k] = acc;
            acc += (nk[k] - prev) * (K - k);
            prev = nk[k];
        }
        cum[K] = acc;
    }
    __syncwarp();
    // --- one pass over out-edges in settle order, 32 nodes at a time: circuit-rank counts, the
    // predecessor replay and, with betweenness, sigma (f64 path counts, as the reference's
    // BrandesTraversalState.sigma) of the chunk: a node is ready once its in-chunk predecessors are
    // done.  The same pass zeroes each node's dependency lanes for the backward sweep.
    bool bad = false;
    double *sig = s.sig;
    double *dl = s.dl;  // dependency lanes, packed (lane_index)
    for (int base = 0; base < R; base += 32) {
        const int i = base + lane;
        const bool act = i < R;
        unsigned pm = 0u;
        Nb<PM> nb;
        if (act) {
            const int v = s.ord[i];
            const float dv = s.sd[i];
            const float cv = route_cost(dv, p.speed);
            const int k0v = first_k(p, cv);
            if (k0v < K) atomicAdd(&cnt[k0v], 1);
            load_nb<PM>(p, s, v, R, nb, bad);
            if (closeness) {
#pragma unroll
                for (int j = 0; j < PM; j++) {
                    if (nb.pos[j] < 0 || !__ldg(&p.g.out_cnt_dev[nb.beg + j])) continue;
                    const float ec = fmaxf(cv, route_cost(nb.d[j], p.speed));
                    const int k0e = first_k(p, ec);
                    if (k0e < K) atomicAdd(&cnt[MAXK + k0e], 1);
                }
            }
            if (p.betweenness) {
                if (i == 0) {
                    s.np[0] = 0;
                } else {
                    bool ok = true;
                    pm = replay_brandes<PM>(p, nb, i, dv, ok);
                    if (!ok) { bad = true; pm = 0u; }
                    int r = 0;
#pragma unroll
                    for (int j = 0; j < PM; j++)
                        if ((pm >> j) & 1u) s.pr[(size_t)i * P + r++] = nb.pos[j];
                    s.np[i] = (uint8_t)r;
                }
            }
        }
        if (!p.betweenness || failed) continue;  // uniform across the warp
        unsigned blk = 0u;  // in-chunk predecessors, as lane bits
#pragma unroll
        for (int j = 0; j < PM; j++)
            if (((pm >> j) & 1u) && nb.pos[j] >= base) blk |= 1u << (nb.pos[j] - base);
        unsigned done = __ballot_sync(FULL, !act);
        bool mine = !act;
        int guard = 0;
        while (done != FULL) {
            const bool ready = !mine && ((blk & ~done) == 0u);
            if (ready) {
                double sg = (i == 0) ? 1.0 : 0.0;
                const unsigned rest = pm & (pm - 1u);
#pragma unroll
                for (int j = 0; j < PM; j++)
                    if (((pm & ~rest) >> j) & 1u) sg = sig[nb.pos[j]];  // the first predecessor: nothing to add to
                if (rest) {
#pragma unroll
                    for (int j = 0; j < PM; j++)
                        if ((rest >> j) & 1u) sg = __dadd_rn(sg, sig[nb.pos[j]]);
                }
                sig[i] = sg;
                const int li0 = lane_index(i, K, nk, cum);
                for (int k = first_k(p, route_cost(s.sd[i], p.speed)); k < K; k++) {
                    dl[li0 + 2 * k] = 0.0;
                    dl[li0 + 2 * k + 1] = 0.0;
                }
                mine = true;
            }
            __syncwarp();
            done |= __ballot_sync(FULL, ready);
            if (++guard > 64) break;
        }
        if (done != FULL) {
            if (lane == 0) raise_err(p.hdr, CS_ERR_INTERNAL, 2);
            failed = true;
        }
    }
    if (__any_sync(FULL, bad)) {
        if (lane == 0) raise_err(p.hdr, CS_ERR_INTERNAL, 1);
    }
    __syncwarp();
    phase_barrier<SYNC>();
    phase_mark(ph, 2, tph);
    // --- closeness (rust/src/centrality.rs:1733-1780).  Density, farness and harmonic terms do not
    // depend on the threshold: they go once into the bucket of the first qualifying threshold and a
    // prefix over thresholds after the launch completes them.  Cycles and beta terms are per k.
    if (closeness) {
        // per-threshold circuit-rank weights, computed by lane 0 into the (now free) edge-count half
        // of the warp's shared counters
        float *rankw = (float *)(cnt + MAXK);
        if (lane == 0) {
            long long nc = 0, ec = 0;
            for (int k = 0; k < K; k++) {
                nc += cnt[k];
                ec += cnt[MAXK + k];
                const long long r = ec - nc + 1;
                const float rank = (nc == 0) ? 0.0f : (float)(r > 0 ? r : 0);
                rankw[k] = fmul(rank, cycles_wt);
                if (p.track_reach && nc > 1) atomicAdd(&p.reach[k], (unsigned)(nc - 1));
            }
        }
        __syncwarp();
        const double wt_d = f2d(wt);
        const size_t KN = (size_t)K * N;
        for (int i = 1 + lane; i < R; i += 32) {
            const int t = s.ord[i];
            const float c = route_cost(s.sd[i], p.speed);
            const int k0 = first_k(p, c);
            if (k0 >= K) continue;
            double *bk = p.bucket + (size_t)k0 * N + t;
            atomicAdd(bk, wt_d);
            atomicAdd(bk + KN, f2d(fmul(c, wt)));
            atomicAdd(bk + 2 * KN, f2d(fmul(__fdiv_rn(1.0f, c), wt)));
            for (int k = k0; k < K; k++) {
                double *row = p.out + (size_t)k * N + t;
                atomicAdd(row + 2 * KN, f2d(rankw[k]));
                atomicAdd(row + 4 * KN, f2d(fmul(expf(fmul(-p.beta[k], c)), wt)));
            }
        }
    }
    phase_barrier<SYNC>();
    phase_mark(ph, 3, tph);
    if constexpr (SYNC == 0) {
        if (!p.betweenness) return;
    }
    // in the block-synchronous form the flag can differ between a block's warps (batched jobs):
    // a warp without betweenness runs the remaining phases empty, so every warp meets the barriers
    const int Rb = (SYNC != 0 && !p.betweenness) ? 0 : R;
    // (sigma was built in the replay pass)
    phase_mark(ph, 4, tph);
    // --- backward Brandes sweep, all K thresholds in one pass (rust/src/centrality.rs:823-873,
    // 1782-1835), in the reference's f64: path counts, predecessor factors sigma_v / sigma_w, seeds
    // (pair count, and pair count * exp(-beta * cost) with the product and exp in f64) and
    // dependencies.  GB300 runs f64 at 1/64 of the f32 rate, so f64 instructions are spent on sums and shares
    // alone: comparisons go by the bits, the seed's double-float is put together in integers, and what a
    // node received is its credit as it is.
    __syncwarp();
    const bool unit_wt = (wt == 1.0f);
    const double wtd = f2d(wt);
    const int nchunks = failed ? 0 : (Rb + 31) / 32;
    constexpr int BW = (PM < BW_COLS) ? PM : BW_COLS;  // predecessors kept in this lane's shared column
    for (int ch = nchunks - 1; ch >= 0; ch--) {
        const int base = ch * 32;
        const int i = base + lane;
        const bool act = i < Rb;
        int pl[PM];
        const int np = act ? load_preds<PM>(s, i, P, pl) : 0;
        unsigned pm = 0;
#pragma unroll
        for (int r = 0; r < PM; r++)
            if (r < np && pl[r] >= base) pm |= 1u << (pl[r] - base);
        bool mine = !act;
        unsigned done = __ballot_sync(FULL, mine);
        int guard = 0;
        while (done != FULL) {
            const unsigned blocked = __reduce_or_sync(FULL, mine ? 0u : pm);
            const bool ready = !mine && !((blocked >> lane) & 1u);
            if (ready) {
                const int v = s.ord[i];
                const float cost = route_cost(s.sd[i], p.speed);
                const double sw = sig[i];
                float pairf;
                if constexpr (OD) pairf = od_weight(p, src, v);
                else pairf = __ldg(&p.eligible[v]) ? 0.5f : 1.0f;
                const double pair = f2d(pairf);
                // the reference's credit is dependency - seed: NaN, never positive, at a destination of such trips
                const bool credited = !OD || fabsf(pairf) < __int_as_float(INF_BITS);
                // predecessor rows and factors go to this lane's shared-memory column, so that the
                // push loop below is a plain (not unrolled) loop over the np predecessors
#pragma unroll
                for (int r = 0; r < BW; r++) {
                    if (r < np) {
                        const double sv = sig[pl[r]];
                        bw_pl[r * 32 + lane] = lane_index(pl[r], K, nk, cum);
                        bw_fr[r * 32 + lane] = same_bits(sv, sw) ? 1.0 : __ddiv_rn(sv, sw);
                    }
                }
                double *dli = dl + lane_index(i, K, nk, cum);
                const int k0 = first_k(p, cost);
                for (int k = k0; k < K; k++) {
                    if (is_zero(sw)) break;
                    const double credit = __ldcg(&dli[2 * k]), creditb = __ldcg(&dli[2 * k + 1]);
                    double dep = (i == 0) ? 0.0 : pair;
                    double depb = (i == 0 || pairf == 0.0f) ? 0.0 : seed_exp(pairf, p.beta[k], cost);
                    if (!is_zero(credit) || !is_zero(creditb)) {  // a leaf of the paths has its seed only
                        dep = __dadd_rn(dep, credit);
                        depb = __dadd_rn(depb, creditb);
                    }
                    if (is_zero(dep) && is_zero(depb)) continue;
#pragma unroll 1
                    for (int r = 0; r < np; r++) {
                        int q;
                        double f;
                        if (r < BW) {
                            q = bw_pl[r * 32 + lane];
                            f = bw_fr[r * 32 + lane];
                        } else {  // beyond the shared column (high-degree graphs): from the scratch
                            const int qp = s.pr[(size_t)i * P + r];
                            const double sv = sig[qp];
                            f = same_bits(sv, sw) ? 1.0 : __ddiv_rn(sv, sw);
                            q = lane_index(qp, K, nk, cum);
                        }
                        if (is_zero(f)) continue;
                        double *pd = dl + q;
                        double f0 = dep, f1 = depb;
                        if (!same_bits(f, 1.0)) {
                            f0 = __dmul_rn(f, f0);
                            f1 = __dmul_rn(f, f1);
                        }
                        atomicAdd(&pd[2 * k], f0);
                        atomicAdd(&pd[2 * k + 1], f1);
                    }
                    if (v == src || !credited) continue;
                    constexpr size_t row_b = OD ? 0 : 5;
                    // trips can have any weight; without them a credit is a sum of terms >= 0
                    if (OD ? positive(credit) : __double_as_longlong(credit) > 0ll)
                        atomicAdd(p.out + (row_b * K + k) * N + v, unit_wt ? credit : __dmul_rn(credit, wtd));
                    if (OD ? positive(creditb) : __double_as_longlong(creditb) > 0ll)
                        atomicAdd(p.out + ((row_b + 1) * K + k) * N + v, unit_wt ? creditb : __dmul_rn(creditb, wtd));
                }
                mine = true;
            }
            __syncwarp();
            done |= __ballot_sync(FULL, ready);
            if (++guard > 64) break;
        }
        if (done != FULL) {
            if (lane == 0) raise_err(p.hdr, CS_ERR_INTERNAL, 3);
            break;
        }
    }
    phase_barrier<SYNC>();
    phase_mark(ph, 5, tph);
}

// ------------------------------------------------------------------------------------------
// 4b. Segment centrality for one source.
// ------------------------------------------------------------------------------------------
// The shadow term of one half street from a to c: log of c below 1 m, else of the ratio.
__device__ __forceinline__ float segment_log(float a, float c) {
    return (a < 1.0f) ? logf(c) : logf(fmaxf(__fdiv_rn(c, a), 1.1920929e-07f));
}

__device__ __forceinline__ void f64_acc(double &a, float x) { a = __dadd_rn(a, f2d(x)); }
constexpr int SEG_QUEUE = 160;  // visited streets a warp collects: up to 31 left over and 4 per lane
constexpr int WORK = BW_COLS * 32 * 12;  // bytes a warp shares: the backward sweep's columns, or the streets
static_assert(SEG_QUEUE * sizeof(float4) <= WORK, "the streets outgrow the warp's share");

template <int PM>
CS_PHASE_INLINE __device__ void segment_accumulate(const PrimalParams &p, const SlotPtrs &s, int src, int R,
                                                   float4 *queue, long long *ph) {
    const int lane = lane_id();
    long long tph = clock64();
    const int K = p.k;
    const int N = p.g.n_bound;
    double *const out = (p.mode == MODE_BOTH) ? p.out2 : p.out;  // segment rows
    bool bad = false;
    // single predecessor (strict <) with its last segment length; pred position in pr[i*P]
    for (int i = lane; i < R; i += 32) {
        if (i == 0) { s.pr[0] = -1; s.fa[0] = 0.0f; continue; }
        const int v = s.ord[i];
        Nb<PM> nb;
        load_nb<PM>(p, s, v, R, nb, bad);
        bool ok = true;
        const int q = replay_first_min<PM>(p, nb, i, s.sd[i], ok);
        if (!ok || q < 0) { bad = true; s.pr[(size_t)i * p.P] = -1; continue; }
        int pos = 0;
        float last = 0.0f;
#pragma unroll
        for (int j = 0; j < PM; j++)
            if (j == q) { pos = nb.pos[j]; last = __ldg(&p.g.out_seglen_dev[nb.beg + j]); }
        s.pr[(size_t)i * p.P] = pos;
        s.fa[i] = last;  // last segment length
    }
    if (__any_sync(FULL, bad)) {
        if (lane == 0) raise_err(p.hdr, CS_ERR_INTERNAL, 4);
        return;
    }
    __syncwarp();
    // origin segment length: inherited along the tree (settle order, chunked)
    for (int base = 0; base < R; base += 32) {
        const int i = base + lane;
        const bool act = i < R;
        const int pp = (act && i > 0) ? s.pr[(size_t)i * p.P] : -1;
        const unsigned pm = (pp >= base) ? (1u << (pp - base)) : 0u;
        bool mine = !act;
        if (act && i == 0) { s.fb[0] = 0.0f; mine = true; }
        unsigned done = __ballot_sync(FULL, mine);
        int guard = 0;
        while (done != FULL) {
            const bool ready = !mine && ((pm & ~done) == 0u);
            if (ready) {
                s.fb[i] = (pp == 0) ? s.fa[i] : s.fb[pp];
                mine = true;
            }
            __syncwarp();
            done |= __ballot_sync(FULL, ready);
            if (++guard > 64) break;
        }
        if (done != FULL) {
            if (lane == 0) raise_err(p.hdr, CS_ERR_INTERNAL, 5);
            return;
        }
    }
    phase_mark(ph, 2, tph);
    // closeness integrals over visited edges (rust/src/centrality.rs:2201-2317), into the source's rows;
    // thresholds in groups of 4, one pass over the visited edges per group.  Bound by the chain of loads
    // that finds a street's farther end (edge -> neighbour -> its position -> its distance) and by lanes
    // idle on streets visited from their other end: a lane loads four streets at once, and the visited ones
    // queue up in shared memory until 32 fill the warp (62,500 sources at 2 km: 19.5 -> 17.9 ms per call,
    // with one exponential for the middle of both halves and the logs once per street).  Tried and not
    // faster: sums in pairs of f32 instead of f64 (20.4 ms), the same without the queue (19.5 ms).
    if (p.closeness) for (int kb = 0; kb < K; kb += 4) {
        const int nk = min(4, K - kb);
        const float dtop = p.dk[kb + nk - 1];
        double acc[12];
#pragma unroll
        for (int q = 0; q < 12; q++) acc[q] = 0.0;
        int qn = 0;
        // one visited street per lane: the nearer end at A, the farther at B (inf: not reached)
        auto integrals = [&](float4 st) {
            const float A = st.x, B = st.y, elen = st.z, imp = st.w;
            const float C = fmul(fadd(fadd(elen, A), B), 0.5f);
            const float Ci = fadd(A, fmul(__fadd_rn(C, -A), imp));
            const bool two = B != C;
            float shA = 0.0f, shB = 0.0f;
            if (C <= dtop) {
                shA = segment_log(A, Ci);
                if (two) shB = segment_log(B, Ci);
            }
#pragma unroll
            for (int q = 0; q < 4; q++) {
                if (q >= nk) break;
                const int k = kb + q;
                const float df = p.dk[k];
                const bool inA = A < df, inB = two && B <= df;
                if (!inA && !inB) continue;
                const float beta = p.beta[k], nbeta = -beta, inb = p.inb[k];
                const bool clip = C > df;
                const float ec = (clip || beta == 0.0f) ? 0.0f : expf(fmul(nbeta, Ci));  // serves both halves
                if (inA) {
                    float cc = C, cci = Ci, sh = shA, e2 = ec;
                    if (clip) {
                        cc = df;
                        cci = fadd(A, fmul(__fadd_rn(df, -A), imp));
                        sh = segment_log(A, cci);
                        e2 = expf(fmul(nbeta, cci));
                    }
                    f64_acc(acc[q], __fadd_rn(cc, -A));
                    f64_acc(acc[4 + q], sh);
                    f64_acc(acc[8 + q], (beta == 0.0f) ? __fadd_rn(cci, -A)
                                                       : fmul(__fadd_rn(e2, -expf(fmul(nbeta, A))), inb));
                }
                if (inB) {
                    float cd = C, cdi = Ci, sh = shB, e2 = ec;
                    if (clip) {
                        cd = df;
                        cdi = fadd(B, fmul(__fadd_rn(df, -B), imp));
                        sh = segment_log(B, cdi);
                        e2 = expf(fmul(nbeta, cdi));
                    }
                    f64_acc(acc[q], __fadd_rn(cd, -B));
                    f64_acc(acc[4 + q], sh);
                    f64_acc(acc[8 + q], (beta == 0.0f) ? __fadd_rn(cdi, -B)
                                                       : fmul(__fadd_rn(e2, -expf(fmul(nbeta, B))), inb));
                }
            }
        };
        for (int base = 0; base < R; base += 32) {
            const int i = base + lane;
            int u = 0, beg = 0, end = 0;
            float au = 0.0f;
            if (i < R) {
                u = s.ord[i];
                au = route_cost(s.sd[i], p.speed);
                if (au <= dtop) {  // no threshold of this group reaches a street from farther on
                    beg = __ldg(&p.g.in_ptr_dev[u]);
                    end = __ldg(&p.g.in_ptr_dev[u + 1]);
                }
            }
            const int most = warp_max_i(end - beg);
            for (int j0 = 0; j0 < most; j0 += 4) {
                // four streets' loads at once: neighbour, its position, its distance
                int nb[4];
                uint32_t at[4];
                float B[4];
#pragma unroll
                for (int j = 0; j < 4; j++) nb[j] = (beg + j0 + j < end) ? __ldg(&p.g.in_nb_dev[beg + j0 + j]) : -1;
#pragma unroll
                for (int j = 0; j < 4; j++) at[j] = (nb[j] >= 0 && nb[j] != u) ? s.aux[nb[j]] : 0u;
#pragma unroll
                for (int j = 0; j < 4; j++)
                    B[j] = (at[j] != 0u && at[j] <= (uint32_t)R) ? route_cost(s.sd[at[j] - 1], p.speed)
                                                                 : __int_as_float(INF_BITS);
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    // visited from here: a self loop, or a neighbour not settled earlier
                    const bool take = nb[j] >= 0 && (nb[j] == u || at[j] == 0u || ((int)(at[j] - 1) >= i && at[j] <= (uint32_t)R));
                    const unsigned m = __ballot_sync(FULL, take);
                    if (take) {
                        const int e = beg + j0 + j;
                        queue[qn + __popc(m & lanemask_lt())] =
                            make_float4(au, nb[j] == u ? au : B[j], __ldg(&p.g.in_seglen_dev[e]), __ldg(&p.g.in_segimp_dev[e]));
                    }
                    qn += __popc(m);
                }
                __syncwarp();
                while (qn >= 32) {
                    qn -= 32;
                    integrals(queue[qn + lane]);
                }
                __syncwarp();
            }
        }
        if (lane < qn) integrals(queue[lane]);
        __syncwarp();
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const int k = kb + q;
            if (k >= K) break;
            const double a0 = warp_sum_d(acc[q]);
            const double a1 = warp_sum_d(acc[4 + q]);
            const double a2 = warp_sum_d(acc[8 + q]);
            if (lane == 0) {
                atomicAdd(out + ((size_t)0 * K + k) * N + src, a0);
                atomicAdd(out + ((size_t)1 * K + k) * N + src, a1);
                atomicAdd(out + ((size_t)2 * K + k) * N + src, a2);
            }
        }
    }
    phase_mark(ph, 3, tph);
    if (!p.betweenness) return;
    // betweenness: subtree sums of per-target auc (rust/src/centrality.rs:2319-2401)
    double *acc = s.dl;  // [R][K]
    for (int i = lane; i < R; i += 32)
        for (int k = 0; k < K; k++) acc[(size_t)i * K + k] = 0.0;
    __syncwarp();
    const int nchunks = (R + 31) / 32;
    for (int ch = nchunks - 1; ch >= 0; ch--) {
        const int base = ch * 32;
        const int i = base + lane;
        const bool act = i < R;
        const int pp = (act && i > 0) ? s.pr[(size_t)i * p.P] : -1;
        const unsigned pm = (pp >= base) ? (1u << (pp - base)) : 0u;
        bool mine = !act;
        unsigned done = __ballot_sync(FULL, mine);
        int guard = 0;
        while (done != FULL) {
            const unsigned blocked = __reduce_or_sync(FULL, mine ? 0u : pm);
            const bool ready = !mine && !((blocked >> lane) & 1u);
            if (ready) {
                const int v = s.ord[i];
                const float sdist = route_cost(s.sd[i], p.speed);
                const float o_len = s.fb[i], l_len = s.fa[i];
                const float min_span = __fadd_rn(__fadd_rn(sdist, -o_len), -l_len);
                const float o_2 = fadd(min_span, o_len), l_2 = fadd(min_span, l_len);
                const bool own = (i > 0) && (v > src);
                for (int k = 0; k < K; k++) {
                    const double below = __ldcg(&acc[(size_t)i * K + k]);
                    double total = below;
                    if (own) {
                        const float df = p.dk[k];
                        const float beta = p.beta[k];
                        if (min_span <= df) {
                            const float o2s = fminf(o_2, df), l2s = fminf(l_2, df);
                            float auc;
                            if (beta == 0.0f) auc = fadd(__fadd_rn(o2s, -min_span), __fadd_rn(l2s, -min_span));
                            else {
                                const float nb = -beta, inb = p.inb[k];
                                const float e1 = expf(fmul(nb, min_span));  // both segments start at the span
                                auc = fadd(fmul(__fadd_rn(expf(fmul(nb, o2s)), -e1), inb),
                                           fmul(__fadd_rn(expf(fmul(nb, l2s)), -e1), inb));
                            }
                            if (isfinite(auc) && auc > 0.0f) total = __dadd_rn(total, f2d(auc));
                        }
                    }
                    // sums of terms > 0: their bits tell zero from more without the f64 pipe
                    if (i > 0 && v != src && __double_as_longlong(below) > 0ll)
                        atomicAdd(out + ((size_t)3 * K + k) * N + v, below);
                    if (pp >= 0 && __double_as_longlong(total) != 0ll) atomicAdd(&acc[(size_t)pp * K + k], total);
                }
                mine = true;
            }
            __syncwarp();
            done |= __ballot_sync(FULL, ready);
            if (++guard > 64) break;
        }
        if (done != FULL) {
            if (lane == 0) raise_err(p.hdr, CS_ERR_INTERNAL, 6);
            return;
        }
    }
    phase_mark(ph, 5, tph);
}

// ------------------------------------------------------------------------------------------
// 4c. Shortest-path tree rows (isochrone query).
// ------------------------------------------------------------------------------------------
template <int PM>
CS_PHASE_INLINE __device__ void tree_rows(const PrimalParams &p, const SlotPtrs &s, int qidx, int R) {
    const int lane = lane_id();
    if (R > p.row_cap) {
        if (lane == 0) p.t_count[qidx] = -R;  // rows too narrow: report the reach only
        return;
    }
    bool bad = false;
    for (int i = lane; i < R; i += 32) {
        const int v = s.ord[i];
        int pred = -1;
        if (i > 0) {
            Nb<PM> nb;
            load_nb<PM>(p, s, v, R, nb, bad);
            bool ok = true;
            const int q = replay_first_min<PM>(p, nb, i, s.sd[i], ok);
            if (!ok || q < 0) bad = true;
            else {
#pragma unroll
                for (int j = 0; j < PM; j++)
                    if (j == q) pred = s.ord[nb.pos[j]];
            }
        }
        const size_t o = (size_t)qidx * p.row_cap + i;
        p.t_node[o] = v;
        p.t_agg[o] = s.sd[i];
        p.t_pred[o] = pred;
    }
    if (__any_sync(FULL, bad) && lane == 0) raise_err(p.hdr, CS_ERR_INTERNAL, 7);
    if (lane == 0) p.t_count[qidx] = R;
}

// ------------------------------------------------------------------------------------------
// 4d. Accessibility of one source (rust/src/data.rs:513-602 aggregate_to_src_idx, :688-731).
//     Over the reached nodes (the search's distances are dijkstra_tree_shortest's), each assigned
//     entry's total distance (network + assignment, f32); an entry counts when it is the nearest
//     of its dedupe key (ties: the lower (node seconds, node, rank in the node's list), the
//     reference keeping the first one it meets), and adds to its class's rows.
// ------------------------------------------------------------------------------------------
__device__ __forceinline__ void access_accumulate(const PrimalParams &p, const SlotPtrs &s, int src, int R) {
    const int lane = lane_id();
    const cs_data_map &dm = p.dm;
    const int K = p.k, N = p.g.n_bound;
    const float maxs = p.maxsec;
    const float max_walk = fmul(maxs, p.speed);
    for (int i = lane; i < R; i += 32) {
        const int v = s.rl[i];
        const float sec = __ldcg(&s.dist[v]);
        if (!(sec < maxs)) continue;
        const float net = fmul(sec, p.speed);
        const int a_end = __ldg(&dm.node_ptr_dev[v + 1]);
        for (int a = __ldg(&dm.node_ptr_dev[v]); a < a_end; a++) {
            const float tot = fadd(net, __ldg(&dm.assign_dist_dev[a]));
            if (!(tot <= max_walk)) continue;
            const int e = __ldg(&dm.assign_entry_dev[a]);
            const int grp = __ldg(&dm.entry_group_dev[e]);
            const int rank = __ldg(&dm.assign_rank_dev[a]);
            bool win = true;
            const int g_end = __ldg(&dm.group_ptr_dev[grp + 1]);
            for (int b = __ldg(&dm.group_ptr_dev[grp]); b < g_end && win; b++) {
                const int a2 = __ldg(&dm.group_assign_dev[b]);
                if (a2 == a) continue;
                const int v2 = __ldg(&dm.assign_node_dev[a2]);
                const float sec2 = __ldcg(&s.dist[v2]);  // +inf when not reached
                if (!(sec2 < maxs)) continue;
                const float tot2 = fadd(fmul(sec2, p.speed), __ldg(&dm.assign_dist_dev[a2]));
                if (!(tot2 <= max_walk)) continue;
                if (tot2 < tot) win = false;
                else if (tot2 == tot) {
                    const int r2 = __ldg(&dm.assign_rank_dev[a2]);
                    if (sec2 < sec || (sec2 == sec && (v2 < v || (v2 == v && r2 < rank)))) win = false;
                }
            }
            if (!win) continue;
            const int c = __ldg(&dm.entry_class_dev[e]);
            if (c < 0) continue;
            for (int k = 0; k < K; k++) {
                if (!(tot <= p.dk[k])) continue;
                const size_t o = ((size_t)c * K + k) * N + src;
                atomicAdd(&p.acc_unw[o], 1.0);
                // clipped_beta_wt (rust/src/common.rs:339-348)
                const float raw = expf(fmul(-p.beta[k], tot));
                atomicAdd(&p.acc_wt[o], f2d(__fdiv_rn(fminf(raw, p.mcw[k]), p.mcw[k])));
                if (p.dk[k] == p.max_dist) atomicMin(&p.acc_near[(size_t)c * N + src], __float_as_uint(tot));
            }
        }
    }
}

// ------------------------------------------------------------------------------------------
// Persistent kernel: each warp owns one scratch slot and pulls sources until the list is empty.
// ------------------------------------------------------------------------------------------
// One source on this warp's slot: search, sort, mode-specific accumulation, scratch reset.
// Returns false when the source overflowed the slot's capacity (recorded for the retry).
// MODE is the accumulation compiled in (a kernel per mode keeps each kernel's code, and so its
// instruction-cache footprint, to what that mode runs); -1 dispatches on p.mode at run time.
template <int PM, int MODE>
__device__ __forceinline__ bool run_source(const PrimalParams &p, const SlotPtrs &s, int li, int src, uint32_t *hist,
                                           int *cnt, int *bw_pl, double *bw_fr, long long *ph, long long &relaxed,
                                           long long &settled) {
    const int lane = lane_id();
    long long t0 = clock64();
    float dmax = 0.0f;
    const int R = warp_search<deg_fast(PM)>(p, s, src, relaxed, dmax);
    phase_mark(ph, 0, t0);
    if (R < 0) {
        // Reach exceeded this slot's capacity: the reached list lost track of touched entries, so
        // reset the slot's whole dense state, record the source for the full-capacity retry and
        // carry on with the next source.
        for (int j = lane; j < p.g.n_bound; j += 32) {
            s.dist[j] = __int_as_float(INF_BITS);
            s.aux[j] = 0u;
        }
        if (lane == 0) {
            const unsigned f = atomicAdd(&p.hdr->n_failed, 1u);
            if (f < (unsigned)p.fail_cap) p.failed[f] = li;
            else raise_err(p.hdr, CS_ERR_CAPACITY, 8);
        }
        __syncwarp();
        return false;
    }
    if constexpr (MODE == MODE_ACCESS) {
        // no settle order needed: the reached list and the distances suffice
        access_accumulate(p, s, src, R);
        __syncwarp();
        for (int i = lane; i < R; i += 32) s.dist[s.rl[i]] = __int_as_float(INF_BITS);
        __syncwarp();
        settled += R;
        return true;
    }
    warp_sort(p, s, R, dmax, hist);
    __syncwarp();
    for (int i = lane; i < R; i += 32) s.aux[s.ord[i]] = (uint32_t)(i + 1);
    __syncwarp();
    phase_mark(ph, 1, t0);
    if constexpr (MODE == MODE_SHORTEST) {
        shortest_accumulate<PM, 0>(p, s, src, R, ph, cnt, bw_pl, bw_fr);
    } else if constexpr (MODE == MODE_SEGMENT) {
        segment_accumulate<PM>(p, s, src, R, (float4 *)bw_fr, ph);
    } else if constexpr (MODE == MODE_TREE) {
        tree_rows<PM>(p, s, li, R);
    } else if constexpr (MODE == MODE_OD) {
        shortest_accumulate<PM, 0, true>(p, s, src, R, ph, cnt, bw_pl, bw_fr);
    } else {
        if (p.mode == MODE_SHORTEST) shortest_accumulate<PM, 0>(p, s, src, R, ph, cnt, bw_pl, bw_fr);
        else if (p.mode == MODE_SEGMENT) segment_accumulate<PM>(p, s, src, R, (float4 *)bw_fr, ph);
        else if (p.mode == MODE_BOTH) {
            // one search and settle order serve both: shortest rows, then segment rows (its own
            // single-predecessor replay over the same positions)
            shortest_accumulate<PM, 0>(p, s, src, R, ph, cnt, bw_pl, bw_fr);
            __syncwarp();
            segment_accumulate<PM>(p, s, src, R, (float4 *)bw_fr, ph);
        } else tree_rows<PM>(p, s, li, R);
    }
    __syncwarp();
    t0 = clock64();
    for (int i = lane; i < R; i += 32) {
        const int v = s.ord[i];
        s.dist[v] = __int_as_float(INF_BITS);
        s.aux[v] = 0u;
    }
    __syncwarp();
    phase_mark(ph, 6, t0);
    settled += R;
    return true;
}

__device__ __forceinline__ void flush_counters(const PrimalParams &p, long long *ph, long long relaxed,
                                               long long settled, long long done_src) {
    const long long rsum = warp_sum_ll(relaxed);
    __syncwarp();
    if (lane_id() == 0) {
        for (int q = 0; q < 8; q++) atomicAdd(&p.hdr->pad[q], (unsigned long long)ph[q]);
        atomicAdd(&p.hdr->edges_relaxed, (unsigned long long)rsum);
        atomicAdd(&p.hdr->nodes_settled, (unsigned long long)settled);
        atomicAdd(&p.hdr->sources_done, (unsigned long long)done_src);
    }
}

// ------------------------------------------------------------------------------------------
// Persistent kernel: each warp owns one scratch slot and pulls sources until the list is empty.
// ------------------------------------------------------------------------------------------
// Segment centrality with a block's warps in lockstep (as primal_sync_kernel for shortest paths):
// search | sort | accumulation + scratch reset, each phase closed by a block barrier that every warp
// meets (a warp without a source, or whose source overflowed, runs the phases empty).
template <int PM>
__device__ __forceinline__ bool run_segment_sync(const PrimalParams &p, const SlotPtrs &s, bool mine, int li, int src,
                                                 uint32_t *hist, float4 *queue, long long *ph, long long &relaxed,
                                                 long long &settled) {
    const int lane = lane_id();
    long long t0 = clock64();
    float dmax = 0.0f;
    int R = 0;
    if (mine) R = warp_search<deg_fast(PM)>(p, s, src, relaxed, dmax);
    phase_mark(ph, 0, t0);
    __syncthreads();
    const bool live = mine && R >= 0;
    if (mine && R < 0) {
        for (int j = lane; j < p.g.n_bound; j += 32) {
            s.dist[j] = __int_as_float(INF_BITS);
            s.aux[j] = 0u;
        }
        if (lane == 0) {
            const unsigned f = atomicAdd(&p.hdr->n_failed, 1u);
            if (f < (unsigned)p.fail_cap) p.failed[f] = li;
            else raise_err(p.hdr, CS_ERR_CAPACITY, 8);
        }
        __syncwarp();
    }
    if (live) {
        warp_sort(p, s, R, dmax, hist);
        __syncwarp();
        for (int i = lane; i < R; i += 32) s.aux[s.ord[i]] = (uint32_t)(i + 1);
        __syncwarp();
    }
    phase_mark(ph, 1, t0);
    __syncthreads();
    if (live) {
        segment_accumulate<PM>(p, s, src, R, queue, ph);
        __syncwarp();
        t0 = clock64();
        for (int i = lane; i < R; i += 32) {
            const int v = s.ord[i];
            s.dist[v] = __int_as_float(INF_BITS);
            s.aux[v] = 0u;
        }
        __syncwarp();
        phase_mark(ph, 6, t0);
        settled += R;
    }
    __syncthreads();
    return live;
}

template <int PM, int MINB>
__global__ void __launch_bounds__(256, MINB) segment_sync_kernel(const PrimalParams p) {
    __shared__ uint32_t hist_all[8][256];
    __shared__ float4 queue_all[8][SEG_QUEUE];
    __shared__ long long ph_all[8][8];
    __shared__ unsigned long long blk_base;
    __shared__ unsigned blk_err;
    const int lane = lane_id();
    const int wib = threadIdx.x >> 5;
    const int slot0 = blockIdx.x * (blockDim.x >> 5);
    const int nw = min((int)(blockDim.x >> 5), p.n_slots - slot0);
    const bool has_slot = wib < nw;
    const SlotPtrs s = slot_ptrs(p.dense, p.dense_stride, p.compact, (size_t)p.cap, p.P, p.L,
                                 has_slot ? slot0 + wib : 0, p.g.n_bound);
    long long relaxed = 0, settled = 0, done_src = 0;
    long long *ph = ph_all[wib];
    if (lane < 8) ph[lane] = 0;
    __syncwarp();
    const int claim = block_claim(nw, p.n_src);
    while (true) {
        if (threadIdx.x == 0) {
            blk_base = atomicAdd(p.rerun ? &p.hdr->work_next2 : &p.hdr->work_next, (unsigned long long)claim);
            blk_err = __ldcg(&p.hdr->err);
        }
        __syncthreads();
        const unsigned long long b0 = blk_base;
        const unsigned berr = blk_err;
        __syncthreads();
        if (nw <= 0 || b0 >= (unsigned long long)p.n_src || berr != 0u) break;
        const unsigned long long idx = b0 + wib;
        const bool mine = wib < claim && idx < (unsigned long long)p.n_src;
        const int li = mine ? (p.remap ? p.remap[idx] : (int)idx) : 0;
        const int src = mine ? p.src_list[li] : 0;
        if (run_segment_sync<PM>(p, s, mine, li, src, hist_all[wib], queue_all[wib], ph, relaxed, settled)) {
            done_src++;
            if (lane == 0) count_progress(p.hdr);
        }
    }
    if (has_slot) flush_counters(p, ph, relaxed, settled, done_src);
}

template <int PM, int MINB, int MODE>
__global__ void __launch_bounds__(256, MINB) primal_kernel(const PrimalParams p) {
    __shared__ uint32_t hist_all[8][256];
    __shared__ int cnt_all[8][4 * MAXK + 2];
    __shared__ long long ph_all[8][8];
    // per warp: the backward sweep's columns (each lane's sigma fractions and predecessor rows), or the
    // visited streets of the segment integrals
    __shared__ __align__(16) double work_all[8][WORK / 8];
    const int lane = lane_id();
    const int wib = threadIdx.x >> 5;
    const int slot = (int)((blockIdx.x * (blockDim.x >> 5)) + wib);
    if (slot >= p.n_slots) return;
    const SlotPtrs s = slot_ptrs(p.dense, p.dense_stride, p.compact, (size_t)p.cap, p.P, p.L, slot, p.g.n_bound);
    long long relaxed = 0, settled = 0, done_src = 0;
    long long *ph = ph_all[wib];
    if (lane < 8) ph[lane] = 0;
    __syncwarp();
    while (true) {
        unsigned long long idx = 0;
        if (lane == 0) idx = atomicAdd(p.rerun ? &p.hdr->work_next2 : &p.hdr->work_next, 1ull);
        idx = __shfl_sync(FULL, idx, 0);
        if (idx >= (unsigned long long)p.n_src) break;
        if (__ldcg(&p.hdr->err) != 0u) break;
        const int li = p.remap ? p.remap[idx] : (int)idx;
        if (run_source<PM, MODE>(p, s, li, p.src_list[li], hist_all[wib], cnt_all[wib],
                                 (int *)(work_all[wib] + bw_cols(PM) * 32), work_all[wib], ph, relaxed, settled)) {
            done_src++;
            if (lane == 0) count_progress(p.hdr);
        }
    }
    flush_counters(p, ph, relaxed, settled, done_src);
}

// ------------------------------------------------------------------------------------------
// Shortest-path form with block-synchronous phases: a block claims one source per warp, and its
// warps run search, sort, replay, closeness, sigma, backward and reset together, a block barrier
// between phases.  At any time a block fetches one phase's code, so the SM's instruction caches
// hold the code of at most one phase per resident block.  Every warp reaches every barrier: a warp
// without a source (or whose source overflowed) runs the phases with R = 0.
// ------------------------------------------------------------------------------------------
template <int PM, int MINB, int WPB, int GW>
__global__ void __launch_bounds__(WPB * 32, MINB) primal_sync_kernel(const PrimalParams p) {
    __shared__ uint32_t hist_all[WPB][256];
    __shared__ int cnt_all[WPB][4 * MAXK + 2];
    __shared__ long long ph_all[WPB][8];
    __shared__ int bw_pl_all[WPB][bw_cols(PM) * 32];
    __shared__ double bw_fr_all[WPB][bw_cols(PM) * 32];
    __shared__ long long blk_base[WPB / GW];
    __shared__ unsigned blk_err[WPB / GW];
    const int lane = lane_id();
    const int wib = threadIdx.x >> 5;
    const int grp = wib / GW, gw = wib % GW;  // phase group of GW warps
    const int slot0 = blockIdx.x * (blockDim.x >> 5) + grp * GW;
    const int nw = min(GW, p.n_slots - slot0);  // warps of this group with a slot
    const bool has_slot = gw < nw;
    const SlotPtrs s = slot_ptrs(p.dense, p.dense_stride, p.compact, (size_t)p.cap, p.P, p.L,
                                 has_slot ? slot0 + gw : 0, p.g.n_bound);
    long long relaxed = 0, settled = 0, done_src = 0;
    long long *ph = ph_all[wib];
    if (lane < 8) ph[lane] = 0;
    __syncwarp();
    const long long n = p.n_src;
    const int claim = block_claim(nw, n);  // one group per block (GW = WPB)
    while (true) {
        if (gw == 0 && lane == 0) {
            blk_base[grp] = (long long)atomicAdd(p.rerun ? &p.hdr->work_next2 : &p.hdr->work_next,
                                                 (unsigned long long)claim);
            blk_err[grp] = __ldcg(&p.hdr->err);
        }
        phase_barrier<GW>();
        const long long base = blk_base[grp];
        const unsigned berr = blk_err[grp];
        phase_barrier<GW>();
        if (nw <= 0 || base >= n || berr != 0u) break;
        const long long idx = base + gw;
        const bool mine = gw < claim && idx < n;
        const int li = mine ? (p.remap ? p.remap[idx] : (int)idx) : 0;
        const int src = mine ? p.src_list[li] : 0;
        long long t0 = clock64();
        int R = 0;
        float dmax = 0.0f;
        if (mine) R = warp_search<deg_fast(PM)>(p, s, src, relaxed, dmax);
        phase_mark(ph, 0, t0);
        phase_barrier<GW>();
        const bool ok = mine && R >= 0;
        if (mine && R < 0) {
            for (int j = lane; j < p.g.n_bound; j += 32) {
                s.dist[j] = __int_as_float(INF_BITS);
                s.aux[j] = 0u;
            }
            if (lane == 0) {
                const unsigned f = atomicAdd(&p.hdr->n_failed, 1u);
                if (f < (unsigned)p.fail_cap) p.failed[f] = li;
                else raise_err(p.hdr, CS_ERR_CAPACITY, 8);
            }
        }
        if (ok) {
            warp_sort(p, s, R, dmax, hist_all[wib]);
            __syncwarp();
            for (int i = lane; i < R; i += 32) s.aux[s.ord[i]] = (uint32_t)(i + 1);
        }
        __syncwarp();
        phase_mark(ph, 1, t0);
        phase_barrier<GW>();
        shortest_accumulate<PM, GW>(p, s, src, ok ? R : 0, ph, cnt_all[wib], bw_pl_all[wib], bw_fr_all[wib]);
        __syncwarp();
        t0 = clock64();
        if (ok) {
            for (int i = lane; i < R; i += 32) {
                const int v = s.ord[i];
                s.dist[v] = __int_as_float(INF_BITS);
                s.aux[v] = 0u;
            }
            settled += R;
            done_src++;
            if (lane == 0) count_progress(p.hdr);
        }
        __syncwarp();
        phase_mark(ph, 6, t0);
        phase_barrier<GW>();
    }
    flush_counters(p, ph, relaxed, settled, done_src);
}

// ------------------------------------------------------------------------------------------
// Batched persistent kernel: one launch over the (job, source) items of many graphs, thresholds
// and modes.  Item i belongs to the job whose item_begin is the largest <= i.  Every warp's slot
// is sized for the largest graph, capacity and lane count of the batch.
// ------------------------------------------------------------------------------------------
__device__ __forceinline__ int job_of(const cs_batch_job *jobs, int n_jobs, long long item) {
    int lo = 0, hi = n_jobs - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (jobs[mid].item_begin <= item) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

__device__ __forceinline__ void job_params(const PrimalParams &base, const cs_batch_job &j, PrimalParams &p) {
    p = base;
    p.g = j.g;
    p.k = j.k;
    uint32_t maxs = 0;
    for (int i = 0; i < MAXK; i++) {
        p.dk[i] = i < j.k ? (float)j.distances[i] : 0.0f;
        p.beta[i] = i < j.k ? j.betas[i] : 0.0f;
        p.inb[i] = __fdiv_rn(1.0f, -p.beta[i]);
        if (i < j.k) maxs = max(maxs, j.seconds[i]);
    }
    p.maxsec = (float)maxs;
    p.speed = j.speed_m_s;
    p.tol = j.tolerance;
    p.delta = j.delta_seconds > 0.0f ? j.delta_seconds : fmaxf(1.0f, p.maxsec / 48.0f);
    p.closeness = j.compute_closeness;
    p.betweenness = j.compute_betweenness;
    p.track_reach = 0;
    p.src_list = j.sources_dev;
    p.n_src = j.n_sources;
    p.src_wt = j.src_wt_dev;
    p.eligible = j.eligible_dev;
    p.out = j.out_dev;
    p.bucket = j.bucket_dev;
    p.out2 = j.out2_dev;
    p.mode = j.mode;
}

// MODE: the accumulation compiled in (0 shortest, 1 segment), or -1 to dispatch on each job's
// mode; a launch covers items [item_lo, item_hi) (or, in a re-run, the listed items).
template <int PM, int MINB, int MODE>
__global__ void __launch_bounds__(256, MINB) batch_kernel(const PrimalParams base, const cs_batch_job *jobs,
                                                          int n_jobs, long long item_lo, long long item_hi) {
    __shared__ uint32_t hist_all[8][256];
    __shared__ int cnt_all[8][4 * MAXK + 2];
    __shared__ long long ph_all[8][8];
    // per warp: the backward sweep's columns (each lane's sigma fractions and predecessor rows), or the
    // visited streets of the segment integrals
    __shared__ __align__(16) double work_all[8][WORK / 8];
    const int lane = lane_id();
    const int wib = threadIdx.x >> 5;
    const int slot = (int)((blockIdx.x * (blockDim.x >> 5)) + wib);
    if (slot >= base.n_slots) return;
    // slot geometry from the batch maxima (base.g.n_bound = largest graph)
    const SlotPtrs s = slot_ptrs(base.dense, base.dense_stride, base.compact, (size_t)base.cap, base.P, base.L, slot,
                                 base.g.n_bound);
    long long relaxed = 0, settled = 0, done_src = 0;
    long long *ph = ph_all[wib];
    if (lane < 8) ph[lane] = 0;
    // the warp's job parameters live in shared memory: a local copy of the (large) parameter block
    // sits in the stack frame, and its loads then miss L1 under the kernel's global traffic
    __shared__ PrimalParams pj_all[8];
    PrimalParams &p = pj_all[wib];
    __syncwarp();
    int cur_job = -1;
    const long long n = !base.rerun ? item_hi - item_lo : (base.n_remap ? (long long)*base.n_remap : base.n_src);
    while (true) {
        unsigned long long idx = 0;
        if (lane == 0) idx = atomicAdd(base.rerun ? &base.hdr->work_next2 : &base.hdr->work_next, 1ull);
        idx = __shfl_sync(FULL, idx, 0);
        if ((long long)idx >= n) break;
        if (__ldcg(&base.hdr->err) != 0u) break;
        const long long item = base.remap ? (long long)base.remap[idx] : item_lo + (long long)idx;
        const int jb = job_of(jobs, n_jobs, item);
        if (jb != cur_job) {
            if (lane == 0) job_params(base, jobs[jb], p);
            __syncwarp();
            cur_job = jb;
        }
        const int li = (int)(item - jobs[jb].item_begin);
        // failures record the global item index
        if (run_source<PM, MODE>(p, s, (int)item, p.src_list[li], hist_all[wib], cnt_all[wib],
                                 (int *)(work_all[wib] + bw_cols(PM) * 32), work_all[wib], ph, relaxed, settled)) {
            done_src++;
            if (lane == 0) count_progress(base.hdr);
        }
    }
    flush_counters(base, ph, relaxed, settled, done_src);
}

// Batched shortest-path or segment items with block-synchronous phases (as primal_sync_kernel and
// segment_sync_kernel): a block claims one item per warp; each warp looks its item's job up.  Every warp
// reaches every barrier.
template <int PM, int MINB, int MODE>
__global__ void __launch_bounds__(256, MINB) batch_sync_kernel(const PrimalParams base, const cs_batch_job *jobs,
                                                               int n_jobs, long long item_lo, long long item_hi) {
    __shared__ uint32_t hist_all[8][256];
    __shared__ int cnt_all[8][4 * MAXK + 2];
    __shared__ long long ph_all[8][8];
    __shared__ __align__(16) double work_all[8][WORK / 8];
    __shared__ long long blk_base;
    __shared__ unsigned blk_err;
    const int lane = lane_id();
    const int wib = threadIdx.x >> 5;
    const int slot0 = blockIdx.x * (blockDim.x >> 5);
    const int nw = min((int)(blockDim.x >> 5), base.n_slots - slot0);
    const bool has_slot = wib < nw;
    const SlotPtrs s = slot_ptrs(base.dense, base.dense_stride, base.compact, (size_t)base.cap, base.P, base.L,
                                 has_slot ? slot0 + wib : 0, base.g.n_bound);
    long long relaxed = 0, settled = 0, done_src = 0;
    long long *ph = ph_all[wib];
    if (lane < 8) ph[lane] = 0;
    __syncwarp();
    const long long n = item_hi - item_lo;
    __shared__ PrimalParams pj_all[8];  // the warps' job parameters (as in batch_kernel)
    PrimalParams &p = pj_all[wib];
    int cur_job = -1;
    const int claim = block_claim(nw, n);
    while (true) {
        if (threadIdx.x == 0) {
            blk_base = (long long)atomicAdd(&base.hdr->work_next, (unsigned long long)claim);
            blk_err = __ldcg(&base.hdr->err);
        }
        __syncthreads();
        const long long b0 = blk_base;
        const unsigned berr = blk_err;
        __syncthreads();
        if (nw <= 0 || b0 >= n || berr != 0u) break;
        const long long idx = b0 + wib;
        const bool mine = wib < claim && idx < n;
        int src = 0, li = 0;
        const long long item = item_lo + idx;
        if (mine) {
            const int jb = job_of(jobs, n_jobs, item);
            if (jb != cur_job) {
                if (lane == 0) job_params(base, jobs[jb], p);
                __syncwarp();
                cur_job = jb;
            }
            li = (int)(item - jobs[jb].item_begin);
            src = p.src_list[li];
        } else if (cur_job < 0) {
            if (lane == 0) job_params(base, jobs[0], p);  // an idle warp still runs the phases (R = 0)
            __syncwarp();
            cur_job = 0;
        }
        long long t0 = clock64();
        int R = 0;
        float dmax = 0.0f;
        if (mine) R = warp_search<deg_fast(PM)>(p, s, src, relaxed, dmax);
        phase_mark(ph, 0, t0);
        __syncthreads();
        const bool ok = mine && R >= 0;
        if (mine && R < 0) {
            for (int j = lane; j < p.g.n_bound; j += 32) {
                s.dist[j] = __int_as_float(INF_BITS);
                s.aux[j] = 0u;
            }
            if (lane == 0) {
                const unsigned f = atomicAdd(&base.hdr->n_failed, 1u);
                if (f < (unsigned)base.fail_cap) base.failed[f] = (int)item;
                else raise_err(base.hdr, CS_ERR_CAPACITY, 8);
            }
        }
        if (ok) {
            warp_sort(p, s, R, dmax, hist_all[wib]);
            __syncwarp();
            for (int i = lane; i < R; i += 32) s.aux[s.ord[i]] = (uint32_t)(i + 1);
        }
        __syncwarp();
        phase_mark(ph, 1, t0);
        __syncthreads();
        // every warp of the block runs the phases with the same closeness / betweenness flags
        // only when its jobs agree on them; the barrier count must not depend on the job
        if constexpr (MODE == MODE_SEGMENT) {
            if (ok) segment_accumulate<PM>(p, s, src, R, (float4 *)work_all[wib], ph);
        } else {
            shortest_accumulate<PM, 8>(p, s, ok ? src : 0, ok ? R : 0, ph, cnt_all[wib],
                                       (int *)(work_all[wib] + bw_cols(PM) * 32), work_all[wib]);
        }
        __syncwarp();
        t0 = clock64();
        if (ok) {
            for (int i = lane; i < R; i += 32) {
                const int v = s.ord[i];
                s.dist[v] = __int_as_float(INF_BITS);
                s.aux[v] = 0u;
            }
            settled += R;
            done_src++;
            if (lane == 0) count_progress(p.hdr);
        }
        __syncwarp();
        phase_mark(ph, 6, t0);
        __syncthreads();
    }
    flush_counters(base, ph, relaxed, settled, done_src);
}


// ------------------------------------------------------------------------------------------
// Launchers (one translation unit per group of modes).  P: the graph's maximum out-degree, minb:
// resident blocks per SM (2-4), sync: block-synchronous phases where the mode has them.
// ------------------------------------------------------------------------------------------
cudaError_t occupancy_primal(int P, int minb, int *blocks_per_sm);
void launch_shortest(const PrimalParams &p, int P, int minb, int blocks, bool sync, cudaStream_t stream);
void launch_od(const PrimalParams &p, int P, int minb, int blocks, cudaStream_t stream);
void launch_segment(const PrimalParams &p, int P, int minb, int blocks, bool sync, cudaStream_t stream);
void launch_tree(const PrimalParams &p, int P, int minb, int blocks, cudaStream_t stream);
void launch_access(const PrimalParams &p, int P, int minb, int blocks, cudaStream_t stream);
// A batch's items [lo, hi) of one mode (MODE_SHORTEST or MODE_SEGMENT), or of any (-1).
void launch_batch_items(const PrimalParams &p, int mode, int minb, int blocks, bool sync, const cs_batch_job *jobs,
                        int n_jobs, long long lo, long long hi, cudaStream_t stream);
// Each unit whose kernels read the seed table fills its own copy (cs_seed.cuh).
void launch_seed_table_shortest(cudaStream_t stream);
void launch_seed_table_batch(cudaStream_t stream);

// The kernel of one mode for a maximum out-degree and register budget.  The per-edge arrays and loops
// are sized and unrolled for 4, 8 or 32 out-edges; street networks without diagonals have at most 4, where
// the kernels of 8 spent a third of their issue slots on absent edges (nine batched towns: shortest
// paths 43.8 -> 37.2 ms, segments 21.9 -> 17.8; 3,001 origins' trips 1.30 -> 1.18 ms; 4,000 sources to
// 3.2 km of 90,000 nodes: trees 0.643 -> 0.572, accessibility 0.557 -> 0.497, both unchanged at 10,201
// sources to 1.6 km).  With 2 blocks per SM
// registers do not matter, and the kernels of 8 serve every smaller degree.
template <int MODE>
void launch_per_warp(const PrimalParams &p, int P, int minb, int blocks, cudaStream_t stream) {
    if (P > 8) primal_kernel<CS_MAX_DEGREE, 2, MODE><<<blocks, 256, 0, stream>>>(p);
    else if (P <= 4 && minb == 4) primal_kernel<4, 4, MODE><<<blocks, 256, 0, stream>>>(p);
    else if (P <= 4 && minb == 3) primal_kernel<4, 3, MODE><<<blocks, 256, 0, stream>>>(p);
    else if (minb == 4) primal_kernel<8, 4, MODE><<<blocks, 256, 0, stream>>>(p);
    else if (minb == 3) primal_kernel<8, 3, MODE><<<blocks, 256, 0, stream>>>(p);
    else primal_kernel<8, 2, MODE><<<blocks, 256, 0, stream>>>(p);
}

}  // namespace cs
