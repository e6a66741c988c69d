// cs_tile.cu -- shortest-path node centrality and OD-weighted betweenness for tiles of nearby sources:
// one thread block per tile of up to 32 sources, one source per lane of every warp.
//
// Reference behaviour (cityseer-api v4.24.0):
//   centrality_shortest        rust/src/centrality.rs:1624-1874
//   dijkstra_brandes_shortest  rust/src/centrality.rs:1344-1494
//   circuit_ranks_from_traversal rust/src/centrality.rs:470-526
//   brandes_backprop_with_beta rust/src/centrality.rs:823-873
//   betweenness_od_shortest    rust/src/centrality.rs:2419-2540
//
// Sources that lie near one another reach almost the same nodes.  A tile numbers the union of its
// sources' reached sets and keeps every per-source value as a row of 32 lanes: dist[node][lane],
// sigma[node][lane], dependency[node][k][lane].  A warp takes one node at a time for all 32 sources, so
// the graph is read once per tile and not once per source, every access to per-source state is one
// whole 128- or 256-byte line, and edge loops, degrees and addresses are uniform across the warp.
// Phases of one tile, the block's warps together:
//  1. Union: a banded label-correcting search ("near-far" delta-stepping) from all sources at once
//     gives each node its least distance over the sources.  Nodes are numbered as they are found, so
//     numbers ascend with that distance up to about a band's width.  Then the tile's adjacency
//     (neighbour number, both directions' seconds, the neighbour's slot of the edge back).
//  2. Search: nodes whose row may improve are bits in shared memory; each round takes the lowest
//     numbered 64 of them, and a warp pulls min(row, neighbour row + seconds).  A node that improved
//     marks the neighbours it can improve.  fl(d + w) with w >= 0 is monotone, so the least fixpoint is
//     unique and equals the reference's heap Dijkstra bit for bit, whatever the order.
//  3. Replay of the offers to each node in settle order through the reference's Phase-1 tie rules (and
//     Phase 2 when tolerance > 1e-4), per lane: only offers within a small factor of the best can end up
//     as predecessors, so a lane with one such offer is done at once.  Predecessors are kept as one
//     32-lane mask per out-edge.  The same pass counts the circuit ranks.
//  4. Schedule: a topological order of (node, lanes) items over all lanes' predecessor graphs, in
//     levels, and sigma along it.  A node waits until all its lanes are ready, but for the 16 lowest
//     numbered of the partly ready ones (two sources can pass a street in opposite directions), whose
//     ready lanes go first.
//  5. Closeness into target rows: a node's 32 terms are summed in the warp before one atomic.
//  6. The dependencies along the levels in reverse, pulled from the successors; a node's 32 credits are
//     summed in the warp before one atomic.
// Sources that do not fit (a tile beyond its scratch, a graph whose edges are not paired, equal
// distances whose order decides a predecessor) are listed before the tile writes any output, and the
// host runs them through the per-warp kernel.
//
// What bounds it, and what it measured (202,500-node lattice, every source, thresholds to 5 km; a tile has
// 9,006 nodes on average and its lanes are 86% full; 377 ms with one warp per source):
//  - First form 352 ms: the f64 pipe, which GB300 runs at 1/64 of the f32 rate.  Warp sums in integers, no
//    add for a lane's first successor, seeds combined by integer ops: 300 ms, f64 pipe 15% busy.
//  - Then instructions and the latency of each level's chain of loads.  Four nodes per warp share the
//    loads of their edges, the edges lie at fixed places, a Link per edge holds what the sweep asks of the
//    target, and the next level's lines are prefetched: 205 ms.
//  - Consecutive items to different warps: 182 ms.  Blocks of 512 threads, 2 per SM: 256 x 4 ran 200 ms, 384 x 2 211 ms, 1024 x 1 226 ms.
//  - Cheaper seeds and f64 only for sums and shares: 175 ms.  A wider union band, the next node's line
//    loaded while closeness sums the last: 172 ms.  Now (16,900 nodes, 3.2 km) 2.0 instructions per cycle
//    and busy SM, f64 pipe 14% busy, DRAM 9%; of 14.5 cycles between two instructions of a warp 3.7 wait
//    at barriers, 2.9 for fixed latencies, 2.7 for loads from memory.
//  - 16 partly ready nodes per level give 10,608 items in 114 levels per tile; letting all of them go
//    gave 13,317 items (+25% sweep), 4 per level 370 levels (+60% time).
#include <algorithm>
#include <cmath>

#include "cs_seed.cuh"
#include "cs_tile.cuh"

namespace cs {
namespace tile {

constexpr int BATCH = 64;         // nodes of one search round
constexpr int LIST = 256;         // candidates of one schedule step
// The union search only orders and bounds the tile: wider bands than a search's (fewer rounds, each a
// chain of loads and barriers) suit it; 2x and 4x took 2.2 and 3.0 of a city pass's 175 ms off.
constexpr float UNION_BAND = 4.0f;
// Header words: one bit per job of a batch (a plain call is job 0; the 513th job shares the first one's),
// set when its graph turns out to have an edge without one back.  No tile of it can be served.
constexpr int UNPAIRED_SLOT = 16, UNPAIRED_WORDS = 8;
static_assert(UNPAIRED_SLOT + UNPAIRED_WORDS <= 24, "beyond the header");
constexpr int PART = 16;          // partly ready nodes that each step lets go
constexpr int MAX_ROUNDS = 1 << 17;  // bounded loops (never reached on a consistent graph)
constexpr float TIE_WINDOW = 1.00115f;  // offers above best * this cannot stay predecessors (8 steps of 1e-4)

struct FixSum {  // a warp's sum in fixed point: value = sum * 2^(e - bias)
    unsigned long long sum;
    int e;  // -1: the terms need f64 adds
};

struct Vars {
    int R, nnear, nnext, nfar, nfar2;
    int fmn;             // bits of the smallest distance queued far
    int fail;            // the tile goes to the per-warp kernel
    unsigned ok;         // lanes with a source that are still served here
    unsigned tcount;
    int n_items, n_level;
    int sched, sched_all;  // (node, lane) pairs in the schedule, and reached
    long long base;
    unsigned herr;
    int nl;
    int job;
    unsigned long long settled, relaxed;
    int wsum[NW + 1];
    int src[32], loc[32];
    float wt[32];
    FixSum rank_sum[MAXK];
    int list[LIST];
};

// Shared memory: Vars, then per threshold and lane the circuit-rank counts (nodes, edges) and weights,
// then two bit sets over the tile's nodes.
struct Smem {
    Vars &v;
    int (*cnt)[32];       // [2 K]
    float (*rankw)[32];   // [K]
    uint32_t *bits, *part;
};

constexpr size_t smem_bytes(int k, int mcap) {
    return ((sizeof(Vars) + 15) & ~size_t(15)) + 3 * 128 * (size_t)k + 2 * ((size_t)mcap / 8);
}
// No launch asks for more than a kernel may have without an attribute, which would be the kernel's and
// not the launch's: another thread could change it between a call's setting and its launch.
static_assert(smem_bytes(MAXK, MMAX) + sizeof(Params) <= 48 * 1024, "a launch needs more shared memory than the default");

__device__ __forceinline__ Smem smem(char *raw, int k, int mcap) {
    char *c = raw + ((sizeof(Vars) + 15) & ~size_t(15));
    int(*cnt)[32] = (int(*)[32])c;
    float(*rankw)[32] = (float(*)[32])(c + 256 * (size_t)k);
    uint32_t *bits = (uint32_t *)(c + 384 * (size_t)k);
    return Smem{*(Vars *)raw, cnt, rankw, bits, bits + mcap / 32};
}

// One node of the tile: first dependency row; degree | circuit flags << 8 | first threshold << 16 |
// eligible << 24; graph node.
struct __align__(16) Node {
    uint32_t dep, info;
    int32_t id;
    uint32_t pad;
};
// One edge, eight per node (a full line): neighbour number (-1 none), seconds out and back, index of the
// edge back.
struct __align__(16) Edge {
    int32_t to;
    float out, in;
    uint32_t back;
};
// What the schedule and the sweep ask of an edge's target: the lanes it is a successor in, of those the
// ones in which it has other predecessors too, its first threshold, and where its dependency row of
// threshold 0 would lie.
struct __align__(16) Link {
    uint32_t succ, multi;
    int32_t k0, row;
};

struct Arrays {
    int32_t *rl;
    Node *node;
    Edge *adj;
    Link *link;
    float *dist;
    uint32_t *pm;    // per edge: lanes whose predecessor its target is
    uint32_t *left;  // of those, the lanes whose predecessor is not scheduled yet
    uint32_t *reach, *done, *multi;
    double *sig;
    uint2 *items;
    uint32_t *lvl;
    double *dep;
    float *trip;
};

__device__ __forceinline__ Arrays arrays(const Params &p) {
    char *b = p.region + p.geo.total * (size_t)blockIdx.x;
    const Geometry &g = p.geo;
    Arrays a;
    a.rl = (int32_t *)(b + g.o_rl);
    a.node = (Node *)(b + g.o_node);
    a.adj = (Edge *)(b + g.o_adj);
    a.dist = (float *)(b + g.o_dist);
    a.pm = (uint32_t *)(b + g.o_pm);
    a.left = a.pm + (size_t)g.mcap * PMAX;
    a.link = (Link *)(b + g.o_link);
    a.reach = (uint32_t *)(b + g.o_masks);
    a.done = a.reach + g.mcap;
    a.multi = a.done + g.mcap;
    a.sig = (double *)(b + g.o_sig);
    a.items = (uint2 *)(b + g.o_items);
    a.lvl = (uint32_t *)(b + g.o_lvl);
    a.dep = (double *)(b + g.o_dep);
    a.trip = (float *)(b + g.o_trip);
    return a;
}

__device__ __forceinline__ float inf_f() { return __int_as_float(INF_BITS); }

// Takes up to cmax of the lowest set bits below n_bits out of `bits` into list, ascending.  Every thread
// of the block calls it; the list is complete after the closing barrier.
__device__ int collect(uint32_t *bits, int n_bits, int *list, int cmax, int *wsum) {
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int words = (n_bits + 31) >> 5;
    const int per = (words + TPB - 1) / TPB;
    const int w0 = tid * per, w1 = min(words, w0 + per);
    int mine = 0;
    for (int i = w0; i < w1; i++) mine += __popc(bits[i]);
    int inc = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(FULL, inc, o);
        if (lane >= o) inc += t;
    }
    if (lane == 31) wsum[w] = inc;
    __syncthreads();
    int before = 0, total = 0;
    {
        const int s = (lane < NW) ? wsum[lane] : 0;
        total = __reduce_add_sync(FULL, s);
        before = __reduce_add_sync(FULL, lane < w ? s : 0);
    }
    int pos = before + inc - mine;
    if (mine && pos < cmax) {
        for (int i = w0; i < w1 && pos < cmax; i++) {
            uint32_t b = bits[i], took = 0u;
            while (b && pos < cmax) {
                const int j = __ffs(b) - 1;
                b &= b - 1;
                took |= 1u << j;
                list[pos++] = i * 32 + j;
            }
            if (took) bits[i] &= ~took;
        }
    }
    __syncthreads();
    return min(total, cmax);
}

// Sums over a warp without f64 adds.  GB300 runs f64 at 1/64 of the f32 rate: the five shuffled f64 adds
// of a warp sum hold an SM's f64 pipe for 80 cycles.  Instead the terms (nonnegative, finite) become fixed
// point at the largest term's exponent, integer warp reductions add them, and the total goes back to f64
// by integer arithmetic.  A sum of f32 terms keeps 54 bits from the largest term's top bit down, so it is
// exact while the terms span at most 30 binary orders, and beyond loses less than f64 adds of them (1,500
// sums of terms over 60 orders: 4.3e-16 at most, f64 5.4e-16); a sum of f64 terms keeps 59.
constexpr int BIAS_F = 180, BIAS_D = 1081;
__device__ __forceinline__ unsigned long long shift_right(unsigned long long x, int n) {  // 0 from n = 64 on
    unsigned long long r;
    asm("shr.u64 %0, %1, %2;" : "=l"(r) : "l"(x), "r"(n));
    return r;
}
__device__ __forceinline__ FixSum fix_sum(float x) {  // BIAS_F
    const uint32_t b = __float_as_uint(x);
    const uint32_t top = __reduce_max_sync(FULL, b);
    if (top >= 0x7f800000u) return {0ull, -1};
    const int e = max((int)(b >> 23), 1), emax = max((int)(top >> 23), 1);
    const uint32_t m = (b & 0x7fffffu) | (b >= 0x800000u ? 0x800000u : 0u);
    const unsigned long long t = (shift_right((unsigned long long)m << 31, emax - e) + 1ull) >> 1;  // to nearest
    const unsigned lo = __reduce_add_sync(FULL, (unsigned)t & 0x7ffffffu);
    const unsigned hi = __reduce_add_sync(FULL, (unsigned)(t >> 27));
    return {((unsigned long long)hi << 27) + lo, emax};
}
__device__ __forceinline__ FixSum fix_sum(double x) {  // BIAS_D
    const uint32_t h = (uint32_t)__double2hiint(x);
    const uint32_t top = __reduce_max_sync(FULL, h);
    if (top >= 0x7ff00000u) return {0ull, -1};
    const int e = max((int)(h >> 20), 1), emax = max((int)(top >> 20), 1);
    const uint32_t mh = (h & 0xfffffu) | (h >= 0x100000u ? 0x100000u : 0u);
    const unsigned long long m = ((unsigned long long)mh << 32) | (uint32_t)__double2loint(x);
    const unsigned long long t = shift_right(m << 6, emax - e);
    const unsigned p0 = __reduce_add_sync(FULL, (unsigned)t & 0x7ffffffu);
    const unsigned p1 = __reduce_add_sync(FULL, (unsigned)(t >> 27) & 0x7ffffffu);
    const unsigned p2 = __reduce_add_sync(FULL, (unsigned)(t >> 54));
    return {((unsigned long long)p2 << 54) + ((unsigned long long)p1 << 27) + p0, emax};
}
// Rounded to nearest (halves up).  Totals below the normal f64 range are left to the f64 adds.
__device__ __forceinline__ double fix_to_d(FixSum f, int bias) {
    if (f.sum == 0ull) return 0.0;
    const int lz = __clzll((long long)f.sum);
    const unsigned long long m = f.sum << lz;
    const unsigned long long ex = (unsigned long long)(63 - lz + f.e - bias + 1022);
    return __longlong_as_double((long long)((ex << 52) + (m >> 11) + ((m >> 10) & 1ull)));
}
__device__ __forceinline__ double slow_sum(double d) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) d += __shfl_xor_sync(FULL, d, o);
    return d;
}

// ------------------------------------------------------------------------------------------
// 1. The union of the reached sets, numbered; the tile's adjacency.
// ------------------------------------------------------------------------------------------
__device__ void discover(const Params &p, const Arrays &a, const Smem &sm, float *d1, uint32_t *aux) {
    Vars &v = sm.v;
    const int tid = threadIdx.x;
    const int mcap = p.geo.mcap, qcap = 2 * mcap;
    // the four queues lie in the path-count rows, which are written later
    uint2 *cur = (uint2 *)a.sig, *nxt = cur + qcap, *far = nxt + qcap, *far2 = far + qcap;
    if (tid == 0) {
        v.R = v.nnear = v.nnext = v.nfar = v.nfar2 = 0;
        v.fmn = INF_BITS;
    }
    __syncthreads();
    if (tid < v.nl) {
        const int s = v.src[tid];
        if (atomicExch((int *)&d1[s], 0) == INF_BITS) {
            const int q = atomicAdd(&v.R, 1);
            if (q < mcap) {
                a.rl[q] = s;
                aux[s] = (uint32_t)(q + 1);
                cur[atomicAdd(&v.nnear, 1)] = make_uint2((unsigned)s, 0u);
            }
        }
    }
    __syncthreads();
    const float band = p.delta * UNION_BAND;
    float T = band;
    int nnear = v.nnear;
    for (int round = 0; round < MAX_ROUNDS; round++) {
        if (nnear > 0) {
            for (int i = tid; i < nnear; i += TPB) {
                const uint2 ent = cur[i];
                const int u = (int)ent.x;
                const float du = __ldcg(&d1[u]);
                if (__float_as_uint(du) != ent.y) continue;
                const int end = __ldg(&p.in_ptr[u + 1]);
                for (int e = __ldg(&p.in_ptr[u]); e < end; e++) {
                    const int x = __ldg(&p.in_nb[e]);
                    const float c = fadd(du, __ldg(&p.in_w[e]));
                    if (x == u || !(c <= p.maxsec)) continue;
                    const int old = atomicMin((int *)&d1[x], __float_as_int(c));
                    if (__float_as_int(c) >= old) continue;
                    if (old == INF_BITS) {
                        const int q = atomicAdd(&v.R, 1);
                        if (q < mcap) {
                            a.rl[q] = x;
                            aux[x] = (uint32_t)(q + 1);
                        }
                    }
                    if (c < T) {
                        const int q = atomicAdd(&v.nnext, 1);
                        if (q < qcap) nxt[q] = make_uint2((unsigned)x, __float_as_uint(c));
                    } else {
                        const int q = atomicAdd(&v.nfar, 1);
                        if (q < qcap) far[q] = make_uint2((unsigned)x, __float_as_uint(c));
                        atomicMin(&v.fmn, __float_as_int(c));
                    }
                }
            }
            __syncthreads();
            nnear = v.nnext;
            const bool over = v.R > mcap || nnear > qcap || v.nfar > qcap;
            __syncthreads();
            if (tid == 0) v.nnext = 0;
            if (over) {
                if (tid == 0) v.fail = 1;
                __syncthreads();
                return;
            }
            uint2 *t = cur;
            cur = nxt;
            nxt = t;
            __syncthreads();
            continue;
        }
        const int nfar = v.nfar;
        if (nfar == 0) return;
        const float mn = __int_as_float(v.fmn);
        T = fmaxf(fadd(mn, band), __int_as_float(__float_as_int(mn) + 1));
        __syncthreads();
        if (tid == 0) {
            v.fmn = INF_BITS;
            v.nfar = 0;
            v.nnear = 0;
        }
        __syncthreads();
        for (int i = tid; i < nfar; i += TPB) {
            const uint2 ent = far[i];
            if (__uint_as_float(ent.y) < T) {
                cur[atomicAdd(&v.nnear, 1)] = ent;
            } else {
                far2[atomicAdd(&v.nfar, 1)] = ent;
                atomicMin(&v.fmn, (int)ent.y);
            }
        }
        __syncthreads();
        nnear = v.nnear;
        uint2 *t = far;
        far = far2;
        far2 = t;
        __syncthreads();
    }
    if (tid == 0) v.fail = 1;
    __syncthreads();
}

__device__ __forceinline__ unsigned long long *unpaired_word(WsHeader *h, int job) {
    return &h->pad[UNPAIRED_SLOT + (job >> 6) % UNPAIRED_WORDS];
}
__device__ __forceinline__ void mark_unpaired(WsHeader *h, int job) { atomicOr(unpaired_word(h, job), 1ull << (job & 63)); }
__device__ __forceinline__ int is_unpaired(WsHeader *h, int job) {
    return (int)((__ldcg(unpaired_word(h, job)) >> (job & 63)) & 1ull);
}

// Eight lanes per node, one per edge.
__device__ void adjacency(const Params &p, const Arrays &a, const Smem &sm, const float *d1, const uint32_t *aux) {
    Vars &v = sm.v;
    const int R = v.R, K = p.k;
    const int lane = lane_id(), j = lane & 7, g = lane & 24;
    bool bad = false, unpaired = false;
    for (int i0 = (threadIdx.x >> 5) * 4; i0 < R; i0 += NW * 4) {
        const int i = i0 + (lane >> 3);
        const bool on = i < R;
        const int id = on ? a.rl[i] : 0;
        const int ob = __ldg(&p.out_ptr[id]), deg = on ? __ldg(&p.out_ptr[id + 1]) - ob : 0;
        const int ideg = on ? __ldg(&p.in_ptr[id + 1]) - __ldg(&p.in_ptr[id]) : 0;
        if (deg != ideg || deg > PMAX) bad = unpaired = true;
        const bool flag = j < deg && __ldg(&p.out_cnt[ob + j]) && __ldg(&p.out_to[ob + j]) != id;
        const unsigned flags = (__ballot_sync(FULL, flag) >> g) & 0xffu;
        if (on && j == 0) {
            const float c = fmul(__ldcg(&d1[id]), p.speed);
            int k0 = 0;
            while (k0 < K && !(c <= p.dk[k0])) k0++;
            Node n;
            n.id = id;
            n.info = (uint32_t)deg | (flags << 8) | ((uint32_t)k0 << 16);
            if (p.eligible && __ldg(&p.eligible[id])) n.info |= 1u << 24;
            n.dep = p.betweenness ? atomicAdd(&v.tcount, (unsigned)(K - k0)) : 0u;
            n.pad = 0u;
            if (n.dep + (unsigned)(K - k0) > p.geo.tcap) bad = true;
            a.node[i] = n;
        }
    }
    if (unpaired) mark_unpaired(p.hdr, v.job);
    // every thread takes the same way on: a flag read after the barrier could be one set beyond it
    if (__syncthreads_or(bad)) {
        if (threadIdx.x == 0) v.fail = 1;
        __syncthreads();
        return;
    }
    for (int i0 = (threadIdx.x >> 5) * 4; i0 < R; i0 += NW * 4) {
        const int i = i0 + (lane >> 3);
        Node n{0u, 0u, 0, 0u};
        if (i < R) n = a.node[i];
        const int deg = n.info & 0xff;
        const bool on = j < deg;
        const int ob = __ldg(&p.out_ptr[n.id]), ib = __ldg(&p.in_ptr[n.id]);
        const int x = on ? __ldg(&p.out_to[ob + j]) : -1;
        const int y = on ? __ldg(&p.in_nb[ib + j]) : -2;
        const bool other = on && x != n.id;
        int r = 0, c = 0, back = -1;  // this is the r-th edge to x: pair it with the r-th edge back
#pragma unroll
        for (int q = 0; q < PMAX; q++) {
            const bool same = __shfl_sync(FULL, x, g + q) == x;
            r += same && q < j;
        }
#pragma unroll
        for (int q = 0; q < PMAX; q++) {
            const bool hit = __shfl_sync(FULL, y, g + q) == x;
            if (hit && c == r) back = q;
            c += hit;
        }
        Edge e{-1, 0.0f, 0.0f, 0u};
        if (other) {
            const uint32_t at = aux[x];
            if (back < 0 || at > (uint32_t)R) {
                bad = true;  // unpaired edge, or scratch not clean
                unpaired |= back < 0;
            } else if (at != 0u) {
                const int xb = __ldg(&p.out_ptr[x]), xdeg = a.node[at - 1].info & 0xff;
                int slot = -1;
                c = 0;
                for (int q = 0; q < xdeg; q++)
                    if (__ldg(&p.out_to[xb + q]) == n.id && c++ == r) slot = q;
                if (slot < 0) bad = unpaired = true;
                e = Edge{(int)at - 1, __ldg(&p.out_w[ob + j]), __ldg(&p.in_w[ib + back]), (at - 1) * PMAX + (uint32_t)max(slot, 0)};
            }
        }
        if (i < R) a.adj[(size_t)i * PMAX + j] = e;
    }
    if (bad) v.fail = 1;
    if (unpaired) mark_unpaired(p.hdr, v.job);
    __syncthreads();
}

__device__ __forceinline__ void prefetch(const void *at) { asm volatile("prefetch.global.L2 [%0];" ::"l"(at)); }
__device__ __forceinline__ void mark(uint32_t *bits, int i) { atomicOr(&bits[i >> 5], 1u << (i & 31)); }

// Four nodes of a warp at once: lane 8 t + j holds edge j of node t, so the latency of loading nodes' edges
// is paid once per four nodes.  edges: lanes that hold one.
struct Quad {
    int i;  // node number, -1 none
    Edge e;
    unsigned edges;
};
__device__ __forceinline__ Quad load_quad(const Arrays &a, int i) {
    Quad q;
    q.i = i;
    q.e = Edge{-1, 0.0f, 0.0f, 0u};
    if (i >= 0) q.e = a.adj[(size_t)i * PMAX + (lane_id() & 7)];
    q.edges = __ballot_sync(FULL, q.e.to >= 0);
    return q;
}

// Node t's distance row and its neighbours' (inf: no such neighbour).
__device__ __forceinline__ void load_rows(const Arrays &a, const Quad &q, int t, float &dv, float *du) {
    const int lane = lane_id();
    const int i = __shfl_sync(FULL, q.i, t * 8);
    dv = i < 0 ? 0.0f : a.dist[(size_t)i * 32 + lane];
#pragma unroll
    for (int j = 0; j < PMAX; j++) {
        du[j] = inf_f();
        if ((q.edges >> (t * 8 + j)) & 1u) du[j] = a.dist[(size_t)__shfl_sync(FULL, q.e.to, t * 8 + j) * 32 + lane];
    }
}

// ------------------------------------------------------------------------------------------
// 2. Search.
// ------------------------------------------------------------------------------------------
__device__ void search(const Params &p, const Arrays &a, const Smem &sm) {
    Vars &v = sm.v;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int R = v.R;
    for (int i = tid; i < (R + 31) / 32; i += TPB) sm.bits[i] = 0u;
    float4 *rows = (float4 *)a.dist;
    for (int i = tid; i < R * 8; i += TPB) rows[i] = make_float4(inf_f(), inf_f(), inf_f(), inf_f());
    __syncthreads();
    if (tid < v.nl) a.dist[(size_t)v.loc[tid] * 32 + tid] = 0.0f;
    for (int s = w * 4; s < v.nl; s += NW * 4) {
        const int t = s + (lane >> 3);
        const Quad q = load_quad(a, t < v.nl ? v.loc[t] : -1);
        if (q.e.to >= 0) mark(sm.bits, q.e.to);
    }
    __syncthreads();
    for (int round = 0; round < MAX_ROUNDS; round++) {
        const int n = collect(sm.bits, R, v.list, BATCH, v.wsum);
        if (n == 0) return;
        for (int q0 = w; q0 < n; q0 += NW * 4) {
            const int qi = q0 + (lane >> 3) * NW;
            const Quad q = load_quad(a, qi < n ? v.list[qi] : -1);
            unsigned marks = 0u;  // this lane's edge: its target can improve
            auto pull = [&](int t, float dv, const float *du) {
                const int i = __shfl_sync(FULL, q.i, t * 8);
                if (i < 0) return;
                const unsigned ed = q.edges >> (t * 8);
                float nv = dv;
#pragma unroll
                for (int j = 0; j < PMAX; j++) {
                    if ((ed >> j) & 1u) {
                        const float c = fadd(du[j], __shfl_sync(FULL, q.e.out, t * 8 + j));
                        if (c <= p.maxsec) nv = fminf(nv, c);
                    }
                }
                if (!__any_sync(FULL, nv < dv)) return;
                a.dist[(size_t)i * 32 + lane] = nv;
#pragma unroll
                for (int j = 0; j < PMAX; j++) {
                    if ((ed >> j) & 1u) {
                        const float c = fadd(nv, __shfl_sync(FULL, q.e.in, t * 8 + j));
                        if (__any_sync(FULL, c < du[j] && c <= p.maxsec)) marks |= 1u << (t * 8 + j);
                    }
                }
            };
            // two nodes' rows in flight
            float dva, dvb, ua[PMAX], ub[PMAX];
            load_rows(a, q, 0, dva, ua);
            load_rows(a, q, 1, dvb, ub);
            pull(0, dva, ua);
            load_rows(a, q, 2, dva, ua);
            pull(1, dvb, ub);
            load_rows(a, q, 3, dvb, ub);
            pull(2, dva, ua);
            pull(3, dvb, ub);
            if ((marks >> lane) & 1u) {
                mark(sm.bits, q.e.to);
                prefetch(&a.adj[(size_t)q.e.to * PMAX]);
            }
        }
        __syncthreads();
    }
    if (tid == 0) v.fail = 1;
    __syncthreads();
}

// ------------------------------------------------------------------------------------------
// 3. Predecessors and circuit ranks.
// ------------------------------------------------------------------------------------------
// Next offer in settle order: the offering node's distance, then its slot (one node's parallel edges keep
// list order).
__device__ __forceinline__ int next_offer(const float *du, const float *c, unsigned todo, float &bc) {
    int best = -1;
    float bd = 0.0f;
    bc = 0.0f;
#pragma unroll
    for (int j = 0; j < PMAX; j++) {
        if (((todo >> j) & 1u) && (best < 0 || du[j] < bd)) {
            best = j;
            bd = du[j];
            bc = c[j];
        }
    }
    return best;
}

// Does pm hold an edge to the node of edge `best`?
__device__ __forceinline__ bool node_in(const Edge *ed, unsigned pm, int best) {
    const int x = ed[best].to;
    bool has = false;
    for (; pm; pm &= pm - 1) has |= ed[__ffs(pm) - 1].to == x;
    return has;
}

__device__ void replay(const Params &p, const Arrays &a, const Smem &sm) {
    Vars &v = sm.v;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int R = v.R, K = p.k;
    const float one_plus = 1.0f + TIE_EPSILON, one_minus = 1.0f - TIE_EPSILON;
    const bool phase2 = p.tol > TIE_EPSILON;
    const float wide = phase2 ? fmaxf(TIE_WINDOW, 1.0f + p.tol) : TIE_WINDOW;
    const int my_loc = v.loc[lane];
    const bool counts = p.closeness != 0;
    long long settled = 0, relaxed = 0;
    for (int i0 = w * 4; i0 < R; i0 += NW * 4) {
      const int it = i0 + (lane >> 3);
      const Quad q = load_quad(a, it < R ? it : -1);
      const uint32_t infos = it < R ? a.node[it].info : 0u;
      if (it + NW * 4 < R && (lane & 7) == 0) prefetch(&a.adj[(size_t)(it + NW * 4) * PMAX]);
      float dn, un[PMAX];
      load_rows(a, q, 0, dn, un);
#pragma unroll 1
      for (int t = 0; t < 4 && i0 + t < R; t++) {
        const int i = i0 + t;
        const uint32_t info = __shfl_sync(FULL, infos, t * 8);
        const int deg = info & 0xff;
        const unsigned eds = q.edges >> (t * 8);
        const Edge *ed = a.adj + (size_t)i * PMAX;
        const float dv = dn;
        float du[PMAX], c[PMAX];
#pragma unroll
        for (int j = 0; j < PMAX; j++) du[j] = un[j];
        if (t < 3) load_rows(a, q, t + 1, dn, un);  // the next node's rows while this one is replayed
        const bool here = dv < inf_f();
        const bool own = i == my_loc;  // this lane's source (lanes without one hold inf everywhere)
        const float lim1 = fmul(dv, TIE_WINDOW), limh = fmul(dv, wide);
        unsigned todo = 0u;
        bool hazard = false;
        float lo = own || !here ? dv : inf_f();
        int best = 0;
#pragma unroll
        for (int j = 0; j < PMAX; j++) {
            c[j] = inf_f();
            if ((eds >> j) & 1u) {
                c[j] = fadd(du[j], __shfl_sync(FULL, q.e.out, t * 8 + j));
                if (here && du[j] < dv) {
                    if (c[j] < lo) {
                        lo = c[j];
                        best = j;
                    }
                    if (c[j] <= lim1) todo |= 1u << j;
                }
                // equal distances: the settle order between the two decides, and it is not kept here
                if (du[j] == dv && c[j] <= limh && here) hazard = true;
            }
        }
        const unsigned m_reach = __ballot_sync(FULL, here);
        if (lane == 0) {
            settled += __popc(m_reach);
            relaxed += __popc(m_reach) * deg;
        }
        hazard |= __float_as_int(lo) != __float_as_int(dv);
        if (__any_sync(FULL, hazard)) {
            const unsigned m = __ballot_sync(FULL, hazard);
            if (lane == 0) atomicAnd(&v.ok, ~m);
        }
        if (p.betweenness) {
            if (!here || own) todo = 0u;
            unsigned pm = todo;
            if (phase2) {
                const float lim = fmul(dv, 1.0f + p.tol);
                unsigned t = 0u;
#pragma unroll
                for (int j = 0; j < PMAX; j++)
                    if (here && !own && du[j] < dv && c[j] <= lim) t |= 1u << j;
                pm = 0u;
                while (t) {
                    float bc;
                    const int b = next_offer(du, c, t, bc);
                    t &= ~(1u << b);
                    if (!node_in(ed, pm, b)) pm |= 1u << b;
                }
            } else if (todo & (todo - 1u)) {  // near ties, through Phase 1
                if (__popc(todo) == 2) {
                    // the best offer and one other: it stays if, coming first, the best is not clearly
                    // better, or if, coming second, it ties
                    const int o = __ffs(todo & ~(1u << best)) - 1;
                    float co = 0.0f, uo = 0.0f, ub = 0.0f;
#pragma unroll
                    for (int j = 0; j < PMAX; j++) {
                        if (j == o) {
                            co = c[j];
                            uo = du[j];
                        }
                        if (j == best) ub = du[j];
                    }
                    const bool first = uo < ub || (uo == ub && o < best);
                    bool stays;
                    if (first) stays = co <= p.maxsec && !(dv < fmul(co, one_minus));
                    else stays = co <= p.maxsec && co <= fmul(dv, one_plus) && ed[o].to != ed[best].to;
                    // equal offers: the first one met is `best` or the other alike, and the second ties
                    if (first && co == dv) stays = ed[o].to != ed[best].to;
                    if (!stays) pm = 1u << best;
                } else {
                    unsigned t = todo;
                    pm = 0u;
                    float cur = inf_f();
                    while (t) {
                        float bc;
                        const int b = next_offer(du, c, t, bc);
                        t &= ~(1u << b);
                        if (bc > p.maxsec) continue;
                        if (bc < cur) {
                            if (bc < fmul(cur, one_minus)) pm = 0u;
                            pm |= 1u << b;
                            cur = bc;
                        } else if (bc <= fmul(cur, one_plus) && !node_in(ed, pm, b)) {
                            pm |= 1u << b;
                        }
                    }
                }
            }
            __syncwarp();
            unsigned mine = 0u;
#pragma unroll
            for (int j = 0; j < PMAX; j++) {
                if ((eds >> j) & 1u) {
                    const unsigned m = __ballot_sync(FULL, (pm >> j) & 1u);
                    if (lane == j) mine = m;
                }
            }
            if (lane < PMAX) a.pm[(size_t)i * PMAX + lane] = a.left[(size_t)i * PMAX + lane] = mine;
            const unsigned mm = __ballot_sync(FULL, (pm & (pm - 1u)) != 0u);
            if (lane == 0) {
                a.reach[i] = m_reach;
                a.multi[i] = mm;
                a.done[i] = 0u;
            }
        }
        if (counts) {
            // the first threshold of the node (no lane's lies below the nearest source's) and of its edges
            const float cv = fmul(dv, p.speed);
            const int kmin = (info >> 16) & 0xff;
            int k0 = kmin;
            while (k0 < K && !(cv <= p.dk[k0])) k0++;
            if (here && k0 < K) {
                atomicAdd(&sm.cnt[k0][lane], 1);
#pragma unroll
                for (int j = 0; j < PMAX; j++) {
                    if (!((info >> (8 + j)) & 1u)) continue;
                    const float ce = fmul(du[j], p.speed);
                    int ke = k0;
                    while (ke < K && !(ce <= p.dk[ke])) ke++;
                    if (ke < K && du[j] < inf_f()) atomicAdd(&sm.cnt[K + ke][lane], 1);
                }
            }
        }
      }
    }
    if (lane == 0 && settled) {
        atomicAdd(&v.settled, (unsigned long long)settled);
        atomicAdd(&v.relaxed, (unsigned long long)relaxed);
    }
    __syncthreads();
}

__device__ void links(const Params &p, const Arrays &a, const Smem &sm) {
    const int R = sm.v.R, lane = lane_id();
    for (int i0 = (threadIdx.x >> 5) * 4; i0 < R; i0 += NW * 4) {
        const int i = i0 + (lane >> 3);
        if (i >= R) continue;
        const size_t o = (size_t)i * PMAX + (lane & 7);
        const Edge e = a.adj[o];
        Link l{0u, 0u, p.k, 0};
        if (e.to >= 0) {
            l.succ = a.pm[e.back];
            const Node nx = a.node[e.to];
            l.multi = a.multi[e.to] & l.succ;
            l.k0 = (int)((nx.info >> 16) & 0xff);
            l.row = (int)nx.dep - l.k0;
        }
        a.link[o] = l;
    }
    __syncthreads();
}

// ------------------------------------------------------------------------------------------
// 4. Schedule, and the path counts (sigma, f64) along it.
// ------------------------------------------------------------------------------------------
__device__ void schedule(const Params &p, const Arrays &a, const Smem &sm) {
    Vars &v = sm.v;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int R = v.R, words = (R + 31) / 32;
    const unsigned ok = v.ok;
    for (int i = tid; i < words; i += TPB) {
        sm.bits[i] = 0u;
        sm.part[i] = 0u;
    }
    if (tid == 0) {
        v.n_items = 0;
        v.n_level = 0;
        v.sched = __popc(ok);
        v.sched_all = 0;
        a.lvl[0] = 0u;
    }
    __syncthreads();
    int reached = 0;
    for (int i = tid; i < R; i += TPB) reached += __popc(a.reach[i] & ok);
    reached = __reduce_add_sync(FULL, reached);
    if (lane == 0) atomicAdd(&v.sched_all, reached);
    if (tid < 32) {  // level 0: the sources, one item per distinct node
        const bool on = (ok >> lane) & 1u;
        const unsigned same = __match_any_sync(FULL, on ? v.loc[lane] : -1 - lane);
        if (on && (__ffs(same) - 1) == lane) a.items[atomicAdd(&v.n_items, 1)] = make_uint2((unsigned)v.loc[lane], same);
    }
    __syncthreads();
    int lo = 0;
    for (int lev = 0; lev < MAX_ROUNDS; lev++) {
        const int hi = v.n_items;
        __syncthreads();
        if (lev + 2 >= (int)p.geo.lcap || hi + R > (int)p.geo.icap) {
            if (tid == 0) v.fail = 1;
            __syncthreads();
            return;
        }
        if (tid == 0) {
            v.n_level = lev + 1;
            a.lvl[lev + 1] = (uint32_t)hi;
        }
        // this level's items: path counts from the predecessors; the successors become candidates
        for (int q0 = lo + w; q0 < hi; q0 += NW * 4) {
            const int qi = q0 + (lane >> 3) * NW;
            const uint2 it = qi < hi ? a.items[qi] : make_uint2(0xffffffffu, 0u);
            const Quad q = load_quad(a, (int)it.x);
            unsigned m = 0u, many = 0u;
            if (q.e.to >= 0) {
                const size_t o = (size_t)q.i * PMAX + (lane & 7);
                m = a.pm[o] & it.y;
                const unsigned next = a.link[o].succ & it.y;
                if (next) {
                    atomicAnd(&a.left[q.e.back], ~next);
                    mark(sm.bits, q.e.to);
                    prefetch(&a.adj[(size_t)q.e.to * PMAX]);
                    prefetch(&a.link[(size_t)q.e.to * PMAX]);
                    prefetch(&a.pm[(size_t)q.e.to * PMAX]);
                }
            }
            if ((lane & 7) == 0 && q.i >= 0) {
                many = a.multi[q.i] & it.y;
                a.done[q.i] |= it.y;
            }
            const unsigned from = __ballot_sync(FULL, m != 0u);
#pragma unroll 1
            for (int t = 0; t < 4 && q0 + t * NW < hi; t++) {
                const int i = __shfl_sync(FULL, q.i, t * 8);
                const unsigned lanes = __shfl_sync(FULL, it.y, t * 8);
                const bool add = __shfl_sync(FULL, many, t * 8) != 0u;
                double s = (lev == 0) ? 1.0 : 0.0;
                for (unsigned f = (from >> (t * 8)) & 0xffu; f; f &= f - 1u) {
                    const int j = t * 8 + __ffs(f) - 1;
                    const unsigned mj = __shfl_sync(FULL, m, j);
                    const int xj = __shfl_sync(FULL, q.e.to, j);
                    const bool use = (mj >> lane) & 1u;
                    const double sx = use ? a.sig[(size_t)xj * 32 + lane] : 0.0;
                    if (add) s = __dadd_rn(s, sx);
                    else if (use) s = sx;
                }
                if ((lanes >> lane) & 1u) a.sig[(size_t)i * 32 + lane] = s;
            }
        }
        __syncthreads();
        // pass 0: candidates whose remaining lanes are all ready; pass 1: the ready lanes of a few others
        // (two sources can pass a street in opposite directions, so some nodes have to be split; each split
        // is another item for the sweeps, each node held back another level)
        for (int pass = 0; pass < 2; pass++) {
            uint32_t *bits = pass ? sm.part : sm.bits;
            for (int chunk = 0; chunk < MAX_ROUNDS; chunk++) {
                const int n = collect(bits, R, v.list, pass ? PART : LIST, v.wsum);
                for (int q = tid; q < n; q += TPB) {
                    const int i = v.list[q];
                    const unsigned rem = a.reach[i] & ok & ~a.done[i];
                    const uint4 *lf = (const uint4 *)&a.left[(size_t)i * PMAX];
                    const uint4 l0 = __ldcg(lf), l1 = __ldcg(lf + 1);
                    const unsigned wait = l0.x | l0.y | l0.z | l0.w | l1.x | l1.y | l1.z | l1.w;
                    const unsigned ready = rem & ~wait;
                    if (!ready) continue;
                    if (ready == rem || pass) {
                        const int o = atomicAdd(&v.n_items, 1);
                        a.items[o] = make_uint2((unsigned)i, ready);
                        atomicAdd(&v.sched, __popc(ready));
                        if (!pass) atomicAnd(&sm.part[i >> 5], ~(1u << (i & 31)));
                    } else {
                        atomicOr(&sm.part[i >> 5], 1u << (i & 31));
                    }
                }
                __syncthreads();
                if (pass || n < LIST) break;
            }
        }
        lo = hi;
        if (v.n_items == hi) {
            // every reached lane has its item, or the tile is left to the per-warp kernel
            if (tid == 0 && v.sched != v.sched_all) v.fail = 1;
            __syncthreads();
            return;
        }
    }
    if (tid == 0) v.fail = 1;
    __syncthreads();
}

// ------------------------------------------------------------------------------------------
// 5. Closeness (rust/src/centrality.rs:1733-1780).
// ------------------------------------------------------------------------------------------
__device__ void closeness(const Params &p, const Arrays &a, const Smem &sm) {
    Vars &v = sm.v;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int R = v.R, K = p.k, N = p.n_bound;
    const unsigned ok = v.ok;
    if (w == 0 && ((ok >> lane) & 1u)) {
        const float cycles_wt = __fdiv_rn(v.wt[lane], __ldg(&p.node_w[v.src[lane]]));
        long long nc = 0, ec = 0;
        for (int k = 0; k < K; k++) {
            nc += sm.cnt[k][lane];
            ec += sm.cnt[K + k][lane];
            const long long r = ec - nc + 1;
            const float rank = (nc == 0) ? 0.0f : (float)(r > 0 ? r : 0);
            sm.rankw[k][lane] = fmul(rank, cycles_wt);
            if (p.track_reach && nc > 1) atomicAdd(&p.reach[k], (unsigned)(nc - 1));
        }
    }
    __syncthreads();
    for (int k = w; k < K; k += NW) {  // the sum over all the tile's sources, of most nodes within k
        const FixSum f = fix_sum(((ok >> lane) & 1u) ? sm.rankw[k][lane] : 0.0f);
        if (lane == 0) v.rank_sum[k] = f;
    }
    __syncthreads();
    const size_t KN = (size_t)K * N;
    const bool on = (ok >> lane) & 1u;
    const int my_loc = v.loc[lane];
    const float wt = on ? v.wt[lane] : 0.0f;
    const bool unit = __all_sync(FULL, !on || wt == 1.0f);
    float d_next = w < R ? a.dist[(size_t)w * 32 + lane] : 0.0f;
    uint4 n_next = w < R ? *(const uint4 *)&a.node[w] : make_uint4(0u, 0u, 0u, 0u);
    for (int i = w; i < R; i += NW) {
        const float d = d_next;
        const Node nd{n_next.x, n_next.y, (int)n_next.z, 0u};
        if (i + NW < R) {  // the next node's row while this one is summed
            d_next = a.dist[(size_t)(i + NW) * 32 + lane];
            n_next = *(const uint4 *)&a.node[i + NW];
        }
        const int kmin = (nd.info >> 16) & 0xff;
        const int t = nd.id;
        const float c = fmul(d, p.speed);
        const bool live = on && d < inf_f() && i != my_loc;
        unsigned seen = 0u;  // lanes within a smaller threshold
        const float far = fmul(c, wt), har = fmul(__frcp_rn(c), wt);
        for (int k = kmin; k < K; k++) {
            const bool in = live && c <= p.dk[k];
            const unsigned m = __ballot_sync(FULL, in);
            if (m == 0u) continue;
            // lane q keeps sum q: 0 cycles, 1 beta, and for the lanes that this threshold is the first of,
            // 2 density, 3 farness, 4 harmonic
            const unsigned fresh = m & ~seen;
            const bool mine = in && ((fresh >> lane) & 1u);
            seen |= m;
            FixSum mys{0ull, 0};
            double slow = 0.0;
            auto keep = [&](int q, float x) {
                const FixSum f = fix_sum(x);
                if (f.e < 0) {
                    const double d = slow_sum(f2d(x));
                    if (lane == q) slow = d;
                }
                if (lane == q) mys = f;
            };
            if (m == ok && v.rank_sum[k].e >= 0) {
                if (lane == 0) mys = v.rank_sum[k];
            } else {
                keep(0, in ? sm.rankw[k][lane] : 0.0f);
            }
            keep(1, in ? fmul(expf(fmul(-p.beta[k], c)), wt) : 0.0f);
            if (fresh) {
                if (unit) {
                    if (lane == 2) mys = FixSum{(unsigned long long)__popc(fresh), BIAS_F};
                } else {
                    keep(2, mine ? wt : 0.0f);
                }
                keep(3, mine ? far : 0.0f);
                keep(4, mine ? har : 0.0f);
            }
            const double val = mys.e < 0 ? slow : fix_to_d(mys, BIAS_F);
            if (__double_as_longlong(val) == 0ll) continue;
            double *dst = (lane < 2) ? p.out + (lane == 0 ? 2 : 4) * KN : p.bucket + (size_t)(lane - 2) * KN;
            atomicAdd(dst + (size_t)k * N + t, val);
        }
    }
}

// ------------------------------------------------------------------------------------------
// 6. Dependencies, backward along the schedule (rust/src/centrality.rs:823-873, 1782-1835).
// ------------------------------------------------------------------------------------------
template <bool OD>
__device__ void backward(const Params &p, const Arrays &a, const Smem &sm) {
    Vars &v = sm.v;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int levels = v.n_level, K = p.k, N = p.n_bound;
    const int my_loc = v.loc[lane];
    const float wt = OD ? 1.0f : v.wt[lane];
    const bool unit = OD || __all_sync(FULL, !((v.ok >> lane) & 1u) || wt == 1.0f);
    const bool weighted = OD || !unit;
    constexpr int row0 = OD ? 0 : 5;
    for (int L = levels - 1; L >= 0; L--) {
        const int lo = (int)a.lvl[L], hi = (int)a.lvl[L + 1];
        {  // the level after this one: what its items will ask for
            const int qn = lo - 1 - (w * 4 + (lane >> 3));
            if (qn >= 0) {
                const size_t n = a.items[qn].x;
                const int j = lane & 7;
                if (j == 0) prefetch(&a.node[n]);
                else if (j == 1) prefetch(&a.link[n * PMAX]);
                else if (j == 2) prefetch(&a.dist[n * 32]);
            }
        }
        for (int q0 = lo + w; q0 < hi; q0 += NW * 4) {
            const int qi = q0 + (lane >> 3) * NW;
            const uint2 it = qi < hi ? a.items[qi] : make_uint2(0xffffffffu, 0u);
            const int my_i = (int)it.x;
            Link l{0u, 0u, K, 0};
            Node nd{0u, 0u, 0, 0u};
            if (my_i >= 0) {
                l = a.link[(size_t)my_i * PMAX + (lane & 7)];
                nd = a.node[my_i];
            }
            const unsigned m = l.succ & it.y, mult = l.multi & it.y;
            const unsigned mults = __ballot_sync(FULL, mult != 0u);
            float dd[4];
#pragma unroll
            for (int t = 0; t < 4; t++) {
                const int i = __shfl_sync(FULL, my_i, t * 8);
                dd[t] = i >= 0 ? a.dist[(size_t)i * 32 + lane] : 0.0f;
            }
#pragma unroll 1
            for (int t = 0; t < 4 && q0 + t * NW < hi; t++) {
                const uint32_t info = __shfl_sync(FULL, nd.info, t * 8);
                const int kmin = (info >> 16) & 0xff;
                const float d = t == 0 ? dd[0] : t == 1 ? dd[1] : t == 2 ? dd[2] : dd[3];
                if (kmin >= K) continue;
                const int i = __shfl_sync(FULL, my_i, t * 8);
                const unsigned lanes = __shfl_sync(FULL, it.y, t * 8);
                const unsigned dep0 = __shfl_sync(FULL, nd.dep, t * 8);
                const bool on = (lanes >> lane) & 1u;
                const bool src = i == my_loc;
                const float cost = fmul(d, p.speed);
                float pairf;
                if constexpr (OD) pairf = on ? a.trip[(size_t)i * 32 + lane] : 0.0f;
                else pairf = ((info >> 24) & 1u) ? 0.5f : 1.0f;
                const bool any_mult = (mults >> (t * 8)) & 0xffu;
                const double sv = any_mult ? a.sig[(size_t)i * 32 + lane] : 1.0;
                for (int k = kmin; k < K; k++) {
                    const bool seeded = on && cost <= p.dk[k] && !src && pairf != 0.0f;
                    double dep = 0.0, depb = 0.0;
                    if (seeded) {
                        if constexpr (OD) dep = f2d(pairf);
                        else dep = __hiloint2double(pairf == 1.0f ? 0x3ff00000 : 0x3fe00000, 0);
                        depb = seed_exp(pairf, p.beta[k], cost);
                    }
                    double *row = a.dep + (size_t)(dep0 + (k - kmin)) * 64 + lane;
                    // rows below a successor's first threshold do not exist: it is beyond k for every lane
                    unsigned f = (__ballot_sync(FULL, m != 0u && k >= l.k0) >> (t * 8)) & 0xffu;
                    if (f == 0u) {
                        if (on) {
                            row[0] = dep;
                            row[32] = depb;
                        }
                        continue;
                    }
                    double acc = 0.0, accb = 0.0;
                    unsigned seen = 0u;  // lanes that have a successor so far
                    for (; f; f &= f - 1u) {
                        const int j = t * 8 + __ffs(f) - 1;
                        const unsigned mj = __shfl_sync(FULL, m, j);
                        const double *r = a.dep + (size_t)(__shfl_sync(FULL, l.row, j) + k) * 64 + lane;
                        const bool use = (mj >> lane) & 1u;
                        double f0 = use ? r[0] : 0.0, f1 = use ? r[32] : 0.0;
                        if (any_mult) {  // a successor with several predecessors: its paths' share through here
                            const unsigned mm = __shfl_sync(FULL, mult, j);
                            const int xj = a.adj[(size_t)i * PMAX + (j & 7)].to;
                            if ((mm >> lane) & 1u) {
                                const double g = __ddiv_rn(sv, a.sig[(size_t)xj * 32 + lane]);
                                f0 = __dmul_rn(g, f0);
                                f1 = __dmul_rn(g, f1);
                            }
                        }
                        if (seen & mj) {
                            acc = __dadd_rn(acc, f0);
                            accb = __dadd_rn(accb, f1);
                        } else if (use) {  // first successors: nothing to add to
                            acc = f0;
                            accb = f1;
                        }
                        seen |= mj;
                    }
                    dep = __dadd_rn(dep, acc);
                    depb = __dadd_rn(depb, accb);
                    if (on) {
                        row[0] = dep;
                        row[32] = depb;
                    }
                    if (src || !on) acc = accb = 0.0;
                    if (weighted) {
                        // a source credits a node only with what is positive, as the reference does per source
                        // (its dependency - seed is NaN at a destination whose trips have no finite weight);
                        // without weights what is not positive is NaN, which the sums below notice
                        const bool credited = !OD || fabsf(pairf) < inf_f();
                        acc = credited && positive(acc) ? (unit ? acc : __dmul_rn(acc, f2d(wt))) : 0.0;
                        accb = credited && positive(accb) ? (unit ? accb : __dmul_rn(accb, f2d(wt))) : 0.0;
                    }
                    const FixSum s0 = fix_sum(acc), s1 = fix_sum(accb);
                    double val = fix_to_d(lane ? s1 : s0, BIAS_D);
                    if ((s0.e < 64 && (s0.e < 0 || s0.sum)) || (s1.e < 64 && (s1.e < 0 || s1.sum))) {
                        // not finite, of a negative source weight, or close to the smallest f64
                        if (!weighted && !positive(acc)) acc = 0.0;
                        if (!weighted && !positive(accb)) accb = 0.0;
                        const double d0 = slow_sum(acc), d1 = slow_sum(accb);
                        val = lane ? d1 : d0;
                    }
                    const int id = __shfl_sync(FULL, nd.id, t * 8);
                    if (lane < 2 && __double_as_longlong(val) != 0ll)
                        atomicAdd(p.out + ((size_t)(row0 + lane) * K + k) * N + id, val);
                }
            }
        }
        __syncthreads();
    }
}

// Trip weights of the tile's origins as rows over the tile's nodes.
__device__ void trips(const Params &p, const Arrays &a, const Smem &sm, const uint32_t *aux) {
    Vars &v = sm.v;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int R = v.R;
    float4 *rows = (float4 *)a.trip;
    for (int i = tid; i < R * 8; i += TPB) rows[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    __syncthreads();
    for (int s = w; s < v.nl; s += NW) {
        const int end = __ldg(&p.od_ptr[v.src[s] + 1]);
        for (int q = __ldg(&p.od_ptr[v.src[s]]) + lane; q < end; q += 32) {
            const int to = __ldg(&p.od_dst[q]);
            if (to < 0 || to >= p.n_bound) continue;
            const uint32_t id = aux[to];
            if (id != 0u && id <= (uint32_t)R) a.trip[(size_t)(id - 1) * 32 + s] = __ldg(&p.od_w[q]);
        }
    }
    __syncthreads();
}

// What a block counts over its tiles, added to the header at its end.
struct Counts {
    unsigned long long done = 0;
    long long ph[7] = {0, 0, 0, 0, 0, 0, 0};  // cycles: union, adjacency, search, replay, schedule, closeness, betweenness
};

// One tile: sources [base, base + nl) of p.src_list.  v.fail on entry: list them at once.
template <bool OD>
__device__ void run_tile(const Params &p, const Arrays &a, const Smem &sm, float *d1, uint32_t *aux, long long base,
                         int nl, Counts &n) {
    Vars &v = sm.v;
    const int tid = threadIdx.x;
    long long t0 = clock64();
    auto mark_phase = [&](int q) {
        const long long now = clock64();
        n.ph[q] += now - t0;
        t0 = now;
    };
    if (tid < 32) {
        const int s = tid < nl ? __ldg(&p.src_list[base + tid]) : 0;
        v.src[tid] = s;
        v.loc[tid] = -1;
        v.wt[tid] = (tid < nl && !OD) ? __ldg(&p.src_wt[s]) : 1.0f;
        if (tid == 0) {
            v.nl = nl;
            v.ok = nl == 32 ? FULL : (1u << nl) - 1u;
            v.tcount = 0u;
        }
    }
    for (int i = tid; i < 2 * 32 * p.k; i += TPB) ((int *)sm.cnt)[i] = 0;
    __syncthreads();
    bool whole = false;  // the numbering lost nodes: reset the whole dense state
    const bool skip = v.fail != 0;
    __syncthreads();
    if (!skip) {
        discover(p, a, sm, d1, aux);
        mark_phase(0);
        whole = v.fail != 0;
        __syncthreads();
        if (!whole) {
            if (tid < nl) v.loc[tid] = (int)aux[v.src[tid]] - 1;
            __syncthreads();
            adjacency(p, a, sm, d1, aux);
        }
    }
    mark_phase(1);
    if (!v.fail) search(p, a, sm);
    mark_phase(2);
    if (!v.fail) {
        replay(p, a, sm);
        mark_phase(3);
        if (p.betweenness) {
            links(p, a, sm);
            schedule(p, a, sm);
        }
        mark_phase(4);
    }
    __syncthreads();
    const bool fail = v.fail != 0;
    const unsigned ok = fail ? 0u : v.ok;
    if (tid < nl && !((ok >> tid) & 1u)) {
        // nothing was written for this source: the per-warp kernel redoes it
        const unsigned f = atomicAdd(p.n_failed, 1u);
        if (f < (unsigned)p.fail_cap) p.failed[f] = (int)(p.item0 + base + tid);
        else raise_err(p.hdr, CS_ERR_CAPACITY, 50);
    }
    if (ok) {
        if (!OD && p.closeness) closeness(p, a, sm);
        mark_phase(5);
        if (p.betweenness) {
            if (OD) trips(p, a, sm, aux);
            backward<OD>(p, a, sm);
        }
        mark_phase(6);
        n.done += __popc(ok);
        if (tid == 0) atomicAdd(&p.hdr->pad[PROGRESS_SLOT], (unsigned long long)__popc(ok));
    }
    __syncthreads();
    if (whole) {
        for (int i = tid; i < p.n_bound; i += TPB) {
            d1[i] = inf_f();
            aux[i] = 0u;
        }
    } else if (!skip) {
        const int R = v.R;
        for (int i = tid; i < R; i += TPB) {
            const int x = a.rl[i];
            d1[x] = inf_f();
            aux[x] = 0u;
        }
    }
    __syncthreads();
}

__device__ __forceinline__ void flush_counts(WsHeader *h, const Vars &v, const Counts &n) {
    if (threadIdx.x != 0) return;
    atomicAdd(&h->edges_relaxed, v.relaxed);
    atomicAdd(&h->nodes_settled, v.settled);
    atomicAdd(&h->sources_done, n.done);
    atomicAdd(&h->pad[SERVED_SLOT], n.done);
    for (int q = 0; q < 7; q++) atomicAdd(&h->pad[q], (unsigned long long)n.ph[q]);
}

template <bool OD>
__global__ void __launch_bounds__(TPB, BPSM) tile_kernel(const __grid_constant__ Params p) {
    extern __shared__ __align__(16) char sm_raw[];
    const Smem sm = smem(sm_raw, p.k, p.geo.mcap);
    Vars &v = sm.v;
    const Arrays a = arrays(p);
    float *d1 = (float *)(p.dense + p.dense_stride * (size_t)blockIdx.x);
    uint32_t *aux = (uint32_t *)(p.dense + p.dense_stride * (size_t)blockIdx.x + p.aux_off);
    Counts n;
    if (threadIdx.x == 0) {
        v.settled = v.relaxed = 0ull;
        v.job = 0;
    }
    while (true) {
        if (threadIdx.x == 0) {
            v.base = (long long)atomicAdd(&p.hdr->work_next, 1ull) * p.lanes;
            v.herr = __ldcg(&p.hdr->err);
            v.fail = is_unpaired(p.hdr, 0);
        }
        __syncthreads();
        const long long base = v.base;
        if (base >= p.n_src || v.herr != 0u) break;
        run_tile<OD>(p, a, sm, d1, aux, base, (int)min((long long)p.lanes, p.n_src - base), n);
    }
    flush_counts(p.hdr, v, n);
}

// A batch's jobs [lo, hi), their sources in tiles of 32: block-wide parameters in shared memory, rewritten
// when the block's job changes (the tiles come in job order).
__global__ void __launch_bounds__(TPB, BPSM) tile_batch_kernel(const __grid_constant__ Params base,
                                                               const cs_batch_job *jobs, int lo, int hi, int kmax) {
    extern __shared__ __align__(16) char sm_raw[];
    __shared__ Params p;
    const Smem sm = smem(sm_raw, kmax, base.geo.mcap);
    Vars &v = sm.v;
    const Arrays a = arrays(base);
    float *d1 = (float *)(base.dense + base.dense_stride * (size_t)blockIdx.x);
    uint32_t *aux = (uint32_t *)(base.dense + base.dense_stride * (size_t)blockIdx.x + base.aux_off);
    Counts n;
    int cur = -1;                 // thread 0: the job p holds, and the tiles of the jobs before the next one
    long long before = 0, first = 0;
    if (threadIdx.x == 0) {
        v.settled = v.relaxed = 0ull;
        cur = lo - 1;
    }
    while (true) {
        if (threadIdx.x == 0) {
            const long long t = (long long)atomicAdd(&base.hdr->work_next, 1ull);
            v.herr = __ldcg(&base.hdr->err);
            int j = cur;
            while (j < hi && t >= before) {
                j++;
                first = before;
                if (j < hi) before += (max(jobs[j].n_sources, 0) + 31) / 32;
            }
            if (j >= hi) {
                v.base = -1;
            } else {
                if (j != cur) {
                    const cs_batch_job &b = jobs[j];
                    p = base;
                    p.n_bound = b.g.n_bound;
                    p.in_ptr = b.g.in_ptr_dev;
                    p.in_nb = b.g.in_nb_dev;
                    p.in_w = b.g.in_w_dev;
                    p.out_ptr = b.g.out_ptr_dev;
                    p.out_to = b.g.out_to_dev;
                    p.out_w = b.g.out_w_dev;
                    p.out_cnt = b.g.out_cnt_dev;
                    p.node_w = b.g.node_w_dev;
                    p.k = b.k;
                    uint32_t maxs = 0;
                    for (int i = 0; i < b.k; i++) {
                        p.dk[i] = (float)b.distances[i];
                        p.beta[i] = b.betas[i];
                        maxs = max(maxs, b.seconds[i]);
                    }
                    p.maxsec = (float)maxs;
                    p.speed = b.speed_m_s;
                    p.tol = b.tolerance;
                    p.delta = b.delta_seconds;
                    p.closeness = b.compute_closeness;
                    p.betweenness = b.compute_betweenness;
                    p.src_list = b.sources_dev;
                    p.n_src = b.n_sources;
                    p.src_wt = b.src_wt_dev;
                    p.eligible = b.eligible_dev;
                    p.out = b.out_dev;
                    p.bucket = b.bucket_dev;
                    p.item0 = b.item_begin;
                    cur = j;
                }
                v.base = (t - first) * 32;
                v.job = j;
                v.fail = is_unpaired(base.hdr, j);
            }
        }
        __syncthreads();
        const long long at = v.base;
        if (at < 0 || v.herr != 0u) break;
        run_tile<false>(p, a, sm, d1, aux, at, (int)min(32ll, p.n_src - at), n);
    }
    flush_counts(base.hdr, v, n);
}

// ==========================================================================================
// Host side.
// ==========================================================================================
Geometry geometry(size_t region_bytes, int k, const float *dk, bool od) {
    Geometry g{};
    // dependency rows per node: a node holds those of the thresholds that its nearest source lies within;
    // reach grows with the square of the threshold, with room for the tile's own extent
    double rows = 0.1;
    for (int i = 0; i < k; i++) {
        const double r = (dk[i] + 0.1 * dk[k - 1]) / (1.1 * dk[k - 1]);
        rows += std::min(1.0, r * r);
    }
    rows = std::min((double)k, rows * 1.1);
    const size_t lcap = 16384;
    const double per = 4 + 16 + 40.0 * PMAX + 128 + 12 + 256 + 3 * 8 + 512 * rows + (od ? 128 : 0);
    const double room = (double)region_bytes - 4.0 * lcap - 16 * 256;
    if (room <= per * 64) return g;
    g.mcap = (int32_t)std::min<double>(MMAX, std::floor(room / per));
    g.mcap &= ~31;
    g.tcap = (uint32_t)((double)g.mcap * rows);
    g.icap = 3u * (uint32_t)g.mcap;
    g.lcap = (uint32_t)lcap;
    auto al = [](size_t x) { return (x + 255) & ~size_t(255); };
    size_t o = 0;
    const size_t m = (size_t)g.mcap;
    g.o_rl = o; o += al(4 * m);
    g.o_node = o; o += al(16 * m);
    g.o_adj = o; o += al(16 * m * PMAX);
    g.o_link = o; o += al(16 * m * PMAX);
    g.o_dist = o; o += al(128 * m);
    g.o_pm = o; o += al(8 * m * PMAX);
    g.o_masks = o; o += al(12 * m);
    g.o_sig = o; o += al(256 * m);
    g.o_items = o; o += al(8 * (size_t)g.icap);
    g.o_lvl = o; o += al(4 * lcap);
    g.o_dep = o; o += al(512 * (size_t)g.tcap);
    g.o_trip = o; o += od ? al(128 * m) : 0;
    g.total = o;
    if (g.total > region_bytes) g.mcap = 0;
    return g;
}

template <bool OD>
cudaError_t launch_t(const Params &p, int blocks, cudaStream_t stream) {
    tile_kernel<OD><<<blocks, TPB, smem_bytes(p.k, p.geo.mcap), stream>>>(p);
    return cudaGetLastError();
}

cudaError_t launch(const Params &p, bool od, int blocks, cudaStream_t stream) {
    return od ? launch_t<true>(p, blocks, stream) : launch_t<false>(p, blocks, stream);
}

cudaError_t launch_batch(const Params &p, const cs_batch_job *jobs_dev, int lo, int hi, int kmax, int blocks,
                         cudaStream_t stream) {
    tile_batch_kernel<<<blocks, TPB, smem_bytes(kmax, p.geo.mcap), stream>>>(p, jobs_dev, lo, hi, kmax);
    return cudaGetLastError();
}

cudaError_t launch_seed_table(cudaStream_t stream) {
    seed_table_kernel<<<(SEED_TAB + 255) / 256, 256, 0, stream>>>();
    return cudaGetLastError();
}

}  // namespace tile
}  // namespace cs
