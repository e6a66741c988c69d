"""What a user of the framework has it compute, as cases that can be timed and compared.

A case is one call (or one round of calls) through the public entry points on synthetic street
networks: jittered lattices of the sizes, spacings and thresholds of the benchmark configurations and
the tests.  `listed()` gives the fixed cases, `draw(rng)` another one of the same ranges,
`prepare(case, seed)` the inputs (the graph a program has ingested, its sources, data or plans),
`run(state)` one pass, `work(case)` what a pass cannot do without, and `exact(case, seed)` the same
outputs from plain torch in 64 bits.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from cityseer_gb300 import synth
from cityseer_gb300.batch import Batch
from cityseer_gb300.centrality import OdMatrix
from cityseer_gb300.data import DataMap
from cityseer_gb300.graph import NetworkStructure
from cityseer_gb300.metrics import networks
from cityseer_gb300.serve import Query, Server

SPEED = 1.33333
BETA_LOG = -math.log(0.01831563888873418)
TIE = 1e-4

SHORTEST = ("node_density", "node_farness", "node_cycles", "node_harmonic", "node_beta", "node_betweenness",
            "node_betweenness_beta")
SIMPLEST = ("node_density", "node_farness", "node_harmonic", "node_betweenness")
SEGMENT = ("segment_density", "segment_harmonic", "segment_beta", "segment_betweenness")


def _dists(case) -> list[int]:
    return [int(d) for d in str(case["distances"]).split(",")]


# ---------------------------------------------------------------------------------------------
# Cases
# ---------------------------------------------------------------------------------------------
def listed():
    return [
        # one address asked for interactively on a neighbourhood graph: latency and launches
        dict(name="one_address", kind="subset", side=40, spacing=100.0, jitter=20.0, drop=0.15, diag=0.0,
             distances="400,800", sources=1, tolerance=0.0),
        # a small town, every node a source (the 1,600-node configuration), written to columns
        dict(name="town", kind="shortest", side=40, spacing=100.0, jitter=20.0, drop=0.15, diag=0.0,
             distances="500,1000,2000"),
        # a city, every node a source, to 5 km (the 202,500-node configuration): the largest
        dict(name="city", kind="shortest", side=450, spacing=80.0, jitter=15.0, drop=0.10, diag=0.05,
             distances="500,1000,2000,5000"),
        # a tenth of a district's nodes as sources, with a route tolerance: sampled estimates
        dict(name="district_sample", kind="subset", side=141, spacing=100.0, jitter=20.0, drop=0.15, diag=0.0,
             distances="800,1600,3200", sources=1989, tolerance=1.0),
        # a few hundred addresses spread over a city, long distances: a planning query
        dict(name="city_addresses", kind="subset", side=300, spacing=80.0, jitter=15.0, drop=0.10, diag=0.05,
             distances="1000,5000", sources=700, tolerance=0.0),
        # metric segments of a city with curved streets (the 62,500-node configuration)
        dict(name="segments", kind="segment", side=250, spacing=80.0, jitter=15.0, drop=0.0, diag=0.0,
             distances="500,1000,2000"),
        # angular centrality on the dual of a district, every street a source
        dict(name="angular", kind="simplest", side=150, spacing=80.0, jitter=15.0, drop=0.05, diag=0.0,
             distances="500,1000,2000", sources=0),
        # angular centrality of a few streets: an interactive query on the dual
        dict(name="angular_streets", kind="simplest", side=91, spacing=80.0, jitter=15.0, drop=0.05, diag=0.0,
             distances="800,1600", sources=37),
        # betweenness of trips between homes and work places
        dict(name="trips", kind="od", side=121, spacing=100.0, jitter=20.0, drop=0.15, diag=0.0,
             distances="1600,3200", origins=3001, trips=9),
        # land uses within walking distance of every node
        dict(name="land_uses", kind="access", side=101, spacing=100.0, jitter=20.0, drop=0.15, diag=0.0,
             distances="400,800,1600", points=257, classes=4),
        # many towns of uneven size in one persistent launch (the batched configuration's recipe)
        dict(name="towns_batched", kind="batch", graphs=9, min_side=45, max_side=160),
        # queries of mixed kinds and sizes arriving together at the server
        dict(name="queries_served", kind="serve", side=161, spacing=100.0, jitter=20.0, drop=0.15, diag=0.0,
             queries=24, max_distance=3000, max_sources=600),
    ]


def _log_int(rng, lo, hi) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _some(rng, choices, lo, hi) -> str:
    return ",".join(str(d) for d in sorted(rng.sample(list(choices), rng.randint(lo, hi))))


def draw(rng):
    kind = rng.choice(["shortest", "shortest", "subset", "subset", "segment", "simplest", "simplest", "od", "access",
                       "batch", "serve"])
    if rng.random() < 0.5:
        street = dict(spacing=100.0, jitter=20.0, drop=0.15, diag=0.0)
    else:
        street = dict(spacing=80.0, jitter=15.0, drop=0.10, diag=0.05)
    if kind == "shortest":
        return dict(kind=kind, side=_log_int(rng, 30, 300), **street,
                    distances=_some(rng, (400, 500, 800, 1000, 1600, 2000, 3200, 5000), 1, 4))
    if kind == "subset":
        side = _log_int(rng, 30, 300)
        return dict(kind=kind, side=side, **street, distances=_some(rng, (400, 800, 1000, 1600, 3200, 5000), 1, 3),
                    sources=min(_log_int(rng, 1, 8192), side * side // 2), tolerance=rng.choice([0.0, 0.0, 0.0, 1.0, 2.5]))
    if kind == "segment":
        return dict(kind=kind, side=_log_int(rng, 30, 230), spacing=80.0, jitter=15.0, drop=rng.choice([0.0, 0.1]),
                    diag=0.0, distances=_some(rng, (400, 500, 800, 1000, 1600, 2000), 1, 4))
    if kind == "simplest":
        side = _log_int(rng, 25, 140)
        return dict(kind=kind, side=side, spacing=80.0, jitter=15.0, drop=rng.choice([0.0, 0.05, 0.15]), diag=0.0,
                    distances=_some(rng, (400, 500, 800, 1000, 1600, 2000), 1, 3),
                    sources=rng.choice([0, 0, min(_log_int(rng, 1, 4096), side * side)]))
    if kind == "od":
        side = _log_int(rng, 40, 160)
        return dict(kind=kind, side=side, **street, distances=_some(rng, (800, 1600, 2000, 3200), 1, 3),
                    origins=min(_log_int(rng, 50, 6000), side * side // 2), trips=rng.randint(1, 20))
    if kind == "access":
        return dict(kind=kind, side=_log_int(rng, 30, 110), **street, distances=_some(rng, (400, 800, 1600, 2000), 1, 3),
                    points=_log_int(rng, 20, 280), classes=rng.randint(1, 6))
    if kind == "batch":
        return dict(kind=kind, graphs=rng.randint(3, 10), min_side=45, max_side=_log_int(rng, 60, 160))
    return dict(kind="serve", side=_log_int(rng, 60, 170), spacing=100.0, jitter=20.0, drop=0.15, diag=0.0,
                queries=rng.randint(8, 28), max_distance=rng.choice([1600, 2400, 3000]), max_sources=_log_int(rng, 50, 600))


# ---------------------------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------------------------
def _streets(case, seed: int) -> synth.Primal:
    """A jittered lattice: streets dropped at random, some nodes with one diagonal shortcut of
    Euclidean length x U(1, 1.3); lengths in f32."""
    rng = np.random.default_rng(seed)
    side, sp, jit = int(case["side"]), float(case["spacing"]), float(case["jitter"])
    n = side * side
    ii, jj = np.divmod(np.arange(n), side)
    x = jj * sp + rng.uniform(-jit, jit, n)
    y = ii * sp + rng.uniform(-jit, jit, n)
    right, down = np.nonzero(jj < side - 1)[0], np.nonzero(ii < side - 1)[0]
    u = np.concatenate([right, down])
    v = np.concatenate([right + 1, down + side])
    keep = np.sort(rng.permutation(len(u))[int(round(float(case["drop"]) * len(u))):])  # as many for every seed
    u, v = u[keep], v[keep]
    stretch = np.ones(len(u))
    if case["kind"] == "segment":  # curved streets are longer than their chords
        curved = rng.random(len(u)) < 0.3
        stretch[curved] = rng.uniform(1.0, 1.1, int(curved.sum()))
    if case["diag"] > 0:
        who = np.nonzero((rng.random(n) < float(case["diag"])) & (ii < side - 1) & (jj < side - 1) & (jj > 0))[0]
        to = who + side + rng.choice([-1, 1], len(who))
        u, v = np.concatenate([u, who]), np.concatenate([v, to])
        stretch = np.concatenate([stretch, rng.uniform(1.0, 1.3, len(who))])
    length = (np.hypot(x[v] - x[u], y[v] - y[u]) * stretch).astype(np.float32)
    return synth.Primal(x=x, y=y, u=u, v=v, length=length, angle_sum=np.zeros(len(u), np.float32),
                        geoms=[None] * len(u), stretched=stretch)


def _picked(n: int, count: int, seed: int) -> np.ndarray:
    return np.sort(np.random.default_rng(seed + 77).choice(n, size=min(count, n), replace=False))


def _trips(case, seed: int, n: int):
    rng = np.random.default_rng(seed + 78)
    o = np.repeat(_picked(n, int(case["origins"]), seed), int(case["trips"]))
    side = int(case["side"])
    oi, oj = np.divmod(o, side)
    reach = max(2, int(max(_dists(case)) / float(case["spacing"]) / 2))
    di = np.clip(oi + rng.integers(-reach, reach + 1, len(o)), 0, side - 1)
    dj = np.clip(oj + rng.integers(-reach, reach + 1, len(o)), 0, side - 1)
    d = di * side + dj
    w = rng.uniform(0.5, 20.0, len(o)).astype(np.float32)
    _, first = np.unique(o * n + d, return_index=True)  # a pair is named once
    first = np.sort(first)
    return o[first], d[first], w[first]


def _batch_graphs(case, seed: int):
    rng = np.random.default_rng(79)  # the same sizes for every seed
    for g in range(int(case["graphs"])):
        side = int(round(math.exp(rng.uniform(math.log(case["min_side"]), math.log(case["max_side"])))))
        dists = sorted(int(d) for d in rng.choice(synth.BATCH_THRESHOLDS[:5], size=int(rng.integers(2, 4)), replace=False))
        one = dict(kind="shortest", side=side, spacing=100.0, jitter=20.0, drop=0.15, diag=0.0,
                   distances=",".join(map(str, dists)))
        yield one, seed * 1000 + g, dists


def _queries(case, seed: int, n: int, n_dual: int) -> list[Query]:
    """Log-uniform source counts, a fifth on the dual; the kinds and sizes are the same for every seed."""
    rng, size = np.random.default_rng(seed + 80), np.random.default_rng(80)
    out = []
    for q in range(int(case["queries"])):
        mode = "simplest" if q % 5 == 4 else ("segment" if q % 8 == 6 else "shortest")
        count = int(round(math.exp(size.uniform(0.0, math.log(case["max_sources"])))))
        count = min(count, 60) if mode == "simplest" else count
        top = int(rng.uniform(400, 1200 if mode == "simplest" else case["max_distance"]))
        dists = sorted([int(d) for d in rng.choice(np.arange(200, top), int(size.integers(0, 3)), replace=False)] + [top])
        if mode == "segment":
            count = n  # segments take every node
        src = rng.choice(n_dual if mode == "simplest" else n, size=count, replace=False)
        out.append(Query(graph=0, sources=[int(s) for s in src], distances=dists, mode=mode))
    return out


def prepare(case, seed):
    kind = case["kind"]
    st = dict(kind=kind, case=case)
    if kind == "batch":
        jobs = []
        for one, s, dists in _batch_graphs(case, seed):
            ns = synth.primal_structure(_streets(one, s))
            jobs.append(dict(ns=ns, mode="shortest", distances=dists))
            if len(jobs) % 3 == 0:
                jobs.append(dict(ns=ns, mode="segment", distances=dists))
        st["jobs"], st["batch"] = jobs, Batch(jobs)
        st["batch"].capture()
        return st
    p = _streets(case, seed)
    n = int(case["side"]) ** 2
    if kind != "simplest":
        st["ns"] = synth.primal_structure(p)
    if kind in ("simplest", "serve"):
        st["dual"] = synth.dual_structure(p)
    if kind == "subset":
        st["sources"] = [int(s) for s in _picked(n, int(case["sources"]), seed)]
    elif kind == "simplest":
        st["sources"] = [int(s) for s in _picked(len(p.u), int(case["sources"]), seed)] if case["sources"] else None
    elif kind == "od":
        st["od"] = OdMatrix(*_trips(case, seed, n))
    elif kind == "access":
        pts = _points(case, seed)
        dm = DataMap()
        for i, (x, y) in enumerate(pts):
            dm.insert(i, f"POINT ({x} {y})")
        dm.assign_data_to_network(st["ns"], 400.0, 20)
        st["data"] = dm
        st["keys"] = [f"c{c}" for c in range(int(case["classes"]))]
        st["uses"] = {i: f"c{i % int(case['classes'])}" for i in range(len(pts))}
    elif kind == "serve":
        st["queries"] = _queries(case, seed, n, len(p.u))
        st["server"] = Server({0: st["ns"]}, {0: st["dual"]}, max_distance=int(case["max_distance"]),
                              max_thresholds=3, max_slots=2432, dual_slots=608, hbm_budget_bytes=8 << 30)
    return st


def _points(case, seed: int) -> np.ndarray:
    rng = np.random.default_rng(seed + 81)
    span = (int(case["side"]) - 1) * float(case["spacing"])
    return np.round(rng.uniform(0.0, span, (int(case["points"]), 2)), 3)


# ---------------------------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------------------------
def _rows(res, names) -> dict:
    return {f"{name}_{d}": col for name in names for d, col in getattr(res, name).items()}


def _stacked(res, mode) -> np.ndarray:
    names = {"shortest": SHORTEST, "simplest": SIMPLEST, "segment": SEGMENT}[mode]
    return np.stack([np.stack(list(getattr(res, m).values())) for m in names])


def run(state):
    kind, case = state["kind"], state["case"]
    if kind == "batch":
        state["batch"].replay()
        return [_stacked(r, job["mode"]) for r, job in zip(state["batch"].results(), state["jobs"])]
    if kind == "serve":
        with state["server"] as server:
            tickets = [server.submit(q) for q in state["queries"]]
            out = []
            for t in tickets:
                res = t.result(timeout=60)
                t.release()
                out.append(_stacked(res, t.query.mode))
        return out
    if kind == "simplest":
        if state["sources"] is None:
            cols = networks.node_centrality_simplest(state["dual"], {}, distances=_dists(case))
            return {k: v for k, v in cols.items() if k != "index"}
        return _rows(state["dual"].centrality_simplest(distances=_dists(case), source_indices=state["sources"]), SIMPLEST)
    ns = state["ns"]
    if kind == "shortest":
        cols = networks.node_centrality_shortest(ns, {}, distances=_dists(case))
        return {k: v for k, v in cols.items() if k != "index"}
    if kind == "subset":
        tol = float(case["tolerance"])
        res = ns.centrality_shortest(distances=_dists(case), source_indices=state["sources"],
                                     tolerance=tol if tol > 0 else None)
        return {**_rows(res, SHORTEST), "reachability": np.array(res.reachability_totals, np.int64)}
    if kind == "segment":
        cols = networks.segment_centrality(ns, {}, distances=_dists(case))
        return {k: v for k, v in cols.items() if k != "index"}
    if kind == "od":
        res = ns.betweenness_od_shortest(state["od"], distances=_dists(case))
        return _rows(res, ("node_betweenness", "node_betweenness_beta"))
    res = state["data"].accessibility(ns, state["uses"], state["keys"], distances=_dists(case))
    out = {}
    for key, acc in res.result.items():
        for d in _dists(case):
            out[f"{key}_{d}_nw"], out[f"{key}_{d}_wt"] = acc.unweighted[d], acc.weighted[d]
        out[f"{key}_nearest"] = acc.distance[max(_dists(case))]
    return out


# ---------------------------------------------------------------------------------------------
# What a pass cannot do without
# ---------------------------------------------------------------------------------------------
def _work_one(side, spacing, dists, n_src, kind):
    """Graph and rows once; per source, each street within reach relaxed once from both ends (an add
    and a compare) and each metric's sum per node and threshold within."""
    n = side * side
    nodes, edges = (n, 4.0 * n) if kind != "simplest" else (2.0 * n, 12.0 * n)
    metrics = {"shortest": 7, "subset": 7, "segment": 4, "simplest": 4, "od": 2}.get(kind, 2)
    reach = [min(nodes, 1.5 * (d / spacing) ** 2 * nodes / n) for d in dists]
    byts = edges * 8 + nodes * (8 + 8 * metrics * len(dists)) + 4 * n_src
    return dict(bytes=byts, flops=n_src * (2 * edges / nodes * max(reach) + metrics * 2 * sum(reach)))


def work(case):
    kind = case["kind"]
    if kind == "batch":
        total = dict(bytes=0.0, flops=0.0)
        for one, _, dists in _batch_graphs(case, 0):
            w = _work_one(one["side"], 100.0, dists, one["side"] ** 2, "shortest")
            total = {k: total[k] + w[k] for k in total}
        return total
    n = case["side"] ** 2
    if kind == "serve":
        total = dict(bytes=0.0, flops=0.0)
        for q in _queries(case, 0, n, int(1.6 * n)):
            w = _work_one(case["side"], case["spacing"], q.distances, len(q.sources),
                          "simplest" if q.mode == "simplest" else "shortest")
            total = {k: total[k] + w[k] for k in total}
        return total
    n_src = case.get("sources") or case.get("origins") or (2 * n if kind == "simplest" else n)
    return _work_one(case["side"], case["spacing"], _dists(case), n_src, kind)


# ---------------------------------------------------------------------------------------------
# The same in 64 bits
# ---------------------------------------------------------------------------------------------
class _Exact:
    """Distances, predecessors and path counts from a block of sources, dense over the nodes."""

    def __init__(self, p: synth.Primal, n: int):
        self.dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
        src = np.concatenate([p.u, p.v])
        dst = np.concatenate([p.v, p.u])
        ln = np.concatenate([p.length, p.length]).astype(np.float64)
        order = np.lexsort((dst, src))
        src, dst, ln = src[order], dst[order], ln[order]
        deg = np.bincount(src, minlength=n)
        first = np.concatenate([[0], np.cumsum(deg)])
        self.n, self.deg = n, int(deg.max())
        nbr = np.full((n, self.deg), n, np.int64)
        w = np.full((n, self.deg), np.inf)
        slot = np.arange(len(src)) - first[src]
        nbr[src, slot], w[src, slot] = dst, ln
        rev = np.zeros((n, self.deg), np.int64)  # the slot of v's list that names u
        rev[src, slot] = slot[np.searchsorted(src * n + dst, dst * n + src)]
        self.nbr = torch.from_numpy(nbr).to(self.dev)
        self.w = torch.from_numpy(w).to(self.dev)
        self.rev = torch.from_numpy(rev).to(self.dev)

    def distances(self, sources, cutoff):
        """[S, n + 1] metres, inf beyond the cutoff; the last column stands for no neighbour."""
        S = len(sources)
        D = torch.full((S, self.n + 1), float("inf"), dtype=torch.float64, device=self.dev)
        D[torch.arange(S, device=self.dev), sources] = 0.0
        while True:
            new = D[:, :-1].clone()
            for j in range(self.deg):
                new = torch.minimum(new, D[:, self.nbr[:, j]] + self.w[:, j])
            new[new > cutoff] = float("inf")
            if torch.equal(new, D[:, :-1]):
                return D
            D[:, :-1] = new

    def preds(self, D, cutoff, tol):
        d = D[:, :-1]
        out = []
        for j in range(self.deg):
            du = D[:, self.nbr[:, j]]
            c = du + self.w[:, j]
            out.append((c <= d * (1 + tol)) & (du < d) & (c <= cutoff) & torch.isfinite(d))
        return out

    def counts(self, sources, preds):
        S = len(sources)
        start = torch.zeros((S, self.n + 1), dtype=torch.float64, device=self.dev)
        start[torch.arange(S, device=self.dev), sources] = 1.0
        sig = start.clone()
        while True:
            new = start[:, :-1].clone()
            for j in range(self.deg):
                new += torch.where(preds[j], sig[:, self.nbr[:, j]], 0.0)
            if torch.equal(new, sig[:, :-1]):
                return sig
            sig[:, :-1] = new

    def credits(self, seed, preds, sig):
        """Each node's dependency (without its own seed) of the seeds on all targets."""
        full = torch.stack(preds, -1)
        full = torch.cat([full, torch.zeros_like(full[:, :1])], 1)
        dep = torch.zeros_like(seed)
        inv = torch.where(sig > 0, 1.0 / sig, 0.0)
        while True:
            t = torch.cat([(seed + dep), torch.zeros_like(seed[:, :1])], 1) * inv
            new = torch.zeros_like(seed)
            for j in range(self.deg):
                v = self.nbr[:, j]
                new += torch.where(full[:, v, self.rev[:, j]], t[:, v], 0.0)
            new *= sig[:, :-1]
            if torch.allclose(new, dep, rtol=1e-13, atol=0.0):
                return new
            dep = new


def _cutoff(dists) -> float:
    return round(max(dists) / SPEED) * SPEED


def _exact_shortest(p, n, dists, sources, tol, subset):
    """The seven rows [7][K][n] of shortest-path centrality and the reach counts."""
    ex = _Exact(p, n)
    K, cut = len(dists), _cutoff(dists)
    out = torch.zeros((7, K, n), dtype=torch.float64, device=ex.dev)
    reach = torch.zeros(K, dtype=torch.int64, device=ex.dev)
    pair = torch.ones(n, dtype=torch.float64, device=ex.dev)
    src_all = torch.from_numpy(np.asarray(sources, np.int64)).to(ex.dev)
    pair[src_all] = 0.5
    step = max(1, int(1.5e8 / 8 / n))
    a = torch.from_numpy(p.u).to(ex.dev)
    b = torch.from_numpy(p.v).to(ex.dev)
    for lo in range(0, len(sources), step):
        src = src_all[lo:lo + step]
        D = ex.distances(src, cut)
        P = ex.preds(D, cut, max(TIE, tol / 100.0))
        sig = ex.counts(src, P)
        d = D[:, :-1]
        other = torch.ones_like(d, dtype=torch.bool)
        other[torch.arange(len(src), device=ex.dev), src] = False
        for k, dk in enumerate(dists):
            m = d <= dk
            edges = (torch.maximum(d[:, a], d[:, b]) <= dk).sum(1)
            rank = torch.clamp(edges - m.sum(1) + 1, min=0).double()
            reach[k] += (m.sum(1) - 1).sum()
            m &= other
            safe = torch.where(m, d, 1.0)
            out[0, k] += m.double().sum(0)
            out[1, k] += torch.where(m, d, 0.0).sum(0)
            out[2, k] += torch.where(m, rank[:, None], 0.0).sum(0)
            out[3, k] += torch.where(m, 1.0 / safe, 0.0).sum(0)
            wt = torch.exp(-BETA_LOG / dk * safe)
            out[4, k] += torch.where(m, wt, 0.0).sum(0)
            out[5, k] += torch.where(other, ex.credits(torch.where(m, pair, 0.0), P, sig), 0.0).sum(0)
            out[6, k] += torch.where(other, ex.credits(torch.where(m, pair * wt, 0.0), P, sig), 0.0).sum(0)
    if subset:
        out[5:] *= n / len(sources)
    return out.cpu().numpy(), reach.cpu().numpy()


def _exact_segment(p, n, dists):
    """Closeness integrals over every source's visited streets; betweenness has no value here."""
    ex = _Exact(p, n)
    K, cut = len(dists), _cutoff(dists)
    out = torch.zeros((3, K, n), dtype=torch.float64, device=ex.dev)
    a = torch.from_numpy(p.u).to(ex.dev)
    b = torch.from_numpy(p.v).to(ex.dev)
    ln = torch.from_numpy(p.length.astype(np.float64)).to(ex.dev)
    step = max(1, int(1e8 / 8 / n))
    for lo in range(0, n, step):
        src = torch.arange(lo, min(n, lo + step), device=ex.dev)
        D = ex.distances(src, cut)
        near, far = torch.minimum(D[:, a], D[:, b]), torch.maximum(D[:, a], D[:, b])
        s, e = torch.nonzero(torch.isfinite(near), as_tuple=True)
        A, B = near[s, e], far[s, e]
        mid = (ln[e] + A + B) / 2.0
        for k, dk in enumerate(dists):
            beta = BETA_LOG / dk
            for start, ok in ((A, A < dk), (B, (B <= dk) & (B != mid))):
                lo_, hi = torch.where(ok, start, 1.0), torch.where(ok, torch.clamp(mid, max=float(dk)), 1.0)
                dens = hi - lo_
                harm = torch.where(lo_ < 1.0, torch.log(hi), torch.log(hi / torch.clamp(lo_, min=1e-30)))
                bet = (torch.exp(-beta * hi) - torch.exp(-beta * lo_)) / -beta
                for m, val in enumerate((dens, harm, bet)):
                    out[m, k].index_add_(0, src[s], torch.where(ok, val, 0.0))
    return out.cpu().numpy()


def exact(case, seed):
    kind = case["kind"]
    if kind in ("simplest", "batch", "serve"):
        return None  # angular routes follow the heap's order; the others repeat the plain calls' rows
    p = _streets(case, seed)
    n, dists = int(case["side"]) ** 2, _dists(case)
    n_src = {"subset": case.get("sources"), "od": case.get("origins")}.get(kind, n)
    depth = 2.5 * max(dists) / float(case["spacing"])
    if depth * n_src * n * 8 * 8 * (2 + 2 * len(dists) if kind not in ("segment", "access") else 2) > 1.5e13:
        return None  # minutes in this form
    if kind in ("shortest", "subset"):
        sources = _picked(n, int(case["sources"]), seed) if kind == "subset" else np.arange(n)
        rows, reach = _exact_shortest(p, n, dists, sources, float(case.get("tolerance", 0.0)), kind == "subset")
        if kind == "subset":
            return {**{f"{m}_{d}": rows[i, k] for i, m in enumerate(SHORTEST) for k, d in enumerate(dists)},
                    "reachability": None}
        names = dict(density=0, farness=1, cycles=2, harmonic=3, beta=4, betweenness=5, betweenness_beta=6)
        out = {f"cc_{m}_{d}": rows[i, k] for m, i in names.items() for k, d in enumerate(dists)}
        with np.errstate(divide="ignore", invalid="ignore"):
            out.update({f"cc_hillier_{d}": rows[0, k] ** 2 / rows[1, k] for k, d in enumerate(dists)})
        return out
    if kind == "segment":
        rows = _exact_segment(p, n, dists)
        return {f"cc_seg_{m}_{d}": rows[i, k] for i, m in enumerate(("density", "harmonic", "beta"))
                for k, d in enumerate(dists)}
    if kind == "od":
        o, d, w = _trips(case, seed, n)
        ex, cut = _Exact(p, n), _cutoff(dists)
        out = torch.zeros((2, len(dists), n), dtype=torch.float64, device=ex.dev)
        origins = np.unique(o)
        step = max(1, int(1.5e8 / 8 / n))
        for lo in range(0, len(origins), step):
            src = torch.from_numpy(origins[lo:lo + step]).to(ex.dev)
            D = ex.distances(src, cut)
            P = ex.preds(D, cut, TIE)
            sig = ex.counts(src, P)
            row = np.searchsorted(origins, o) - lo
            mine = (row >= 0) & (row < len(src))
            trip = torch.zeros((len(src), n), dtype=torch.float64, device=ex.dev)
            trip[torch.from_numpy(row[mine]).to(ex.dev), torch.from_numpy(d[mine]).to(ex.dev)] = \
                torch.from_numpy(w[mine].astype(np.float64)).to(ex.dev)
            trip[torch.arange(len(src), device=ex.dev), src] = 0.0
            other = torch.ones_like(trip, dtype=torch.bool)
            other[torch.arange(len(src), device=ex.dev), src] = False
            for k, dk in enumerate(dists):
                s = torch.where(D[:, :-1] <= dk, trip, 0.0)
                wt = torch.exp(-BETA_LOG / dk * torch.clamp(D[:, :-1], max=1e6))
                out[0, k] += torch.where(other, ex.credits(s, P, sig), 0.0).sum(0)
                out[1, k] += torch.where(other, ex.credits(s * wt, P, sig), 0.0).sum(0)
        rows = out.cpu().numpy()
        return {f"{m}_{dk}": rows[i, k] for i, m in enumerate(("node_betweenness", "node_betweenness_beta"))
                for k, dk in enumerate(dists)}
    return None  # which nodes a point is assigned to is the framework's own result
