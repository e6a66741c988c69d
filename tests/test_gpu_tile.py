"""The tile kernel (32 sources per block, one per lane) against the other shortest-path kernels.

Both sum the same f32 terms and f64 dependencies in another order: rows of at most 2^18 nonnegative f64
terms differ by at most 2^18 * 2^-53 = 3e-11 of their norm, so 1e-10 bounds them.  Counts are exact."""
import numpy as np
import pytest

from cityseer_gb300 import centrality, synth
from cityseer_gb300.batch import Batch
from cityseer_gb300.graph import NetworkStructure

pytestmark = pytest.mark.gpu

ROWS = ("node_density", "node_farness", "node_cycles", "node_harmonic", "node_beta", "node_betweenness",
        "node_betweenness_beta")


def _lattice(side, seed=3, **kw):
    return synth.primal_structure(synth.lattice(side=side, spacing=80.0, jitter=15.0, drop=0.1, seed=seed, **kw))


def _edited(side, edit):
    """A lattice with more edges: `edit(rng, n)` gives (src, dst, length) of directed edges to add."""
    p = synth.lattice(side=side, spacing=80.0, jitter=15.0, drop=0.1, seed=5)
    rng = np.random.default_rng(7)
    es, ed, el = edit(rng, side * side)
    src = np.concatenate([p.u, p.v, es])
    dst = np.concatenate([p.v, p.u, ed])
    ln = np.concatenate([p.length, p.length, el]).astype(np.float32)
    idx = np.concatenate([np.zeros(2 * len(p.u), np.int64), 1 + np.arange(len(es)) // 2])
    return NetworkStructure.from_arrays(p.x, p.y, src, dst, ln, edge_idx=idx)


def _parallel(rng, n):  # second, slightly longer streets between neighbours, in both directions
    a = rng.choice(n - 1, 40, replace=False)
    ln = rng.uniform(60.0, 90.0, 40)
    return np.repeat(a, 2) + np.tile([0, 1], 40), np.repeat(a, 2) + np.tile([1, 0], 40), np.repeat(ln, 2)


def _equal_distances():
    """An exact grid with 4 mm links between nodes that many sources reach at equal distances: the settle
    order decides which of the two is a predecessor, so those sources go to the per-warp kernel."""
    p = synth.lattice(side=20, spacing=80.0, jitter=0.0, drop=0.0, seed=2)
    a = np.array([21, 105, 190, 262])
    src = np.concatenate([p.u, p.v, a + 1, a + 20])
    dst = np.concatenate([p.v, p.u, a + 20, a + 1])
    ln = np.concatenate([p.length, p.length, np.full(8, 0.004)]).astype(np.float32)
    return NetworkStructure.from_arrays(p.x, p.y, src, dst, ln)


def _one_way(rng, n):  # edges without one back: no tile can be served
    a = rng.choice(n - 1, 5, replace=False)
    return a, a + 1, rng.uniform(50.0, 90.0, 5)


GRAPHS = {
    "plain": lambda: _lattice(24),
    "diagonals": lambda: _lattice(24, diag_frac=0.3),
    "two_nodes": lambda: NetworkStructure.from_arrays(np.array([0.0, 50.0]), np.zeros(2), np.array([0, 1]),
                                                      np.array([1, 0]), np.array([50.0, 50.0], np.float32)),
    "exact_grid": lambda: synth.primal_structure(synth.lattice(side=20, spacing=80.0, jitter=0.0, drop=0.1, seed=2)),
    "parallel": lambda: _edited(20, _parallel),
    "equal_distances": _equal_distances,
    "one_way": lambda: _edited(20, _one_way),
}


@pytest.fixture
def tile(monkeypatch):
    # the comparison runs one warp per source
    monkeypatch.setenv("CS_BLOCK_PER_SOURCE", "0")

    def choose(on):
        monkeypatch.setenv("CS_TILE", "1" if on else "0")
    return choose


def _compare(a, b, names):
    for name in names:
        for d, want in getattr(b, name).items():
            got = getattr(a, name)[d]
            if name == "node_density" and np.all(want == np.round(want)):
                assert np.array_equal(got, want), (name, d)
            assert np.linalg.norm(got - want) <= 1e-10 * np.linalg.norm(want), (name, d)


@pytest.mark.parametrize("graph,distances,n_src,kw", [
    ("plain", [300, 700, 1500], 576, {}),                               # every node: full tiles and a remainder
    ("plain", [900], 33, {}),                                           # one lane more than a tile
    ("plain", [100 + 90 * i for i in range(16)], 200, {}),              # the most thresholds of a launch
    ("plain", [1200], 1, {}),
    ("plain", [500, 1500], 300, dict(compute_betweenness=False)),
    ("plain", [500, 1500], 300, dict(compute_closeness=False)),
    ("plain", [500, 1500], 300, dict(tolerance=3.0)),
    ("diagonals", [400, 1600], 576, {}),
    ("diagonals", [400, 1600], 100, dict(tolerance=20.0)),
    ("two_nodes", [40, 60], 2, {}),
    ("exact_grid", [400, 1200], 400, {}),
    ("parallel", [400, 1200], 400, {}),
    ("equal_distances", [400, 1200], 400, {}),
    ("one_way", [400, 1200], 400, {}),
])
def test_tile_equals_the_per_source_kernels(tile, graph, distances, n_src, kw):
    ns = GRAPHS[graph]()
    n = ns.node_bound()
    src = np.random.default_rng(1).choice(n, min(n_src, n), replace=False)
    args = dict(distances=distances, source_indices=[int(s) for s in src], **kw)
    tile(False)
    want = ns.centrality_shortest(**args)
    tile(True)
    got = ns.centrality_shortest(**args)
    names = [m for m in ROWS if (kw.get("compute_closeness", True) or "between" in m)
             and (kw.get("compute_betweenness", True) or "between" not in m)]
    _compare(got, want, names)
    assert got.reachability_totals == want.reachability_totals


def test_tile_weights_and_repeated_sources(tile):
    p = synth.lattice(side=20, spacing=80.0, jitter=15.0, drop=0.1, seed=5)
    src, dst = np.concatenate([p.u, p.v]), np.concatenate([p.v, p.u])
    w = np.random.default_rng(3).choice([0.0, 0.25, 1.0, 7.5], 400)
    ns = NetworkStructure.from_arrays(p.x, p.y, src, dst, np.concatenate([p.length, p.length]), weight=w)
    args = dict(distances=[500, 1100], source_indices=[3, 3, 399, 0, 3] + list(range(100, 160)), sample_probability=0.5)
    tile(False)
    want = ns.centrality_shortest(**args)
    tile(True)
    got = ns.centrality_shortest(**args)
    for name in ROWS:
        for d, col in getattr(want, name).items():
            new = getattr(got, name)[d]
            assert np.array_equal(np.isfinite(new), np.isfinite(col))
            ok = np.isfinite(col)  # a source of weight 0 has no cycles weight
            assert np.linalg.norm(new[ok] - col[ok]) <= 1e-10 * np.linalg.norm(col[ok])


@pytest.mark.parametrize("distance,n_src", [(240, 1), (240, 152), (240, 153), (2800, 608), (2800, 609)])
def test_blocks_or_warps_by_reach_and_count(monkeypatch, distance, n_src):
    """One block per source or one warp per source, at the edges of the rule (few and many hops)."""
    monkeypatch.setenv("CS_TILE", "0")
    ns = _lattice(60)
    src = [int(s) for s in np.random.default_rng(2).choice(3600, n_src, replace=False)]
    by_rule = ns.centrality_shortest(distances=[distance], source_indices=src)
    monkeypatch.setenv("CS_BLOCK_PER_SOURCE", "0")
    _compare(by_rule, ns.centrality_shortest(distances=[distance], source_indices=src), ROWS)


@pytest.mark.parametrize("graphs", [
    ["plain", "diagonals"], ["two_nodes", "equal_distances", "plain"], ["exact_grid", "one_way", "parallel"],
])
def test_batched_tiles(tile, graphs):
    """Jobs of one tiled launch, with another mode beside them; run at once and replayed from a capture."""
    flags = [{}, dict(compute_betweenness=False), dict(compute_closeness=False)]
    jobs = [dict(ns=GRAPHS[g](), mode="shortest", distances=[[300, 700, 1500], [900], [400, 1200]][i], **flags[i])
            for i, g in enumerate(graphs)]
    jobs.insert(1, dict(ns=jobs[0]["ns"], mode="segment", distances=[500]))
    jobs.append(dict(ns=jobs[0]["ns"], mode="shortest", distances=[1100], source_indices=[0, 1]))
    tile(False)
    plain = Batch(jobs)
    plain.run()
    want = plain.results()
    tile(True)
    b = Batch(jobs)
    b.run()
    for got in (b.results(), None):
        if got is None:
            b.capture()
            b.replay()
            b.replay()
            assert b.status()[0] == 0
            got = b.results()
        for g, w, j in zip(got, want, jobs):
            if j["mode"] == "segment":
                _compare(g, w, ("segment_density", "segment_betweenness"))
            else:
                _compare(g, w, [m for m in ROWS if (j.get("compute_closeness", True) or "between" in m)
                                and (j.get("compute_betweenness", True) or "between" not in m)])


def test_batched_tiles_beyond_one_list(tile):
    ns = _lattice(300)  # three jobs of 90,000 sources: more than one launch's list of 2^18 holds
    jobs = [dict(ns=ns, mode="shortest", distances=[d]) for d in (320, 240, 160)]
    tile(False)
    plain = Batch(jobs)
    plain.run()
    want = plain.results()
    tile(True)
    b = Batch(jobs)
    b.run()
    for g, w in zip(b.results(), want):
        _compare(g, w, ROWS)


@pytest.mark.parametrize("graph", ["diagonals", "exact_grid", "parallel"])
def test_tile_trips(tile, graph):
    ns = GRAPHS[graph]()
    n = ns.node_bound()
    rng = np.random.default_rng(4)
    o = np.repeat(rng.choice(n, 70, replace=False), 4)
    od = centrality.OdMatrix(o, rng.integers(0, n, len(o)), rng.uniform(1e-3, 1e3, len(o)))
    tile(False)
    want = ns.betweenness_od_shortest(od, distances=[600, 1300])
    tile(True)
    got = ns.betweenness_od_shortest(od, distances=[600, 1300])
    _compare(got, want, ("node_betweenness", "node_betweenness_beta"))


def test_spatial_order_is_a_permutation_that_keeps_repeats():
    ns = _lattice(92)  # 8,464 nodes
    every = centrality.spatial_order(ns, np.arange(92 * 92))
    step = np.hypot(np.diff(ns._x.view()[every]), np.diff(ns._y.view()[every]))
    assert sorted(every.tolist()) == list(range(92 * 92)) and step.max() < 4 * 80.0
    twice = np.concatenate([np.arange(92 * 92), [5, 5, 17]])
    assert sorted(centrality.spatial_order(ns, twice).tolist()) == sorted(twice.tolist())
    assert centrality.spatial_order(ns, [9, 3, 3]).tolist() == [9, 3, 3]
