"""Calls that take the tile kernel by the rule of the shortest-path calls: 10,000 sources, 40 hops."""
import ctypes as C

import numpy as np
import pytest
import torch

import oracle
from cityseer_gb300 import _native, abi, centrality, common, device, synth
from cityseer_gb300.batch import Batch
from cityseer_gb300.graph import NetworkStructure
from helpers import assert_close_sums

pytestmark = pytest.mark.gpu

ROWS = ("node_density", "node_farness", "node_cycles", "node_harmonic", "node_beta", "node_betweenness",
        "node_betweenness_beta")
SIDE = 100
DISTANCES = [700, 3200]


def _streets(side=SIDE):
    return synth.lattice(side=side, spacing=80.0, jitter=15.0, drop=0.1, seed=11)


def _left() -> int:
    """Sources of the last call that its kernel left to another pass."""
    left = C.c_int64()
    _native.check(_native.load().cs_last_retries(C.byref(left), None), "cs_last_retries")
    return left.value


def _served() -> int:
    """Sources of the last call whose rows came from tiles."""
    entries = (C.c_int64 * 16)()
    _native.check(_native.load().cs_last_phase_cycles(entries, 16), "cs_last_phase_cycles")
    return entries[11]


def _per_warp(ns, monkeypatch, distances):
    with monkeypatch.context() as m:
        m.setenv("CS_TILE", "0")
        m.setenv("CS_BLOCK_PER_SOURCE", "0")
        return ns.centrality_shortest(distances=distances)


def _same(got, want, names=ROWS):
    """The same f32 terms and f64 dependencies, summed in another order: at most 2^18 nonnegative terms,
    2^18 * 2^-53 = 3e-11 of their norm."""
    for name in names:
        for d, col in getattr(want, name).items():
            assert np.linalg.norm(getattr(got, name)[d] - col) <= 1e-10 * np.linalg.norm(col), (name, d)


def _with_loops(side=SIDE):
    """One-way loops of three streets: nodes with as many edges in as out, but no edge back for some."""
    p = _streets(side)
    at = side * np.arange(side // 5, side - side // 5, 12)[:, None] + np.arange(side // 5, side - side // 5, 12)
    a = at.reshape(-1)
    b, c = a + 2, a + 2 * side + 1
    src = np.concatenate([p.u, p.v, a, b, c])
    dst = np.concatenate([p.v, p.u, b, c, a])
    ln = np.concatenate([p.length, p.length, np.full(3 * len(a), 170.0)]).astype(np.float32)
    idx = np.concatenate([np.zeros(2 * len(p.u), np.int64), 1 + np.arange(3 * len(a))])
    return NetworkStructure.from_arrays(p.x, p.y, src, dst, ln, edge_idx=idx)


def test_one_way_loops(monkeypatch):
    """The tiles that meet an edge without one back find out in their second pass over the edges, and leave
    every source to the per-warp kernel."""
    ns = _with_loops()
    got = ns.centrality_shortest(distances=DISTANCES)
    assert _left() > 0
    _same(got, _per_warp(ns, monkeypatch, DISTANCES))


@pytest.fixture(scope="module")
def lattice():
    return synth.primal_structure(_streets())


@pytest.mark.parametrize("distances,kw", [
    ([700, 3200, 4000], {}),  # unions of up to 5,000 nodes
    ([3200], dict(tolerance=2.0)),
    ([3200], dict(compute_closeness=False)),
])
def test_every_source_against_the_oracle(lattice, distances, kw):
    """Counts are exact, betweenness differs in the order of its f64 sums, closeness also in the last bits
    of its f32 exponentials and quotients."""
    n = lattice.node_bound()
    d, b, s = common.pair_distances_betas_time(1.33333, distances=distances)
    closeness = kw.get("compute_closeness", True)
    ref, _ = oracle.centrality_shortest(oracle.OracleGraph(lattice), d, b, s, closeness=closeness,
                                        tol=centrality.validate_tolerance(kw.get("tolerance")),
                                        plan=oracle.plan_from(centrality.prepare_source_sampling(
                                            lattice, None, None, None, None), n),
                                        nthreads=oracle.default_threads())
    res = lattice.centrality_shortest(distances=distances, **kw)
    assert (_served(), _left()) == (n, 0)
    for m, name in enumerate(ROWS):
        if m < 5 and not closeness:
            continue
        for i, dist in enumerate(d):
            got = getattr(res, name)[dist]
            if name in ("node_density", "node_cycles"):
                np.testing.assert_array_equal(got, ref[m, i], err_msg=f"{name}[{dist}]")
            else:
                assert_close_sums(got, ref[m, i], rtol=1e-9 if m >= 5 else 1e-5, what=f"{name}[{dist}]")


def test_trips_of_every_node_against_the_oracle(lattice):
    n = lattice.node_bound()
    rng = np.random.default_rng(9)
    o = np.repeat(np.arange(n), 2)
    od = centrality.OdMatrix(o, np.clip(o + rng.integers(-900, 900, len(o)), 0, n - 1), rng.uniform(0.1, 9.0, len(o)))
    d, b, s = common.pair_distances_betas_time(1.33333, distances=DISTANCES)
    ref = oracle.betweenness_od(oracle.OracleGraph(lattice), d, b, s, od.rows(n), ns=lattice,
                                nthreads=oracle.default_threads())
    res = lattice.betweenness_od_shortest(od, distances=DISTANCES)
    assert (_served(), _left()) == (n, 0)
    for m, name in enumerate(("node_betweenness", "node_betweenness_beta")):
        for i, dist in enumerate(d):
            assert_close_sums(getattr(res, name)[dist], ref[m, i], rtol=1e-9, what=f"{name}[{dist}]")


def test_unions_beyond_the_scratch(lattice, monkeypatch):
    """A plan of small capacity: the tiles' unions outgrow it, their sources go to the per-warp kernel and
    its capacity chain, and the scratch is clean for the next call, whose tiles fit."""
    n = lattice.node_bound()
    for distances, left in (([3200], n), ([400], 0)):
        call = abi.shortest_call(lattice, distances)
        if left:
            plan = device.plan_primal(centrality._primal_csr(lattice), 0, 1, 1.33333, cap=256, mem_budget=8 << 30)
            plan.variant |= _native.CS_PLAN_NEAR_SOURCES
            ws = device.Workspace(plan, n, call.out.device)
        else:
            monkeypatch.setenv("CS_TILE", "1")  # few hops: not by the rule
        call.plan, call.workspace = plan, ws
        abi.check(abi.library().cs_centrality_shortest(*call.args()))
        served = _served()
        got = call.out.cpu().numpy()
        assert served == n - left and (_left() > 0) == (left > 0)
        want = _per_warp(lattice, monkeypatch, distances)
        for m, name in enumerate(ROWS):
            col = getattr(want, name)[distances[0]]
            assert np.linalg.norm(got[m, 0] - col) <= 1e-10 * np.linalg.norm(col), (name, distances)


@pytest.mark.parametrize("order", ["curve", "rows", "random"])
def test_only_vouched_orders_are_tiled(lattice, order):
    """Sources in rows or at random run one by one unless the plan says that neighbours follow one another:
    tiles of them hold many reaches each and take longer (3.2 km: 14.7 and 13.9 ms against 11.0 and 13.2)."""
    n = lattice.node_bound()
    call = abi.shortest_call(lattice, [3200])
    plan = _native.Plan.from_buffer_copy(call.plan)
    if order != "curve":
        plan.variant &= ~_native.CS_PLAN_NEAR_SOURCES
        src = np.arange(n) if order == "rows" else np.random.default_rng(1).permutation(n)
        call.query._keep[0].copy_(torch.from_numpy(src.astype(np.int32)))
    call.plan = plan
    abi.check(abi.library().cs_centrality_shortest(*call.args()))
    assert _served() == (n if order == "curve" else 0)


def test_one_way_loops_of_one_job_of_a_batch(lattice, monkeypatch):
    """The other jobs' sources stay in tiles."""
    loops = _with_loops(40)
    jobs = [dict(ns=g, mode="shortest", distances=[d]) for g, d in ((loops, 1500), (lattice, 1500), (loops, 3000))]
    monkeypatch.setenv("CS_TILE", "1")  # every job, the loops first
    batch = Batch(jobs)
    batch.run()
    entries = (C.c_int64 * 16)()
    _native.check(_native.load().cs_last_phase_cycles(entries, 16), "cs_last_phase_cycles")
    assert entries[11] >= lattice.node_bound() and 0 < entries[10] <= 2 * loops.node_bound()
    monkeypatch.setenv("CS_TILE", "0")
    plain = Batch(jobs)
    plain.run()
    for got, want in zip(batch.results(), plain.results()):
        _same(got, want)


@pytest.mark.parametrize("distances,tiled", [([2000], False), ([800, 1200, 1600, 2000], False), ([2800], True),
                                             ([1000, 1500, 2000, 2500], False), ([1280, 1920, 2560, 3200], True)])
def test_reach_and_thresholds_decide(lattice, distances, tiled):
    """Tiles pay from a reach on that grows with the dependency rows a node needs (10,000 sources: 25 hops
    2.5 against 2.3 ms, with four thresholds 3.7 against 2.9; 36 hops 3.6 against 4.5)."""
    lattice.centrality_shortest(distances=distances)
    assert _served() == (lattice.node_bound() if tiled else 0)


def test_jobs_that_pay_are_consecutive(lattice):
    """A batch's table is sorted by what decides, not by reach alone: of jobs of 40, 32, 26 and 25 hops the
    third has too many thresholds for its reach."""
    sets = ([1280, 1920, 2560, 3200], [2560], [832, 1248, 1664, 2080], [2080])
    batch = Batch([dict(ns=lattice, mode="shortest", distances=d) for d in sets])
    batch.run()
    entries = (C.c_int64 * 16)()
    _native.check(_native.load().cs_last_phase_cycles(entries, 16), "cs_last_phase_cycles")
    assert entries[11] == 3 * lattice.node_bound()
