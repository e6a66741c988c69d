"""Source and trip weights of any sign and size, in each schedule of the shortest-path kernels: one warp
per source, one block per source, and tiles of 32 sources."""
import ctypes as C
import math

import numpy as np
import pytest
import torch
from scipy.sparse import coo_matrix
from scipy.sparse.csgraph import connected_components

import oracle
from cityseer_gb300 import _native, common, synth
from cityseer_gb300.batch import Batch
from cityseer_gb300.centrality import OdMatrix
from cityseer_gb300.graph import NetworkStructure
from helpers import assert_close_sums

pytestmark = pytest.mark.gpu

SCHEDULES = {"warp": {"CS_TILE": "0", "CS_BLOCK_PER_SOURCE": "0"}, "block": {"CS_TILE": "0", "CS_BLOCK_PER_SOURCE": "1"},
             "tile": {"CS_TILE": "1"}}
DISTANCES = [700, 2400]


def _choose(monkeypatch, schedule):
    for name in ("CS_TILE", "CS_BLOCK_PER_SOURCE"):
        monkeypatch.delenv(name, raising=False)
    for name, value in SCHEDULES[schedule].items():
        monkeypatch.setenv(name, value)


@pytest.fixture(scope="module")
def lattice():
    return synth.primal_structure(synth.lattice(side=100, spacing=80.0, jitter=15.0, drop=0.1, seed=11))


def _trips(n, weights):
    """Three destinations within a few streets of every node."""
    rng = np.random.default_rng(6)
    o = np.repeat(np.arange(n), 3)
    d = np.clip(o + rng.choice([-305, -204, -103, -7, 8, 98, 207, 303], len(o)), 0, n - 1)
    return OdMatrix(o, d, weights(rng, len(o)))


def test_negative_weights_in_the_seed_exponentials():
    """w * exp(-(beta * cost)) is as exact for w < 0 as for w > 0 (5e-14, the bound of the positive ones)."""
    rng = np.random.default_rng(3)
    n = 1 << 16
    d = rng.uniform(100.0, 20000.0, n)
    beta = np.round(4.0 / d, 5).astype(np.float32)
    cost = (rng.uniform(0.0, 2.0, n) * d).astype(np.float32)
    w = -rng.uniform(1e-3, 1e3, n).astype(np.float32)
    w[:4096] = -np.exp2(rng.integers(-8, 8, 4096)).astype(np.float32)  # powers of two
    tw, tb, tc = (torch.from_numpy(x).cuda() for x in (w, beta, cost))
    out = torch.empty(n, dtype=torch.float64, device="cuda")
    _native.check(_native.load().cs_debug_seed_exp(tw.data_ptr(), tb.data_ptr(), tc.data_ptr(), out.data_ptr(), n, None),
                  "cs_debug_seed_exp")
    want = w.astype(np.float64) * np.exp(-(beta.astype(np.float64) * cost.astype(np.float64)))
    assert np.max(np.abs(out.cpu().numpy() / want - 1.0)) < 5e-14


@pytest.mark.parametrize("schedule", SCHEDULES)
def test_trips_of_both_signs(lattice, schedule, monkeypatch):
    """A node is credited with what an origin's trips through it come to only where that is positive."""
    n = lattice.node_bound()
    od = _trips(n, lambda rng, m: rng.uniform(-3.0, 5.0, m))
    d, b, s = common.pair_distances_betas_time(1.33333, distances=DISTANCES)
    ref = oracle.betweenness_od(oracle.OracleGraph(lattice), d, b, s, od.rows(n), ns=lattice,
                                nthreads=oracle.default_threads())
    _choose(monkeypatch, schedule)
    res = lattice.betweenness_od_shortest(od, distances=DISTANCES)
    for m, name in enumerate(("node_betweenness", "node_betweenness_beta")):
        for i, dist in enumerate(d):
            assert_close_sums(getattr(res, name)[dist], ref[m, i], rtol=1e-9, atol=1e-9, what=f"{schedule} {name}[{dist}]")


@pytest.mark.parametrize("schedule", ["warp", "tile"])
def test_trips_without_a_finite_weight(lattice, schedule, monkeypatch):
    """Trips of weight NaN or infinity leave NaN in no row; the block kernel's rows are the measure."""
    n = lattice.node_bound()

    def weights(rng, m):
        w = rng.uniform(0.5, 5.0, m)
        w[rng.choice(m, 30, replace=False)] = np.nan
        w[rng.choice(m, 30, replace=False)] = np.inf
        return w

    od = _trips(n, weights)
    _choose(monkeypatch, "block")
    want = lattice.betweenness_od_shortest(od, distances=DISTANCES)
    _choose(monkeypatch, schedule)
    got = lattice.betweenness_od_shortest(od, distances=DISTANCES)
    for name in ("node_betweenness", "node_betweenness_beta"):
        for dist in DISTANCES:
            a, b = getattr(got, name)[dist], getattr(want, name)[dist]
            assert not np.isnan(a).any() and np.isfinite(b).sum() > n // 2
            assert_close_sums(a, b, rtol=1e-9, atol=1e-9, what=f"{schedule} {name}[{dist}]")


def test_tile_sums_keep_every_bit_of_small_terms(monkeypatch):
    """One source of weight 1 among sources of about 1e-9: a tile's sums of 32 terms are as exact as f64
    adds of them, and the tiles' sums (and the sources that tiles leave) are added in f64: at most
    32 + 32 + left roundings of 2^-53."""
    p = synth.lattice(side=32, spacing=80.0, jitter=15.0, drop=0.1, seed=5)
    n = 32 * 32
    w = np.random.default_rng(8).uniform(0.5e-9, 1.5e-9, n).astype(np.float32)
    w[527] = 1.0
    src, dst = np.concatenate([p.u, p.v]), np.concatenate([p.v, p.u])
    ns = NetworkStructure.from_arrays(p.x, p.y, src, dst, np.concatenate([p.length, p.length]), weight=w)
    monkeypatch.setenv("CS_TILE", "1")
    batch = Batch([dict(ns=ns, mode="shortest", distances=[6000])])  # to every node of the component
    batch.run()
    entries = (C.c_int64 * 16)()
    _native.check(_native.load().cs_last_phase_cycles(entries, 16), "cs_last_phase_cycles")
    served = entries[11]
    assert served > n // 2
    got = batch.results()[0].node_density[6000]
    _, part = connected_components(coo_matrix((np.ones(len(src)), (src, dst)), shape=(n, n)), directed=False)
    want = np.array([math.fsum(float(w[i]) for i in np.nonzero(part == part[v])[0] if i != v) for v in range(n)])
    assert np.all(np.abs(got - want) <= (64 + n - served) * 2.0 ** -53 * want)
