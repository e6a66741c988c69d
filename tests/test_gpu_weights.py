"""Trip weights of any value, in each schedule of the shortest-path kernels: one warp per source, one
block per source, and tiles of 32 sources (which calls of 10,000 sources of this reach take by themselves)."""
import numpy as np
import pytest
import torch

import oracle
from cityseer_gb300 import _native, common, synth
from cityseer_gb300.centrality import OdMatrix
from helpers import assert_close_sums

pytestmark = pytest.mark.gpu

SCHEDULES = {"warp": {"CS_TILE": "0", "CS_BLOCK_PER_SOURCE": "0"}, "block": {"CS_TILE": "0", "CS_BLOCK_PER_SOURCE": "1"},
             "tile": {}}
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
