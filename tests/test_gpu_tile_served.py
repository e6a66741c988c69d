"""Calls that take the tile kernel by the rule of the shortest-path calls: 10,000 sources, 30 hops."""
import ctypes as C

import numpy as np
import pytest

from cityseer_gb300 import _native, synth
from cityseer_gb300.graph import NetworkStructure

pytestmark = pytest.mark.gpu

ROWS = ("node_density", "node_farness", "node_cycles", "node_harmonic", "node_beta", "node_betweenness",
        "node_betweenness_beta")
SIDE = 100
DISTANCES = [700, 2400]


def _streets():
    return synth.lattice(side=SIDE, spacing=80.0, jitter=15.0, drop=0.1, seed=11)


def _left() -> int:
    """Sources of the last call that its kernel left to another pass."""
    left = C.c_int64()
    _native.check(_native.load().cs_last_retries(C.byref(left), None), "cs_last_retries")
    return left.value


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


def test_one_way_loops(monkeypatch):
    """Nodes with as many edges in as out, but no edge back for some: the tiles that meet one find out in
    their second pass over the edges, and leave every source to the per-warp kernel."""
    p = _streets()
    at = SIDE * np.arange(20, 80, 12)[:, None] + np.arange(20, 80, 12)
    a = at.reshape(-1)
    b, c = a + 2, a + 2 * SIDE + 1
    src = np.concatenate([p.u, p.v, a, b, c])
    dst = np.concatenate([p.v, p.u, b, c, a])
    ln = np.concatenate([p.length, p.length, np.full(3 * len(a), 170.0)]).astype(np.float32)
    idx = np.concatenate([np.zeros(2 * len(p.u), np.int64), 1 + np.arange(3 * len(a))])
    ns = NetworkStructure.from_arrays(p.x, p.y, src, dst, ln, edge_idx=idx)
    got = ns.centrality_shortest(distances=DISTANCES)
    assert _left() > 0
    _same(got, _per_warp(ns, monkeypatch, DISTANCES))
