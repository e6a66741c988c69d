"""Calls from several host threads at once, each on its own stream and workspace."""
import ctypes as C
import threading

import numpy as np
import pytest
import torch

from cityseer_gb300 import _native, abi, synth

pytestmark = pytest.mark.gpu


def test_tile_calls_of_different_shapes_at_once(monkeypatch):
    """Tile launches with different amounts of shared memory (as many as thresholds ask for) do not disturb
    one another: what one call sets on the kernel is not what another call's launch is checked against."""
    monkeypatch.setenv("CS_TILE", "1")
    shapes = [[100], [60 + 20 * i for i in range(16)]] * 4
    calls = 3000
    errors, rows = [], {}
    start = threading.Barrier(len(shapes))

    def work(t, distances):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                ns = synth.primal_structure(synth.lattice(side=24, spacing=80.0, jitter=15.0, drop=0.1, seed=t))
                call = abi.shortest_call(ns, distances, source_indices=[200])
                fn, args = abi.library().cs_centrality_shortest, call.args()
                entries = (C.c_int64 * 16)()
                start.wait(timeout=60)
                for i in range(calls):
                    if i in (0, calls - 1):
                        call.out.zero_()
                    abi.check(fn(*args))
                    if i in (0, calls - 1):
                        rows[t, i] = call.out.cpu().numpy()
                        _native.check(_native.load().cs_last_phase_cycles(entries, 16), "cs_last_phase_cycles")
                        assert entries[11] == 1  # a tile served the source
        except Exception as e:
            errors.append(f"{len(distances)} thresholds: {e!r}")
            start.abort()

    threads = [threading.Thread(target=work, args=(t, d)) for t, d in enumerate(shapes)]
    for t in threads:
        t.start()
    for t in threads:
        t.join(timeout=120)
    assert not errors
    for t in range(len(shapes)):
        assert np.array_equal(rows[t, 0], rows[t, calls - 1], equal_nan=True)  # one source: one term per sum
