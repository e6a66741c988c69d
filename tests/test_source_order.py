"""The device arrays of a call over every node, kept with the graph, in the order that the call asks for."""
import numpy as np
import torch

from cityseer_gb300 import centrality, synth


def test_each_order_has_its_own_arrays():
    """Simplest paths keep the listed order, shortest paths want neighbours in a row: calls of both kinds
    on one graph (a dual one takes both) each get their own, whichever comes first."""
    n = 96 * 96
    cpu = torch.device("cpu")
    for first in (False, True):
        ns = synth.primal_structure(synth.lattice(side=96, spacing=80.0, jitter=15.0, drop=0.1, seed=4))
        sp = centrality.prepare_source_sampling(ns, None, None, None, None)
        want = {False: np.arange(n), True: centrality.spatial_order(ns, sp.process)}
        assert not np.array_equal(want[False], want[True])
        for order in (first, not first, first):
            got = centrality.plan_tensors(ns, sp, sp.process, cpu, order=order)
            assert np.array_equal(got[0].numpy(), want[order]), (first, order)
        kept = centrality.plan_tensors(ns, sp, sp.process, cpu, order=True)
        assert kept[0].data_ptr() == centrality.plan_tensors(ns, sp, sp.process, cpu, order=True)[0].data_ptr()
        centrality.drop_device_state(ns)
        assert not any(k.startswith("every_source") for k in ns._cache if isinstance(k, str))


def test_coordinates_without_an_order_still_give_a_permutation(recwarn):
    """Coordinates only order the sources: NaN, infinite and overflowing ones are no reason to complain."""
    n = 96 * 96
    ns = synth.primal_structure(synth.lattice(side=96, spacing=80.0, jitter=15.0, drop=0.1, seed=4))
    x = ns._x.view()
    x[[3, 70, 700]] = [np.inf, -np.inf, np.nan]
    x[[5, 50]] = [1.5e308, -1.5e308]
    assert sorted(centrality.spatial_order(ns, np.arange(n)).tolist()) == list(range(n))
    assert not [w for w in recwarn if issubclass(w.category, RuntimeWarning)]
