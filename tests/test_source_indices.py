"""What source_indices may be: an iterable with one node index per entry."""
import numpy as np
import pytest

from cityseer_gb300 import synth
from cityseer_gb300.centrality import prepare_source_sampling


@pytest.fixture(scope="module")
def ns():
    return synth.primal_structure(synth.lattice(side=6, spacing=80.0, jitter=15.0, drop=0.0, seed=5))


@pytest.mark.parametrize("given,error", [
    ([[0, 1], [2, 3]], ValueError), (np.array([[0, 1]]), ValueError), (np.array(3), TypeError), (3, TypeError),
    (np.array([2 ** 63 + 5], np.uint64), OverflowError), (np.array([1e30]), OverflowError),
    (np.array([np.nan]), ValueError), (np.ma.array([1, 2], mask=[0, 1]), np.ma.MaskError),
    (np.array([1], "datetime64[s]"), TypeError), ([36], ValueError), ([-1], ValueError),
])
def test_refused(ns, given, error):
    with pytest.raises(error):
        prepare_source_sampling(ns, None, None, None, given)


@pytest.mark.parametrize("given", [
    [4, 1, 4], np.array([4, 1, 4]), np.array([4, 1, 4], np.int32), np.array([4, 1, 4], np.uint8), (i for i in (4, 1, 4)),
    np.array([4, 1, 4], object), np.array([[4], [1], [4]]), np.array([4.0, 1.0, 4.0]),
])
def test_taken_in_order_with_repeats(ns, given):
    plan = prepare_source_sampling(ns, None, None, None, given)
    assert plan.process.tolist() == [4, 1, 4] and plan.n_sources == 3


def test_none_listed(ns):
    assert len(prepare_source_sampling(ns, None, None, None, np.array([])).process) == 0
