"""Negative and zero cutoffs, which the reference takes (only their square enters
the pair test): the lists have room and are the oracle's."""
import numpy as np
import pytest

from conftest import assert_same_lists

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [60, 200, 201, 1025])
@pytest.mark.parametrize("cutoff", [-0.5, -3.9, -4.0, 0.0])
def test_negative_cutoffs(oracle, n, cutoff):
    from matscipy_neighbours import neighbour_list
    rng = np.random.default_rng(n)
    cell = 4.0 * np.eye(3)
    pos = rng.uniform(size=(n, 3)) @ cell
    pbc = np.array([True, True, False])
    want = oracle.oracle_neighbour_list("ijdDS", cell, pos, cutoff, pbc)
    for _ in range(3):
        got = neighbour_list("ijdDS", positions=pos, cell=cell, pbc=pbc, cutoff=cutoff)
        assert_same_lists(got, want, "ijdDS")
