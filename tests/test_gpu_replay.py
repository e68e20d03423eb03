"""The captured count phase is replayed only for calls it was captured for: systems
of the same atom count and cell table that differ in the visited offsets (a
cutoff that crosses the cell's height), taking turns on one plan, each get the
oracle's list."""
import numpy as np
import pytest

from conftest import assert_same_lists

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [150, 400])
@pytest.mark.parametrize("cutoffs", [(2.99, 3.01), (3.01, 2.99), (5.99, 6.01), (1.49, 3.02)])
def test_cutoffs_around_the_cell_height(oracle, n, cutoffs):
    from matscipy_neighbours import neighbour_list
    rng = np.random.default_rng(n)
    cell = 3.0 * np.eye(3)
    pos = rng.uniform(size=(n, 3)) @ cell
    pbc = np.array([True, True, True])
    want = [oracle.oracle_neighbour_list("ijdDS", cell, pos, c, pbc) for c in cutoffs]
    for k in (0, 0, 0, 1, 0, 1, 1, 1, 0):
        got = neighbour_list("ijdDS", positions=pos, cell=cell, pbc=pbc, cutoff=cutoffs[k])
        assert_same_lists(got, want[k], "ijdDS")
