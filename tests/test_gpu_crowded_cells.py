"""Atoms crowded into few cells: below and above the mean occupancy at which the cell
order is sorted instead of ranked (192), and one crowded cell among empty ones; the
lists are the oracle's, rows in ascending order."""
import numpy as np
import pytest

from conftest import assert_same_lists

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cells,n", [((1, 1, 1), 191), ((1, 1, 1), 192), ((1, 1, 1), 193),
                                     ((2, 2, 1), 768), ((2, 2, 1), 769), ((9, 1, 1), 2100)])
@pytest.mark.parametrize("clump", [False, True])
@pytest.mark.parametrize("kind", ["scalar", "type"])
def test_crowded_cells(oracle, cells, n, clump, kind):
    from matscipy_neighbours import neighbour_list
    rng = np.random.default_rng(n)
    cell = np.diag([1.01 * c for c in cells])
    u = rng.uniform(size=(n, 3))
    if clump:
        u = (0.3 + u * 0.9) / cells
    pos = np.ascontiguousarray(u @ cell)
    pbc = np.array([False, True, False])
    cut, types = 1.0, None
    if kind == "type":
        cut, types = np.array([[1.0, 0.3], [0.3, 0.1]]), (rng.uniform(size=n) < 0.9).astype(np.int32)
    want = oracle.oracle_neighbour_list("ijdDS", cell, pos, cut, pbc, types=types)
    for _ in range(3):
        got = neighbour_list("ijdDS", positions=pos, cell=cell, pbc=pbc, cutoff=cut, numbers=types)
        assert_same_lists(got, want, "ijdDS")
