"""Atoms ordered by counting them into cells: cell tables at the edges of a scan
tile (2,048 cells), crowded cells, hashed slots, and tables too large for it
(radix sort): the lists are the oracle's bit for bit, rows in ascending order."""
import numpy as np
import pytest

from conftest import assert_same_lists

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cells,n,grid", [
    ((1, 1, 1), 700, "dense"), ((16, 16, 8), 3000, "dense"), ((2047, 1, 1), 3000, "dense"),
    ((683, 3, 1), 3000, "dense"), ((64, 64, 1), 5000, "dense"), ((2, 2, 2), 2500, "dense"),
    ((2, 2, 2), 2500, "hashed"), ((16, 16, 8), 3000, "hashed"), ((130, 127, 127), 900, "dense"),
    ((16, 16, 8), 3000, "morton"), ((1, 1, 1), 1, "dense"), ((40, 1, 1), 2, "dense")])
def test_cell_tables(oracle, cells, n, grid):
    from matscipy_neighbours.batch import NeighbourListBatch
    rng = np.random.default_rng(sum(cells) + n)
    box = np.diag([1.001 * c for c in cells])
    pos = rng.uniform(0, 1, size=(n, 3)) @ box
    if max(cells) > 100:  # keep some pairs in a long box
        pos[n // 2:] = pos[: n - n // 2] + rng.normal(scale=0.3, size=(n - n // 2, 3))
    # two systems: the second one's cells follow the first one's
    systems = [dict(positions=pos, cell=box, pbc=np.array([True, False, True]), cutoff=1.0),
               dict(positions=pos[: n // 3 + 1], cell=box, pbc=np.array([False] * 3), cutoff=1.0)]
    b = NeighbourListBatch(systems, grid=grid, autotune=False)
    for _ in range(2):
        b.run()
        off = b.sys_offsets()
        outs = [t.cpu().numpy() for t in b.results()]
        for s, sd in enumerate(systems):
            want = oracle.oracle_neighbour_list("ijdDS", sd["cell"], sd["positions"], 1.0,
                                                sd["pbc"])
            assert_same_lists(tuple(o[off[s]:off[s + 1]] for o in outs), want, "ijdDS")
    b.close()
