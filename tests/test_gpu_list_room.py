"""Room of the neighbour lists: what the plan keeps stays in proportion to the pairs
a system can have, whatever its shape, and the lists are the oracle's."""
import numpy as np
import pytest

from _lists import list_info
from conftest import assert_same_lists

pytestmark = pytest.mark.gpu


def _plan():
    import torch
    from matscipy_neighbours import _matscipy_neighbours as ext
    torch.cuda.set_device(0)
    ext.check(ext.lib.nbl_plan_trim(ext.plan_for(0)))
    return ext.plan_for(0)


@pytest.mark.parametrize("shape,cutoff", [("cube", 5.0), ("sheet", 2.5), ("chain", 2.5)])
@pytest.mark.parametrize("n", [129, 3000])
def test_open_systems_of_every_shape(oracle, n, shape, cutoff):
    """All atoms within each other's cutoff; flat and thin shrink-wrapped cells, whose
    volume says nothing about their neighbours."""
    from matscipy_neighbours import neighbour_list
    rng = np.random.default_rng(n)
    side = {"cube": (1.0, 1.0, 1.0), "sheet": (60.0, 50.0, 1e-4),
            "chain": (900.0, 0.05, 0.05)}[shape]
    pos = rng.uniform(size=(n, 3)) * side
    cell = np.diag(side)
    pbc = np.array([False] * 3)
    want = oracle.oracle_neighbour_list("ijdDS", cell, pos, cutoff, pbc)
    plan = _plan()
    for _ in range(2):
        got = neighbour_list("ijdDS", positions=pos, cell=cell, pbc=pbc, cutoff=cutoff)
        assert_same_lists(got, want, "ijdDS")
        info = list_info(plan)
        assert info.lists and not info.short_of_room
        # an entry is 4 bytes; a MB for chains, and the scatter of short rows
        assert info.list_bytes <= 8 * len(want[0]) + 400 * n + (2 << 20)
