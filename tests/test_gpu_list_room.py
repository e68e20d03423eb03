"""Room of the neighbour lists: what the plan keeps stays in proportion to the pairs
a system can have, whatever its shape, and the lists are the oracle's."""
import ctypes

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


def _bulk(n=20000, seed=0):
    rng = np.random.default_rng(seed)
    box = (n / 0.085) ** (1.0 / 3.0)
    cell = box * np.array([[1.0, 0.0, 0.0], [0.1, 1.0, 0.0], [0.0, -0.2, 1.0]])
    return np.ascontiguousarray(rng.uniform(size=(n, 3)) @ cell), cell


def test_rows_of_a_range_and_full_lists_in_turn(oracle):
    """A range's lists hold its rows only, and a call of one range leaves the next
    call of another one with all the room it needs."""
    import torch
    from matscipy_neighbours.distributed import neighbour_list_rows
    pos, cell = _bulk()
    pbc = np.array([True, True, False])
    want = oracle.oracle_neighbour_list("ijdDS", cell, pos, 4.0, pbc)
    dev = torch.from_numpy(pos).cuda()
    plan = _plan()
    room = {}
    for rows in ((0, 20000), (5000, 7500), (0, 20000), (5000, 7500), (0, 2500), (19999, 20000),
                 (0, 20000), (17, 17)):
        got = neighbour_list_rows("ijdDS", dev, cell, pbc, 4.0, rows)
        torch.cuda.synchronize()
        keep = (want[0] >= rows[0]) & (want[0] < rows[1])
        assert_same_lists(tuple(g.cpu().numpy() for g in got), tuple(w[keep] for w in want),
                          "ijdDS")
        info = list_info(plan)
        assert not info.short_of_room, rows
        assert room.setdefault(rows, info.list_bytes) == info.list_bytes, rows
    own = lambda rows: room[rows] - (1 << 20)   # (a MB for chains)
    assert own((5000, 7500)) < own((0, 20000)) / 6


def test_cutoff_kinds_and_densities_in_turn(oracle):
    """Few pairs, then many, of the same sizes: no call's room follows the other's."""
    from matscipy_neighbours import neighbour_list
    pos, cell = _bulk(n=6000)
    rng = np.random.default_rng(4)
    types = rng.integers(0, 2, size=6000).astype(np.int32)
    few = np.array([[4.0, 1.0], [1.0, 1.0]])
    types[:] = 1
    types[0] = 0
    squeezed = pos.copy()
    squeezed[:, 0] *= 0.3
    pbc = np.array([True, False, True])
    calls = [(pos, few, types), (pos, 4.0, None), (squeezed, 4.0, None), (pos, few, types),
             (squeezed, 4.0, None), (pos, 4.0, None)]
    plan = _plan()
    sizes = []
    for p, cut, ty in calls + calls:
        want = oracle.oracle_neighbour_list("ijdDS", cell, p, cut, pbc, types=ty)
        got = neighbour_list("ijdDS", positions=p, cell=cell, pbc=pbc, cutoff=cut, numbers=ty)
        assert_same_lists(got, want, "ijdDS")
        sizes.append(list_info(plan).list_bytes)
    assert len(set(sizes[len(calls):])) == 1, sizes
    assert not list_info(plan).short_of_room


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("place", ["droplet", "blob", "half"])
@pytest.mark.parametrize("n", [300, 2500])
def test_first_count_of_crowded_atoms_has_room(oracle, n, place, precision):
    """Atoms crowded into a small part of their box, where the mean density lets expect
    hardly any neighbours: every row has its list after the first call already."""
    from matscipy_neighbours import _matscipy_neighbours as ext
    from matscipy_neighbours import neighbour_list
    rng = np.random.default_rng(n)
    cell = np.diag([120.0, 130.0, 110.0])
    u = rng.uniform(size=(n, 3))
    if place == "droplet":
        pos = 50.0 + u * (n / 0.08) ** (1.0 / 3.0)
    else:
        pos = 50.0 + u
        if place == "half":
            pos[::2] = u[::2] @ cell
    pbc = np.array([False] * 3)
    want = oracle.oracle_neighbour_list("ijdDS", cell, pos, 3.0, pbc)
    plan = _plan()
    neighbour_list("i", positions=u[:200] * 20.0, cell=cell, pbc=pbc, cutoff=3.0)  # other sizes
    prev = ext.set_options(precision=precision)
    try:
        for _ in range(2):
            got = neighbour_list("ijdDS", positions=pos, cell=cell, pbc=pbc, cutoff=3.0)
            assert_same_lists(got, want, "ijdDS")
            info = list_info(plan)
            assert info.lists and not info.short_of_room
    finally:
        ext.set_options(**prev)


@pytest.mark.parametrize("blob,by_atoms", [(0, 1), (1500, 0)])
def test_a_blob_in_a_gas_is_counted_by_cells(oracle, blob, by_atoms):
    """Few atoms per occupied cell on average, but most pairs in one cell."""
    from matscipy_neighbours import neighbour_list
    rng = np.random.default_rng(blob)
    cell = 100.0 * np.eye(3)
    pos = rng.uniform(size=(3000, 3)) @ cell
    pos[:blob] = 50.0 + rng.uniform(size=(blob, 3))
    pbc = np.array([False, True, False])
    want = oracle.oracle_neighbour_list("ijdDS", cell, pos, 2.5, pbc)
    plan = _plan()
    for _ in range(3):
        got = neighbour_list("ijdDS", positions=pos, cell=cell, pbc=pbc, cutoff=2.5)
        assert_same_lists(got, want, "ijdDS")
    assert list_info(plan).by_atoms == by_atoms


@pytest.mark.parametrize("capacity", [None, 3 << 20])
def test_batch_of_droplets_has_room(oracle, capacity):
    """The lists of a batch are sized by a count, also where the caller gives the
    output's capacity."""
    from matscipy_neighbours.batch import NeighbourListBatch
    rng = np.random.default_rng(2)
    cell = 90.0 * np.eye(3)
    systems = [dict(positions=40.0 + rng.uniform(size=(n, 3)) * w, cell=cell,
                    pbc=np.array([False, True, False]), cutoff=3.0)
               for n, w in ((600, 2.0), (1500, 25.0), (3, 1.0), (400, 1.0))]
    b = NeighbourListBatch(systems, autotune=False, capacity=capacity)
    for _ in range(2):
        b.run()
        off = b.sys_offsets()
        outs = [t.cpu().numpy() for t in b.results()]
        for s, sd in enumerate(systems):
            want = oracle.oracle_neighbour_list("ijdDS", cell, sd["positions"], 3.0, sd["pbc"])
            assert_same_lists(tuple(o[off[s]:off[s + 1]] for o in outs), want, "ijdDS")
    info = list_info(batch=b._h)
    assert info.lists and not info.by_atoms
    assert info.list_bytes >= 4 * off[-1]
    b.close()


@pytest.mark.parametrize("place", ["bulk", "droplet"])
@pytest.mark.parametrize("failures", [0, 1, 2, 3, 4])
def test_device_without_room_for_the_lists(oracle, place, failures):
    """Workspace growths that fail leave fewer lists, and rows without one to the
    thread-per-atom fill; what there was room for is kept for these sizes, so that
    later calls neither release nor grow the workspace."""
    import torch
    from matscipy_neighbours import _matscipy_neighbours as ext
    ext.lib.nbl_debug_inject.argtypes = [ctypes.c_int, ctypes.c_int64]
    n = 24000
    pos, cell = _bulk(n)
    if place == "droplet":
        cell = 8.0 * cell
    pbc = np.array([False] * 3)
    want = oracle.oracle_neighbour_list("ijdDS", cell, pos, 6.0, pbc)
    plan = _plan()
    from matscipy_neighbours import neighbour_list
    call = lambda: neighbour_list("ijdDS", positions=pos, cell=cell, pbc=pbc, cutoff=6.0)
    if place == "droplet":   # room for a gas of the same sizes: only the second count grows
        neighbour_list("i", positions=8.0 * pos, cell=cell, pbc=pbc, cutoff=6.0)
    try:
        ext.check(ext.lib.nbl_debug_inject(1, failures))
        try:
            got = call()
        except MemoryError:   # more failures than smaller layouts
            assert failures > 1
            return
        assert_same_lists(got, want, "ijdDS")
        ext.check(ext.lib.nbl_debug_inject(1, 0))
        first = list_info(plan)
        assert bool(first.short_of_room) == (failures > 0 and first.list_bytes < 4 * len(want[0]))
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        ext.check(ext.lib.nbl_debug_inject(1, 1))   # a growth would fail
        for _ in range(3):
            assert_same_lists(call(), want, "ijdDS")
            info = list_info(plan)
            assert info.list_bytes == first.list_bytes
            assert info.workspace_bytes == first.workspace_bytes
        assert torch.cuda.mem_get_info()[0] == free
    finally:
        ext.check(ext.lib.nbl_debug_inject(1, 0))
