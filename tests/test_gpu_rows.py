"""Neighbour lists written by the count and expanded by the output-ordered fill:
rows shorter and far longer than the mean density lets expect (chained chunks,
rows that found no room), the first call of a size and the next one (which knows
the size of the lists), every cutoff kind and grid, entries of one and two words.
All of it is the oracle's list bit for bit."""
import numpy as np
import pytest

from conftest import assert_same_lists

pytestmark = pytest.mark.gpu


def _positions(place, n, rng):
    box = np.array([[24.0, 0.0, 0.0], [2.0, 26.0, 0.0], [-1.0, 1.5, 22.0]])
    u = rng.uniform(0.0, 1.0, size=(n, 3))
    if place == "uniform":
        box = box * (n / 400.0) ** (1.0 / 3.0) * 0.6
    elif place == "blob":          # everyone's neighbour: rows of n - 1 in a box of ~1
        u = 0.5 + 0.02 * (u - 0.5)
    elif place == "mixed":         # a dense corner in a dilute box
        u[: n // 3] *= 0.06
    return np.ascontiguousarray(u @ box), box


def _cutoff(kind, n, rng):
    if kind == "atom":             # one radius above half of the widest pair cutoff
        r = rng.uniform(0.5, 1.1, size=n)
        r[0] = 1.9
        return r, None
    if kind == "type":
        return np.array([[2.4, 1.1], [1.1, 0.7]]), rng.integers(0, 2, size=n).astype(np.int32)
    return 2.1, None


@pytest.mark.parametrize("kind", ["scalar", "atom", "type"])
@pytest.mark.parametrize("place,n", [("uniform", 129), ("uniform", 1025), ("uniform", 2999),
                                     ("blob", 131), ("blob", 300), ("blob", 1500),
                                     ("mixed", 900), ("mixed", 4001)])
def test_rows_of_every_length(oracle, place, n, kind):
    from matscipy_neighbours import neighbour_list, neighbour_matrix
    rng = np.random.default_rng(n)
    pos, cell = _positions(place, n, rng)
    cut, types = _cutoff(kind, n, rng)
    pbc = np.array([True, place != "mixed", n % 2 == 0])
    want = oracle.oracle_neighbour_list("ijdDS", cell, pos, cut, pbc, types=types)
    kw = dict(positions=pos, cell=cell, pbc=pbc, cutoff=cut, numbers=types)
    neighbour_list("i", positions=pos[:50], cell=cell, pbc=pbc, cutoff=1.0)  # another size
    for q in ("ijdDS", "ijdDS", "jS", "d"):   # unknown, then known list sizes; subsets
        got = neighbour_list(q, **kw)
        assert_same_lists(got if len(q) > 1 else (got,), tuple(want["ijdDS".index(c)] for c in q), q)
    i, j, _, D, _ = want
    deg = np.bincount(i, minlength=n)
    K = int(deg.max())
    idx, dist, count = neighbour_matrix(max_neighbours=K + 3, **kw)
    used = np.arange(K + 3)[None, :] < deg[:, None]
    assert np.array_equal(count, deg)
    assert np.array_equal(idx[used], j) and not idx[~used].any()
    assert np.array_equal(dist[used].view(np.int64), D.view(np.int64)) and not dist[~used].any()


@pytest.mark.parametrize("grid", ["dense", "hashed", "morton"])
@pytest.mark.parametrize("precision", ["fp32", "fp64"])
def test_rows_of_a_batch_with_two_word_entries(oracle, grid, precision):
    """Many visits (a cutoff far beyond a small cell) and many atoms: an entry's
    atom and visit no longer share one word.  Also many candidates per atom
    beside few, on every grid."""
    from matscipy_neighbours.batch import NeighbourListBatch
    rng = np.random.default_rng(5)
    tiny = np.array([[1.0, 0.0, 0.0], [0.2, 1.1, 0.0], [0.1, -0.3, 0.9]])
    gas = np.diag([100.0, 101.0, 99.0])
    systems = [dict(positions=rng.uniform(0, 1, size=(2, 3)) @ tiny, cell=tiny,
                    pbc=np.array([True] * 3), cutoff=14.0),
               dict(positions=rng.uniform(0, 1, size=(33000, 3)) @ gas, cell=gas,
                    pbc=np.array([True, False, True]), cutoff=2.5),
               dict(positions=np.zeros((1, 3)), cell=gas, pbc=np.array([False] * 3), cutoff=2.5)]
    b = NeighbourListBatch(systems, grid=grid, precision=precision, autotune=False)
    for _ in range(2):
        b.run()
        off = b.sys_offsets()
        outs = [t.cpu().numpy() for t in b.results()]
        for s, sd in enumerate(systems):
            want = oracle.oracle_neighbour_list("ijdDS", sd["cell"], sd["positions"],
                                                sd["cutoff"], sd["pbc"])
            assert_same_lists(tuple(o[off[s]:off[s + 1]] for o in outs), want, "ijdDS")
    b.close()


@pytest.mark.parametrize("rows", [(0, 1), (0, 257), (255, 256), (300, 2048), (2047, 2048)])
def test_rows_of_a_range(oracle, rows):
    import torch
    from matscipy_neighbours.distributed import neighbour_list_rows
    rng = np.random.default_rng(8)
    pos, cell = _positions("uniform", 2048, rng)
    pbc = np.array([True, True, False])
    want = oracle.oracle_neighbour_list("ijdDS", cell, pos, 2.1, pbc)
    keep = (want[0] >= rows[0]) & (want[0] < rows[1])
    got = neighbour_list_rows("ijdDS", torch.from_numpy(pos).cuda(), cell, pbc, 2.1, rows)
    torch.cuda.synchronize()
    assert_same_lists(tuple(g.cpu().numpy() for g in got), tuple(w[keep] for w in want), "ijdDS")


@pytest.mark.parametrize("n,edge,cutoff", [(1, 1.0, 52.0), (2, 1.3, 5.0), (700, 9.0, 2.5)])
def test_forces_then_the_list(oracle, n, edge, cutoff):
    """The force pass walks without a visit table (more visits than a table
    holds) and with one; a list built right after it is the oracle's."""
    import matscipy_neighbours as m
    rng = np.random.default_rng(n)
    cell = edge * np.array([[1.0, 0.0, 0.0], [0.1, 1.0, 0.0], [0.0, -0.2, 1.0]])
    g = int(np.ceil(n ** (1.0 / 3.0)))
    site = np.stack(np.meshgrid(*[np.arange(g)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n]
    pos = (site + 0.2 * rng.uniform(size=(n, 3))) / g @ cell
    i, D = oracle.oracle_neighbour_list("iD", cell, pos, cutoff, np.array([True] * 3))
    r2 = (D * D).sum(axis=1)
    s6 = (0.8 / r2) ** 3   # sigma^2 = 0.8
    f = np.zeros((n, 3))
    np.add.at(f, i, (-24.0 * s6 * (2.0 * s6 - 1.0) / r2)[:, None] * D)
    scale = np.abs(24.0 * s6 * (2.0 * s6 + 1.0) / np.sqrt(r2)).sum()
    e, got = m.lennard_jones(pos, cutoff, cell=cell, pbc=[True] * 3, sigma=np.sqrt(0.8))
    assert np.abs(got - f).max() <= 1e-12 * scale
    assert abs(e - 2.0 * np.sum(s6 * s6 - s6)) <= 1e-12 * np.sum(2.0 * (s6 * s6 + s6))
    want = oracle.oracle_neighbour_list("ijS", cell, pos, cutoff, np.array([True] * 3))
    assert_same_lists(m.neighbour_list("ijS", positions=pos, cell=cell, pbc=[True] * 3,
                                       cutoff=cutoff), want, "ijS")


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("n,edge,cutoff", [(33, 4.0, 1.9), (1000, 10.0, 2.5), (4097, 14.0, 2.5),
                                           (900, 60.0, 2.5), (400, 6.2, 3.0)])
def test_forces_by_items_and_by_atoms(oracle, n, edge, cutoff, precision):
    """Force passes by work items (tiles of every size, many candidates) and by
    atoms (sparse, plain FP64) against the pair list."""
    import matscipy_neighbours as m
    from matscipy_neighbours import _matscipy_neighbours as ext
    rng = np.random.default_rng(n)
    cell = edge * np.array([[1.0, 0.0, 0.0], [0.1, 1.0, 0.0], [0.0, -0.2, 1.0]])
    g = int(np.ceil(n ** (1.0 / 3.0)))
    site = np.stack(np.meshgrid(*[np.arange(g)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n]
    pos = (site + 0.2 * rng.uniform(size=(n, 3))) / g @ cell
    pbc = np.array([True, False, True])
    i, D = oracle.oracle_neighbour_list("iD", cell, pos, cutoff, pbc)
    r2 = (D * D).sum(axis=1)
    s6 = (0.8 / r2) ** 3
    f = np.zeros((n, 3))
    np.add.at(f, i, (-24.0 * s6 * (2.0 * s6 - 1.0) / r2)[:, None] * D)
    scale = np.abs(24.0 * s6 * (2.0 * s6 + 1.0) / np.sqrt(r2)).sum() + 1e-300
    prev = ext.set_options(precision=precision)
    try:
        e, got = m.lennard_jones(pos, cutoff, cell=cell, pbc=pbc, sigma=np.sqrt(0.8))
    finally:
        ext.set_options(**prev)
    assert np.abs(got - f).max() <= 1e-12 * scale
    assert abs(e - 2.0 * np.sum(s6 * s6 - s6)) <= 1e-12 * (np.sum(2.0 * (s6 * s6 + s6)) + 1e-300)
