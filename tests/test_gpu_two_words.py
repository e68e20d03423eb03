"""List entries of two words: where the visited offsets are so many that an atom's
number and a visit's no longer share one word.  A sheet in an open cell a ten-
thousandth of the cutoff high (450,009 visited offsets, of which nine are inside)
and a batch with a tiny periodic cell; the sparse and the dense count, the split and
the whole walk, fill, matrix and forces.  All of it is the oracle's."""
import numpy as np
import pytest

from _lists import list_info
from conftest import assert_same_lists

pytestmark = pytest.mark.gpu

HEIGHT = 1e-4


def _sheet(n, per_cell, rng, clump=0):
    side = 2.5 * np.sqrt(n / per_cell)
    cell = np.diag([side, 1.1 * side, HEIGHT])
    u = rng.uniform(size=(n, 3))
    u[:clump, :2] = 0.4 + 1.5 / side * u[:clump, :2]   # one crowd: chained rows
    return np.ascontiguousarray(u @ cell), cell


def _cutoff(kind, n, rng):
    if kind == "atom":
        return rng.uniform(0.8, 1.25, size=n), None
    if kind == "type":
        return np.array([[2.5, 1.3], [1.3, 0.9]]), rng.integers(0, 2, size=n).astype(np.int32)
    return 2.5, None


@pytest.mark.parametrize("kind", ["scalar", "atom", "type"])
@pytest.mark.parametrize("n,per_cell,clump", [(8300, 1.5, 0), (8300, 9.0, 0), (8300, 1.5, 400),
                                              (33000, 1.5, 300)])
def test_sheets(oracle, n, per_cell, clump, kind):
    from matscipy_neighbours import _matscipy_neighbours as ext
    from matscipy_neighbours import neighbour_list, neighbour_matrix
    rng = np.random.default_rng(n)
    pos, cell = _sheet(n, per_cell, rng, clump)
    cut, types = _cutoff(kind, n, rng)
    pbc = np.array([True, False, False])
    kw = dict(positions=pos, cell=cell, pbc=pbc, cutoff=cut, numbers=types)
    want = oracle.oracle_neighbour_list("ijdDS", cell, pos, cut, pbc, types=types)
    plan = ext.plan_for(0)
    for _ in range(2):
        assert_same_lists(neighbour_list("ijdDS", **kw), want, "ijdDS")
        info = list_info(plan)
        assert info.lists and info.two_words
        assert clump or info.by_atoms == (per_cell < 4)
    i, j, _, D, _ = want
    deg = np.bincount(i, minlength=n)
    K = int(deg.max()) + 1
    idx, dist, count = neighbour_matrix(max_neighbours=K, **kw)
    used = np.arange(K)[None, :] < deg[:, None]
    assert np.array_equal(count, deg)
    assert np.array_equal(idx[used], j) and not idx[~used].any()
    assert np.array_equal(dist[used].view(np.int64), D.view(np.int64)) and not dist[~used].any()


@pytest.mark.parametrize("per_cell", [0.5, 1.5, 9.0])
def test_forces_of_a_sheet(oracle, per_cell):
    import matscipy_neighbours as m
    from matscipy_neighbours import _matscipy_neighbours as ext
    rng = np.random.default_rng(3)
    n = 8300
    side = 2.5 * np.sqrt(n / per_cell)
    g = int(np.ceil(np.sqrt(n)))
    site = np.stack(np.meshgrid(np.arange(g), np.arange(g), indexing="ij"), -1).reshape(-1, 2)[:n]
    cell = np.diag([side, side, HEIGHT])
    pos = np.ascontiguousarray(np.c_[(site + 0.3 * rng.uniform(size=(n, 2))) / g,
                                     rng.uniform(size=n)] @ cell)
    pbc = np.array([True, True, False])
    sigma = 0.4 * side / g
    i, D = oracle.oracle_neighbour_list("iD", cell, pos, 2.5, pbc)
    r2 = (D * D).sum(axis=1)
    s6 = (sigma * sigma / r2) ** 3
    f = np.zeros((n, 3))
    np.add.at(f, i, (-24.0 * s6 * (2.0 * s6 - 1.0) / r2)[:, None] * D)
    scale = np.abs(24.0 * s6 * (2.0 * s6 + 1.0) / np.sqrt(r2)).sum()
    e, got = m.lennard_jones(pos, 2.5, cell=cell, pbc=pbc, sigma=sigma)
    assert list_info(ext.plan_for(0)).two_words
    assert np.abs(got - f).max() <= 1e-12 * scale
    assert abs(e - 2.0 * np.sum(s6 * s6 - s6)) <= 1e-12 * np.sum(2.0 * (s6 * s6 + s6))


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("n,edge", [(17000, 80.0), (33000, 100.0), (33000, 45.0)])
def test_batch_with_a_tiny_cell(oracle, n, edge, precision):
    """Few candidates per atom on average (the count without culling)."""
    from matscipy_neighbours.batch import NeighbourListBatch
    rng = np.random.default_rng(n)
    tiny = np.diag([1.0, 1.01, 0.99])
    gas = np.diag([edge, 1.01 * edge, 0.99 * edge])
    systems = [dict(positions=np.array([[0.3, 0.2, 0.1]]), cell=tiny, pbc=np.array([True] * 3),
                    cutoff=25.5),
               dict(positions=rng.uniform(0, 1, size=(n, 3)) @ gas, cell=gas,
                    pbc=np.array([True, False, True]), cutoff=2.5)]
    b = NeighbourListBatch(systems, precision=precision, autotune=False)
    for _ in range(2):
        b.run()
        off = b.sys_offsets()
        outs = [t.cpu().numpy() for t in b.results()]
        for s, sd in enumerate(systems):
            want = oracle.oracle_neighbour_list("ijdDS", sd["cell"], sd["positions"],
                                                sd["cutoff"], sd["pbc"])
            assert_same_lists(tuple(o[off[s]:off[s + 1]] for o in outs), want, "ijdDS")
    assert list_info(batch=b._h).two_words
    b.close()
