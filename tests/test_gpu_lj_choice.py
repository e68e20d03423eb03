"""Forces of a droplet and of a gas with the same atoms, box and cell table, in turn: the
device chooses the pass at first, the plan knows it afterwards, and whichever runs the
forces are those of the pair list.  A droplet in a wide box is not taken for a gas."""
import numpy as np
import pytest

from _lists import list_info

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [5000, 30001])
def test_droplet_and_gas_in_turn(oracle, n):
    import torch
    import matscipy_neighbours as m
    from matscipy_neighbours import _matscipy_neighbours as ext
    rng = np.random.default_rng(n)
    g = int(np.ceil(n ** (1.0 / 3.0)))
    site = np.stack(np.meshgrid(*[np.arange(g)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n]
    u = site + 0.2 * rng.uniform(size=(n, 3))
    edge = 5.0 * g
    cell, pbc = edge * np.eye(3), np.array([False] * 3)
    systems = {}
    for name, spacing in (("droplet", 1.1), ("gas", 3.4)):
        pos = u * spacing + 0.1
        i, D = oracle.oracle_neighbour_list("iD", cell, pos, 2.6, pbc)
        r2 = (D * D).sum(axis=1)
        s6 = 1.0 / r2 ** 3
        f = np.zeros((n, 3))
        np.add.at(f, i, (-24.0 * s6 * (2.0 * s6 - 1.0) / r2)[:, None] * D)
        scale = np.abs(24.0 * s6 * (2.0 * s6 + 1.0) / np.sqrt(r2)).sum() + 1e-300
        systems[name] = (pos, f, 2.0 * np.sum(s6 * s6 - s6), scale)
    plan = ext.plan_for(0)
    ext.check(ext.lib.nbl_plan_trim(plan))
    for name in ("droplet", "droplet", "gas", "gas", "droplet", "gas", "droplet", "droplet"):
        pos, f, energy, scale = systems[name]
        e, got = m.lennard_jones(pos, 2.6, cell=cell, pbc=pbc)
        assert np.abs(got - f).max() <= 1e-12 * scale
        assert abs(e - energy) <= 1e-12 * scale
    assert not list_info(plan).by_atoms
    for _ in range(2):
        m.lennard_jones(systems["gas"][0], 2.6, cell=cell, pbc=pbc)
        torch.cuda.synchronize()
    assert list_info(plan).by_atoms == (n > 16384)
