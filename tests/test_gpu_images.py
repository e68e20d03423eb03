"""Packed image indices: a candidate's record carries its image index in three
10-bit fields as long as every |q| <= 127 and open axes contribute nothing;
other atoms take the full record.  Pairs of both kinds, at the edges of the
packed range and mixed within one cell, are the oracle's bit for bit."""
import numpy as np
import pytest

from conftest import assert_same_lists

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pbc", [(True, True, True), (True, True, False), (False, True, True)])
@pytest.mark.parametrize("images", [(126, 127), (127, 128), (-127, -128), (0, 700), (-3, 5)])
@pytest.mark.parametrize("n,atoms", [(60, -1), (400, -1), (400, 1)])
def test_far_images(oracle, pbc, images, n, atoms):
    import ctypes
    from matscipy_neighbours import _matscipy_neighbours as ext
    from matscipy_neighbours import neighbour_list
    rng = np.random.default_rng(n + 10 * abs(images[1]))
    cell = np.array([[7.0, 0.0, 0.0], [1.5, 8.0, 0.0], [0.5, -0.7, 9.0]])
    pos = rng.uniform(0.0, 1.0, size=(n, 3)) @ cell
    pos += rng.choice(images, size=(n, 3)) * np.asarray(pbc) @ cell
    pos += (rng.integers(-2, 3, size=(n, 3)) * ~np.asarray(pbc)) @ cell  # outside open axes
    plan = ext.plan_for(0)
    cfg = ext.LaunchConfig()
    cfg.thread_per_atom = atoms
    try:
        ext.check(ext.lib.nbl_plan_set_launch_config(plan, ctypes.byref(cfg)))
        got = neighbour_list("ijdDS", positions=pos, cell=cell, pbc=pbc, cutoff=2.3)
    finally:
        cfg.thread_per_atom = 0
        ext.lib.nbl_plan_set_launch_config(plan, ctypes.byref(cfg))
    want = oracle.oracle_neighbour_list("ijdDS", cell, pos, 2.3, np.asarray(pbc))
    assert len(want[0]) > 0
    assert_same_lists(got, want, "ijdDS")
