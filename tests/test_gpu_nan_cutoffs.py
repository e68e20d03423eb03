"""Radii and per-type cutoffs that are not numbers (the reference takes them: such a
pair's distance is never below its cutoff, and they do not enter the widest one), on
every pass."""
import ctypes

import numpy as np
import pytest

from conftest import assert_same_lists

pytestmark = pytest.mark.gpu


def _brute(pos, box, pair_cutoff, pbc):
    """All pairs by brute force in the oracle's row order of i; (i, j, S) sets."""
    out = set()
    shifts = [np.array(s) for s in np.ndindex(3, 3, 3)]
    for s in shifts:
        s = s - 1
        if np.any((s != 0) & ~pbc):
            continue
        d = np.linalg.norm(pos[None, :, :] + s * box - pos[:, None, :], axis=-1)
        with np.errstate(invalid="ignore"):
            hit = d < pair_cutoff
        if not s.any():
            np.fill_diagonal(hit, False)
        out |= {(i, j, *s) for i, j in zip(*np.nonzero(hit))}
    return out


@pytest.mark.parametrize("kind", ["atom", "type"])
@pytest.mark.parametrize("n,box,atoms", [(90, 8.0, 0), (300, 12.0, 0), (300, 12.0, -1),
                                         (300, 12.0, 1), (300, 25.0, 0), (300, 25.0, -1)])
def test_nan_cutoffs(oracle, n, box, atoms, kind):
    from matscipy_neighbours import _matscipy_neighbours as ext
    from matscipy_neighbours import neighbour_list
    rng = np.random.default_rng(n)
    pos = rng.uniform(size=(n, 3)) * box
    cell = box * np.eye(3)
    pbc = np.array([True, False, True])
    types = None
    if kind == "atom":
        cut = rng.uniform(0.5, 1.4, size=n)
        cut[::7] = np.nan
        pair = cut[:, None] + cut[None, :]
    else:
        types = rng.integers(0, 3, size=n).astype(np.int32)
        cut = np.array([[2.8, np.nan, 1.5], [np.nan, 2.0, 1.0], [1.5, 1.0, np.nan]])
        pair = cut[types[:, None], types[None, :]]
    want = oracle.oracle_neighbour_list("ijdDS", cell, pos, cut, pbc, types=types)
    assert {(i, j, *s) for i, j, s in zip(want[0], want[1], want[4])} == \
        _brute(pos, box, pair, pbc)
    plan = ext.plan_for(0)
    cfg = ext.LaunchConfig(thread_per_atom=atoms)
    try:
        ext.check(ext.lib.nbl_plan_set_launch_config(plan, ctypes.byref(cfg)))
        for _ in range(2):
            got = neighbour_list("ijdDS", positions=pos, cell=cell, pbc=pbc, cutoff=cut,
                                 numbers=types)
            assert_same_lists(got, want, "ijdDS")
    finally:
        cfg.thread_per_atom = 0
        ext.lib.nbl_plan_set_launch_config(plan, ctypes.byref(cfg))
