"""Outputs that find no room beside the lists of their count: the lists are given back,
the pairs counted again by hit words, and the call succeeds as it did without lists."""
import ctypes

import numpy as np
import pytest

from _lists import list_info
from conftest import assert_same_lists

pytestmark = pytest.mark.gpu


def _system(n=3000):
    rng = np.random.default_rng(n)
    cell = (n / 0.08) ** (1.0 / 3.0) * np.array([[1.0, 0, 0], [0.1, 1.0, 0], [0, -0.2, 1.0]])
    return np.ascontiguousarray(rng.uniform(size=(n, 3)) @ cell), cell, np.array([True, True, False])


@pytest.fixture
def failing(monkeypatch):
    """torch.empty on a device runs out of memory once, after `skip` allocations."""
    import torch
    real = torch.empty

    def arm(skip):
        left = [skip]

        def empty(*a, **k):
            if k.get("device") is not None and left[0] is not None:
                if left[0] == 0:
                    left[0] = None
                    raise torch.OutOfMemoryError("no room (injected)")
                left[0] -= 1
            return real(*a, **k)
        monkeypatch.setattr(torch, "empty", empty)
        return left
    return arm


@pytest.mark.parametrize("skip", [0, 3])
@pytest.mark.parametrize("call", ["list", "rows", "matrix", "autograd"])
def test_device_outputs(oracle, failing, call, skip):
    import torch
    from matscipy_neighbours import _matscipy_neighbours as ext
    from matscipy_neighbours import neighbour_list, neighbour_matrix
    from matscipy_neighbours.autograd import neighbour_list_autograd
    from matscipy_neighbours.distributed import neighbour_list_rows
    pos, cell, pbc = _system()
    dev = torch.from_numpy(pos).cuda()
    want = oracle.oracle_neighbour_list("ijDdS", cell, pos, 4.0, pbc)
    K = int(np.bincount(want[0]).max())
    left = failing(min(skip, 2) if call == "matrix" else skip)
    if call == "list":
        got = neighbour_list("ijDdS", positions=dev, cell=cell, pbc=pbc, cutoff=4.0,
                             array_namespace=torch)
    elif call == "rows":
        got = neighbour_list_rows("ijDdS", dev, cell, pbc, 4.0, (700, 2000))
        keep = (want[0] >= 700) & (want[0] < 2000)
        want = tuple(w[keep] for w in want)
    elif call == "autograd":
        got = [t.detach() for t in neighbour_list_autograd(
            dev, torch.from_numpy(cell), pbc, 4.0)]
    else:
        idx, _, count = neighbour_matrix(positions=dev, cell=cell, pbc=pbc, cutoff=4.0,
                                         max_neighbours=K, array_namespace=torch)
        used = np.arange(K)[None, :] < count.cpu().numpy()[:, None]
        got, want = (idx[torch.from_numpy(used).cuda()],), (want[1],)
    assert left[0] is None
    for g, w in zip(got, want):
        np.testing.assert_array_equal(g.cpu().numpy(), w)
    plan = ext.plan_for(0)
    assert not list_info(plan).lists
    cfg = ext.LaunchConfig()
    ext.check(ext.lib.nbl_plan_get_launch_config(plan, ctypes.byref(cfg)))
    assert cfg.thread_per_atom == 0
    neighbour_list("i", positions=pos, cell=cell, pbc=pbc, cutoff=4.0)
    assert list_info(plan).lists


def test_host_outputs(oracle, monkeypatch):
    from matscipy_neighbours import _matscipy_neighbours as ext
    from matscipy_neighbours import neighbour_list
    ext.lib.nbl_debug_inject.argtypes = [ctypes.c_int, ctypes.c_int64]
    pos, cell, pbc = _system()
    want = oracle.oracle_neighbour_list("ijDdS", cell, pos, 4.0, pbc)
    plan = ext.plan_for(0)
    ext.check(ext.lib.nbl_plan_trim(plan))
    real, calls = ext._host_outputs, []

    def outputs(*a, **k):
        if not calls:   # the scratch of the outputs cannot grow, the first time
            ext.check(ext.lib.nbl_debug_inject(1, 1))
        calls.append(1)
        return real(*a, **k)
    monkeypatch.setattr(ext, "_host_outputs", outputs)
    try:
        got = neighbour_list("ijDdS", positions=pos, cell=cell, pbc=pbc, cutoff=4.0)
    finally:
        ext.check(ext.lib.nbl_debug_inject(1, 0))
    assert len(calls) == 1 and not list_info(plan).lists
    assert_same_lists(got, want, "ijDdS")
