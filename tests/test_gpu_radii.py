"""Per-atom radii in device memory belong to the caller: a fill that has to test
candidates again (thread-per-atom passes, rows or items that found no room) uses
the radii its count saw, even if the caller's have changed since."""
import ctypes

import numpy as np
import pytest

from conftest import assert_same_lists

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("place", ["uniform", "mixed"])
@pytest.mark.parametrize("atoms", [-1, 0, 1])
@pytest.mark.parametrize("n", [90, 1500])
def test_radii_changed_between_count_and_fill(oracle, n, atoms, place):
    import torch
    from matscipy_neighbours import _matscipy_neighbours as ext
    rng = np.random.default_rng(n)
    cell = np.array([[24.0, 0.0, 0.0], [2.0, 26.0, 0.0], [-1.0, 1.5, 22.0]])
    u = rng.uniform(size=(n, 3))
    if place == "mixed":   # rows far longer than the density lets expect
        u[: n // 2] *= 0.04
    pos = np.ascontiguousarray(u @ cell)
    r = rng.uniform(0.5, 1.4, size=n)
    pbc = np.array([True, True, False])
    want = oracle.oracle_neighbour_list("ijdDS", cell, pos, r, pbc)
    origin, inv = np.zeros(3), np.ascontiguousarray(np.linalg.inv(cell.T))
    pbc8 = pbc.astype(np.uint8)
    dpos, dr = torch.from_numpy(pos).cuda(), torch.from_numpy(r).cuda()
    req = ext.make_request(31, origin, cell, inv, pbc8, n, ctypes.c_void_p(dpos.data_ptr()), True,
                           float(2.0 * r.max()), dr.data_ptr(), None, 0, None, 0,
                           aux_on_device=True)
    plan, npairs = ctypes.c_void_p(), ctypes.c_int64()
    ext.check(ext.lib.nbl_plan_create(0, ctypes.byref(plan)))
    cfg = ext.LaunchConfig(thread_per_atom=atoms)
    try:
        ext.check(ext.lib.nbl_plan_set_launch_config(plan, ctypes.byref(cfg)))
        torch.cuda.synchronize()
        ext.check(ext.lib.nbl_count(plan, ctypes.byref(req), None, ctypes.byref(npairs)))
        assert npairs.value == len(want[0])
        dr.zero_()
        torch.cuda.synchronize()
        P = npairs.value
        outs = {"i": torch.empty(P, dtype=torch.int32, device="cuda"),
                "j": torch.empty(P, dtype=torch.int32, device="cuda"),
                "D": torch.empty((P, 3), dtype=torch.float64, device="cuda"),
                "d": torch.empty(P, dtype=torch.float64, device="cuda"),
                "S": torch.empty((P, 3), dtype=torch.int32, device="cuda")}
        o = ext._outputs_struct(outs, lambda t: t.data_ptr())
        ext.check(ext.lib.nbl_fill(plan, ctypes.byref(o), None))
        ext.check(ext.lib.nbl_check(plan, None))
    finally:
        ext.check(ext.lib.nbl_plan_destroy(plan))
    assert_same_lists(tuple(outs[q].cpu().numpy() for q in "ijdDS"), want, "ijdDS")
