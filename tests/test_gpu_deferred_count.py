"""Counts made after a force pass: nbl_lj_forces leaves them to the call that
first reads them, for the row range the forces had, whatever the plan's range is
by then; rows outside it count zero."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,edge", [(700, 9.0), (900, 60.0)])   # dense and sparse grids
@pytest.mark.parametrize("rows", [(0, 1), (100, 257), (699, 700)])
@pytest.mark.parametrize("reader", ["counts", "offsets", "matrix"])
def test_range_reset_between_forces_and_counts(oracle, n, edge, rows, reader):
    import torch
    from matscipy_neighbours import _matscipy_neighbours as ext
    rng = np.random.default_rng(n)
    cell = edge * np.array([[1.0, 0.0, 0.0], [0.1, 1.0, 0.0], [0.0, -0.2, 1.0]])
    pos = np.ascontiguousarray(rng.uniform(size=(n, 3)) @ cell)
    pbc = np.array([True, False, True])
    first = oracle.oracle_neighbour_list("i", cell, pos, 2.5, pbc)
    deg = np.bincount(first, minlength=n)
    want = np.where((np.arange(n) >= rows[0]) & (np.arange(n) < rows[1]), deg, 0)
    K = int(deg.max()) + 1
    origin, inv = np.zeros(3), np.ascontiguousarray(np.linalg.inv(cell.T))
    pbc8 = pbc.astype(np.uint8)
    dev = torch.from_numpy(pos).cuda()
    req = ext.make_request(1, origin, cell, inv, pbc8, n, ctypes.c_void_p(dev.data_ptr()), True,
                           2.5, None, None, 0, None, 0)
    force = torch.zeros((n, 3), dtype=torch.float64, device="cuda")
    energy = torch.zeros((), dtype=torch.float64, device="cuda")
    counts = torch.full((n,), -1, dtype=torch.int32, device="cuda")
    off = torch.full((n + 1,), -1, dtype=torch.int64, device="cuda")
    idx = torch.full((n, K), -1, dtype=torch.int32, device="cuda")
    dist = torch.empty((n, K, 3), dtype=torch.float64, device="cuda")
    p = lambda t: ctypes.c_void_p(t.data_ptr())
    plan, npairs, over = ctypes.c_void_p(), ctypes.c_int64(), ctypes.c_int()
    ext.check(ext.lib.nbl_plan_create(0, ctypes.byref(plan)))
    try:
        torch.cuda.synchronize()
        # a full count first: its degrees are what stale counts would show
        ext.check(ext.lib.nbl_count(plan, ctypes.byref(req), None, ctypes.byref(npairs)))
        ext.check(ext.lib.nbl_set_atom_range(plan, *rows))
        ext.check(ext.lib.nbl_lj_forces(plan, ctypes.byref(req), 1.0, 1.0, p(force), p(energy),
                                        None))
        ext.check(ext.lib.nbl_set_atom_range(plan, 0, -1))
        if reader == "matrix":
            ext.check(ext.lib.nbl_fill_matrix(plan, K, p(idx), p(dist), p(counts),
                                              ctypes.byref(over), None))
        if reader == "offsets":
            ext.check(ext.lib.nbl_row_offsets(plan, p(off), None))
        ext.check(ext.lib.nbl_counts(plan, p(counts), None))
        ext.check(ext.lib.nbl_row_offsets(plan, p(off), None))
        ext.check(ext.lib.nbl_check(plan, None))
    finally:
        ext.check(ext.lib.nbl_plan_destroy(plan))
    assert np.array_equal(counts.cpu().numpy(), want)
    assert np.array_equal(off.cpu().numpy(), np.concatenate([[0], np.cumsum(want)]))
    if reader == "matrix":
        got = idx.cpu().numpy()
        keep = np.arange(K)[None, :] < want[:, None]
        j = oracle.oracle_neighbour_list("j", cell, pos, 2.5, pbc)
        assert np.array_equal(got[keep], j[(first >= rows[0]) & (first < rows[1])])
