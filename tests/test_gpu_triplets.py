"""Triplets on the device at the edges of a row's shared-memory list (128 kept
pairs) and of the lane rounds, with and without distances: the host's list."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lengths", [[0], [1], [2, 0, 1, 32, 33], [127, 128, 129, 3], [300, 0, 5],
                                     [64] * 300, [0, 0, 260]])
@pytest.mark.parametrize("distances", [False, True])
def test_triplets_of_rows(lengths, distances):
    import torch
    import matscipy_neighbours as m
    first = np.concatenate([[0], np.cumsum(lengths)]).astype(np.int32)
    if lengths[0] == 0 and len(lengths) > 2:
        first[:1] = -1   # an atom before the first one with pairs
    rng = np.random.default_rng(len(lengths))
    d = rng.uniform(0.0, 1.0, size=int(first[-1]))
    args = (d, 0.6) if distances else ()
    # the host walks rows from a non-negative start only
    want = m.triplet_list(np.maximum(first, 0), *args)
    dev = (torch.from_numpy(d).cuda(), 0.6) if distances else ()
    got = m.triplet_list(torch.from_numpy(first).cuda(), *dev)
    for g, w in zip(got, want):
        assert np.array_equal(g.cpu().numpy(), w)
