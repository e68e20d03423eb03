"""Triplets of rows that keep more pairs than a warp's shared-memory list holds (256: a
CTA takes over, up to 2,048 in its shared memory): the host's list, and no cliff in time
where a row grows past the list."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lengths", [[255, 256, 257], [511, 512, 513, 7], [640, 0, 900], [1300],
                                     [2047, 2048], [2049, 3], [2500]])
@pytest.mark.parametrize("keep", [None, 0.15, 0.97])
def test_long_rows(lengths, keep):
    import torch
    import matscipy_neighbours as m
    first = np.concatenate([[0], np.cumsum(lengths)]).astype(np.int32)
    d = np.random.default_rng(len(lengths)).uniform(size=int(first[-1]))
    args = () if keep is None else (d, keep)
    want = m.triplet_list(first, *args)
    dev = () if keep is None else (torch.from_numpy(d).cuda(), keep)
    got = m.triplet_list(torch.from_numpy(first).cuda(), *dev)
    for g, w in zip(got, want):
        assert np.array_equal(g.cpu().numpy(), w)


@pytest.mark.parametrize("length,shorter,longer", [(2000, 120, 136), (2000, 490, 530)])
def test_no_cliff(length, shorter, longer):
    """Rows of 2,000 pairs: as long as the number of triplets is about the same, so is
    the time (a walk over the row per kept pair took six times as long)."""
    import torch
    import matscipy_neighbours as m
    rows = 1000
    first = torch.arange(rows + 1, dtype=torch.int32, device="cuda") * length

    def best(kept):
        d = torch.ones((rows, length), dtype=torch.float64, device="cuda")
        d[:, torch.linspace(0, length - 1, kept).long().cuda()] = 0.0
        d = d.reshape(-1)
        times = []
        for _ in range(6):
            t0, t1 = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            t0.record()
            out = m.triplet_list(first, d, 0.5)
            t1.record()
            t1.synchronize()
            times.append(t0.elapsed_time(t1))
            assert len(out[0]) == rows * kept * (kept - 1)
            del out
        return min(times)
    assert best(longer) < 2.5 * best(shorter)
