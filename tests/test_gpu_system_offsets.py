"""Offsets of the systems' atoms (kups_system_offsets) against numpy: empty systems, runs across the 16 atoms
of a thread and the 4096 of a block, more systems than the scan's block, no atoms, indices out of range."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,s,order", [(0, 1, "sorted"), (1, 1, "sorted"), (17, 3, "sorted"), (4096, 255, "sorted"),
                                       (4097, 256, "sorted"), (50000, 257, "sorted"), (50000, 1000, "any"),
                                       (3, 700, "any")])
def test_offsets(n, s, order):
    from kups_gb300.ewald import _offsets

    rng = np.random.default_rng(n + s)
    sysi = rng.integers(0, s, n)
    if order == "sorted":
        sysi = np.sort(sysi)
    off, most = _offsets(torch.as_tensor(sysi, dtype=torch.int32).cuda(), s)
    counts = np.bincount(sysi, minlength=s)
    np.testing.assert_array_equal(off.cpu().numpy(), np.concatenate([[0], np.cumsum(counts)]))
    assert most == counts.max()


def test_indices_out_of_range_are_refused():
    from kups_gb300.ewald import _offsets

    for bad in ([0, 1, 2], [0, -1, 1]):
        with pytest.raises(RuntimeError):
            _offsets(torch.tensor(bad, dtype=torch.int32).cuda(), 2)
