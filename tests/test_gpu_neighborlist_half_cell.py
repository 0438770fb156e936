"""Skewed cells whose cutoff reaches half a cell width: two particles half a cell apart along a face normal
are within the cutoff by one image and far away by the other, and float32 coordinates may round to either.
Bit-exact against the float64 oracle."""

import numpy as np
import pytest

from test_gpu_neighborlist_search import check

pytestmark = pytest.mark.gpu


def widths(L):
    return abs(np.linalg.det(L)) / np.array([np.linalg.norm(np.cross(L[(a + 1) % 3], L[(a + 2) % 3])) for a in range(3)])


@pytest.mark.parametrize("tril", [[30.0, 3.0, 30.0, -6.0, 8.0, 11.0], [11.0, 3.0, 30.0, -6.0, 8.0, 30.0],
                                  [30.0, 14.0, 12.0, 5.0, -5.0, 40.0], [12.0, 0.0, 12.0, 0.0, 0.0, 12.0]])
@pytest.mark.parametrize("pairs", [20, 2000])  # a batch of one wave, and one that defers
def test_half_a_cell_apart(tril, pairs):
    L = np.array([[tril[0], 0, 0], [tril[1], tril[2], 0], [tril[3], tril[4], tril[5]]])
    w = widths(L)
    a = int(w.argmin())
    rc = 0.5 * w[a] * (1 - 1e-10)
    normal = np.cross(L[(a + 1) % 3], L[(a + 2) % 3])
    normal /= np.linalg.norm(normal)
    rng = np.random.default_rng(pairs)
    gap = np.concatenate([10.0 ** rng.uniform(-9, -6, pairs // 2), -(10.0 ** rng.uniform(-9, -6, pairs - pairs // 2))])
    first = rng.uniform(-1.5, 1.5, (pairs, 3)) @ L
    pos = np.stack([first, first + (rc - gap)[:, None] * rng.choice([-1, 1], (pairs, 1)) * normal], 1).reshape(-1, 3)
    system = np.repeat(np.arange(pairs // 10), 20)
    found = check(pos, system, np.tile(tril, (pairs // 10, 1)), np.full(pairs // 10, rc))
    assert found >= pairs  # both directions of the pairs inside the cutoff, at least
