"""Cells left out of a particle's search because the cutoff does not reach them: edge sets bit-exact against
the float64 oracle for 1 to 7 cells along each axis, cubic and skewed cells, particles on cell faces, edges
and corners and one ulp beside them, pairs at exactly the cutoff, and coordinates many cells away."""

import numpy as np
import pytest

from oracle import neighborlist as onl
from oracle import unitcell as ouc
from test_gpu_core import assert_same_edges, gpu_edges

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cells", [(1, 2, 3), (3, 3, 3), (3, 4, 5), (4, 4, 4), (7, 4, 3), (6, 6, 6)])
@pytest.mark.parametrize("angles", [(90, 90, 90), (75, 100, 115)])
@pytest.mark.parametrize("slack", [1.001, 1.2])
def test_reach(cells, angles, slack):
    rng = np.random.default_rng(sum(cells) + angles[0])
    rc = 1.0
    L = ouc.lattice_from_lengths_angles([1.0, 1.0, 1.0], angles)
    widths = abs(np.linalg.det(L)) / np.array([np.linalg.norm(np.cross(L[1], L[2])), np.linalg.norm(np.cross(L[0], L[2])),
                                               np.linalg.norm(np.cross(L[0], L[1]))])
    L = L * (np.array(cells) * rc * slack / widths)[:, None]  # `cells` widths of slack rc along each axis
    tril = ouc.tril_from_lattice(L)[None]
    grid = np.stack(np.meshgrid(*[np.arange(c) / c for c in cells], indexing="ij"), -1).reshape(-1, 3)
    f = np.concatenate([grid, np.nextafter(grid, 1.0), np.nextafter(grid, -1.0), grid + 0.5 / np.array(cells),
                        rng.uniform(0, 1, (200, 3))])
    f = f + rng.integers(-5, 6, f.shape)
    pos = f @ L
    # partners at the cutoff, and an ulp to either side of it
    step = rng.normal(size=(60, 3))
    step /= np.linalg.norm(step, axis=1)[:, None]
    pos = np.concatenate([pos, pos[:60] + rc * step, pos[:60] + np.nextafter(rc, 0) * step])
    system = np.zeros(len(pos), np.int64)
    exp = onl.neighbor_list(pos, system, tril, np.array([rc]))
    got, _ = gpu_edges(pos, system, tril, np.array([rc]))
    assert_same_edges(got, onl.sort_edges(*exp))
