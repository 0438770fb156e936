"""k vectors beyond the kernels' tables (|n| > 16): the potential and its patched call refuse them, wherever in
the list they stand, and take those at the limit."""

import numpy as np
import pytest
import torch

from test_gpu_ewald_streams import salt

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n, refused", [(16, False), (-16, False), (17, True), (-17, True), (47, True)])
@pytest.mark.parametrize("row, axis", [(0, 0), (1, 2), (-1, 1)])
def test_components_beyond_the_tables_are_refused(n, refused, row, axis):
    from kups_gb300 import _lib, ewald, potential

    parts, tril, prm, lj, _, _ = salt()
    good = prm.reciprocal_lattice_shifts
    kn = good.clone()
    kn[0, row, axis] = n
    patch = potential.ParticlePatch(torch.arange(2, device="cuda"), parts.positions[:2] + 0.1)
    pot = ewald.LJEwaldPotential(prm, *lj)
    cache = pot(parts, tril).cache
    pot.ewald = ewald.EwaldParameters(prm.alpha, prm.cutoff, kn)
    if not refused:
        out = pot(parts, tril)
        assert np.isfinite(out.total_energies.cpu().numpy()).all()
        assert np.isfinite(pot(parts, tril, patch, out.cache).total_energies.cpu().numpy()).all()
        return
    with pytest.raises(_lib.KupsError, match="unsupported"):
        pot(parts, tril)
    with pytest.raises(_lib.KupsError, match="unsupported"):
        pot(parts, tril, patch, cache)
