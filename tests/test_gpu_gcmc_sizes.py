"""The change of the reciprocal-space energy for molecules of every size that has its own phase sum (1 to 4
atoms unrolled, 5 to 8 in a loop), with old, new and both ends, against the float64 sum over k of the
positions that the device holds.  Tolerance per k: float32 fractional coordinates are off by up to 3e-7 and
the phase products by 1e-6, so a unit charge's phase by e_k = 2 pi 3e-7 (|n_x| + |n_y| + |n_z|) + 1e-6; S and
its change carry that times the charges, and the float32 terms of the sum 1e-6 of their sizes."""

import numpy as np
import pytest

from oracle import unitcell as ouc
from test_gpu_gcmc import random_molecule, small_setup, wrapped

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("atoms", [1, 2, 3, 4, 5, 6, 7, 8])
@pytest.mark.parametrize("kind", ["translate", "insert", "delete"])
def test_reciprocal_energy_change_of_molecules_of_any_size(atoms, kind):
    from kups_gb300 import gcmc, units

    setup = small_setup(n_sys=3, rc=5.0)
    rng = np.random.default_rng(10 * atoms + len(kind))
    tril = setup.tril[0]
    L = ouc.lattice_from_tril(tril)
    setup.motif_positions = 1.2 * np.arange(atoms)[:, None] * np.array([[0.6, 0.64, 0.48]])
    setup.motif_species = np.resize([4, 5], atoms)
    setup.motif_charges = np.resize([0.3, -0.2, -0.1], atoms)
    place = lambda: wrapped(random_molecule(rng, L, setup.motif_positions), tril)
    guests = [np.concatenate([place() for _ in range(4)]) for _ in range(3)]
    mc = gcmc.GCMC(setup, seed=5)
    mc.set_guests(guests)
    mols = [int(m) for m in rng.integers(0, 4, 3)]
    old = [g.reshape(4, atoms, 3)[m] for g, m in zip(guests, mols)]
    news = [None if kind == "delete" else place() if kind == "insert" else wrapped(o + rng.normal(0, 0.5, 3), tril)
            for o in old]
    got = mc.evaluate([gcmc.MOVES.index(kind)] * 3, mols, news)[:, 2]
    n = np.asarray(setup.kvec_n[0], float)
    P = gcmc.prefactor(tril, n, setup.alpha[0])
    k = 2 * np.pi * n @ np.linalg.inv(L).T
    held = lambda x: np.asarray(x, np.float32).astype(float)
    S = lambda x, q: np.exp(1j * held(x) @ k.T).T @ q
    q = setup.motif_charges
    eps = 2 * np.pi * 3e-7 * np.abs(n).sum(1) + 1e-6
    for i in range(3):
        s = S(setup.fw_positions, setup.fw_charges) + S(guests[i], np.tile(q, 4))
        d = np.zeros(len(n), complex)
        if kind != "insert":
            d -= S(old[i], q)
        if kind != "delete":
            d += S(news[i], q)
        want = units.TO_STANDARD_UNITS * (P * (np.abs(s + d) ** 2 - np.abs(s) ** 2)).sum()
        every = np.abs(setup.fw_charges).sum() + 4 * np.abs(q).sum()
        tol = (2 * (np.abs(s) + np.abs(d)) * 2 * np.abs(q).sum() + 2 * np.abs(d) * every) * eps
        tol = units.TO_STANDARD_UNITS * (P * (tol + 1e-6 * (2 * np.abs(s) * np.abs(d) + np.abs(d) ** 2))).sum()
        assert abs(got[i] - want) <= tol, (i, got[i], want, tol)
