"""kups_virial_stress over the forms a group can take: runs of 1, 15, 16 (the most one thread takes), 17 and
40 neighbouring atoms, groups in pieces, molecules across the faces and wider than a quarter of the cell,
systems whose borders fall inside a warp, counts around the 128-atom chunk, groups without atoms, and
coordinates far outside the cell; against the float64 oracle (relative 1e-11 of the largest component: the
sums run in a different order)."""

import numpy as np
import pytest
import torch

from oracle import observables as ob
from oracle.md import kinetic_energy
from oracle.unitcell import lattice_from_tril, wrap
from test_gpu_observables import close

pytestmark = pytest.mark.gpu


def _case(size, n_mol, width, order, images, seed):
    """Three systems of n_mol groups of ``size`` atoms, ``width`` times the cell wide."""
    rng = np.random.default_rng(seed)
    trils = np.array([[9.0, 0.7, 10.0, -1.1, 0.6, 8.0], [30.0, 0.0, 31.0, 0.0, 0.0, 32.0],
                      [15.0, -2.0, 14.0, 3.0, 1.0, 16.0]])
    pos, sysi, grp = [], [], []
    for s, t in enumerate(trils):
        L = lattice_from_tril(t)
        f = rng.uniform(-0.5, 0.5, (n_mol, 1, 3)) + width * rng.uniform(-0.5, 0.5, (n_mol, size, 3))
        p = f.reshape(-1, 3) @ L
        pos.append(p if images else wrap(p, t[None]))
        if images:  # each atom in an image of its own
            pos[-1] = pos[-1] + rng.integers(-3, 4, (len(p), 3)) @ L
        sysi.append(np.full(len(p), s))
        grp.append(2 * s + (n_mol + 2) * s + np.repeat(np.arange(n_mol), size))  # some groups without atoms
    pos, sysi, grp = np.concatenate(pos), np.concatenate(sysi), np.concatenate(grp)
    o = {"as is": np.arange(len(pos)), "pieces": np.argsort(np.arange(len(pos)) % 7, kind="stable"),
         "reversed": np.arange(len(pos))[::-1].copy(),
         "mixed systems": np.argsort(np.tile(np.arange(n_mol), 3).repeat(size), kind="stable")}[order]
    return pos[o], sysi[o], grp[o], int(grp.max()) + 4, trils, rng


@pytest.mark.parametrize("size,n_mol,width,order,images", [
    (1, 300, 0.0, "as is", False), (2, 21, 0.1, "as is", True), (3, 14, 0.1, "as is", False),
    (3, 14, 0.1, "as is", True), (3, 1000, 0.2, "mixed systems", False), (3, 40, 0.1, "reversed", False),
    (3, 400, 0.9, "as is", False), (15, 9, 0.2, "as is", False), (16, 64, 0.2, "as is", True),
    (17, 64, 0.2, "as is", False), (40, 11, 0.3, "as is", False), (5, 200, 0.1, "pieces", False)])
def test_group_forms_match_the_oracle(size, n_mol, width, order, images):
    from kups_gb300 import observables

    pos, sysi, grp, n_groups, tril, rng = _case(size, n_mol, width, order, images, size + n_mol)
    n = len(pos)
    grad, mom, mass = rng.normal(size=(n, 3)), rng.normal(size=(n, 3)), rng.uniform(1, 40, n)
    dtril = rng.normal(size=(3, 6))
    for momenta in (mom, None):
        out = observables.virial_observables(pos, grad, sysi, tril, dtril, group=grp, n_groups=n_groups,
                                             momenta=momenta, masses=mass, molecular=True)
        out = {k: v.cpu().numpy() for k, v in out.items()}
        st = ob.virial_stress(pos, grad, sysi, tril, dtril)
        ke = kinetic_energy(mom, mass, sysi, 3) if momenta is not None else np.zeros(3)
        close(out["stress"], st)
        close(out["molecular_stress"], ob.molecular_virial_stress(pos, grad, sysi, grp, n_groups, tril, dtril))
        close(out["lattice_stress"], ob.lattice_stress(tril, dtril))
        close(out["pressure"], ob.instantaneous_pressure(ke, st, tril))
        if momenta is not None:
            close(out["kinetic"], ke)


@pytest.mark.parametrize("n", [0, 1, 31, 33, 127, 129, 152 * 3 * 128 + 5])
def test_atomic_stress_of_few_and_many_atoms(n):
    from kups_gb300 import observables

    rng = np.random.default_rng(n)
    tril = np.array([[9.0, 0.7, 10.0, -1.1, 0.6, 8.0], [30.0, 0.0, 31.0, 0.0, 0.0, 32.0]])
    pos, grad, sysi = rng.normal(size=(n, 3)), rng.normal(size=(n, 3)), np.arange(n) * 2 // max(n, 1)
    out = observables.stress_via_virial_theorem(pos, grad, sysi, tril).cpu().numpy()
    close(out, ob.virial_stress(pos, grad, sysi, tril, np.zeros((2, 6))))
