"""The paired edge kernels with species tables that are not symmetric: an edge and its reverse then carry
different terms.  And cutoffs that no pair is within.  Reference and tolerances as for the pair lists' test."""

import numpy as np
import pytest

import test_gpu_pair_lists as lists

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [5, 90])
@pytest.mark.parametrize("sig, eps", [([[2.0, 2.3], [2.1, 2.6]], [[0.01, 0.02], [0.02, 0.03]]),
                                      ([[2.0, 2.3], [2.3, 2.6]], [[0.01, 0.02], [0.0, 0.03]])])
@pytest.mark.parametrize("paired", [False, True])
def test_tables_that_are_not_symmetric(monkeypatch, n, sig, eps, paired):
    monkeypatch.setattr(lists, "SIG", np.array(sig))
    monkeypatch.setattr(lists, "EPS", np.array(eps))
    pos, system, species, q, e, s = lists.system_of(n, n)
    for terms in (1, 3):
        lists.close(lists.pair(pos, system, species, q, e, s, terms, paired),
                    lists.reference(pos, system, species, q, e, s, terms))
    want = lists.reference(pos, system, species, q, e, s, 1)
    lists.close(lists.lj(pos, system, species, e, s, False, paired), want)
    lists.close(lists.lj(pos, system, species, e, s, True, paired), want, 2e-5)  # float32 pairs


def test_potential_with_a_table_that_is_not_symmetric():
    from kups_gb300 import potential
    from kups_gb300.neighborlist import CellListNeighborList

    class Own(CellListNeighborList):
        """A neighbour list of the caller's: nothing is known of its edges."""

    pos, system, species, _, _, _ = lists.system_of(90, 4)
    t = lists.t
    prm = potential.LennardJonesParameters(("A", "B"), t([[2.0, 2.3], [2.1, 2.6]]), t([[0.01, 0.02], [0.015, 0.03]]),
                                           t(lists.RC))
    st = potential.LJState(potential.LJParticles(t(pos), t(species, lists.torch.int32), t(system, lists.torch.int32)),
                           t(lists.CELLS), prm)
    results = []
    for neighbors in (CellListNeighborList(64), Own(64)):
        out = potential.LennardJonesPotential(neighbors, pair_fp32=False)(st)
        results.append([x.cpu().numpy() for x in (out.total_energies, out.gradients.positions, out.gradients.unitcell)])
    lists.close(*results, 1e-10)


@pytest.mark.parametrize("species", [8, 32, 33])  # the largest tables that are looked through, and beyond
@pytest.mark.parametrize("symmetric", [False, True])
def test_large_tables(monkeypatch, species, symmetric):
    rng = np.random.default_rng(species)
    sig, eps = rng.uniform(1.8, 2.6, (2, species, species)) * np.array([[[1.0]], [[0.01]]])
    if symmetric:
        sig, eps = (sig + sig.T) / 2, (eps + eps.T) / 2
    monkeypatch.setattr(lists, "SIG", sig)
    monkeypatch.setattr(lists, "EPS", eps)
    pos, system, _, q, e, s = lists.system_of(90, species)
    kinds = rng.integers(0, species, len(pos))
    for terms in (1, 3):
        lists.close(lists.pair(pos, system, kinds, q, e, s, terms, True),
                    lists.reference(pos, system, kinds, q, e, s, terms))
    lists.close(lists.lj(pos, system, kinds, e, s, False, True), lists.reference(pos, system, kinds, q, e, s, 1))


@pytest.mark.parametrize("paired", [False, True])
@pytest.mark.parametrize("cutoff", [0.0, -4.0])
def test_no_pair_is_within_a_cutoff_of_nothing(monkeypatch, paired, cutoff):
    """One system's real-space electrostatics switched off by its cutoff: r < cutoff holds for no pair."""
    monkeypatch.setattr(lists, "RCE", np.array([5.0, cutoff, 5.2]))
    pos, system, species, q, e, s = lists.system_of(90, 7)
    lists.close(lists.pair(pos, system, species, q, e, s, 3, paired),
                lists.reference(pos, system, species, q, e, s, 3))
