"""Edge-list pair kernels where their run layout could go wrong: list lengths around a warp's reads,
shuffled lists (no two neighbours share a particle), padding rows in the middle, several systems in
one warp, self images, skewed cells and shifts beyond one; and the paired form against the directed
one.  Reference: the same sums in float64 numpy.  Tolerance 1e-10 of the largest component: at most
2e4 terms of float64 rounding (2e-12) with room for cancellation between terms."""

import numpy as np
import pytest
import torch
from scipy.special import erfc

from oracle import neighborlist as onl

pytestmark = pytest.mark.gpu
KE = 14.399645

CELLS = np.array([[10.0, 0, 10.0, 0, 0, 10.0], [10.0, 3.0, 9.0, -2.5, 2.0, 11.0], [5.0, 0, 5.5, 0, 0, 6.0]])


def lattice(t):
    return np.array([[t[0], 0, 0], [t[1], t[2], 0], [t[3], t[4], t[5]]])


def system_of(n, seed, cut=5.2):
    """n particles over three cells (the last has a self image inside the cutoff), their full list,
    two species and charges; some particles a lattice vector away, so that shifts reach 2."""
    rng = np.random.default_rng(seed)
    system = np.sort(rng.integers(0, 3, n))
    L = np.stack([lattice(t) for t in CELLS])
    f = rng.uniform(-0.5, 0.5, (n, 3)) + rng.integers(-1, 2, (n, 3)) * (rng.random((n, 1)) < 0.2)
    # a minimum distance keeps the LJ terms of a random table within a few orders of magnitude
    pos = np.einsum("na,nab->nb", f, L[system])
    e, s = onl.neighbor_list(pos, system, CELLS, np.full(3, cut))
    d = pos[e[:, 1]] - pos[e[:, 0]] + np.einsum("na,nab->nb", s, L[system[e[:, 0]]])
    far = (d * d).sum(1) > 1.0  # drop close pairs in both directions
    e, s = onl.sort_edges(e[far], s[far])
    return pos, system, rng.integers(0, 2, n), rng.normal(size=n), e.astype(np.int32), s.astype(np.int32)


SIG, EPS = np.array([[2.0, 2.3], [2.3, 2.6]]), np.array([[0.01, 0.02], [0.02, 0.03]])
RC, RCE, AL = np.array([4.5, 5.0, 5.1]), np.array([5.0, 4.0, 5.2]), np.array([0.3, 0.4, 0.5])


def reference(pos, system, species, q, e, s, terms):
    L = np.stack([lattice(t) for t in CELLS])
    i, j = e[:, 0], e[:, 1]
    si = system[i]
    d = pos[j] - pos[i] + np.einsum("na,nab->nb", s, L[si])
    r2 = (d * d).sum(1)
    r = np.sqrt(r2)
    u, f = np.zeros(len(e)), np.zeros(len(e))  # energy, dE/d(r^2)
    if terms & 1:
        on = r2 < RC[si] ** 2
        c6 = (SIG[species[i], species[j]] ** 2 / r2) ** 3
        ep = EPS[species[i], species[j]]
        u += on * 4 * ep * (c6 * c6 - c6)
        f += on * -12 * ep * c6 * (2 * c6 - 1) / r2
    if terms & 6:
        qq = KE * q[i] * q[j]
        if terms & 2:
            on, a = r < RCE[si], AL[si]
            u += on * qq * erfc(a * r) / r
            f += on * 0.5 * qq * (-erfc(a * r) / r2 - 2 * a / np.sqrt(np.pi) * np.exp(-a * a * r2) / r) / r
        if terms & 4:
            u -= qq / r
            f += 0.5 * qq / (r2 * r)
    g = f[:, None] * d  # half of each directed edge's gradient
    energy = 0.5 * np.bincount(si, u, minlength=3)
    grad = np.zeros_like(pos)
    np.add.at(grad, j, g)
    np.add.at(grad, i, -g)
    low = [(0, 0), (1, 0), (1, 1), (2, 0), (2, 1), (2, 2)]
    gt = np.stack([np.bincount(si, s[:, a] * g[:, b], minlength=3) for a, b in low], 1)
    return energy, grad, gt


def t(x, dt=torch.float64):
    return torch.as_tensor(np.ascontiguousarray(x), dtype=dt).cuda()


def lj(pos, system, species, e, s, fp32, paired):
    from kups_gb300 import potential

    out = potential.lj_from_edges(t(pos), t(system, torch.int32), t(species, torch.int32), t(CELLS), t(SIG), t(EPS),
                                  t(RC), t(e, torch.int32), t(s, torch.int32), len(e), fp32, paired)
    return [x.cpu().numpy() for x in (out.total_energies, out.gradients.positions, out.gradients.unitcell)]


def pair(pos, system, species, q, e, s, terms, paired):
    from kups_gb300 import ewald, units

    out = ewald.pair_edges(t(pos), t(system, torch.int32), t(species, torch.int32),
                           t(q * np.sqrt(KE / units.TO_STANDARD_UNITS)), t(CELLS), t(e, torch.int32),
                           t(s, torch.int32), len(e), terms, t(SIG), t(EPS), t(RC), t(AL), t(RCE), paired=paired)
    return [x.cpu().numpy() for x in out]


def close(got, want, tol=1e-10):
    for g, w in zip(got, want):
        assert np.abs(g - w).max() <= tol * max(np.abs(w).max(), 1e-300)


@pytest.mark.parametrize("n", [2, 5, 17, 90])
@pytest.mark.parametrize("paired", [False, True])
def test_full_lists(n, paired):
    pos, system, species, q, e, s = system_of(n, n)
    for terms in (1, 2, 3, 6):
        close(pair(pos, system, species, q, e, s, terms, paired), reference(pos, system, species, q, e, s, terms))
    want = reference(pos, system, species, q, e, s, 1)
    close(lj(pos, system, species, e, s, False, paired), want)
    close(lj(pos, system, species, e, s, True, paired), want, 2e-5)  # float32 pairs


@pytest.mark.parametrize("length", [1, 31, 32, 127, 128, 129, 255, 257, 511, 512, 1025])
def test_shuffled_lists_with_padding_rows(length):
    pos, system, species, q, e, s = system_of(90, 3)
    rng = np.random.default_rng(length)
    pick = rng.permutation(len(e))[:length]
    e, s = e[pick].copy(), s[pick].copy()
    want_e, want_s = e.copy(), s.copy()
    hole = rng.random(length) < 0.2
    e[hole] = len(pos)  # the index that pads a list
    want = reference(pos, system, species, q, want_e[~hole], want_s[~hole], 3)
    close(pair(pos, system, species, q, e, s, 3, False), want)
    close(lj(pos, system, species, e, s, False, False), reference(pos, system, species, q, want_e[~hole], want_s[~hole], 1))


def test_paired_and_directed_agree_to_rounding_on_a_long_list():
    from kups_gb300 import potential, workloads

    w = workloads.batched_uneven_lj(n_systems=40, n_min=64, n_max=900, seed=5)
    prm = potential.LennardJonesParameters(("Ar",), t(w.sigma), t(w.epsilon), t([w.cutoff]))
    st = potential.LJState(potential.LJParticles(t(w.positions), t(w.species, torch.int32), t(w.system, torch.int32)),
                           t(w.tril), prm)
    for fp32 in (False, True):
        out = potential.LennardJonesPotential(pair_fp32=fp32)(st)  # the paired form

        class Own(type(potential.LennardJonesPotential().neighborlist)):
            """A neighbour list of the caller's: nothing is known of its edges."""

        ref = potential.LennardJonesPotential(Own(64), pair_fp32=fp32)(st)
        close([x.cpu().numpy() for x in (out.total_energies, out.gradients.positions, out.gradients.unitcell)],
              [x.cpu().numpy() for x in (ref.total_energies, ref.gradients.positions, ref.gradients.unitcell)], 1e-12)
