"""Bonded kernels where their launch and row table could go wrong: more parameter rows than the
block's table holds, edge counts around a warp's share, several edges per thread (a tiled edge set
against its multiple of the oracle's sums), non-integer and unlisted dihedral periodicities, and
straight dihedrals.  Tolerances as the kernels' main tests: energies 1e-10 (float64) and 2e-5
(float32), gradients 1e-6 and 2e-4 of the largest component.  Energies against the oracle, gradients
against automatic differentiation of the same formulas (central differences leave 1e-10 of the
energy, which a single far edge's gradient can be as small as)."""

import math

import numpy as np
import pytest
import torch

from oracle import bonded as ob
from test_gpu_bonded import params_object, random_case

pytestmark = pytest.mark.gpu


def energies(kind, v, p):
    """Per-edge energies of difference vectors v (torch, [E, 3] each) with parameter rows p."""
    dot, cross, norm = (lambda a, b: (a * b).sum(-1)), torch.linalg.cross, (lambda a: a.norm(dim=-1))
    if kind == "harmonic_bond":
        return p[1] * (norm(v[0]) - p[0]) ** 2
    if kind == "morse_bond":
        return p[1] * (1 - torch.exp(-p[2] * (norm(v[0]) - p[0]))) ** 2
    if kind in ("harmonic_angle", "cosine_angle"):
        c = (dot(v[0], v[1]) / (norm(v[0]) * norm(v[1]))).clamp(-1, 1)
        if kind == "harmonic_angle":
            return p[1] * (torch.rad2deg(torch.acos(c)) - p[0]) ** 2
        c2 = 1 / (4 * (torch.sin(p[0]) ** 2).clamp(min=1e-10))
        bent = c2 * (2 * torch.cos(p[0]) ** 2 + 1) - 4 * c2 * torch.cos(p[0]) * c + c2 * (2 * c * c - 1)
        return p[1] * torch.where((p[0] - math.pi).abs() < p[2], 1 + c, bent)
    if kind == "dihedral":
        b1, b2, b3 = v[0], v[1] - v[0], v[2] - v[1]
        m, n = cross(b1, b2), cross(b2, b3)
        phi = torch.atan2(dot(cross(m, n), b2) / (norm(b2) + 1e-10), dot(m, n))
        return 0.5 * p[0] * (1 - torch.cos(p[1] * p[2]) * torch.cos(p[1] * phi))
    n = cross(v[1], v[2])
    w = torch.asin((dot(v[0], n) / (norm(n) + 1e-10) / (norm(v[0]) + 1e-10)).clamp(-1, 1))
    planar = p[0].abs() < 1e-6
    s2 = torch.sin(p[0]) ** 2
    c2 = torch.where(planar, 0.0, 1 / (4 * torch.where(s2 > 1e-10, s2, 1.0)))
    c1 = torch.where(planar, -1.0, -4 * c2 * torch.cos(p[0]))
    c0 = torch.where(planar, 1.0, c2 * (2 * torch.cos(p[0]) ** 2 + 1))
    k = torch.where(planar, p[1], p[1] / (c0 + c1 + c2).clamp(min=1e-10))
    return k * (c0 + c1 * torch.cos(w) + c2 * torch.cos(2 * w))


def gradients(kind, pos, system, species, tril, table, T, edges, shifts):
    f = lambda a: torch.as_tensor(np.asarray(a, float))
    x, cell = f(pos).requires_grad_(True), f(tril).requires_grad_(True)
    L = torch.zeros(len(tril), 3, 3, dtype=torch.float64)
    low = [(0, 0), (1, 0), (1, 1), (2, 0), (2, 1), (2, 2)]
    L = L.index_put((torch.arange(len(tril))[:, None], torch.tensor([a for a, _ in low])[None],
                     torch.tensor([b for _, b in low])[None]), cell)
    si = torch.as_tensor(system[edges[:, 0]])
    v = [x[edges[:, m + 1]] - x[edges[:, 0]] + torch.einsum("na,nab->nb", f(shifts[:, m]), L[si])
         for m in range(edges.shape[1] - 1)]
    row = np.ravel_multi_index(species[edges].T, (T,) * edges.shape[1])
    e = energies(kind, v, f(table)[row].T)
    return [g.numpy() for g in torch.autograd.grad(e.sum(), (x, cell))]


def compare(kind, case, times=1, fp32=False):
    from kups_gb300 import bonded

    pos, system, species, tril, edges, shifts, table, T, order = case
    term = bonded.BondedTerm(params_object(kind, table, T, order), np.tile(edges, (times, 1)),
                             np.tile(shifts, (times, 1, 1)), fp32=fp32)
    got = [x.cpu().numpy() for x in bonded.evaluate([term], pos, system, species, tril)]
    args = (kind, pos, system, species, tril, table, T, edges, shifts)
    want = [times * x for x in [ob.bonded(*args)[0]] + gradients(*args)]
    tol = (2e-5, 2e-4, 2e-4) if fp32 else (1e-10, 1e-6, 1e-6)
    for g, w, t in zip(got, want, tol):
        np.testing.assert_allclose(g, w, rtol=0, atol=t * np.abs(w).max())


@pytest.mark.parametrize("kind", list(ob.KINDS))
@pytest.mark.parametrize("fp32", [False, True])
@pytest.mark.parametrize("edges,types", [(1, 1), (31, 2), (33, 5), (129, 7)])
def test_rows_and_edge_counts(kind, fp32, edges, types):
    compare(kind, random_case(kind, np.random.default_rng(edges), E=edges, T=types), fp32=fp32)


@pytest.mark.parametrize("kind", list(ob.KINDS))
@pytest.mark.parametrize("fp32", [False, True])
def test_several_edges_per_thread(kind, fp32):
    compare(kind, random_case(kind, np.random.default_rng(3)), times=1201, fp32=fp32)


@pytest.mark.parametrize("periodicity", [0.0, 0.5, 2.5, -3.0, 1.0, 2.0, 3.0, 4.0, 5.0, 6.0, 7.0])
def test_dihedral_periodicities(periodicity):
    case = list(random_case("dihedral", np.random.default_rng(11)))
    case[6] = case[6].copy()
    case[6][:, 1] = periodicity
    compare("dihedral", case)


def test_straight_dihedral_has_no_gradient_and_the_energy_of_phi_zero():
    from kups_gb300 import bonded

    pos = np.array([[0.0, 0, 0], [1.0, 0, 0], [2.0, 0, 0], [3.0, 0.5, 0]])
    term = bonded.BondedTerm(bonded.DihedralParameters(("A",), np.full((1,) * 4, 2.0), np.full((1,) * 4, 3.0),
                                                       np.full((1,) * 4, np.pi)), np.arange(4)[None])
    e, g, gt = bonded.evaluate([term], pos, np.zeros(4, int), np.zeros(4, int), np.array([[20.0, 0, 20.0, 0, 0, 20.0]]))
    assert abs(float(e[0]) - 2.0) < 1e-12 and float(g.abs().max()) == 0.0 and float(gt.abs().max()) == 0.0
