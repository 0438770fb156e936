"""Ewald kernels at the edges of their tiles against the float64 oracle: atoms around the 32 of a chunk and
the 16 of a block, k vectors around the 256 and 512 of a tile, real space around 32 partners per pass and
with cells exactly twice the cutoff wide, systems many cells from the origin; and the fused integrator steps against
the separate ones.

Bars: those of float32 pair and phase arithmetic in this package: energies relative 1e-5 (reciprocal
1e-6 of the sum of the terms, which are positive), gradients RMS relative 1e-5."""

import numpy as np
import pytest
import torch

from oracle import ewald as oew
from oracle import lennard_jones as olj
from oracle import neighborlist as onl
from oracle import unitcell as ouc
from test_gpu_ewald import KE, cuda, offsets

pytestmark = pytest.mark.gpu


def _cells(rng, counts, low):
    lat = [ouc.lattice_from_lengths_angles(rng.uniform(low, low + 3, 3), rng.uniform(85, 95, 3)) for _ in counts]
    return lat, np.stack([ouc.tril_from_lattice(x) for x in lat])


@pytest.mark.parametrize("counts", [(1, 2), (31, 33), (32, 64, 7), (500, 3)])
@pytest.mark.parametrize("nk", [1, 255, 257, 511, 515])
def test_reciprocal_space_tiles(counts, nk):
    from kups_gb300.ewald import ewald_recip, ewald_recip_energy

    rng = np.random.default_rng(nk + len(counts))
    lat, tril = _cells(rng, counts, 9.0)
    pos = np.concatenate([rng.uniform(-0.5, 0.5, (n, 3)) @ x for n, x in zip(counts, lat)])
    q = rng.normal(size=len(pos))
    sysi = np.repeat(np.arange(len(counts)), counts)
    # half-space vectors of the half-box |n| <= 5, in random order (no run of n_z), some rows zero
    kn = np.stack([rng.permutation(oew.kvecs_cube(5))[:nk] for _ in counts])
    kn[:, ::7] = 0
    alpha = rng.uniform(0.25, 0.4, len(counts))
    e, g, dt, sk = oew.long_range(pos, q, sysi, tril, kn, alpha)
    off, mx = offsets(sysi, len(counts))
    args = (cuda(tril), cuda(kn, torch.int32), cuda(alpha))
    ge, gg, gdt, gsk, _ = (x.cpu().numpy() for x in ewald_recip(cuda(pos), cuda(q), off, mx, *args))
    np.testing.assert_allclose(gsk, sk, atol=2e-6 * np.abs(sk).max())
    np.testing.assert_allclose(ge, e, rtol=1e-5, atol=1e-12)
    np.testing.assert_allclose(ewald_recip_energy(*args, cuda(gsk)).cpu().numpy(), ge, rtol=1e-12, atol=1e-14)
    for s in range(len(counts)):
        d, r = (gg - g)[sysi == s], g[sysi == s]
        assert np.sqrt(np.mean(d**2)) <= 1e-5 * max(np.sqrt(np.mean(r**2)), 1e-3), s
    np.testing.assert_allclose(gdt, dt, rtol=1e-5, atol=1e-5 * np.abs(dt).max())


def _real(pos, q, sp, sysi, tril, sig, eps, rc, alpha):
    import ctypes as C

    from kups_gb300 import _lib
    from kups_gb300.ewald import TERM_EWALD_REAL, TERM_LJ
    from kups_gb300.neighborlist import new_status, read_status

    s = len(tril)
    off, mx = offsets(sysi, s)
    en, gr = torch.full((s,), 7.0, dtype=torch.float64, device="cuda"), torch.zeros((len(q), 3), dtype=torch.float64,
                                                                                   device="cuda")
    lib, st = _lib.load(), new_status()
    keep = [cuda(pos), cuda(q), cuda(sp, torch.int32), cuda(tril), cuda(sig), cuda(eps), cuda(rc), cuda(alpha)]
    ws = torch.empty(lib.kups_lj_ewald_real_forces_workspace_bytes(s, mx), dtype=torch.uint8, device="cuda")
    rcode = lib.kups_lj_ewald_real_forces_packed(
        keep[0].data_ptr(), keep[1].data_ptr(), keep[2].data_ptr(), off.data_ptr(), s, mx, keep[3].data_ptr(),
        keep[4].data_ptr(), keep[5].data_ptr(), len(sig), keep[6].data_ptr(), keep[7].data_ptr(), keep[6].data_ptr(),
        KE, TERM_LJ | TERM_EWALD_REAL, en.data_ptr(), gr.data_ptr(), ws.data_ptr(), ws.numel(), st.data_ptr(),
        C.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rcode == 0 and read_status(st).code == 0
    return en.cpu().numpy(), gr.cpu().numpy()


@pytest.mark.parametrize("counts", [(2, 15), (16, 17, 31), (33, 512), (1025, 40)])
@pytest.mark.parametrize("away", [0, 40])
@pytest.mark.parametrize("narrow", [False, True])
def test_real_space_tiles(counts, away, narrow):
    from kups_gb300.workloads import lattice_positions

    rng = np.random.default_rng(sum(counts))
    low = 1.9 * max(counts) ** (1 / 3) + 8.0
    if narrow:  # cubes exactly twice the cutoff wide: pairs at half the cell are at the cutoff
        rc = np.full(len(counts), np.ceil(low) / 2)
        lat = [np.eye(3) * 2 * r for r in rc]
        tril = np.stack([ouc.tril_from_lattice(x) for x in lat])
    else:
        lat, tril = _cells(rng, counts, low)
        rc = np.full(len(counts), 0.46 * low)
    pos = np.concatenate([(lattice_positions(rng, n, 1.0, 0.6 / low) - 0.5 + away * rng.integers(-1, 2, 3)) @ x
                          for n, x in zip(counts, lat)])  # the system `away` cells from the origin
    q = rng.normal(size=len(pos))
    sysi = np.repeat(np.arange(len(counts)), counts)
    sp = rng.integers(0, 2, len(q))
    sig, eps = olj.lorentz_berthelot([0.9, 1.2], [0.004, 0.006])
    alpha = rng.uniform(0.3, 0.4, len(counts))
    e, s = onl.neighbor_list(pos, sysi, tril, rc)
    el, gl, _ = olj.lj_from_edges(pos, sysi, sp, tril, sig, eps, rc, e, s)
    ee, ge, _ = oew.short_range_from_edges(pos, q, sysi, tril, alpha, rc, e, s)
    en, gr = _real(pos, q, sp, sysi, tril, sig, eps, rc, alpha)
    # the float32 sums of signed pair terms: relative to the terms' sizes
    size = np.zeros(len(counts))
    d = pos[e[:, 1]] - pos[e[:, 0]] + np.einsum("ea,eab->eb", s.reshape(-1, 3), np.stack(lat)[sysi[e[:, 0]]])
    r = np.linalg.norm(d, axis=1)
    np.add.at(size, sysi[e[:, 0]], 0.5 * KE * np.abs(q[e[:, 0]] * q[e[:, 1]]) / r)
    assert (np.abs(en - el - ee) <= 1e-5 * (size + np.abs(el))).all()
    for k in range(len(counts)):
        g = (gl + ge)[sysi == k]
        assert np.sqrt(np.mean((gr[sysi == k] - g) ** 2)) <= 1e-5 * max(np.sqrt(np.mean(g**2)), 1e-3), k


@pytest.mark.parametrize("n", [1, 31, 4001])
def test_fused_integrator_steps_match_the_separate_ones(n):
    from kups_gb300 import _lib
    from kups_gb300.neighborlist import _stream

    rng = np.random.default_rng(n)
    _, tril = _cells(rng, (1, 1), 9.0)
    sysi = cuda(np.sort(rng.integers(0, 2, n)), torch.int32)
    mk = lambda *shape: cuda(rng.normal(size=shape))
    mom, pos, ga, gb, mass = mk(n, 3), mk(n, 3) * 9, mk(n, 3), mk(n, 3), cuda(rng.uniform(1, 40, n))
    dt, tr, lib, st = cuda([0.1, 0.2]), cuda(tril), _lib.load(), _stream()
    m1, p1, m2, p2 = mom.clone(), pos.clone(), mom.clone(), pos.clone()
    lib.kups_md_kick(m1.data_ptr(), ga.data_ptr(), sysi.data_ptr(), dt.data_ptr(), 0.5, n, st)
    lib.kups_md_drift(p1.data_ptr(), m1.data_ptr(), mass.data_ptr(), sysi.data_ptr(), dt.data_ptr(), tr.data_ptr(),
                      0.7, n, st)
    assert lib.kups_md_kick_drift(m2.data_ptr(), ga.data_ptr(), p2.data_ptr(), mass.data_ptr(), sysi.data_ptr(),
                                  dt.data_ptr(), tr.data_ptr(), 0.5, 0.7, n, st) == 0
    torch.testing.assert_close(m2, m1, rtol=0, atol=0)
    torch.testing.assert_close(p2, p1, rtol=0, atol=0)
    e, grad, energy = [mk(2) for _ in range(3)], torch.empty_like(ga), torch.empty(2, dtype=torch.float64, device="cuda")
    assert lib.kups_md_sum_kick(m2.data_ptr(), grad.data_ptr(), ga.data_ptr(), gb.data_ptr(), sysi.data_ptr(),
                                dt.data_ptr(), 0.5, n, energy.data_ptr(), *(x.data_ptr() for x in e), 2, st) == 0
    lib.kups_md_kick(m1.data_ptr(), (ga + gb).data_ptr(), sysi.data_ptr(), dt.data_ptr(), 0.5, n, st)
    torch.testing.assert_close(grad, ga + gb, rtol=0, atol=0)
    torch.testing.assert_close(m2, m1, rtol=0, atol=0)
    torch.testing.assert_close(energy, e[0] + e[1] + e[2], rtol=0, atol=0)
