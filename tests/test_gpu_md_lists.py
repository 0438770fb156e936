"""Verlet lists of the fused MD kernel at the edges of their 16-atom chunks and 32-candidate batches:
systems of 1 to 2048 atoms in one batch, sparse to dense, with one and two image layers; forces and
energies against the float64 oracle at the same float32 positions.

Bars: those of float32 pair arithmetic in this package, force RMS relative error 1e-5 and energy relative
error 1e-5 (a missing or doubled neighbour at the distances drawn is above 1e-4 of either)."""

import numpy as np
import pytest
import torch

from oracle import md as omd
from test_gpu_core import ENERGY_REL_TOL, FORCE_RMS_TOL, md_state

pytestmark = pytest.mark.gpu

SIGMA, EPS = 3.4, 0.0103


def _batch(counts, density, seed):
    from kups_gb300 import workloads

    rng = np.random.default_rng(seed)
    box = np.maximum((np.array(counts) / density) ** (1 / 3) * SIGMA, 2.0 * SIGMA)
    pos = np.concatenate([workloads.lattice_positions(rng, n, float(b), 0.85 * SIGMA) for n, b in zip(counts, box)])
    system = np.repeat(np.arange(len(counts), dtype=np.int32), counts)
    tril = np.zeros((len(counts), 6))
    tril[:, 0] = tril[:, 2] = tril[:, 5] = box
    s = len(counts)
    return workloads.MDWorkload(
        pos.astype(np.float32).astype(np.float64), np.zeros((len(pos), 3)), np.full(len(pos), 40.0),
        np.zeros(len(pos), np.int32), system, tril.astype(np.float32).astype(np.float64), np.full(s, 100.0),
        np.full(s, 0.1), np.full(s, 0.01), np.array([[SIGMA]]), np.array([[EPS]]), 2.2 * SIGMA, 0.3 * SIGMA)


@pytest.mark.parametrize("counts,density", [([1, 2, 15, 16, 17, 31, 32, 33, 47, 48, 49], 0.5),
                                            ([63, 64, 65, 200, 511, 513, 1023], 0.8), ([2048, 1000], 0.05),
                                            ([2048, 2047], 0.8)])
@pytest.mark.parametrize("lanes", [0, 1, 16])
def test_lists_match_the_oracle(counts, density, lanes):
    from kups_gb300 import md

    w = _batch(counts, density, len(counts))
    packed = md.pack(md_state(w))
    prop = md.FusedLennardJonesMD("velocity_verlet", min_lanes_per_atom=lanes)
    prop.run_packed(packed, 0)
    perm = packed.perm.cpu().numpy().astype(int)
    got = np.empty((len(perm), 3))
    got[perm] = packed.frc4.cpu().numpy()[:, :3]
    energy, force, _ = omd.lj_forces(w.positions, w.system, w.species, w.tril, w.sigma, w.epsilon,
                                     np.full(len(counts), w.cutoff))
    for s, n in enumerate(counts):
        f = force[w.system == s]
        rms = np.sqrt(np.mean(f**2))
        assert np.sqrt(np.mean((got[w.system == s] - f) ** 2)) <= FORCE_RMS_TOL * max(rms, 1e-3), (s, n)
        assert abs(packed.energy.cpu().numpy()[s] - energy[s]) <= ENERGY_REL_TOL * max(abs(energy[s]), 1e-3), (s, n)
