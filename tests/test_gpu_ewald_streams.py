"""The second stream of the LJ + Ewald classes: objects that have made one are copied and pickled as before,
and a call that fails on the host leaves no work of that stream unordered with the caller's."""

import copy
import pickle

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def salt(n=64, box=12.0, cutoff=5.0):
    """Rock salt with small displacements: (particles, cell, Ewald parameters, LJ tables, masses, momenta)."""
    from kups_gb300 import ewald

    t = lambda x, dt=torch.float64: torch.as_tensor(np.ascontiguousarray(x), dtype=dt).cuda()
    rng = np.random.default_rng(1)
    g = np.stack(np.meshgrid(*[np.arange(4)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n]
    kind = g.sum(1) % 2
    pos = (g + 0.5) * (box / 4) - box / 2 + rng.normal(scale=0.1, size=g.shape)
    prm = ewald.EwaldParameters(t([0.5]), t([cutoff]), t(ewald.kvecs_cube(3)[None], torch.int32))
    parts = ewald.EwaldParticles(t(pos), t(1.0 - 2.0 * kind), torch.zeros(n, dtype=torch.int32, device="cuda"),
                                 t(kind, torch.int32))
    lj = (t([[2.3, 3.3], [3.3, 4.4]]), t([[4e-3, 5e-3], [5e-3, 6e-3]]), t([cutoff]))
    return parts, t([[box, 0, box, 0, 0, box]]), prm, lj, t(np.full(n, 30.0)), t(rng.normal(size=(n, 3)))


@pytest.mark.parametrize("copied", [copy.deepcopy, lambda x: pickle.loads(pickle.dumps(x))])
def test_objects_with_a_second_stream_are_copied(copied):
    from kups_gb300 import ewald

    parts, tril, prm, lj, masses, momenta = salt()
    pot = ewald.LJEwaldPotential(prm, *lj)
    want = pot(parts, tril)
    got = copied(pot)(parts, tril)
    assert torch.allclose(got.total_energies, want.total_energies, rtol=1e-12, atol=0)
    sim = ewald.LJEwaldMD(parts, masses, tril, prm, 0.01, *lj)
    sim.start(momenta)
    twin = copied(sim)
    for s in (sim, twin):
        s.run(3)
        s.check()
    assert torch.allclose(sim.energy, twin.energy, rtol=1e-9, atol=0)


@pytest.mark.parametrize("what", ["potential", "simulation"])
def test_a_failing_call_waits_for_the_second_stream(monkeypatch, what):
    """The launch on the second stream raises after it has enqueued work; what the caller's stream does next
    comes after that work."""
    from kups_gb300 import ewald

    parts, tril, prm, lj, masses, momenta = salt()
    mark = torch.zeros(1, device="cuda")

    def late(*args, **kwargs):
        torch.cuda._sleep(100_000_000)  # about 50 ms
        mark.fill_(1)
        raise RuntimeError("a launch refused")

    if what == "potential":
        pot = ewald.LJEwaldPotential(prm, *lj)
        call = lambda: pot(parts, tril)
        call()
    else:
        sim = ewald.LJEwaldMD(parts, masses, tril, prm, 0.01, *lj)
        sim.start(momenta)
        assert sim.allpairs
        call = sim._forces
    torch.cuda.synchronize()
    monkeypatch.setattr(ewald, "ewald_recip", late)
    with pytest.raises(RuntimeError, match="a launch refused"):
        call()
    seen = mark.clone()
    assert float(seen) == 1.0
