"""The work a user of kups_gb300 has it do, as measurable cases.

Each case is one call a program makes through the package's public classes: fused molecular
dynamics, GCMC, LJ + Ewald dynamics, potential evaluations, neighbour lists, bonded terms,
virial observables, and training / evaluation of the learned insertion proposal.  ``listed()``
names twelve of them, ``draw(rng)`` gives more of the same ranges; ``prepare`` builds what the
program holds before the call, ``run`` makes it, ``work`` counts what it cannot do without and
``exact`` gives its results from float64 torch / numpy alone.
"""

import math

import numpy as np
import torch

from kups_gb300 import bonded, ewald, gcmc, md, mlp, observables, potential, units, workloads
from kups_gb300.neighborlist import CellListNeighborList, NeighborListPoints

DEV = "cuda"
F64 = torch.float64
KE = units.TO_STANDARD_UNITS
TRIL = ((0, 0), (1, 0), (1, 1), (2, 0), (2, 1), (2, 2))


def listed():
    return [
        # one small system in a production loop: 864 argon atoms, NVT, 20 steps a call
        {"name": "argon_nvt_864", "kind": "md", "systems": 1, "n_min": 864, "n_max": 864, "steps": 20,
         "integrator": "baoab"},
        # a batch of many uneven systems advanced together (the package's headline use)
        {"name": "md_uneven_1024", "kind": "md", "systems": 1024, "n_min": 64, "n_max": 2048, "steps": 20,
         "integrator": "baoab"},
        # adsorption isotherm: 1024 replicas of a CO2-loaded rigid host, 20 Monte Carlo steps a launch
        {"name": "gcmc_co2_1024", "kind": "gcmc", "replicas": 1024, "steps": 20},
        # molten salt dynamics with Ewald electrostatics, steps replayed from the propagator's graph
        {"name": "melt_nve_4000", "kind": "melt_md", "ions": 4000, "cutoff": 12.0, "kmax": 8, "steps": 10},
        # a single energy / force / stress evaluation of a small system, float64 pairs (latency)
        {"name": "lj_argon_864_f64", "kind": "lj", "systems": 1, "n_min": 864, "n_max": 864, "fp32": False},
        # the same over a batch of uneven systems with the default float32 pairs
        {"name": "lj_uneven_256", "kind": "lj", "systems": 256, "n_min": 64, "n_max": 2048, "fp32": True},
        # full LJ + Ewald energies, forces and cell gradients of the salt (float64 reference path)
        {"name": "lj_ewald_4000", "kind": "lj_ewald", "ions": 4000, "cutoff": 12.0, "kmax": 8},
        # neighbour lists of triclinic molecular liquids with intramolecular exclusions
        {"name": "neighbors_molecules_61k", "kind": "neighbors", "systems": 37, "molecules": 550, "cutoff": 6.0},
        # bonded energies, forces and cell gradients of many chain molecules, float64
        {"name": "bonded_chains_2048", "kind": "bonded", "chains": 2048, "beads": 256, "fp32": False},
        # one optimisation step of the learned insertion proposal at its default batch
        {"name": "proposal_train_16384", "kind": "train", "batch": 16384},
        # proposal log densities of a ragged set of points
        {"name": "proposal_forward_300007", "kind": "forward", "points": 300007},
        # stresses, kinetic energy and pressure of sampled configurations of a molecular liquid
        {"name": "virial_molecules_512k", "kind": "virial", "systems": 64, "molecules": 2667},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["md", "md", "gcmc", "melt_md", "lj", "lj", "lj_ewald", "neighbors", "bonded", "bonded", "train",
                       "forward", "virial"])
    c = {"kind": kind}
    if kind == "md":
        lo = _log(rng, 64, 900)
        c.update(systems=_log(rng, 1, 1024), n_min=lo, n_max=min(2048, lo + rng.randrange(0, 1200)),
                 steps=rng.randrange(5, 21), integrator=rng.choice(["baoab", "baoab", "velocity_verlet", "csvr", "csvr_npt"]))
    elif kind == "gcmc":
        c.update(replicas=_log(rng, 16, 1024), steps=rng.randrange(5, 21))
    elif kind in ("melt_md", "lj_ewald"):
        c.update(ions=2 * _log(rng, 150, 2000), cutoff=rng.choice([8.0, 9.5, 12.0]), kmax=rng.randrange(4, 9))
        if kind == "melt_md":
            c.update(steps=rng.randrange(2, 11))
    elif kind == "lj":
        lo = _log(rng, 64, 1200)
        c.update(systems=_log(rng, 1, 256), n_min=lo, n_max=min(2048, lo + rng.randrange(0, 1200)),
                 fp32=rng.random() < 0.6)
    elif kind == "neighbors":
        s = _log(rng, 1, 64)
        c.update(systems=s, molecules=_log(rng, 40, 20000 // s + 40), cutoff=round(rng.uniform(3.0, 6.0), 2))
    elif kind == "bonded":
        c.update(chains=_log(rng, 16, 2048), beads=_log(rng, 8, 256), fp32=rng.random() < 0.5)
    elif kind == "train":
        c.update(batch=2 * _log(rng, 512, 8192))
    elif kind == "forward":
        c.update(points=_log(rng, 1000, 300007))
    else:
        s = _log(rng, 1, 64)
        c.update(systems=s, molecules=_log(rng, 50, 170000 // s))
    return c


# ----------------------------------------------------------------------------- inputs
def _t(x, dtype=F64):
    return torch.as_tensor(np.ascontiguousarray(x), dtype=dtype, device=DEV)


def _liquid(c, seed):
    """Argon liquids: one 864-atom fcc crystal at 94.4 K, or uneven batches at 0.7-0.9 reduced density."""
    if c["systems"] == 1 and c["n_min"] == c["n_max"] == 864:
        w = workloads.argon_fcc(seed=seed)
        w.positions += np.random.default_rng(seed + 1).normal(scale=0.2, size=w.positions.shape)  # thermal displacements
        w.positions -= w.tril[0, 0] * np.floor(w.positions / w.tril[0, 0] + 0.5)
        return w
    rng = np.random.default_rng(seed)
    s, sig = c["systems"], workloads.ARGON_SIGMA
    counts = np.random.default_rng(s).permutation(np.linspace(c["n_min"], c["n_max"], s).round().astype(int))
    box = (counts / rng.uniform(0.7, 0.9, s)) ** (1 / 3) * sig
    pos = np.concatenate([workloads.lattice_positions(rng, int(n), float(b), 0.9 * sig) for n, b in zip(counts, box)])
    system = np.repeat(np.arange(s, dtype=np.int32), counts)
    temp, mass = rng.uniform(80.0, 140.0, s), np.full(len(pos), workloads.ARGON_MASS)
    mom = rng.standard_normal((len(pos), 3)) * np.sqrt(mass * temp[system] * units.BOLTZMANN_CONSTANT)[:, None]
    tril = np.zeros((s, 6))
    tril[:, 0] = tril[:, 2] = tril[:, 5] = box
    return workloads.MDWorkload(pos, mom, mass, np.zeros(len(pos), np.int32), system, tril, temp,
                                np.full(s, 2.0 * units.FEMTO_SECOND), np.full(s, 1e-3 / units.FEMTO_SECOND),
                                np.array([[sig]]), np.array([[workloads.ARGON_EPS]]), 2.5 * sig, 0.3 * sig)


def _salt(c, seed):
    """Molten salt at the density of 4000 ions in a 40 A cube: a rock-salt arrangement with random
    vacancies and displacements, Maxwell-Boltzmann momenta at 1200 K."""
    n = c["ions"]
    box = 40.0 * (n / 4000.0) ** (1 / 3)
    w = workloads.ionic_melt(n_ions=n, box=box, cutoff=c["cutoff"], kmax=c["kmax"], seed=seed)
    rng = np.random.default_rng(seed + 7)
    side = 2 * math.ceil(n ** (1 / 3) / 2)
    g = np.stack(np.meshgrid(*[np.arange(side)] * 3, indexing="ij"), -1).reshape(-1, 3)
    even = g.sum(1) % 2 == 0
    ion = np.empty((n, 3))
    for sp, sites in ((0, g[even]), (1, g[~even])):
        m = int((w.species == sp).sum())
        ion[w.species == sp] = sites[rng.choice(len(sites), m, replace=False)]
    ion = (ion + 0.5) * (box / side) - box / 2 + rng.normal(scale=0.1, size=(n, 3))
    w.positions = ion - box * np.floor(ion / box + 0.5)
    return w


def _co2(c, seed):
    """CO2 replicas with their host's channels filled as at the isotherm's plateau: molecules along
    the channel axes on displaced sites, 80 to 125 in each replica."""
    st = workloads.gcmc_co2_framework(n_replicas=c["replicas"], seed=seed)
    rng = np.random.default_rng(seed + 5)
    t = st.tril[0]
    L = np.array([[t[0], 0, 0], [t[1], t[2], 0], [t[3], t[4], t[5]]])
    ring = [(0.0, 0.0)] + [(3.2 * math.cos(a), 3.2 * math.sin(a)) for a in np.arange(6) * math.pi / 3]
    sites = np.array([np.array([i / 2, j / 2, 0]) @ L + [x, y, 5.0 * (k + 0.5)]
                      for i in range(2) for j in range(2) for x, y in ring for k in range(5)])
    motif = st.motif_positions[:, [1, 2, 0]]  # the molecule's axis along the channel
    guests = []
    for _ in range(c["replicas"]):
        m = int(rng.integers(80, 126))
        p = sites[rng.choice(len(sites), m, replace=False)] + rng.normal(scale=0.12, size=(m, 3))
        f = (p[:, None, :] + motif[None]).reshape(-1, 3) @ np.linalg.inv(L)
        guests.append((f - np.floor(f + 0.5)) @ L)
    mc = gcmc.GCMC(st, seed=seed)
    mc.set_guests(guests)
    return mc


def _molecules(systems, molecules, density, seed):
    """Three-atom molecules at random places of triclinic cells, wrapped atom by atom."""
    rng = np.random.default_rng(seed)
    n = systems * molecules * 3
    a = (molecules * 3 / density) ** (1 / 3)
    tril = np.tile(a * np.array([1.0, 0.05, 0.98, -0.08, 0.03, 1.02]), (systems, 1))
    L = _lattice(tril)
    sysi = np.repeat(np.arange(systems), molecules * 3)
    com = np.repeat(rng.uniform(-0.5, 0.5, (systems * molecules, 3)), 3, axis=0)
    pos = np.einsum("na,nab->nb", com, L[sysi]) + rng.normal(scale=0.6, size=(n, 3))
    f = np.einsum("na,nab->nb", pos, np.linalg.inv(L)[sysi])
    return np.einsum("na,nab->nb", f - np.floor(f + 0.5), L[sysi]), sysi, np.arange(n) // 3, tril, rng


def _lattice(tril):
    L = np.zeros((len(tril), 3, 3))
    for k, (a, b) in enumerate(TRIL):
        L[:, a, b] = np.asarray(tril)[:, k]
    return L


def _chains(c, seed):
    """Random-walk chains of 1.5 A steps, two alternating bead species, in 40 A cubes; the edges
    carry the image shifts of chains stored wrapped."""
    rng = np.random.default_rng(seed)
    s, n = c["chains"], c["beads"]
    steps = rng.normal(size=(s, n, 3))
    steps *= rng.normal(1.5, 0.03, (s, n, 1)) / np.linalg.norm(steps, axis=-1, keepdims=True)
    walk = np.cumsum(steps, axis=1) + rng.uniform(0, 40, (s, 1, 3))
    image = np.floor(walk / 40.0 + 0.5).astype(np.int64)
    pos = (walk - 40.0 * image).reshape(-1, 3)
    image = image.reshape(-1, 3)
    base = (np.arange(s) * n)[:, None]

    def edges(offs, lo, hi):
        e = ((base + np.arange(lo, hi)[None])[..., None] + np.asarray(offs)).reshape(-1, len(offs))
        return e, (image[e[:, 1:]] - image[e[:, :1]]).astype(np.int32)

    var = lambda order, x: x * (1.0 + 0.1 * np.sin(np.arange(2 ** order).reshape((2,) * order)))
    return {
        "pos": pos, "system": np.repeat(np.arange(s), n), "species": (np.arange(s * n) % 2).astype(np.int32),
        "tril": np.tile([40.0, 0, 40.0, 0, 0, 40.0], (s, 1)),
        "bond": edges([0, 1], 0, n - 1), "angle": edges([0, -1, 1], 1, n - 1),
        "dihedral": edges([0, 1, 2, 3], 0, n - 3), "inversion": edges([0, -1, 1, 2], 1, n - 2),
        "x0": var(2, 1.5), "kb": var(2, 2.0), "theta0": var(3, 109.5), "ka": var(3, 0.01),
        "V": var(4, 0.1), "per": np.full((2,) * 4, 3.0), "phi0": np.full((2,) * 4, np.pi),
        "omega0": np.zeros((2,) * 4), "ki": var(4, 0.05),
    }


def _network(c, seed):
    """A proposal in the middle of its training: initial weights of the seed, nonzero biases, Adam moments."""
    net = mlp.LearnedInsertionProposal(seed=seed)
    g = torch.Generator(device=DEV).manual_seed(seed)
    rnd = lambda: torch.randn(mlp.N_PARAMS, generator=g, device=DEV)
    net.m.copy_(1e-4 * rnd())
    net.v.copy_((1e-3 * rnd()) ** 2 + 1e-6)
    net.t = 200
    return net, g


# ----------------------------------------------------------------------------- prepare and run
def prepare(case, seed):
    k = case["kind"]
    if k == "md":
        w = _liquid(case, seed)
        prm = potential.LennardJonesParameters(("Ar",), _t(w.sigma), _t(w.epsilon), _t([w.cutoff]))
        sy = md.MDSystems(_t(w.tril), _t(w.time_step), _t(w.temperature), _t(w.friction))
        if case["integrator"].startswith("csvr"):
            ones = torch.ones(w.n_systems, dtype=F64, device=DEV)
            sy.thermostat_time_constant = 100.0 * units.FEMTO_SECOND * ones
            sy.target_pressure = units.BAR * ones
            sy.pressure_coupling_time = 1000.0 * units.FEMTO_SECOND * ones
            sy.compressibility = 1e-4 / units.BAR * ones
            sy.minimum_scale_factor = 0.99 * ones
        state = md.MDState(md.MDParticles(_t(w.positions), _t(w.momenta), _t(w.masses), _t(w.species, torch.int32),
                                          _t(w.system, torch.int32)), sy, prm, skin=w.skin)
        return {"kind": k, "prop": md.FusedLennardJonesMD(case["integrator"], case["steps"]), "state": state, "key": seed}
    if k == "gcmc":
        return {"kind": k, "mc": _co2(case, seed), "steps": case["steps"]}
    if k in ("melt_md", "lj_ewald"):
        w = _salt(case, seed)
        prm = ewald.EwaldParameters(_t([w.alpha]), _t([w.cutoff]), _t(w.kvec_n, torch.int32))
        parts = ewald.EwaldParticles(_t(w.positions), _t(w.charges), torch.zeros(case["ions"], dtype=torch.int32, device=DEV),
                                     _t(w.species, torch.int32))
        if k == "lj_ewald":
            pot = ewald.LJEwaldPotential(prm, _t(w.sigma), _t(w.epsilon), _t([w.cutoff]))
            return {"kind": k, "pot": pot, "particles": parts, "tril": _t(w.tril)}
        sim = ewald.LJEwaldMD(parts, _t(w.masses), _t(w.tril), prm, w.time_step, _t(w.sigma), _t(w.epsilon),
                              _t([w.cutoff]))
        sim.start(_t(w.momenta))
        return {"kind": k, "sim": sim, "steps": case["steps"]}
    if k == "lj":
        w = _liquid(case, seed)
        state = potential.LJState(potential.LJParticles(_t(w.positions), _t(w.species, torch.int32),
                                                        _t(w.system, torch.int32)), _t(w.tril),
                                  potential.LennardJonesParameters(("Ar",), _t(w.sigma), _t(w.epsilon), _t([w.cutoff])))
        return {"kind": k, "pot": potential.make_lennard_jones_potential(pair_fp32=case["fp32"]), "state": state}
    if k == "neighbors":
        pos, sysi, mol, tril, _ = _molecules(case["systems"], case["molecules"], 0.1, seed)
        pts = NeighborListPoints(_t(pos), _t(sysi, torch.int32), None, _t(mol, torch.int32))
        return {"kind": k, "nl": CellListNeighborList(128), "points": pts, "tril": _t(tril),
                "cutoffs": torch.full((case["systems"],), case["cutoff"], dtype=F64, device=DEV)}
    if k == "bonded":
        d = _chains(case, seed)
        lab = ("A", "B")
        prm = {"bond": bonded.HarmonicBondParameters(lab, d["x0"], d["kb"]),
               "angle": bonded.HarmonicAngleParameters(lab, d["theta0"], d["ka"]),
               "dihedral": bonded.DihedralParameters(lab, d["V"], d["per"], d["phi0"]),
               "inversion": bonded.InversionParameters(lab, d["omega0"], d["ki"])}
        terms = [bonded.BondedTerm(p, *d[name], fp32=case["fp32"]) for name, p in prm.items()]
        return {"kind": k, "terms": terms, "args": (_t(d["pos"]), _t(d["system"], torch.int32),
                                                    _t(d["species"], torch.int32), _t(d["tril"]))}
    if k == "train":
        net, g = _network(case, seed)
        b = case["batch"]
        data = 0.5 + 0.1 * torch.randn((b // 2, 3), generator=g, device=DEV, dtype=F64)  # a pore around the cell's centre
        x = torch.cat([data - torch.floor(data), torch.rand((b // 2, 3), generator=g, device=DEV, dtype=F64)])
        y = torch.cat([torch.ones(b // 2, device=DEV), torch.zeros(b // 2, device=DEV)])
        return {"kind": k, "net": net, "x": x, "y": y, "loss": torch.zeros(1, device=DEV)}
    if k == "forward":
        net, g = _network(case, seed)
        return {"kind": k, "net": net, "x": torch.rand((case["points"], 3), generator=g, device=DEV, dtype=F64)}
    if k == "virial":
        pos, sysi, mol, tril, rng = _molecules(case["systems"], case["molecules"], 0.1, seed)
        n = len(pos)
        return {"kind": k, "args": (_t(pos), _t(rng.normal(size=(n, 3))), _t(sysi, torch.int32), _t(tril),
                                    _t(rng.normal(size=(case["systems"], 6)))),
                "more": dict(group=_t(mol, torch.int32), n_groups=case["systems"] * case["molecules"],
                             momenta=_t(rng.normal(size=(n, 3))), masses=_t(rng.uniform(1, 16, n)), molecular=True)}
    raise ValueError(k)


def run(s):
    k = s["kind"]
    if k == "md":  # the simulation loop's body: the returned state is the next call's input
        s["state"] = out = s["prop"](s["key"], s["state"])
        p, y = out.particles, out.systems
        res = {"positions": p.positions, "momenta": p.momenta, "forces": p.forces, "energy": y.potential_energy,
               "kinetic": y.kinetic_energy, "cell_gradient": y.unitcell_gradients, "pressure": y.pressure}
        if s["prop"].integrator == "csvr_npt":
            res["tril"] = y.tril
        return res
    if k == "gcmc":
        mc = s["mc"](None, s["steps"])
        return {"guest": mc.guest, "n_mol": mc.n_mol, "structure_factor": mc.sk, "energy": mc.energy, "width": mc.width,
                "history": mc.history, "attempted": mc.attempted, "accepted": mc.accepted, "sums": mc.obs}
    if k == "melt_md":
        sim = s["sim"]
        sim.run(s["steps"])
        return {"positions": sim.p.positions, "momenta": sim.mom, "gradient": sim.grad, "energy": sim.energy}
    if k == "lj":
        out = s["pot"](s["state"])
        return {"energy": out.total_energies, "gradient": out.gradients.positions, "cell_gradient": out.gradients.unitcell}
    if k == "lj_ewald":
        out = s["pot"](s["particles"], s["tril"])
        return {"energy": out.total_energies, "gradient": out.gradients.positions, "cell_gradient": out.gradients.unitcell,
                "structure_factor": out.cache.structure_factor}
    if k == "neighbors":
        e = s["nl"](s["points"], None, s["tril"], s["cutoffs"])
        return {"edges": e.indices, "shifts": e.shifts, "count": e.n_edges}
    if k == "bonded":
        return dict(zip(("energy", "gradient", "cell_gradient"), bonded.evaluate(s["terms"], *s["args"])))
    if k == "train":
        net = s["net"]
        s["loss"].zero_()
        net.backward(s["x"], s["y"], s["loss"])
        net.adam(1e-3)
        return {"param": net.param, "moment1": net.m, "moment2": net.v, "loss": s["loss"]}
    if k == "forward":
        return s["net"].forward(s["x"])
    return observables.virial_observables(*s["args"], **s["more"])


def work(case):
    """Inputs read once, outputs written once, and the arithmetic of the pairs inside the cutoffs
    (or edges, k vectors, matrix products) each counted once."""
    k = case["kind"]
    if k in ("md", "lj"):
        n = case["systems"] * (case["n_min"] + case["n_max"]) / 2
        pairs = n * 4 / 3 * math.pi * 2.5**3 * 0.8 / 2
        if k == "lj":
            return {"bytes": n * (24 + 4 + 4 + 24) + case["systems"] * 112.0, "flops": 40 * pairs}
        return {"bytes": n * (48 + 8 + 8 + 72) + case["systems"] * 136.0, "flops": case["steps"] * (30 * pairs + 60 * n)}
    if k == "gcmc":
        r, nk = case["replicas"], 2400
        # each step: one molecule's new and old ends against the atoms within the cutoff, and the k sum
        near = 4 / 3 * math.pi * 12.0**3 * 8300 / 54127.0
        return {"bytes": 8000 * 20 + r * (2 * 105 * 3 * 16 + 2 * nk * 16.0),
                "flops": case["steps"] * r * (6 * near * 40 + nk * 6 * 16.0)}
    if k in ("melt_md", "lj_ewald"):
        n, m = case["ions"], case["kmax"]
        nk = (m + 1) * (2 * m + 1) ** 2
        flops = n * 4 / 3 * math.pi * case["cutoff"] ** 3 * 0.0625 / 2 * 80 + 2 * n * nk * 20.0
        if k == "lj_ewald":
            return {"bytes": n * (24 + 8 + 8 + 24) + nk * 28.0, "flops": flops}
        return {"bytes": n * (2 * 48 + 24 + 24) + nk * 12.0, "flops": case["steps"] * flops}
    if k == "neighbors":
        n = case["systems"] * case["molecules"] * 3
        edges = n * 4 / 3 * math.pi * case["cutoff"] ** 3 * 0.1
        return {"bytes": n * 32 + edges * 20.0, "flops": edges * 20.0}
    if k == "bonded":
        n = case["chains"] * case["beads"]
        return {"bytes": n * (24 + 8 + 24) + n * (4 * (2 + 3 + 4 + 4) + 12 * (1 + 2 + 3 + 3)) + case["chains"] * 104.0,
                "flops": n * 600.0}
    gemm = 2.0 * (64 * 256 + 2 * 256 * 256 + 256)
    if k == "train":
        return {"bytes": case["batch"] * 28.0 + mlp.N_PARAMS * 28.0, "flops": case["batch"] * (3 * gemm - 2 * 64 * 256)}
    if k == "forward":
        return {"bytes": case["points"] * 28.0 + mlp.N_PARAMS * 2, "flops": case["points"] * gemm}
    n = case["systems"] * case["molecules"] * 3
    return {"bytes": n * 88.0 + case["systems"] * 350.0, "flops": n * 80.0}


# ----------------------------------------------------------------------------- float64 results
def _lj_system(x, box, s6, e4, rc):
    """Energy, dE/dx and dE/dtril (order TRIL) of one cubic system of equal atoms inside its cell."""
    n = x.shape[0]
    imgs = [-1, 0, 1] if 2 * rc > box else [None]
    e = x.new_zeros(())
    g, w = torch.zeros_like(x), x.new_zeros((3, 3))
    for i0 in range(0, n, 512):
        d0 = x[None, :, :] - x[i0:i0 + 512, None, :]
        for o in [(a, b, c) for a in imgs for b in imgs for c in imgs]:
            s = -torch.round(d0 / box) if o[0] is None else torch.tensor(o, dtype=F64, device=x.device).expand_as(d0)
            d = d0 + s * box
            r2 = (d * d).sum(-1)
            r2 = torch.where((r2 < rc * rc) & (r2 > 0), r2, torch.inf)
            c6 = s6 / r2**3
            e = e + 0.5 * (e4 * (c6 * c6 - c6)).sum()
            gd = (-6.0 * e4 * c6 * (2 * c6 - 1) / r2).masked_fill(~torch.isfinite(r2), 0.0)[..., None] * d
            g[i0:i0 + 512] -= gd.sum(1)
            w += 0.5 * torch.einsum("ija,ijb->ab", s, gd)
    return e, g, torch.stack([w[a, b] for a, b in TRIL])


def _philox_normals(seed, stream, counter):
    """Four normals per stream: Philox4x32-10 words, Box-Muller."""
    c = [np.full(len(stream), counter & 0xFFFFFFFF, np.uint64), np.full(len(stream), counter >> 32, np.uint64),
         (stream & 0xFFFFFFFF).astype(np.uint64), (stream >> 32).astype(np.uint64)]
    k0, k1, m32 = seed & 0xFFFFFFFF, (seed >> 32) & 0xFFFFFFFF, np.uint64(0xFFFFFFFF)
    for _ in range(10):
        p0, p1 = c[0] * np.uint64(0xD2511F53), c[2] * np.uint64(0xCD9E8D57)
        c = [(p1 >> np.uint64(32)) ^ c[1] ^ np.uint64(k0), p1 & m32, (p0 >> np.uint64(32)) ^ c[3] ^ np.uint64(k1), p0 & m32]
        k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
    u = [((v >> np.uint64(8)).astype(np.float64) + 1.0) / 16777216.0 for v in c]
    r0, r1 = np.sqrt(-2 * np.log(u[0])), np.sqrt(-2 * np.log(u[2]))
    return np.stack([r0 * np.cos(2 * np.pi * u[1]), r0 * np.sin(2 * np.pi * u[1]), r1 * np.cos(2 * np.pi * u[3])], -1)


def _exact_md(c, seed):
    if c["integrator"] not in ("baoab", "velocity_verlet"):
        return None
    w = _liquid(c, seed)
    counts = np.bincount(w.system, minlength=w.n_systems)
    if float((counts.astype(float) ** 2).sum()) * (c["steps"] + 1) > 4e9:
        return None  # minutes of float64 pairs
    s6, e4 = float(w.sigma[0, 0]) ** 6, 4 * float(w.epsilon[0, 0])
    off = np.concatenate([[0], np.cumsum(counts)])
    noise = [_t(_philox_normals(seed, np.arange(w.n_atoms, dtype=np.uint64), k)) for k in range(c["steps"])]
    out = {n: [] for n in ("positions", "momenta", "forces", "energy", "kinetic", "cell_gradient", "pressure")}
    for s in range(w.n_systems):
        a, b = off[s], off[s + 1]
        box, dt, m = float(w.tril[s, 0]), float(w.time_step[s]), float(w.masses[a])
        x, p = _t(w.positions[a:b]), _t(w.momenta[a:b])
        kt = float(w.temperature[s]) * units.BOLTZMANN_CONSTANT
        c1 = math.exp(-float(w.friction[s]) * dt)
        c2 = math.sqrt(kt * (1 - c1 * c1) * m)
        force = lambda y: _lj_system(y - box * torch.floor(y / box + 0.5), box, s6, e4, w.cutoff)
        e, g, wt = force(x)
        for k in range(c["steps"]):
            p = p - 0.5 * dt * g
            x = x + 0.5 * dt * p / m
            if c["integrator"] == "baoab":
                p = c1 * p + c2 * noise[k][a:b]
            x = x + 0.5 * dt * p / m
            e, g, wt = force(x)
            p = p - 0.5 * dt * g
        x = x - box * torch.floor(x / box + 0.5)
        kin = 0.5 * (p * p).sum() / m
        virial = (x * g).sum() + box * (wt[0] + wt[2] + wt[5])
        for n, v in zip(out, (x, p, -g, e, kin, wt, (2 * kin - virial) / (3 * box**3))):
            out[n].append(v)
    return {n: torch.cat(v) if n in ("positions", "momenta", "forces") else torch.stack(v) for n, v in out.items()}


def _exact_salt(w, x):
    """LJ + Ewald energy, dE/dx, dE/dtril and S(k) of the salt in its cube."""
    box, a, rc = float(w.tril[0, 0]), w.alpha, w.cutoff
    q, sp = _t(w.charges), torch.as_tensor(w.species, device=DEV).long()
    sg, ep = _t(w.sigma), _t(w.epsilon)
    e, g, wt = x.new_zeros(()), torch.zeros_like(x), x.new_zeros((3, 3))
    imgs = [-1, 0, 1] if 2 * rc > box else [None]
    for i0 in range(0, x.shape[0], 500):
        d0 = x[None] - x[i0:i0 + 500, None]
        s6 = sg[sp[i0:i0 + 500]][:, sp] ** 6
        e4 = 4 * ep[sp[i0:i0 + 500]][:, sp]
        qq = KE * q[i0:i0 + 500, None] * q[None]
        for o in [(i, j, k) for i in imgs for j in imgs for k in imgs]:
            s = -torch.round(d0 / box) if o[0] is None else torch.tensor(o, dtype=F64, device=DEV).expand_as(d0)
            d = d0 + s * box
            r2 = (d * d).sum(-1)
            on = (r2 < rc * rc) & (r2 > 0)
            r2 = torch.where(on, r2, 1.0)
            r = torch.sqrt(r2)
            c6, er = s6 / r2**3, torch.erfc(a * r)
            u = e4 * (c6 * c6 - c6) + qq * er / r
            f = -6 * e4 * c6 * (2 * c6 - 1) / r2 - qq * (er / r2 + 2 * a / math.sqrt(math.pi) * torch.exp(-a * a * r2) / r) / r
            e = e + 0.5 * torch.where(on, u, 0.0).sum()
            gd = torch.where(on, f, 0.0)[..., None] * d
            g[i0:i0 + 500] -= gd.sum(1)
            wt += 0.5 * torch.einsum("ija,ijb->ab", s, gd)
    kn = _t(w.kvec_n[0])
    k = 2 * math.pi / box * kn
    k2 = (k * k).sum(-1)
    P = (2 - (kn[:, 0] == 0).to(F64)) * 2 * math.pi / box**3 * torch.exp(-k2 / (4 * a * a)) / k2.clamp(min=1e-300)
    P = torch.where(k2 > 0, P, 0.0)
    k2 = torch.where(k2 > 0, k2, 1.0)
    th = x @ k.T
    cs, sn = torch.cos(th), torch.sin(th)
    sc, ss = q @ cs, q @ sn
    el = KE * (P * (sc**2 + ss**2)).sum()
    wk = P * (ss * cs - sc * sn)
    gl = 2 * KE * q[:, None] * (wk @ k)
    ck = KE * (sc**2 + ss**2) * P * (-1 / (2 * a * a) - 2 / k2)
    m = -(x / box).T @ gl - (k / box).T @ (ck[:, None] * k) - torch.eye(3, dtype=F64, device=DEV) * el / box
    es = -KE * a / math.sqrt(math.pi) * (q * q).sum()
    low = lambda t: torch.stack([t[i, j] for i, j in TRIL])
    return {"energy": (e + el + es).reshape(1), "gradient": g + gl, "cell_gradient": (low(wt) + low(m))[None],
            "structure_factor": torch.stack([sc, ss], -1)[None]}


def _exact_melt(c, seed):
    w = _salt(c, seed)
    box, dt = float(w.tril[0, 0]), w.time_step
    x, p, m = _t(w.positions), _t(w.momenta), _t(w.masses)[:, None]
    r = _exact_salt(w, x)
    for _ in range(c["steps"]):
        p = p - 0.5 * dt * r["gradient"]
        x = x + dt * p / m
        x = x - box * torch.floor(x / box + 0.5)
        r = _exact_salt(w, x)
        p = p - 0.5 * dt * r["gradient"]
    return {"positions": x, "momenta": p, "gradient": r["gradient"], "energy": r["energy"]}


def _exact_bonded(c, seed):
    d = _chains(c, seed)
    x = _t(d["pos"]).requires_grad_(True)
    tril = _t(d["tril"]).requires_grad_(True)
    system, species = torch.as_tensor(d["system"], device=DEV), torch.as_tensor(d["species"], device=DEV).long()
    L = torch.zeros((c["chains"], 3, 3), dtype=F64, device=DEV)
    L = L.index_put(([torch.arange(c["chains"], device=DEV)[:, None]] + [torch.tensor([t[i] for t in TRIL], device=DEV)[None] for i in (0, 1)]), tril)
    total = torch.zeros(c["chains"], dtype=F64, device=DEV)
    cross = lambda a, b: torch.linalg.cross(a, b, dim=-1)
    dot = lambda a, b: (a * b).sum(-1)
    for name in ("bond", "angle", "dihedral", "inversion"):
        e, sh = (torch.as_tensor(v, device=DEV) for v in d[name])
        e, si = e.long(), system[e[:, 0].long()]
        v = [x[e[:, i + 1]] - x[e[:, 0]] + torch.einsum("na,nab->nb", sh[:, i].to(F64), L[si]) for i in range(e.shape[1] - 1)]
        row = tuple(species[e[:, i]] for i in range(e.shape[1]))
        par = lambda key: _t(d[key])[row]
        if name == "bond":
            u = par("kb") * (v[0].norm(dim=-1) - par("x0")) ** 2
        elif name == "angle":
            th = torch.rad2deg(torch.atan2(cross(v[0], v[1]).norm(dim=-1), dot(v[0], v[1])))
            u = par("ka") * (th - par("theta0")) ** 2
        elif name == "dihedral":
            b1, b2, b3 = v[0], v[1] - v[0], v[2] - v[1]
            m, n = cross(b1, b2), cross(b2, b3)
            phi = torch.atan2(dot(cross(m, n), b2) / b2.norm(dim=-1), dot(m, n))
            u = 0.5 * par("V") * (1 - torch.cos(par("per") * par("phi0")) * torch.cos(par("per") * phi))
        else:  # planar inversions: k (1 - cos omega)
            n = cross(v[1], v[2])
            sw = dot(v[0], n) / (n.norm(dim=-1) * v[0].norm(dim=-1))
            u = par("ki") * (1 - torch.sqrt((1 - sw * sw).clamp(min=1e-30)))
        total = total.index_add(0, si, u)
    g, gt = torch.autograd.grad(total.sum(), (x, tril))
    return {"energy": total.detach(), "gradient": g, "cell_gradient": gt}


def _layers(flat):
    w = {n: flat[o:o + int(np.prod(s))].reshape(s) for n, (o, s) in mlp.OFFSETS.items()}
    return [(w["W1"], w["b1"]), (w["W2"], w["b2"]), (w["W3"], w["b3"]), (w["w4"][None], w["b4"])]


def _exact_network(flat, x):
    ph = 2 * math.pi * (x @ _t(mlp.default_frequencies()).T)
    h = torch.stack([torch.sin(ph), torch.cos(ph)], -1).reshape(x.shape[0], -1)
    for i, (w, b) in enumerate(_layers(flat)):
        h = h @ w.T + b
        h = torch.nn.functional.softplus(h) if i < 3 else h
    return h[:, 0]


def exact(case, seed):
    k = case["kind"]
    if k == "md":
        return _exact_md(case, seed)
    if k == "melt_md":
        return _exact_melt(case, seed)
    if k == "lj_ewald":
        w = _salt(case, seed)
        return _exact_salt(w, _t(w.positions))
    if k == "lj":
        w = _liquid(case, seed)
        off = np.concatenate([[0], np.cumsum(np.bincount(w.system, minlength=w.n_systems))])
        r = [_lj_system(_t(w.positions[off[s]:off[s + 1]]), float(w.tril[s, 0]), float(w.sigma[0, 0]) ** 6,
                        4 * float(w.epsilon[0, 0]), w.cutoff) for s in range(w.n_systems)]
        return {"energy": torch.stack([v[0] for v in r]), "gradient": torch.cat([v[1] for v in r]),
                "cell_gradient": torch.stack([v[2] for v in r])}
    if k == "bonded":
        return _exact_bonded(case, seed)
    if k == "forward":
        s = prepare(case, seed)
        flat = s["net"].param.to(F64)
        return torch.cat([_exact_network(flat, x) for x in s["x"].split(65536)])
    if k == "train":
        s = prepare(case, seed)
        net, x, y = s["net"], s["x"], s["y"].to(F64)
        flat = net.param.to(F64).requires_grad_(True)
        g = _exact_network(flat, x)
        loss = torch.nn.functional.softplus(torch.where(y > 0.5, -g, g)).mean()
        (gr,) = torch.autograd.grad(loss, (flat,))
        m, v, t = 0.9 * net.m.to(F64) + 0.1 * gr, 0.999 * net.v.to(F64) + 0.001 * gr * gr, net.t + 1
        step = 1e-3 * (m / (1 - 0.9**t)) / (torch.sqrt(v / (1 - 0.999**t)) + 1e-8)
        return {"param": flat.detach() - step, "moment1": m, "moment2": v, "loss": loss.detach().reshape(1)}
    if k == "virial":
        s = prepare(case, seed)
        pos, g, sy, tril, gt = s["args"]
        L = torch.zeros((tril.shape[0], 3, 3), dtype=F64, device=DEV)
        G = torch.zeros_like(L)
        for i, (a, b) in enumerate(TRIL):
            L[:, a, b], G[:, a, b] = tril[:, i], gt[:, i]
        sy, vol = sy.long(), (tril[:, 0] * tril[:, 2] * tril[:, 5]).abs()[:, None, None]
        inv = torch.linalg.inv(L)
        wrap = lambda r, i: r - torch.einsum("na,nab->nb", torch.floor(torch.einsum("na,nab->nb", r, inv[i]) + 0.5), L[i])
        first = pos[0::3].repeat_interleave(3, 0)
        com = wrap(wrap(pos - first, sy).reshape(-1, 3, 3).mean(1) + pos[0::3], sy[0::3]).repeat_interleave(3, 0)
        per = lambda v: torch.zeros((tril.shape[0],) + tuple(v.shape[1:]), dtype=F64, device=DEV).index_add_(0, sy, v)
        outer = lambda a, b: a[:, :, None] * b[:, None, :]
        lg = L.transpose(1, 2) @ G
        mol = per(outer(pos - wrap(pos - com, sy), g))
        stress = -(per(outer(pos, g)) + lg) / vol
        mom, ms = s["more"]["momenta"], s["more"]["masses"]
        kin = per(0.5 * (mom * mom).sum(-1) / ms)
        return {"stress": stress, "lattice_stress": -G / vol,
                "pressure": 2 * kin / (3 * vol[:, 0, 0]) + torch.diagonal(stress, dim1=1, dim2=2).sum(-1) / 3,
                "molecular_stress": -(0.5 * (mol + mol.transpose(1, 2)) + lg) / vol, "kinetic": kin}
    return None
