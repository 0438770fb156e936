"""Systems stepped by teams of 8, 4 and 2 CTAs (few systems of at least 384 atoms) against the same steps by
one CTA each (chosen by a grid size of the caller's own): every output the same to the bit, through list
builds, resumed lists, per-step records, a list overflow, several species and sizes that leave CTAs of a
team with few atoms or none."""

import numpy as np
import pytest
import torch

from test_gpu_core import md_state
from test_gpu_md_lists import _batch

pytestmark = pytest.mark.gpu

INTEGRATORS = ["velocity_verlet", "baoab", "csvr", "csvr_npt"]


def _state(counts, species, seed):
    from kups_gb300 import potential, units

    w = _batch(counts, 0.75, seed)
    rng = np.random.default_rng(seed)
    w.momenta = rng.normal(size=w.momenta.shape) * np.sqrt(40.0 * 100.0 * units.BOLTZMANN_CONSTANT)
    st = md_state(w)
    s = len(counts)
    ones = torch.ones(s, dtype=torch.float64, device="cuda")
    st.systems.time_step = 1.0 * ones
    st.systems.temperature = 100.0 * ones
    st.systems.thermostat_time_constant = 20 * units.FEMTO_SECOND * ones
    st.systems.target_pressure = 100 * units.BAR * ones
    st.systems.pressure_coupling_time = 50 * units.FEMTO_SECOND * ones
    st.systems.compressibility = 1e-3 / units.BAR * ones
    st.systems.minimum_scale_factor = 0.99 * ones
    if species > 1:
        st.particles.species = torch.as_tensor(rng.integers(0, species, len(w.positions)), dtype=torch.int32).cuda()
        st.lj_parameters = potential.LennardJonesParameters.from_lorentz_berthelot_mixing(
            ("A", "B", "C")[:species], [3.4, 3.1, 2.8][:species], [0.0103, 0.008, 0.005][:species],
            [float(st.lj_parameters.cutoff)])
    return st


def _run(state, integrator, ctas, steps, **kw):
    from kups_gb300 import md

    packed = md.pack(state)
    packed.rebuilds = torch.zeros(packed.n_systems, dtype=torch.int32, device="cuda")
    prop = md.FusedLennardJonesMD(integrator, n_ctas=ctas, **kw)
    traces = [prop.run_packed(packed, k, seed=7, step0=17 * i, trace=integrator != "csvr") for i, k in enumerate(steps)]
    out = {k: getattr(packed, k).cpu().numpy() for k in ("pos4", "mom4", "frc4", "energy", "kinetic", "virial",
                                                         "pressure", "rebuilds", "cell")}
    for i, t in enumerate(traces):
        if t is not None:
            out[f"potential {i}"], out[f"kinetic {i}"] = (x.cpu().numpy() for x in t)
    return out


def _same(a, b):
    for k in a:
        np.testing.assert_array_equal(a[k].view(np.uint8), b[k].view(np.uint8), err_msg=k)


@pytest.mark.parametrize("integrator", INTEGRATORS)
@pytest.mark.parametrize("counts,species", [([384], 1), ([864], 1), ([1025], 3), ([2048, 400], 1),
                                            ([1, 1500, 33, 500], 2), ([500] * 25, 1), ([900] * 45, 1)])
def test_team_steps_are_those_of_one_cta(integrator, counts, species):
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    state = _state(counts, species, len(counts) + species)
    one = _run(state, integrator, sms, (17, 1, 30))
    _same(_run(state, integrator, 0, (17, 1, 30)), one)
    assert one["rebuilds"].max() > 1  # lists were rebuilt on the way


def test_team_lists_overflow_and_resume_across_grids():
    """A capacity too small at first; then a call by teams that resumes the lists one CTA built, and back."""
    from kups_gb300 import md

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    state = _state([700, 600], 1, 3)
    _same(_run(state, "baoab", 0, (9,), neighbor_capacity=16), _run(state, "baoab", sms, (9,), neighbor_capacity=16))
    runs = []
    for grids in ((sms, sms, sms), (sms, 0, sms)):
        packed = md.pack(state)
        packed.rebuilds = torch.zeros(2, dtype=torch.int32, device="cuda")
        prop = md.FusedLennardJonesMD("velocity_verlet")
        for i, g in enumerate(grids):
            prop.n_ctas = g
            prop.run_packed(packed, 6, seed=1, step0=6 * i)
        runs.append({k: getattr(packed, k).cpu().numpy() for k in ("pos4", "mom4", "frc4", "energy", "rebuilds")})
    _same(*runs)


def test_team_step_records_of_the_cell_gradient():
    from kups_gb300 import md

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    state = _state([864], 1, 5)
    got = []
    for g in (0, sms):
        packed, rec = md.pack(state), torch.zeros((12, 1, 6), dtype=torch.float64, device="cuda")
        md.FusedLennardJonesMD("baoab", n_ctas=g).launch(packed, 12, 3, 0, trace_virial=rec)
        got.append(rec.cpu().numpy())
    _same({"virial": got[0]}, {"virial": got[1]})
    assert np.abs(got[0]).min() > 0
