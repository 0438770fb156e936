"""Host groups skipped by their boxes leave energy changes bit-identical in cells of every shape: cubic,
skewed along all axes, flat (an axis barely twice the cutoff wide, groups reaching past half of it) and
elongated, with hosts of one group to many and a last group that is not full."""

import numpy as np
import pytest

from oracle import unitcell as ouc
from test_gpu_gcmc import co2_template, random_molecule, small_setup

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lengths,angles", [([30, 30, 30], [90, 90, 90]), ([33, 29, 35], [71, 104, 63]),
                                            ([40, 38, 16.1], [90, 90, 120]), ([17, 18, 60], [100, 80, 110])])
@pytest.mark.parametrize("n_fw", [31, 33, 3000])
def test_host_groups_skipped_by_their_boxes(lengths, angles, n_fw):
    from kups_gb300 import gcmc

    rng = np.random.default_rng(n_fw)
    n_sys = 24
    setup = small_setup(n_sys=n_sys, rc=7.0)
    L = ouc.lattice_from_lengths_angles(lengths, angles)
    tril = ouc.tril_from_lattice(L)
    setup.tril = np.repeat(tril[None], n_sys, 0)
    # in order along a corner of the cell, so that groups are compact and their boxes count
    f = rng.uniform(-0.5, 0.5, (n_fw, 3))
    f = f[np.lexsort((f[:, 2], np.floor(6 * f[:, 1]), np.floor(6 * f[:, 0])))]
    setup.fw_positions = f @ L
    setup.fw_species = rng.integers(0, 4, n_fw)
    setup.fw_charges = rng.normal(0, 0.3, n_fw)
    setup.fw_count = np.full(n_sys, n_fw)
    news = [random_molecule(rng, L, co2_template()[0]) for _ in range(n_sys)]
    news = [ouc.wrap(p, np.repeat(tril[None], 3, 0)) for p in news]
    outs = []
    for groups in (True, False):
        mc = gcmc.GCMC(setup, seed=3)
        mc.set_guests([np.zeros((0, 3))] * n_sys)
        if not groups:
            mc.fw_group = None
        outs.append(mc.evaluate([gcmc.MOVES.index("insert")] * n_sys, [0] * n_sys, news))
    np.testing.assert_array_equal(outs[0], outs[1])
    assert np.isfinite(outs[0]).all() and np.abs(outs[0]).max() > 0
