"""Coordinates that are not finite reach the status word of every bonded kind: NaN of either sign and
infinities, in any atom of an edge and any component, in both precisions."""

import struct

import numpy as np
import pytest

from oracle import bonded as ob
from test_gpu_bonded import params_object, random_case

pytestmark = pytest.mark.gpu
VALUES = {"nan": struct.unpack("<d", struct.pack("<Q", 0x7ff8000000000000))[0],
          "minus nan": struct.unpack("<d", struct.pack("<Q", 0xfff8000000000000))[0], "inf": np.inf}


@pytest.mark.parametrize("kind", list(ob.KINDS))
@pytest.mark.parametrize("value", list(VALUES))
@pytest.mark.parametrize("fp32", [False, True])
@pytest.mark.parametrize("shifted", [False, True])
def test_non_finite_coordinates_are_reported(kind, value, fp32, shifted):
    from kups_gb300 import _lib, bonded

    pos, system, species, tril, edges, shifts, table, T, order = random_case(kind, np.random.default_rng(3))
    edge, shift = edges[:1], shifts[:1] * shifted
    term = bonded.BondedTerm(params_object(kind, table, T, order), edge, shift, fp32=fp32)
    bonded.evaluate([term], pos, system, species, tril)  # finite: no error
    for atom in range(order):
        for component in ((0,), (1,), (2,), (0, 1, 2)):
            x = pos.copy()
            x[edge[0, atom], component] = VALUES[value]
            with pytest.raises(_lib.KupsError, match="non-finite"):
                bonded.evaluate([term], x, system, species, tril)
