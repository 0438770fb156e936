"""The one-pass pair search where its float32 prefilter, its per-warp staging and its packed image
shifts could go wrong: pairs exactly at the cutoff or exactly half a cell apart, particles many
cells outside the primary one (shifts beyond 10 bits), more edges per particle than a warp stages,
particle counts around a block's, and a capacity smaller than the list.  Bit-exact against the
float64 oracle (no tolerance): membership is decided in float64 whenever float32 could not."""

import math

import numpy as np
import pytest
import torch

from oracle import neighborlist as onl

pytestmark = pytest.mark.gpu

CUBE = [10.0, 0, 10.0, 0, 0, 10.0]
SKEW = [10.0, 3.0, 9.0, -2.5, 2.0, 11.0]


def build(pos, system, tril, cut, cap, exclusion=None):
    from kups_gb300 import _lib
    from kups_gb300.neighborlist import new_status, read_status

    lib = _lib.load()
    n, s = len(pos), len(tril)
    t = lambda x, dt: torch.as_tensor(np.ascontiguousarray(x), dtype=dt).cuda()
    p, sy, tr, rc = t(pos, torch.float64), t(system, torch.int32), t(tril, torch.float64), t(cut, torch.float64)
    ex = t(np.arange(n) if exclusion is None else exclusion, torch.int32)
    edges = torch.full((cap, 2), -7, dtype=torch.int32, device="cuda")
    shifts = torch.full((cap, 3), -7, dtype=torch.int32, device="cuda")
    ne = torch.zeros(1, dtype=torch.int64, device="cuda")
    ws = torch.empty(lib.kups_neighborlist_workspace_bytes(n, s), dtype=torch.uint8, device="cuda").fill_(0xa5)
    st = new_status()
    _lib.check(lib.kups_neighborlist_build(p.data_ptr(), sy.data_ptr(), sy.data_ptr(), ex.data_ptr(), n, s,
                                           tr.data_ptr(), rc.data_ptr(), s, edges.data_ptr(), shifts.data_ptr(), cap,
                                           ne.data_ptr(), ws.data_ptr(), ws.numel(), st.data_ptr(), None), "build")
    return int(ne.item()), edges.cpu().numpy(), shifts.cpu().numpy(), read_status(st)


def check(pos, system, tril, cut, exclusion=None):
    pos, system, tril = np.asarray(pos, float), np.asarray(system), np.asarray(tril, float)
    want = onl.neighbor_list(pos, system, tril, np.asarray(cut, float), exclusion=exclusion)
    k = len(want[0])
    count, e, sh, st = build(pos, system, tril, cut, k + 5, exclusion)
    assert st.code == 0 and count == k
    assert (e[k:] == len(pos)).all() and (sh[k:] == 0).all()
    assert (np.diff(e[:k, 0]) >= 0).all()  # grouped by the first particle
    got, ref = onl.sort_edges(e[:k], sh[:k]), onl.sort_edges(*want)
    assert np.array_equal(got[0], ref[0]) and np.array_equal(got[1], ref[1])
    return k


@pytest.mark.parametrize("cell", [CUBE, SKEW])
@pytest.mark.parametrize("cut", [2.5, 4.9, 5.5])
def test_pairs_exactly_at_the_cutoff_and_half_a_cell_apart(cell, cut):
    # a grid of spacing cell / 4: distances equal to 2.5 and differences of exactly half a cell
    g = np.stack(np.meshgrid(*[np.arange(4)] * 3, indexing="ij"), -1).reshape(-1, 3) / 4.0 - 0.5
    L = np.array([[cell[0], 0, 0], [cell[1], cell[2], 0], [cell[3], cell[4], cell[5]]])
    check(g @ L, np.zeros(64, int), [cell], [cut])


def test_half_a_cell_apart_with_an_infinite_cutoff():
    g = np.stack(np.meshgrid(*[np.arange(2)] * 3, indexing="ij"), -1).reshape(-1, 3) * 5.0
    check(np.concatenate([g, g + [0.0, 1.0, 2.0]]), np.zeros(16, int), [CUBE], [math.inf])


@pytest.mark.parametrize("cell", [CUBE, SKEW])
@pytest.mark.parametrize("cut", [3.0, 5.5])
@pytest.mark.parametrize("reach", [3, 400, 700])
def test_particles_many_cells_away(cell, cut, reach):
    """Lattice offsets up to +-reach: shifts beyond +-512 leave the packed form (reach 400 and 700)."""
    rng = np.random.default_rng(reach)
    n = 90
    L = np.array([[cell[0], 0, 0], [cell[1], cell[2], 0], [cell[3], cell[4], cell[5]]])
    f = rng.uniform(-0.5, 0.5, (n, 3)) + rng.integers(-reach, reach + 1, (n, 3)) * (rng.random((n, 1)) < 0.3)
    check(f @ L, np.zeros(n, int), [cell], [cut])


@pytest.mark.parametrize("n", [1, 2, 7, 8, 9, 31, 33, 257])
def test_counts_around_a_block(n):
    rng = np.random.default_rng(n)
    system = np.sort(rng.integers(0, 3, n))
    tril = np.array([CUBE, SKEW, [30.0, 0, 30.0, 0, 0, 30.0]])
    check(rng.uniform(-5, 5, (n, 3)), system, tril, [3.0, 5.6, 4.0])


@pytest.mark.parametrize("cut,images", [(4.9, False), (7.5, True)])
def test_more_edges_than_a_warp_stages(cut, images):
    """700 particles in 10 A: up to about 350 edges each inside 4.9 A, about 1200 with images inside 7.5 A."""
    rng = np.random.default_rng(4)
    n = 1500 if not images else 700
    k = check(rng.uniform(-5, 5, (n, 3)), np.zeros(n, int), [CUBE], [cut], exclusion=np.arange(n) // 3)
    assert k / n > 512


def test_capacity_smaller_than_the_list_writes_the_leading_rows():
    from kups_gb300 import _lib

    rng = np.random.default_rng(8)
    pos = rng.uniform(-5, 5, (200, 3))
    want, _ = onl.neighbor_list(pos, np.zeros(200, int), np.array([CUBE]), np.array([3.0]))
    full = build(pos, np.zeros(200, int), [CUBE], [3.0], len(want))
    cap = len(want) // 2 + 1
    count, e, sh, st = build(pos, np.zeros(200, int), [CUBE], [3.0], cap)
    assert count == len(want) and st.code == _lib.KUPS_ERR_CAPACITY and st.required == len(want)
    assert np.array_equal(e, full[1][:cap]) and np.array_equal(sh, full[2][:cap])
