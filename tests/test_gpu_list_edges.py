"""The list builders where their work splits: groups of eight atoms and
chunks of 32 candidates that end inside a cell, cells far denser than the
average (more candidate chunks than estimated), pairs at exactly the list
radius (settled in FP64), frozen atoms, boxes without the FP32 minimum image,
and systems whose pair masks are made in several slabs.

Reference: the C restatement of MDBas's builders, entry by entry."""
import numpy as np
import pytest

import oracle
from mdbas_b200 import nb, systems
from dropin_util import DropinSystem

pytestmark = pytest.mark.gpu


def _check(s, ratio=1, frozen=None, cell=None, box_type=nb.CUBIC):
    d = DropinSystem(s, linkRatio=ratio, frozen=frozen, cell=cell, box_type=box_type)
    link = d.makelist()
    o = oracle.Oracle()
    box = o.box(s.cell() if cell is None else cell, box_type)
    excl = d.get_excl()
    if link:
        ref = o.link_cell_list(box, d.x, d.y, d.z, excl, linkRatio=ratio, frozen=frozen,
                               box_type=box_type)
    else:
        ref = o.verlet_list(box, d.x, d.y, d.z, excl, frozen=frozen, box_type=box_type)
    got = d.get_list()
    d.free()
    for a, b in zip(got, ref):
        assert np.array_equal(a, b)
    return link


def _atoms(pos, box):
    n = len(pos)
    e2, e3 = np.zeros((0, 2), np.int32), np.zeros((0, 3), np.int32)
    one = np.ones(n)
    return systems.System("atoms", box, *(np.ascontiguousarray(pos[:, k]) for k in range(3)),
                          0.1 * one, one, 1.5 * one, 16.0 * one, e2, e3)


@pytest.mark.parametrize("n", [1, 2, 7, 8, 9, 31, 32, 33, 255, 257, 1030])
def test_all_pairs_remainders(gpu, n):
    rng = np.random.default_rng(n)
    assert _check(_atoms(rng.uniform(-20, 20, (n, 3)), 40.0)) == 0


@pytest.mark.parametrize("n", [1, 9, 33, 500, 4099])
@pytest.mark.parametrize("ratio", [1, 3])
def test_link_cell_remainders(gpu, n, ratio):
    # empty cells, cells of a few atoms, groups across cells
    rng = np.random.default_rng(n)
    assert _check(_atoms(rng.uniform(-30, 30, (n, 3)), 60.0), ratio=ratio) == 1


def test_dense_cells(gpu):
    rng = np.random.default_rng(5)
    pos = np.concatenate([rng.uniform(-30, 30, (2000, 3)), rng.uniform(0, 9, (3000, 3))])
    assert _check(_atoms(pos, 60.0)) == 1


@pytest.mark.parametrize("m,link", [(10, 0), (17, 1)])
def test_pairs_at_the_list_radius(gpu, m, link):
    # a crystal of spacing 3.5 A holds pairs at exactly 14 A
    g = 3.5 * (np.stack(np.meshgrid(*[np.arange(m)] * 3, indexing="ij"), -1).reshape(-1, 3)
               - 0.5 * m)
    assert _check(_atoms(g, 3.5 * m)) == link


@pytest.mark.parametrize("n", [3000, 12000])
def test_frozen(gpu, n):
    frozen = (np.random.default_rng(n).random(n) < 0.4).astype(np.int32)
    _check(systems.water_box_for_atoms(n, seed=n), frozen=frozen)


@pytest.mark.parametrize("n", [3000, 18558])
def test_triclinic(gpu, n):
    s = systems.water_box_for_atoms(n, seed=n)
    cell = s.box * np.array([1, 0, 0, 0.2, 1, 0, 0.1, -0.15, 1])
    p = np.stack([s.x, s.y, s.z], 1) / s.box @ cell.reshape(3, 3)
    s.x, s.y, s.z = (p[:, k].copy() for k in range(3))
    _check(s, cell=cell, box_type=nb.TCLIN)


def test_mask_slabs(gpu):
    """96,000 atoms without link cells: the mask rows exceed one slab; a sample
    of rows against MDBas's expression."""
    n = 96000
    s = systems.water_box_for_atoms(n, seed=2)
    d = DropinSystem(s, noLink=1)
    assert d.makelist() == 0
    lst, pair, order = d.get_list()
    assert np.array_equal(order, np.arange(n))
    off = np.concatenate([[0], np.cumsum(pair.astype(np.int64))])
    u = d.box.u1
    for i in np.random.default_rng(1).integers(0, n - 1, 40).tolist() + [0, n - 2]:
        j = np.arange(i + 1, n)
        r2 = 0.0
        for a in (d.x, d.y, d.z):
            t = a[j] - a[i]
            t = t - s.box * np.trunc(t * u + np.where(t * u >= 0, 0.5, -0.5))
            r2 = r2 + t * t
        j = j[(r2 <= 14.0 * 14.0) & (j // 3 != i // 3)]
        assert np.array_equal(lst[off[i]:off[i + 1]], j)
    d.free()
