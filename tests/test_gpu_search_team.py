"""The cluster-pair search of small systems (a block per cluster, its warps
sharing the candidates) at the sizes around its limit of 12,000 atoms and at
its smallest, sparse and crowded: more survivors than the shared buffer holds
at once, groups of 32 that end inside a round, exclusions, frozen atoms.

Reference: MDBas's all-pairs list in the C restatement, as pair sets (pairs
within FP32 rounding of the radius are settled in FP64, so the sets are equal)."""
import numpy as np
import pytest

import oracle
from mdbas_b200 import nb, systems

pytestmark = pytest.mark.gpu

L = 60.0


def _check(s, frozen=None):
    eng = nb.Engine(s, precision=1, frozen=frozen)
    eng.build()
    p = eng.export_pairs(1e30).astype(np.int64)
    eng.close()
    o = oracle.Oracle()
    lst, pair, order = o.verlet_list(o.box(s.cell()), s.x, s.y, s.z, s.exclusions(symmetric=True),
                                     frozen=frozen)
    i, j = np.repeat(order, pair[order]).astype(np.int64), lst.astype(np.int64)
    ref = np.sort(np.minimum(i, j) * s.n + np.maximum(i, j))
    got = np.sort(np.minimum(p[:, 0], p[:, 1]) * s.n + np.maximum(p[:, 0], p[:, 1]))
    assert np.array_equal(got, ref)


def _atoms(pos):
    one = np.ones(len(pos))
    e2, e3 = np.zeros((0, 2), np.int32), np.zeros((0, 3), np.int32)
    return systems.System("atoms", L, *(np.ascontiguousarray(pos[:, k]) for k in range(3)),
                          0.1 * one, one, 1.5 * one, 16.0 * one, e2, e3)


@pytest.mark.parametrize("n", [27, 65, 1031, 11999, 12000, 12001])
def test_spread(gpu, n):
    _check(_atoms(np.random.default_rng(n).uniform(-L / 2, L / 2, (n, 3))))


@pytest.mark.parametrize("n", [600, 4000])
def test_crowded(gpu, n):
    rng = np.random.default_rng(n)
    pos = np.concatenate([rng.uniform(-7, 7, (n, 3)), rng.uniform(-L / 2, L / 2, (n // 2, 3))])
    _check(_atoms(pos))


@pytest.mark.parametrize("n", [2997, 12000, 12003])
def test_water_frozen(gpu, n):
    s = systems.water_box_for_atoms(n, seed=n)
    _check(s, frozen=(np.random.default_rng(n).random(n) < 0.3).astype(np.int32))
