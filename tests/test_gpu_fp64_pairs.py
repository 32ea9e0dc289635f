"""The FP64 pair kernel where its work splits: rows shorter than, equal to and
just beyond one round of 32 entries, systems below and above the count at
which rows are cut into two items, and pairs that its fast forms do not take
(alpha r beyond their range, almost coinciding atoms).

Reference: the C restatement of MDBas's loop.  Tolerance: the FP64 form's
1e-12 relative (summation order and a few ulp per pair function)."""
import numpy as np
import pytest

import oracle
from mdbas_b200 import nb, systems
from dropin_util import force_rel_rms

pytestmark = pytest.mark.gpu

TOL = 1e-12


def _cluster(n, spacing, seed=1):
    """n neutral-in-sum atoms on a jittered lattice in a 40 A box."""
    rng = np.random.default_rng(seed)
    m = int(np.ceil(n ** (1 / 3) - 1e-9))
    g = np.stack(np.meshgrid(*[np.arange(m)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n]
    p = spacing * (g - 0.5 * (m - 1)) + rng.uniform(-0.1, 0.1, (n, 3))
    q = rng.uniform(-0.8, 0.8, n)
    e2, e3 = np.zeros((0, 2), np.int32), np.zeros((0, 3), np.int32)
    return systems.System("cluster", 40.0, *(p[:, k].copy() for k in range(3)), q - q.mean(),
                          rng.uniform(5.0, 11.0, n), rng.uniform(1.4, 1.9, n), np.full(n, 16.0),
                          e2, e3)


def _check(s, alpha=0.34, vdw=1):
    o = oracle.Oracle()
    box = o.box(s.cell())
    excl = s.exclusions(symmetric=False)
    lst, pair, order = o.verlet_list(box, s.x, s.y, s.z, excl)
    p = o.param(alpha=alpha, vdwSwitch=vdw)
    rx, ry, rz, re = o.ewald_energy(box, s, lst, pair, order, excl, p=p)
    eng = nb.Engine(s, precision=0, alpha=alpha, vdwSwitch=vdw, noLink=1)
    eng.build()
    for _ in range(2):  # the work counter starts over
        eng.compute()
        f, e = eng.forces(), eng.energies()
        assert e["n_pairs"] == re["n_pairs"]
        assert force_rel_rms(f, (rx, ry, rz)) < TOL
        for k, r in (("elec_direct", "e_dir"), ("vdw", "e_vdw"), ("vir_direct", "vir_dir"),
                     ("vir_vdw", "vir_vdw")):
            # the terms cancel in the sums: scale by the forces' work as well
            scale = abs(re[r]) + abs(re["vir_dir"]) + abs(re["vir_vdw"])
            assert abs(e[k] - re[r]) <= TOL * scale, k
    eng.close()


@pytest.mark.parametrize("n", [2, 31, 32, 33, 34, 64, 65, 97])
def test_short_rows(gpu, n):
    _check(_cluster(n, 2.6, seed=n))


@pytest.mark.parametrize("n", [1500, 7101, 7110])
def test_row_split_boundary(gpu, n):
    _check(systems.water_box_for_atoms(n, seed=n))


@pytest.mark.parametrize("alpha,vdw", [(0.0, 1), (0.499, 1), (0.501, 1), (0.8, 1), (0.34, 0)])
def test_alpha_range(gpu, alpha, vdw):
    # alpha * 12 A on either side of the fast form's limit of 6
    _check(_cluster(343, 3.0, seed=3), alpha=alpha, vdw=vdw)


def test_almost_coinciding_atoms(gpu):
    s = _cluster(64, 3.0, seed=4)
    s.eps = np.zeros(s.n)
    s.x[1], s.y[1], s.z[1] = s.x[0] + 5e-4, s.y[0], s.z[0]
    _check(s)
