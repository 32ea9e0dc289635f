"""SPME's half-complex grid where it can go wrong: triclinic boxes (the planes
at half a grid length, whose index MDBas takes as +m/2 on both sides), odd
grid lengths, tiles with more atoms than one staged batch and empty tiles, one
atom, and every order that has its own kernels beside one that shares them.
(Orders are even: an odd B-spline's modulus vanishes at half a grid length,
and the sum is dominated by that 1e86 in MDBas's form as well.)

Reference: the numpy restatement (full complex grid); tolerances of
test_gpu_spme.py, the forces of a lone atom (removed with their mean) by the
energy's size."""
import numpy as np
import pytest

from mdbas_b200 import nb, systems

pytestmark = pytest.mark.gpu

BOX = 24.0
TRI = np.array([BOX, 0, 0, 5.0, BOX, 0, 3.0, -4.0, BOX])


def _atoms(n, seed, spread):
    rng = np.random.default_rng(seed)
    pos = rng.uniform(-spread, spread, (n, 3))
    z = np.zeros(n)
    return systems.System("q", BOX, *(pos[:, i].copy() for i in range(3)), rng.uniform(-1, 1, n),
                          z, z, z + 1, np.zeros((0, 2), np.int32), np.zeros((0, 3), np.int32))


@pytest.mark.parametrize("tri", [False, True])
@pytest.mark.parametrize("grid,nbsp", [((8, 8, 8), 4), ((16, 8, 24), 6), ((24, 16, 16), 8),
                                       ((16, 16, 24), 10), ((9, 8, 15), 8),
                                       ((10, 12, 14), 4)])
@pytest.mark.parametrize("n,spread", [(1, 9.0), (150, 9.0), (400, 2.5)])
def test_half_grid(gpu, oracle_lib, grid, nbsp, tri, n, spread):
    from oracle import spme_oracle as so
    s = _atoms(n, 10 * n + nbsp, spread)
    btype = nb.TCLIN if tri else nb.CUBIC
    cell = TRI if tri else s.cell()
    got = nb.spme(s, alpha=0.4, grid=grid, nbsp=nbsp, cell=cell, box_type=btype)
    box = oracle_lib.box(cell, box_type=btype)
    ref = so.spme_energy(box, s.x, s.y, s.z, s.q, 0.4, systems.CHARGE_CONST, grid, nbsp)
    size = systems.CHARGE_CONST * 0.4 * (s.q ** 2).sum()  # the self term cancels most of it
    assert abs(got[0] - ref[0]) <= 1e-11 * size
    assert abs(got[4] - ref[4]) <= 1e-10 * size
    err = np.sqrt(sum(((a - b) ** 2).sum() for a, b in zip(got[1:4], ref[1:4])))
    norm = np.sqrt(sum((b ** 2).sum() for b in ref[1:4]))
    assert err <= 1e-10 * max(norm, 1e-3 * size / BOX)
