"""The explicit Ewald sum where its work splits: atom counts around a block,
fewer k-vectors than parts, uneven m-ranges, one dimension only, and a
triclinic box, against the sum written out in numpy.

Tolerance: energies, virials and stresses 1e-12 relative, forces 1e-11 of the
largest (the bounds of the comparison with MDBas's own ewald_rec)."""
import numpy as np
import pytest

from mdbas_b200 import nb, systems

pytestmark = pytest.mark.gpu

ALPHA = 0.34


def _numpy(s, mmax, cell, btype):
    p = nb.make_pbc(cell, btype)
    b = 2 * np.pi * np.array([[p.u1, p.u2, p.u3], [p.v1, p.v2, p.v3], [p.w1, p.w2, p.w3]])
    rc = 1.05 * 2 * np.pi * min(m * w for m, w in zip(mmax, (p.u, p.v, p.w)))
    r = [np.arange(-m, m + 1) for m in mmax]
    m = np.stack(np.meshgrid(*r, indexing="ij"), -1).reshape(-1, 3)
    half = (m[:, 0] > 0) | ((m[:, 0] == 0) & ((m[:, 1] > 0) | ((m[:, 1] == 0) & (m[:, 2] > 0))))
    k = m[half] @ b
    # rows m1 = 0, m2 < 0 are left out of MDBas's half space, m2 > 0 kept
    k2 = (k * k).sum(1)
    k, k2 = k[k2 <= rc * rc], k2[k2 <= rc * rc]
    pos = np.stack([s.x, s.y, s.z], 1)
    ph = k @ pos.T
    c, sn = np.cos(ph), np.sin(ph)
    sc, ss = c @ s.q, sn @ s.q
    ra = -0.25 / ALPHA ** 2
    a = np.exp(ra * k2) / k2
    f1 = 2 * (2 * np.pi / p.vol) * systems.CHARGE_CONST
    de = a[:, None] * (sn * sc[:, None] - c * ss[:, None])
    f = 2 * f1 * (de.T @ k) * s.q[:, None]
    s2 = sc ** 2 + ss ** 2
    vam = 2 * a * (1 / k2 - ra) * s2
    erec = f1 * (a * s2).sum()
    st = [-f1 * (vam * k[:, i] * k[:, j]).sum() for i in range(3) for j in range(i, 3)]
    enn = -0.5 * np.pi * systems.CHARGE_CONST * (s.q.sum() / ALPHA) ** 2 / p.vol
    for i in (0, 3, 5):
        st[i] += erec + enn
    eself = -systems.CHARGE_CONST * ALPHA * (s.q ** 2).sum() / np.sqrt(np.pi)
    return erec + eself + enn, f, -(st[0] + st[3] + st[5]), st


@pytest.mark.parametrize("n", [1, 2, 127, 128, 129, 700])
@pytest.mark.parametrize("mmax,tri", [((3, 5, 4), False), ((1, 1, 1), False), ((2, 2, 2), True),
                                      ((6, 5, 7), True)])
def test_parts(gpu, n, mmax, tri):
    rng = np.random.default_rng(n)
    box = 25.0
    pos = rng.uniform(-12, 12, (n, 3))
    z = np.zeros(n)
    s = systems.System("q", box, *(pos[:, i].copy() for i in range(3)), rng.uniform(-1, 1, n), z,
                       z, z + 1, np.zeros((0, 2), np.int32), np.zeros((0, 3), np.int32))
    cell = [box, 0, 0, 2.0, box, 0, 1.0, -3.0, box] if tri else s.cell()
    btype = nb.TCLIN if tri else nb.CUBIC
    ref = _numpy(s, mmax, cell, btype)
    got = nb.ewald_rec(s, ALPHA, mmax, cell=cell, box_type=btype)
    again = nb.ewald_rec(s, ALPHA, mmax, cell=cell, box_type=btype)
    assert got[0] == again[0] and all(np.array_equal(a, b) for a, b in zip(got[1:4], again[1:4]))
    assert abs(got[0] - ref[0]) <= 1e-12 * abs(ref[0])
    f = np.stack(got[1:4], 1)
    # with one or two atoms the terms cancel: scale by the terms' size
    scale = max(np.abs(ref[1]).max(), 1e-3 * np.abs(ref[0]) / box)
    assert np.abs(f - ref[1]).max() <= 1e-11 * scale
    size = max(abs(v) for v in ref[3]) + abs(ref[0])
    assert abs(got[4] - ref[2]) <= 1e-12 * size
    assert max(abs(a - b) for a, b in zip(got[5], ref[3])) <= 1e-12 * size
