"""A captured step (small kernels folded into the two half kicks, the bath's
scaling left to the next step, reciprocal space, bonded terms and exclusions as
branches) against the host-driven step, bit for bit, over the forms a step can
take: no constraints, all atoms in rigid triangles, some, general constraints;
frozen atoms, bonded terms, explicit Ewald and SPME, with and without a bath,
displacement test, fixed cadence and pruning.  The kinetic energy and the
wrapped positions are checked by themselves."""
import numpy as np
import pytest

from mdbas_b200 import nb, systems

pytestmark = pytest.mark.gpu

STEPS = 45  # two launches of 20 and five host-driven steps


def _run(s, graph, cons=None, kspace=None, frozen=None, bonded=None, tau=0.0, update=0, prune=0.0,
         dt=0.0005):
    e = nb.Engine(s, precision=1, frozen=frozen)
    e.md_set_graph(graph)
    if prune:
        e.md_set_prune(prune)
    if bonded:
        e.set_bonded(bonded)
    if kspace:
        e.set_kspace(*kspace)
    e.md_init(s.mass, (s.vx, s.vy, s.vz), time_step=dt, list_update=update, constraints=cons)
    rows = e.md_run(STEPS, energy_every=1, target_temp=300.0, tau_t=tau)
    out = (np.stack(e.positions()), np.stack(e.velocities()), rows)
    e.close()
    return out


def _check(s, **kw):
    a, b = _run(s, 20, **kw), _run(s, 0, **kw)
    for u, v in zip(a, b):
        assert np.array_equal(u, v)
    pos, vel, rows = a
    kin = 0.5 * (s.mass * (vel * vel).sum(0)).sum()
    # fixed point of 2^-24 per atom; the bath scales the sum in FP64
    assert abs(rows[-1, 2] - kin) <= s.n * 2.0 ** -24 + 1e-9 * kin
    assert np.all(np.abs(pos) <= 0.5 * s.box * (1 + 1e-12))


@pytest.fixture(scope="module")
def water():
    return systems.water_box(500, 25.0, seed=4, temperature=300.0)


@pytest.fixture(scope="module")
def chains():
    return systems.flexible_chains(6, 39.0, seed=2, temperature=300.0)


def _some(cons, keep):
    k = np.nonzero(keep)[0]
    return np.asarray(cons[0]).reshape(-1, 2)[k], np.asarray(cons[1])[k]


@pytest.mark.parametrize("which", ["triangles", "some", "general"])
@pytest.mark.parametrize("opt", [dict(), dict(tau=0.1), dict(tau=0.1, prune=0.5),
                                 dict(update=7), dict(tau=0.05, update=7, prune=0.5)])
def test_water(gpu, water, which, opt):
    cons = water.water_constraints()
    mol = np.asarray(cons[0]).reshape(-1, 2).min(1) // 3
    if which == "some":
        cons = _some(cons, mol % 3 > 0)
    elif which == "general":
        first = np.r_[True, mol[1:] != mol[:-1]]
        cons = _some(cons, ~first)  # two constraints a molecule
    frozen = (np.arange(water.n) // 3 % 50 == 0).astype(np.int32) if opt.get("prune") else None
    if frozen is not None:
        water = systems.water_box(500, 25.0, seed=4, temperature=300.0)
        for v in (water.vx, water.vy, water.vz):
            v[frozen > 0] = 0.0
    # (without bonds in their place, free atoms of water collapse within 20 fs)
    _check(water, cons=cons, frozen=frozen, dt=0.0005 if which == "triangles" else 0.0001, **opt)


@pytest.mark.parametrize("kspace", [None, (1, (6, 6, 6)), (2, (32, 32, 32), 6),
                                    (2, (32, 40, 48), 4)])
@pytest.mark.parametrize("opt", [dict(), dict(tau=0.1), dict(update=5)])
def test_chains(gpu, chains, kspace, opt):
    _check(chains, kspace=kspace, bonded=chains.meta["bonded"], **opt)
