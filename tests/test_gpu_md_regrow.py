"""A captured launch whose pair list outgrows its room is taken back and made
again with more.  Until it is, its later steps run on an empty list, and what
they do wrong (constraints that do not converge, positions that are not
finite) is no result: the run made again has to end as the host-driven one,
bit for bit.

The list outgrows its room because free atoms without interactions fly
together; two like charges on a spring, one of them in a rigid pair, are at
rest as long as their pair force is there."""
import numpy as np
import pytest

from mdbas_b200 import nb, systems

pytestmark = pytest.mark.gpu

DT = 0.001


def _system(charge, wall):
    """(system, velocities, constraints, bonded): atoms 0 and 1 the charges,
    atom 2 in the rigid pair with 0; the rest fly inward.  wall: a Morse term
    that is nothing at the charges' distance of 3 A and beyond any number from
    2.993 A on."""
    g = np.stack(np.meshgrid(*[np.arange(-12, 13) * 2.5] * 3, indexing="ij"), -1).reshape(-1, 3)
    g = g[(g * g).sum(1) <= 30.0 ** 2]
    rng = np.random.default_rng(1)
    g = g + rng.uniform(-0.05, 0.05, g.shape)
    probe = np.array([[-40.0, 40.0, 40.0], [-37.0, 40.0, 40.0], [-41.0, 40.0, 40.0]])
    pos = np.concatenate([probe, g])
    n = len(pos)
    q = np.zeros(n)
    q[:2] = charge
    vel = -pos * (0.85 / 20 / DT)
    vel[:3] = 0.0
    s = systems.System("inward", 100.0, *(pos[:, k].copy() for k in range(3)), q, np.zeros(n),
                       np.zeros(n), np.ones(n), np.zeros((0, 2), np.int32),
                       np.zeros((0, 3), np.int32))
    cons = (np.array([[0, 2]], np.int32), np.array([1.0]))
    bond = {"bonds": {"atoms": [[0, 1]], "k": [1.0], "r0": [2.0], "type": [0]}}
    if not charge:
        return s, tuple(vel[:, k].copy() for k in range(3)), None, None
    e = _engine(s)
    e.set_bonded(bond)
    e.build()
    e.compute()
    pull = e.bonded()[1][0][0]       # towards atom 1 (+x)
    push = e.forces()[0][0]          # away from it
    e.close()
    assert pull > 0.0 > push
    bond["bonds"]["k"] = [-push / pull]
    if wall:
        bond["bonds"] = {"atoms": [[0, 1]] * 2, "k": [-push / pull, 1.0], "r0": [2.0, 2.997],
                         "beta": [0.0, 1e5], "type": [nb.BHARM, nb.BMORSE]}
    return s, tuple(vel[:, k].copy() for k in range(3)), cons, bond


def _engine(s):
    return nb.Engine(s, precision=1, exclusions=(np.zeros(s.n + 1, np.int32),
                                                 np.zeros(0, np.int32)))


def _run(graph, s, vel, cons, bond, **kw):
    e = _engine(s)
    e.md_set_graph(graph)
    if bond:
        e.set_bonded(bond)
    e.md_init(s.mass, vel, time_step=DT, constraints=cons, **kw)
    room = e.list_stats()[3]
    rows = e.md_run(20, energy_every=1)
    grown = e.list_stats()[3] > room
    out = np.stack(e.positions()), np.stack(e.velocities()), rows
    e.close()
    return grown, out


@pytest.mark.parametrize("charge,wall,kw", [
    (0.0, False, dict()),  # the list alone
    # any force on the rigid pair takes SHAKE more than its one iteration
    (1.0, False, dict(tol_shake=1e-6, max_cycle=1)),
    (1.0, True, dict()),
])
def test_overflowing_launch_leaves_nothing(gpu, charge, wall, kw):
    system = _system(charge, wall)
    grown, a = _run(20, *system, **kw)
    assert grown
    _, b = _run(0, *system, **kw)
    for u, v in zip(a, b):
        assert np.array_equal(u, v)
