"""A captured launch whose pair list outgrows its room is taken back and made
again with more: it has to end as the host-driven run, bit for bit.  The list
outgrows its room because free atoms without interactions fly together."""
import numpy as np
import pytest

from mdbas_b200 import nb, systems

pytestmark = pytest.mark.gpu

DT = 0.001


def _system():
    g = np.stack(np.meshgrid(*[np.arange(-12, 13) * 2.5] * 3, indexing="ij"), -1).reshape(-1, 3)
    g = g[(g * g).sum(1) <= 30.0 ** 2]
    pos = g + np.random.default_rng(1).uniform(-0.05, 0.05, g.shape)
    n = len(pos)
    vel = -pos * (0.85 / 20 / DT)
    s = systems.System("inward", 100.0, *(pos[:, k].copy() for k in range(3)), np.zeros(n),
                       np.zeros(n), np.zeros(n), np.ones(n), np.zeros((0, 2), np.int32),
                       np.zeros((0, 3), np.int32))
    return s, tuple(vel[:, k].copy() for k in range(3))


def _engine(s):
    return nb.Engine(s, precision=1, exclusions=(np.zeros(s.n + 1, np.int32),
                                                 np.zeros(0, np.int32)))


def _run(graph, s, vel):
    e = _engine(s)
    e.md_set_graph(graph)
    e.md_init(s.mass, vel, time_step=DT)
    room = e.list_stats()[3]
    rows = e.md_run(20, energy_every=1)
    grown = e.list_stats()[3] > room
    out = np.stack(e.positions()), np.stack(e.velocities()), rows
    e.close()
    return grown, out


def test_outgrown_list(gpu):
    system = _system()
    grown, a = _run(20, *system)
    assert grown
    _, b = _run(0, *system)
    for u, v in zip(a, b):
        assert np.array_equal(u, v)
