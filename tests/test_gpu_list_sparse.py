"""Link cells far more numerous than the atoms (a droplet in a wide box): the
list, entry by entry, and the device memory a build takes, which may follow the
number of cells for the cells' counts alone, not for their candidate tables."""
import numpy as np
import pytest
import torch

import oracle
from mdbas_b200 import nb, systems
from dropin_util import DropinSystem

pytestmark = pytest.mark.gpu


def _droplet(n, box, seed=1):
    rng = np.random.default_rng(seed)
    pos = np.concatenate([rng.uniform(-15, 15, (n - n // 10, 3)),          # one droplet,
                          rng.uniform(-0.5 * box, 0.5 * box, (n // 10, 3))])  # some vapour
    one = np.ones(n)
    return systems.System("droplet", box, *(pos[:, k].copy() for k in range(3)), 0.1 * one, one,
                          1.5 * one, 16.0 * one, np.zeros((0, 2), np.int32),
                          np.zeros((0, 3), np.int32))


@pytest.mark.parametrize("ratio", [1, 2, 5])
@pytest.mark.parametrize("n", [20, 3000])
def test_list_in_a_wide_box(gpu, n, ratio):
    s = _droplet(n, 400.0, seed=n)
    d = DropinSystem(s, linkRatio=ratio)
    assert d.makelist() == 1
    excl = d.get_excl()
    o = oracle.Oracle()
    ref = o.link_cell_list(o.box(s.cell()), d.x, d.y, d.z, excl, linkRatio=ratio)
    got = d.get_list()
    d.free()
    for a, b in zip(got, ref):
        assert np.array_equal(a, b)


def test_memory_in_a_wide_box(gpu):
    s = _droplet(3000, 2000.0)
    cells = int(2000.0 / 14.0) ** 3
    e = nb.Engine(s, precision=0, exclusions=(np.zeros(s.n + 1, np.int32),
                                              np.zeros(0, np.int32)))
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    e.build()
    taken = free - torch.cuda.mem_get_info()[0]
    e.close()
    # three counts a cell, and what 3,000 atoms take (lists of all pairs at the most)
    assert taken <= 4 * 4 * cells + 4 * s.n * s.n + (32 << 20)
