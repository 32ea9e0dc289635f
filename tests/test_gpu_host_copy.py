"""Results copied to host arrays: sizes around a slot (512 KB), several slots
and more than all of them, page-locked and pageable arrays, several threads at
once.  Copies are exact."""
import threading

import numpy as np
import pytest

from mdbas_b200 import nb, systems

pytestmark = pytest.mark.gpu


def _atoms(n, seed=1):
    pos = np.random.default_rng(seed).uniform(-20, 20, (3, n))
    z = np.zeros(n)
    return systems.System("a", 40.0, pos[0], pos[1], pos[2], z, z, z + 1, z + 1,
                          np.zeros((0, 2), np.int32), np.zeros((0, 3), np.int32))


def _engine(s):
    return nb.Engine(s, precision=1, exclusions=(np.zeros(s.n + 1, np.int32),
                                                 np.zeros(0, np.int32)))


# 65,536 doubles fill a slot; 700,001 atoms (16.8 MB) take more than 32 slots
@pytest.mark.parametrize("n", [1, 21845, 21846, 65535, 65536, 65537, 200003, 700001])
def test_round_trip(gpu, n):
    s = _atoms(n)
    e = _engine(s)
    for _ in range(2):
        for a, b in zip(e.positions(), (s.x, s.y, s.z)):
            assert np.array_equal(a, b)
    e.close()


def test_page_locked_arrays(gpu):
    import torch
    s = systems.water_box_for_atoms(48000, seed=2)
    e = nb.Engine(s, precision=1)
    plain = [np.zeros(s.n) for _ in range(3)]
    locked = [torch.zeros(s.n, dtype=torch.float64).pin_memory().numpy() for _ in range(3)]
    a = e.evaluate(s.x, s.y, s.z, *plain)
    b = e.evaluate(s.x, s.y, s.z, *locked)
    assert a == b
    for x, y in zip(plain, locked):
        assert np.array_equal(x, y)
    e.close()


def test_threads(gpu):
    """Four engines in four threads: whoever finds the slots taken copies
    directly."""
    wrong = []

    def work(n, seed):
        s = _atoms(n, seed)
        e = _engine(s)
        for _ in range(20):
            for a, b in zip(e.positions(), (s.x, s.y, s.z)):
                if not np.array_equal(a, b):
                    wrong.append(n)
        e.close()

    ts = [threading.Thread(target=work, args=(n, n)) for n in (1000, 50001, 120000, 240001)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not wrong


@pytest.mark.parametrize("n", [1, 21845, 21846, 65536, 65537, 200003, 700001])
def test_round_trip_through_slots(gpu, n):
    """Past the results that are copied before the slots exist."""
    s = _atoms(n)
    e = _engine(s)
    for _ in range(12):
        for a, b in zip(e.positions(), (s.x, s.y, s.z)):
            assert np.array_equal(a, b)
    e.close()


@pytest.mark.parametrize("n", [16383, 16384, 16386, 70002])
def test_locked_and_pageable_in_one_result(gpu, n):
    """Arrays on either side of the 128 KB from which page-locked ones are
    written directly, past the results that are copied before the slots
    exist."""
    import torch
    s = _atoms(n)
    s.eps, s.sig = np.full(n, 1e-3), np.full(n, 1e-3)
    e = _engine(s)
    first = None
    for k in range(14):
        f = [torch.zeros(n, dtype=torch.float64).pin_memory().numpy() if (k >> a) & 1
             else np.zeros(n) for a in range(3)]
        en = e.evaluate(s.x, s.y, s.z, *f)
        if first is None:
            first = en, f
        assert en == first[0]
        for x, y in zip(f, first[1]):
            assert np.array_equal(x, y)
    e.close()


# three arrays in one slot, ending inside a slot, over several slots, in all of
# them, and in more than there are
@pytest.mark.parametrize("n", [1001, 21846, 70001, 680001, 710001])
def test_added_results(gpu, n):
    """Forces added to the caller's: the old value plus the result, once."""
    import ctypes as C
    s = _atoms(n)
    s.q = np.random.default_rng(2).uniform(-0.1, 0.1, n)
    _, *ref, _ = nb.spme(s, grid=(32, 32, 32), nbsp=4)
    assert np.abs(ref).max() > 0.0
    pbc = nb.make_pbc(s.cell())
    out = (C.c_double * 8)()
    before = np.random.default_rng(3).uniform(-100, 100, (3, n))
    hold = _engine(_atoms(1))  # the slots live
    for _ in range(12):
        f = [a.copy() for a in before]
        nb.check(nb.lib().mdbas_nb_spme(n, C.byref(pbc), 0.34, systems.CHARGE_CONST, 32, 32, 32, 4,
                                        *(nb._ptr(a) for a in (s.x, s.y, s.z, s.q, *f)), out, 0,
                                        None), "spme")
        for a, b, c in zip(f, before, ref):
            assert np.array_equal(a, b + c)
    hold.close()
