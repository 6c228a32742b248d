"""Neighbour lists past the 512 entries that are sorted on chip (clumps, which
the models without repulsion allow): in id order, so the trajectory is the
oracle's bit for bit, and soon enough that no block of a resident run gives
up waiting for the others."""
import time

import numpy as np
import pytest

from oracle import oracle as O
from spp_gb300 import System, abi, configs

pytestmark = pytest.mark.gpu


def clump(n, m, L, seed):
    """m particles within a list radius of each other, n - m spread out; ids mixed."""
    g = np.random.default_rng(seed)
    xy = (2 * g.random((n, 2)) - 1) * L
    xy[:m] = 0.4 * g.random((m, 2)) - 0.7 * L
    xy = xy[g.permutation(n)].astype(np.float32)
    return xy[:, 0].copy(), xy[:, 1].copy(), (6.28 * g.random(n) - 3.14).astype(np.float32)


@pytest.mark.parametrize("resident", ["1", "0"])
@pytest.mark.parametrize("lanes", [1, 4])
@pytest.mark.parametrize("m", [512, 513, 514, 1023, 1025, 1600])
def test_order(gpu_lib, monkeypatch, m, lanes, resident):
    monkeypatch.setenv("SPP_RESIDENT", resident)
    n = m + 60
    p = configs.lyapunov_config(n=n, integrator=abi.INT_RK2)
    p.L, p.gather_lanes, p.skin = 16.0, lanes, 0.02
    state = clump(n, m, p.L, m)
    with System(p) as s:
        s.upload(*state)
        assert s.observables().max_neighbors >= m - 1
        s.step(8)
        got = s.download()
        assert s.observables().n_rebuilds >= 2
    want = O.run32(p, O.State32(*state), 8)
    for g, w in zip(got, (want.x, want.y, want.th, want.ix, want.iy)):
        assert np.array_equal(g, w)


def test_large_clump_in_a_resident_run(gpu_lib, monkeypatch):
    """5,000 of 16,384 particles in one clump: an insertion sort of one such
    list takes longer than a barrier of the resident run waits."""
    n, m = 16384, 5000
    p = configs.lyapunov_config(n=n, integrator=abi.INT_RK2)
    p.skin = 0.02
    state = clump(n, m, p.L, 1)
    got = []
    for resident in ("1", "0"):
        monkeypatch.setenv("SPP_RESIDENT", resident)
        with System(p) as s:
            s.upload(*state)
            t = time.perf_counter()
            s.step(6)
            s.sync()
            assert time.perf_counter() - t < 2.0
            o = s.observables()
            assert o.n_rebuilds >= 2 and o.max_neighbors >= m - 1
            got.append(s.download())
    for a, b in zip(*got):
        assert np.array_equal(a, b)
