"""Resident runs (k_run: many steps in one cooperative launch) against the
step graphs, bit for bit, where the launch shape, the list and the barrier
bookkeeping can go wrong: sizes around the edges of blocks and of the
one- and two-blocks-per-SM shapes, the Euler step's alternating buffers,
overflowing and very long lists, and calls of a single step."""
import numpy as np
import pytest

from spp_gb300 import System, abi, configs

pytestmark = pytest.mark.gpu


def run(p, state, chunks, monkeypatch, resident):
    monkeypatch.setenv("SPP_RESIDENT", "1" if resident else "0")
    with System(p) as s:
        s.upload(*state)
        for c in chunks:
            s.step(c)
        out = s.download()
        o = s.observables()
    return out, (o.step, o.n_rebuilds, o.late_rebuilds, o.list_regrowths, o.max_neighbors)


def check(p, state, chunks, monkeypatch):
    a, oa = run(p, state, chunks, monkeypatch, True)
    b, ob = run(p, state, chunks, monkeypatch, False)
    for u, v in zip(a, b):
        assert np.array_equal(u, v)
    assert oa == ob
    return oa


@pytest.mark.parametrize("n", [1, 31, 33, 4096, 16384, 16385, 97280, 97281, 175104, 175105])
@pytest.mark.parametrize("integrator", [abi.INT_EULER, abi.INT_RK2, abi.INT_RK4])
def test_sizes(gpu_lib, monkeypatch, n, integrator):
    L = max(4.0, 0.5 * n ** 0.5)
    p = configs.abp_config(n=n, L=L, integrator=integrator)
    check(p, configs.random_state(n, L, seed=2), (1, 23), monkeypatch)


@pytest.mark.parametrize("rings,swimmers", [(3, 2), (40, 0), (1024, 32)])
def test_vesicles(gpu_lib, monkeypatch, rings, swimmers):
    p = configs.vesicle_config(n_rings=rings, swimmers_per_ring=swimmers)
    p.skin = 0.05   # rebuilds within the run, where swimmers move (the rings start at rest)
    rebuilds = check(p, configs.vesicle_state(p), (25,), monkeypatch)[1]
    assert rebuilds >= 2 or swimmers == 0


@pytest.mark.parametrize("lanes", [1, 4])
@pytest.mark.parametrize("n", [17, 100, 700])
def test_long_lists(gpu_lib, monkeypatch, n, lanes):
    """Every particle is every other's neighbour: lists of n - 1 entries, past
    the in-block sort, past the entries kept in shared memory and past the
    warp's sort; the first capacity overflows and grows."""
    p = configs.lyapunov_config(n=n + 8)
    p.L, p.gather_lanes, p.skin = 16.0, lanes, 0.02
    g = np.random.default_rng(n)
    xy = (0.4 * g.random((2, n + 8))).astype(np.float32)
    xy[:, n:] += 5.0
    th = g.random(n + 8).astype(np.float32)
    o = check(p, (xy[0], xy[1], th), (1, 12), monkeypatch)
    assert o[4] == n - 1 and o[1] >= 2


def test_overflow_inside_a_run(gpu_lib, monkeypatch):
    p = configs.abp_config(n=3000, L=22.0)
    p.list_capacity = 8
    o = check(p, configs.random_state(p.n, p.L, seed=4), (60,), monkeypatch)
    assert o[3] >= 1
