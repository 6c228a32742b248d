"""Resident Lyapunov runs (k_lrun) against the step graphs with their
renormalisation kernels, bit for bit: numbers of vectors around its groups
of four, one and four threads per particle, sizes around the launch shape's
edge, chunks that do not divide the run, rebuilds and overflowing lists
between renormalisations."""
import numpy as np
import pytest

from spp_gb300 import System, abi, configs

pytestmark = pytest.mark.gpu


def run(p, state, K, calls, monkeypatch, resident):
    monkeypatch.setenv("SPP_RESIDENT", "1" if resident else "0")
    with System(p) as s:
        s.upload(*state)
        s.lyap_init(K, seed=5)
        for steps, every in calls:
            s.lyap_step(steps, every)
        lam, T = s.lyap_exponents()
        o = s.observables()
        return (lam, s.lyap_vectors()) + s.download() + ((T, o.step, o.n_rebuilds, o.list_regrowths),)


def check(p, state, K, calls, monkeypatch):
    a = run(p, state, K, calls, monkeypatch, True)
    b = run(p, state, K, calls, monkeypatch, False)
    for u, v in zip(a, b):
        assert np.array_equal(u, v)
    return a[-1]


@pytest.mark.parametrize("integrator", [abi.INT_RK2, abi.INT_RK4])
@pytest.mark.parametrize("K", [1, 3, 4, 5, 8])
@pytest.mark.parametrize("n,lanes", [(150, 4), (150, 1), (2500, 4), (2500, 1)])
def test_vectors(gpu_lib, monkeypatch, n, lanes, K, integrator):
    p = configs.lyapunov_config(n=n, integrator=integrator)
    p.gather_lanes, p.skin, p.Dr = lanes, 0.05, 0.02   # rebuilds within the run
    o = check(p, configs.random_state(n, p.L, seed=7), K, [(13, 5), (1, 3), (4, 4)], monkeypatch)
    assert o[2] >= 2


@pytest.mark.parametrize("n", [16384, 16385, 58368, 58369])
def test_sizes(gpu_lib, monkeypatch, n):
    p = configs.lyapunov_config(n=n)
    check(p, configs.random_state(n, p.L, seed=7), 8, [(6, 4)], monkeypatch)


@pytest.mark.parametrize("lanes", [1, 4])
@pytest.mark.parametrize("steps,every", [(40, 1), (40, 7), (41, 10)])
def test_overflow(gpu_lib, monkeypatch, lanes, steps, every):
    """Four places per list at first: overflows at the upload and again as the
    flocks condense, at any place within a chunk."""
    n = 1500
    p = configs.lyapunov_config(n=n)
    p.list_capacity, p.gather_lanes, p.skin, p.v0 = 4, lanes, 0.1, 2.0
    g = np.random.default_rng(1)
    x, y, th = configs.random_state(n, p.L, seed=7)
    c = n // 3                                    # a third converges on a point
    ang = 2 * np.pi * g.random(c)
    r = 1.5 + 2.0 * g.random(c)
    x[:c], y[:c] = r * np.cos(ang), r * np.sin(ang)
    th[:c] = np.arctan2(-y[:c], -x[:c])
    o = check(p, (x, y, th.astype(np.float32)), 4, [(steps, every), (steps, every)], monkeypatch)
    assert o[3] >= 2
