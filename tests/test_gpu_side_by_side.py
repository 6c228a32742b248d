"""Calls on one handle while another handle works: a long training or a long
resident run is cut into launches short enough to let others in."""
import threading
import time

import numpy as np
import pytest

from spp_gb300 import System, configs, surrogate

pytestmark = pytest.mark.gpu


def vicsek(n):
    p = configs.vicsek_config(n=n, L=0.5 * n ** 0.5, eta=0.3, seed=1)
    s = System(p)
    s.upload(*configs.random_state(n, p.L, seed=1))
    s.step(2)
    s.observables()   # kernels loaded
    return s


def fit_data(E, B, iters, seed=0):
    g = np.random.default_rng(seed)
    return (g.standard_normal((B, 7)).astype(np.float32), g.random(B).astype(np.float32)), dict(iters=iters)


def test_step_beside_a_training(gpu_lib):
    m = surrogate.Mlp(ensemble=5, seed=1)
    data, kw = fit_data(5, 300, 60000)
    m.train(*data, iters=300)
    with vicsek(50001) as s:
        th = threading.Thread(target=lambda: m.train(*data, **kw))
        th.start()
        time.sleep(0.3)
        t = time.perf_counter()
        s.step(20)
        s.observables()
        t = time.perf_counter() - t
        assert th.is_alive() and t < 0.2
        th.join()


def test_step_beside_a_long_run(gpu_lib):
    n = 16384
    p = configs.abp_config(n=n, L=64.0)
    with System(p) as big, vicsek(50001) as s:
        big.upload(*configs.random_state(n, p.L, seed=1))
        big.step(100)
        big.observables()
        big.step(120000)   # about a second
        t = time.perf_counter()
        s.step(2)
        s.observables()
        t = time.perf_counter() - t
        left = time.perf_counter()
        big.sync()
        left = time.perf_counter() - left
        assert t < 0.05 and left > 0.2


def test_training_in_several_launches(gpu_lib, monkeypatch):
    """More iterations than one launch holds: the parameters are those of the
    iteration graphs, bit for bit."""
    got = []
    for cluster in ("1", "0"):
        monkeypatch.setenv("SPP_MLP_CLUSTER", cluster)
        for E, B, iters in ((5, 300, 700), (2, 40, 1001), (6, 3000, 60)):
            m = surrogate.Mlp(ensemble=E, seed=3)
            data, kw = fit_data(E, B, iters, seed=E)
            loss = m.train(*data, lr=2e-3, **kw)
            got.append((np.asarray(loss), m.params()))
    for a, b in zip(got[:3], got[3:]):
        for u, v in zip(a, b):
            assert np.array_equal(u, v)
