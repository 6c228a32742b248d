"""Calls on one handle while another handle works: a long resident run is cut
into launches short enough to let others in."""
import time

import pytest

from spp_gb300 import System, configs

pytestmark = pytest.mark.gpu


def vicsek(n):
    p = configs.vicsek_config(n=n, L=0.5 * n ** 0.5, eta=0.3, seed=1)
    s = System(p)
    s.upload(*configs.random_state(n, p.L, seed=1))
    s.step(2)
    s.observables()   # kernels loaded
    return s


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
