"""Resident Vicsek runs driven by short calls: the owners are sorted in some of
them only, a launch goes on with the counts that the one before left, and the
bits are those of the multi-kernel step."""
import time

import numpy as np
import pytest

from spp_gb300 import System, abi, configs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("model", [abi.MODEL_VICSEK, abi.MODEL_VICSEK_REF_ANGLE, abi.MODEL_VICSEK_REF_VECTOR])
@pytest.mark.parametrize("n,calls,step0", [(5000, [16] * 5, 0), (5000, [1] * 40, 3), (60000, [8] * 5 + [17, 1], 0),
                                           (120000, [16, 16, 5], (1 << 32) - 60)])
def test_short_calls(gpu_lib, monkeypatch, n, calls, step0, model):
    p = configs.vicsek_config(n=n, L=0.5 * n ** 0.5, eta=0.2, seed=6, model=model)
    state = configs.random_state(n, p.L, seed=6)
    got = []
    for resident in ("1", "0"):
        monkeypatch.setenv("SPP_RESIDENT", resident)
        with System(p) as s:
            s.upload(*state, step0=step0)
            for c in calls:
                s.step(c)
            got.append(s.download() + (s.observables().step,))
    for a, b in zip(*got):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("model", [abi.MODEL_VICSEK, abi.MODEL_VICSEK_REF_ANGLE, abi.MODEL_VICSEK_REF_VECTOR])
def test_counts_carried_from_call_to_call(gpu_lib, monkeypatch, model):
    """Calls of every length modulo the three counts, full buckets in some of
    the steps, series and uploads in between."""
    n = 3000
    p = configs.vicsek_config(n=n, L=25.0, eta=0.2, seed=6, model=model)
    spread = configs.random_state(n, p.L, seed=6)
    clump = tuple(np.float32(0.1) * v for v in spread[:2]) + (spread[2],)
    got = []
    for resident in ("1", "0"):
        monkeypatch.setenv("SPP_RESIDENT", resident)
        out = []
        with System(p) as s:
            for state in (spread, clump, spread):
                s.upload(*state)
                for c in (1, 2, 3, 4, 5, 1, 1, 7):
                    s.step(c)
                    out += s.polarization_series(2, c)
                out += s.download()
        got.append(out)
    for a, b in zip(*got):
        assert np.array_equal(a, b)


def test_cost_of_a_call(gpu_lib):
    """Launch and start of a run of one step, in steps of a long run: two
    barriers more than now (2.4 steps) were more than the launch of the kernel
    that this one replaced."""
    p = configs.vicsek_config(n=300, L=9.0, eta=0.3, seed=1)
    with System(p) as s:
        s.upload(*configs.random_state(300, p.L, seed=1))

        def best(calls, steps):
            r = []
            for _ in range(20):
                s.sync()
                t = time.perf_counter()
                for _ in range(calls):
                    s.step(steps)
                s.sync()
                r.append((time.perf_counter() - t) / calls)
            return min(r)
        assert best(100, 1) < 2.2 * best(5, 200) / 200
