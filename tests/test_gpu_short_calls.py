"""Resident Vicsek runs driven by short calls: the owners are sorted in some of
them only, and the bits are those of the multi-kernel step."""
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
