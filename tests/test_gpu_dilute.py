"""Dilute Vicsek systems, whose cells are many for their particles."""
import numpy as np
import pytest

from spp_gb300 import System, abi, configs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("model", [abi.MODEL_VICSEK, abi.MODEL_VICSEK_REF_ANGLE, abi.MODEL_VICSEK_REF_VECTOR])
def test_more_cells_than_buckets_are_kept_for(gpu_lib, monkeypatch, model):
    """4.8 million cells: the step kernels, with the resident run refused by its
    plan or by the environment."""
    n, L = 1000, 1100.0
    p = configs.vicsek_config(n=n, L=L, eta=0.1, seed=3, model=model)
    state = configs.random_state(n, 3.0, seed=3)
    got = []
    for on in ("1", "0"):
        monkeypatch.setenv("SPP_RESIDENT", on)
        with System(p) as s:
            s.upload(*state)
            s.step(20)
            P = s.polarization_series(3, 2)[0]
            assert s.resident_launches() == 0
            got.append(s.download() + (P,))
    for a, b in zip(*got):
        assert np.array_equal(a, b)
