"""Frames and renormalisations further apart than one resident launch is long."""
import numpy as np
import pytest

from spp_gb300 import System, abi, configs

pytestmark = pytest.mark.gpu


def test_series_with_long_gaps(gpu_lib):
    n, every = 64, 40000
    p = configs.vicsek_config(n=n, L=4.0, eta=0.2, seed=4)
    state = configs.random_state(n, p.L, seed=4)
    with System(p) as s, System(p) as t:
        s.upload(*state)
        t.upload(*state)
        before = s.kernel_launches()
        P = s.polarization_series(2, every)[0]
        assert s.kernel_launches() - before >= 2 * every >> 14   # launches of a bounded length
        for f in range(2):
            for _ in range(8):
                t.step(every // 8)
            assert t.observables().polarization == P[f]
        for a, b in zip(s.download(), t.download()):
            assert np.array_equal(a, b)


@pytest.mark.parametrize("steps,every", [(17000, 16500), (700, 300), (513, 512), (512, 1000)])
def test_renormalisations_with_long_gaps(gpu_lib, monkeypatch, steps, every):
    """Against the step graphs, one of which holds all the steps up to a
    renormalisation (the flocks' growing lists overflow on the way: each
    recovery is a renormalisation too, at the same step in both)."""
    p = configs.lyapunov_config(n=60, integrator=abi.INT_RK2)
    p.Dr, p.skin = 0.02, 0.2   # rebuilds between the renormalisations
    state = configs.random_state(p.n, p.L, seed=7)
    got = []
    for resident in ("1", "0"):
        monkeypatch.setenv("SPP_RESIDENT", resident)
        with System(p) as s:
            s.upload(*state)
            s.lyap_init(3, seed=5)
            s.lyap_step(steps, every)
            s.lyap_step(7, 4)
            lam, T = s.lyap_exponents()
            o = s.observables()
            got.append((lam, s.lyap_vectors(), np.float64(T)) + s.download() + ((o.n_rebuilds, o.list_regrowths),))
    assert got[0][-1][0] >= 3
    for a, b in zip(*got):
        assert np.array_equal(a, b)
