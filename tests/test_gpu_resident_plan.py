"""Which systems run resident (one cooperative launch for many steps) and which
step through graphs: the comparisons of the two elsewhere mean something only
where the first is really taken."""
import numpy as np
import pytest

from spp_gb300 import System, abi, configs, surrogate

pytestmark = pytest.mark.gpu

CHUNK = 256   # steps of a resident launch at most


def launches(s, steps, call):
    r0, k0 = s.resident_launches(), s.kernel_launches()
    call(steps)
    s.sync()
    return s.resident_launches() - r0, s.kernel_launches() - k0


@pytest.mark.parametrize("env", ["", "SPP_RESIDENT", "SPP_NO_GRAPHS"])
@pytest.mark.parametrize("n,fits", [(1, True), (31, True), (16384, True), (16385, True), (97280, True), (97281, True),
                                    (175104, True), (175105, False)])
@pytest.mark.parametrize("integrator", [abi.INT_EULER, abi.INT_RK4])
def test_disks(gpu_lib, monkeypatch, n, fits, integrator, env):
    if env:
        monkeypatch.setenv(env, "0" if env == "SPP_RESIDENT" else "1")
    p = configs.abp_config(n=n, L=max(4.0, 0.5 * n ** 0.5), integrator=integrator)
    with System(p) as s:
        s.upload(*configs.random_state(n, p.L, seed=2))
        steps = 20 if env == "SPP_NO_GRAPHS" else CHUNK + 5
        resident, passes = launches(s, steps, s.step)
        assert resident == (2 if fits and not env else 0)
        assert passes >= steps * (2 if integrator == abi.INT_EULER else 4)


@pytest.mark.parametrize("model", [abi.MODEL_VICSEK, abi.MODEL_VICSEK_REF_ANGLE, abi.MODEL_VICSEK_REF_VECTOR])
@pytest.mark.parametrize("n,fits", [(1, True), (16384, True), (16385, True), (24321, True), (48641, True),
                                    (87552, True), (97280, True), (175105, False)])
def test_vicsek(gpu_lib, monkeypatch, n, fits, model):
    p = configs.vicsek_config(n=n, L=max(4.0, 0.5 * n ** 0.5), eta=0.3, seed=2, model=model)
    for off in (False, True):
        if off:
            monkeypatch.setenv("SPP_RESIDENT", "0")
        with System(p) as s:
            s.upload(*configs.random_state(n, p.L, seed=2))
            resident, passes = launches(s, CHUNK + 5, s.step)
            assert resident == (2 if fits and not off else 0)
            assert passes == (CHUNK + 5) * 5
            resident, passes = launches(s, 3, lambda k: s.polarization_series(k, 2))
            assert resident == (1 if fits and not off else 0)
            assert passes == 6 * 5 + 3


@pytest.mark.parametrize("n,lanes,fits", [(150, 4, True), (150, 1, True), (16384, 0, True), (19456, 4, True),
                                          (19457, 4, False), (58368, 1, True), (58369, 1, False)])
def test_lyapunov(gpu_lib, monkeypatch, n, lanes, fits):
    p = configs.lyapunov_config(n=n)
    p.gather_lanes = lanes
    for off in (False, True):
        if off:
            monkeypatch.setenv("SPP_RESIDENT", "0")
        with System(p) as s:
            s.upload(*configs.random_state(n, p.L, seed=2))
            s.lyap_init(8, seed=1)
            resident, passes = launches(s, 25, lambda k: s.lyap_step(k, 10))
            assert resident == (1 if fits and not off else 0)
            assert passes >= 25 * 9 + 3 * 6


def test_vesicles(gpu_lib):
    p = configs.vesicle_config(n_rings=20, swimmers_per_ring=4)
    with System(p) as s:
        s.upload(*configs.vesicle_state(p))
        assert launches(s, 7, s.step)[0] == 1


def test_training(gpu_lib, monkeypatch):
    g = np.random.default_rng(0)
    x, t = g.standard_normal((300, 7)).astype(np.float32), g.random(300).astype(np.float32)
    for env, value, want in (("SPP_MLP_CLUSTER", "1", 4), ("SPP_MLP_CLUSTER", "0", 0), ("SPP_MLP_SCALAR", "1", 0)):
        monkeypatch.setenv(env, value)
        m = surrogate.Mlp(ensemble=5, seed=1)
        m.train(x, t, iters=333)
        m.train(x, t, iters=334)
        m.train(x, t, iters=1)
        assert m.resident_launches() == want
        m.close()
