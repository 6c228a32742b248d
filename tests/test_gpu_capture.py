"""Steps on a stream that is being captured: small Vicsek systems are recorded
and replayed, other systems refused without harm."""
import numpy as np
import pytest

from spp_gb300 import System, abi, configs

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def on_stream(s):
    torch.cuda.init()
    st = torch.cuda.Stream()
    abi.check(abi.lib().spp_set_stream(s.handle, st.cuda_stream), "spp_set_stream")
    return st


def capture(s, st, steps):
    """(graph, status of spp_step) of a capture of `steps` steps."""
    g = torch.cuda.CUDAGraph()
    st.wait_stream(torch.cuda.current_stream())
    with torch.cuda.graph(g, stream=st, capture_error_mode="relaxed"):
        rc = abi.lib().spp_step(s.handle, steps)
    return g, rc


def small(n, D, model):
    return n <= 16384 and D * D < 65536 and (24 if model == abi.MODEL_VICSEK_REF_ANGLE else 20) * n + 8 * D * D <= 229376


@pytest.mark.parametrize("model", [abi.MODEL_VICSEK, abi.MODEL_VICSEK_REF_ANGLE, abi.MODEL_VICSEK_REF_VECTOR])
@pytest.mark.parametrize("n,L", [(1, 4.0), (4096, 32.0), (9000, 30.0), (9100, 47.3), (9600, 40.0), (11400, 9.0),
                                 (11500, 9.0), (100, 84.0), (100, 86.0), (16384, 64.0), (50001, 111.0)])
@pytest.mark.filterwarnings("ignore:The CUDA Graph is empty")
def test_vicsek(gpu_lib, n, L, model):
    p = configs.vicsek_config(n=n, L=L, eta=0.3, seed=5, model=model)
    state = configs.random_state(n, L, seed=5)
    with System(p) as s, System(p) as t:
        st = on_stream(s)
        s.upload(*state)
        t.upload(*state)
        g, rc = capture(s, st, 5)
        taken = small(n, int(2 * L / 1.001), model)
        assert rc == (0 if taken else 3)
        if taken:
            for _ in range(3):
                g.replay()
            torch.cuda.synchronize()
            t.step(15)
        else:   # neither handle is the worse for it
            s.upload(*state)
            s.step(15)
            t.step(15)
        assert s.observables().step == 15
        for a, b in zip(s.download(), t.download()):
            assert np.array_equal(a, b)
        del g


@pytest.mark.parametrize("n", [2000, 200000])
@pytest.mark.filterwarnings("ignore:The CUDA Graph is empty")
def test_list_systems_are_refused(gpu_lib, n):
    p = configs.abp_config(n=n, L=0.5 * n ** 0.5)
    state = configs.random_state(n, p.L, seed=5)
    with System(p) as s, System(p) as t:
        st = on_stream(s)
        s.upload(*state)
        s.step(2)
        s.sync()
        g, rc = capture(s, st, 3)
        assert rc == 3
        s.upload(*state)
        t.upload(*state)
        s.step(4)
        t.step(4)
        for a, b in zip(s.download(), t.download()):
            assert np.array_equal(a, b)
        del g
