"""The Vicsek step of systems too large for a resident run (k_vicsek_step,
reached here by switching resident runs off), bit for bit against the oracle:
three and four cells per side (every cell at an edge), odd grids, crowded and
empty cells, closed boxes, and a size past the resident ones."""
import numpy as np
import pytest

from oracle import oracle as O
from spp_gb300 import System, abi, configs

pytestmark = pytest.mark.gpu

MODELS = [abi.MODEL_VICSEK, abi.MODEL_VICSEK_REF_ANGLE, abi.MODEL_VICSEK_REF_VECTOR]


def check(p, steps, seed=8):
    x, y, th = configs.random_state(p.n, p.L, seed=seed)
    x[: p.n // 3] *= np.float32(0.1)         # a crowded strip
    with System(p) as s:
        s.upload(x, y, th)
        s.step(1)
        s.step(steps - 1)
        got = s.download()
    m = O.run32(p, O.State32(x, y, th), steps)
    for g, want in zip(got, (m.x, m.y, m.th, m.ix, m.iy)):
        assert np.array_equal(g, want)


@pytest.mark.parametrize("model", MODELS)
@pytest.mark.parametrize("n,D", [(1, 3), (40, 3), (300, 4), (257, 5), (2000, 31), (1500, 64)])
def test_grids(gpu_lib, monkeypatch, n, D, model):
    monkeypatch.setenv("SPP_RESIDENT", "0")
    p = configs.vicsek_config(n=n, L=0.5 * 1.001 * D + 0.01, eta=0.2, seed=6, model=model)
    if model == abi.MODEL_VICSEK_REF_VECTOR:
        p.r_push, p.beta_push = 0.8, 0.3
    check(p, 12)


def test_closed_box(gpu_lib, monkeypatch):
    monkeypatch.setenv("SPP_RESIDENT", "0")
    p = configs.vicsek_config(n=700, L=9.0, eta=0.2, seed=6, model=abi.MODEL_VICSEK_REF_ANGLE)
    p.boundary = abi.BOUNDARY_WALLS
    p.v0 = 0.1
    check(p, 12)


@pytest.mark.parametrize("model", MODELS)
def test_large_system(gpu_lib, model):
    p = configs.vicsek_config(n=180001, L=220.0, eta=0.3, seed=6, model=model)
    check(p, 4)
