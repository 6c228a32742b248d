"""Resident Vicsek runs (k_vrun) against the multi-kernel step, bit for bit:
sizes around the edges of its launch shapes (4, 2 and 1 threads per
particle, one and two blocks per SM), cells beyond their buckets, runs past
the owners' sort, and series recorded inside one launch."""
import numpy as np
import pytest

from spp_gb300 import System, abi, configs

pytestmark = pytest.mark.gpu

MODELS = [abi.MODEL_VICSEK, abi.MODEL_VICSEK_REF_ANGLE, abi.MODEL_VICSEK_REF_VECTOR]


def run(p, state, chunks, series, monkeypatch, resident):
    monkeypatch.setenv("SPP_RESIDENT", "1" if resident else "0")
    with System(p) as s:
        s.upload(*state)
        for c in chunks:
            s.step(c)
        P = s.polarization_series(*series) if series else ()
        return s.download() + tuple(P) + (s.observables().step,)


def check(p, state, chunks, monkeypatch, series=None):
    a = run(p, state, chunks, series, monkeypatch, True)
    b = run(p, state, chunks, series, monkeypatch, False)
    for u, v in zip(a, b):
        assert np.array_equal(u, v)


@pytest.mark.parametrize("model", MODELS)
@pytest.mark.parametrize("n", [1, 33, 5000, 24320, 24321, 43776, 43777, 48640, 48641, 87552, 87553, 97281, 175104,
                               175105])
def test_sizes(gpu_lib, monkeypatch, n, model):
    L = max(4.0, 0.5 * n ** 0.5)
    p = configs.vicsek_config(n=n, L=L, eta=0.25, seed=2, model=model)
    check(p, configs.random_state(n, L, seed=2), (1, 18), monkeypatch)


@pytest.mark.parametrize("model", MODELS)
@pytest.mark.parametrize("L", [1.6, 9.0])
@pytest.mark.parametrize("n", [700, 30000])
def test_full_buckets(gpu_lib, monkeypatch, n, L, model):
    """Every cell far beyond its bucket (three cells per side: every cell is a
    neighbour of every other, across the edges too)."""
    if n * n / (L * L) > 1e8:
        n = 3000
    p = configs.vicsek_config(n=n, L=L, eta=0.1, seed=3, model=model)
    p.v0 = 0.2
    check(p, configs.random_state(n, L, seed=3), (1, 20), monkeypatch)


@pytest.mark.parametrize("n,frames,every", [(600, 7, 1), (5000, 5, 3), (60000, 3, 17)])
def test_series(gpu_lib, monkeypatch, n, frames, every):
    p = configs.vicsek_config(n=n, L=0.5 * n ** 0.5, eta=0.2, seed=4)
    check(p, configs.random_state(n, p.L, seed=4), (2,), monkeypatch, series=(frames, every))
