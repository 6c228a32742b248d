"""Dilute Vicsek systems: the cell buckets of a resident run shrink with the
number of cells, down to the multi-kernel step where even small ones would
hold memory by the box's area; the bits stay, in flocks that overflow every
bucket too."""
import numpy as np
import pytest

from spp_gb300 import System, abi, configs

pytestmark = pytest.mark.gpu


def flocks(n, L, seed):
    g = np.random.default_rng(seed)
    c = (2 * g.random((3, 1 + n // 60)) - 1) * np.array([[L], [L], [3.1]])
    q = g.integers(0, c.shape[1], n)
    x, y = (c[k, q] + 0.6 * g.standard_normal(n) for k in (0, 1))
    x, y = (((v + L) % (2 * L) - L).astype(np.float32) for v in (x, y))
    return (np.where(x >= np.float32(L), -np.float32(L), x), np.where(y >= np.float32(L), -np.float32(L), y),
            c[2, q].astype(np.float32))


@pytest.mark.parametrize("model", [abi.MODEL_VICSEK, abi.MODEL_VICSEK_REF_ANGLE, abi.MODEL_VICSEK_REF_VECTOR])
@pytest.mark.parametrize("n,L,resident", [(3000, 100.0, True), (3000, 150.0, True), (3000, 240.0, True),
                                          (3000, 350.0, True), (3000, 420.0, False), (60000, 300.0, True)])
def test_bits(gpu_lib, monkeypatch, n, L, resident, model):
    p = configs.vicsek_config(n=n, L=L, eta=0.1, seed=3, model=model)
    got = []
    for on in ("1", "0"):
        monkeypatch.setenv("SPP_RESIDENT", on)
        with System(p) as s:
            s.upload(*flocks(n, L, 3))
            s.step(20)
            s.sync()
            assert (s.resident_launches() > 0) == (on == "1" and resident)
            got.append(s.download())
    for a, b in zip(*got):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("model", [abi.MODEL_VICSEK, abi.MODEL_VICSEK_REF_ANGLE])
@pytest.mark.parametrize("n,L", [(3000, 420.0), (3000, 350.0), (1000, 900.0), (20000, 400.0)])
def test_memory(gpu_lib, n, L, model):
    """At most 128 bucket places of 40 bytes per particle or 2 million in all,
    next to the cell counts (8 bytes per key, up to 4 keys a cell, and 12 a cell)
    and the particles."""
    torch = pytest.importorskip("torch")
    p = configs.vicsek_config(n=n, L=L, eta=0.3, seed=1, model=model)
    state = configs.random_state(n, L, seed=1)
    with System(p) as s:   # kernels loaded
        s.upload(*state)
        s.step(1)
        s.sync()
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    with System(p) as s:
        s.upload(*state)
        used = free - torch.cuda.mem_get_info()[0]
    cells = (2 * L) ** 2
    assert used < 40 * max(128 * n, 2 << 20) + 44 * cells + 400 * n + (8 << 20)


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
