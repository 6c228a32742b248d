"""Pair histograms at the edges of their kernel (k_obs_hist) against the FP32
mirror, count for count: three cells per side (every cell adjacent to every
other across the boundary), one bin, more copies or bins than shared memory
takes, grids larger than the system's own, and particles on bin edges."""
import numpy as np
import pytest

from oracle import oracle as O
from spp_gb300 import System, configs

pytestmark = pytest.mark.gpu


def frame(n, L, seed, lattice=False):
    g = np.random.default_rng(seed)
    if lattice:
        # separations that fall on bin edges (multiples of 1/4)
        m = int(np.ceil(np.sqrt(n)))
        k = np.arange(m * m)[:n]
        x = (-L + 0.25 + 0.25 * (k % m)).astype(np.float32)
        y = (-L + 0.25 + 0.25 * (k // m)).astype(np.float32)
        return x, y, (np.pi / 4 * g.integers(-4, 4, n)).astype(np.float32)
    x = (g.random(n) * 2 * L - L).astype(np.float32)
    y = (g.random(n) * 2 * L - L).astype(np.float32)
    x[: n // 2] *= np.float32(0.25)   # half the particles four times as close
    x = np.where(x >= np.float32(L), -np.float32(L), x)
    y = np.where(y >= np.float32(L), -np.float32(L), y)
    return x, y, (g.random(n) * 6 - 3).astype(np.float32)


@pytest.mark.parametrize("n,L,lattice", [(1, 6.0, False), (65, 6.0, False), (1000, 8.0, True), (3000, 12.0, False)])
@pytest.mark.parametrize("r,nbins", [("max", 50), (2.0, 1), (2.0, 4), (2.0, 4096), (0.05, 7)])
def test_radial(gpu_lib, n, L, lattice, r, nbins):
    x, y, th = frame(n, L, n, lattice)
    r = 2 * L / 3.01 if r == "max" else r
    with System(configs.vicsek_config(n=n, L=L)) as s:
        s.upload(x, y, th)
        for _ in range(2):   # the scratch is used again
            assert np.array_equal(s.radial_distribution(r, nbins), O.radial32(x, y, L, r, nbins))


@pytest.mark.parametrize("n,L,lattice", [(1, 6.0, False), (65, 6.0, False), (1000, 8.0, True), (3000, 12.0, False)])
@pytest.mark.parametrize("lx,ly,gx,gy", [(1.0, 2.0, 8, 16), (2.5, 2.5, 1, 1), (2.0, 2.0, 256, 256), (0.03, 0.04, 5, 3),
                                         (1.5, 1.0, 200, 250)])
def test_body_frame(gpu_lib, n, L, lattice, lx, ly, gx, gy):
    x, y, th = frame(n, L, n, lattice)
    c, sn = O.math32("cos", th), O.math32("sin", th)
    with System(configs.vicsek_config(n=n, L=L)) as s:
        s.upload(x, y, th)
        got = s.pair_distribution(lx, ly, gx, gy)
    assert np.array_equal(got, O.pair_distribution32(x, y, c, sn, lx, ly, gx, gy))


def test_radial_on_a_grid_of_many_cells(gpu_lib):
    """17.6 million cells: more tiles of the scan than one block scans."""
    L, n = 420.0, 3000
    g = np.random.default_rng(5)
    c = (g.random((n // 3, 2)) * 2 * L - L)
    xy = (np.concatenate([c, c + 0.05 + 0.1 * g.random(c.shape), c - 0.1 * g.random(c.shape)])).astype(np.float32)
    xy = np.clip(xy, -L, np.nextafter(np.float32(L), np.float32(0.0)))
    x, y = np.ascontiguousarray(xy[:, 0]), np.ascontiguousarray(xy[:, 1])
    want = O.radial32(x, y, L, 0.2, 7)
    assert want.sum() > n / 2
    with System(configs.vicsek_config(n=n, L=L)) as s:
        s.upload(x, y, np.zeros(n, np.float32))
        assert np.array_equal(s.radial_distribution(0.2, 7), want)


@pytest.mark.parametrize("gx,gy", [(65536, 1), (1, 65536), (58109, 1), (58110, 1), (1, 58111)])
def test_body_frame_on_a_thin_grid(gpu_lib, gx, gy):
    """The most bins a grid may have, all on one side: more edges than shared
    memory holds (and the last that it holds)."""
    n, L = 500, 8.0
    x, y, th = frame(n, L, 3)
    c, sn = O.math32("cos", th), O.math32("sin", th)
    with System(configs.vicsek_config(n=n, L=L)) as s:
        s.upload(x, y, th)
        got = s.pair_distribution(2.0, 1.5, gx, gy)
    assert np.array_equal(got, O.pair_distribution32(x, y, c, sn, 2.0, 1.5, gx, gy))
