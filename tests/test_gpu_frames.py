"""Frames in and out of a system, through its pinned block (up to 16,384
particles) and straight to the caller's memory: what goes in comes out, with
either, both or none of the box-crossing counters."""
import numpy as np
import pytest

from spp_gb300 import System, configs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 16383, 16384, 16385])
@pytest.mark.parametrize("given", ["none", "x", "y", "both"])
def test_round_trip(gpu_lib, n, given):
    L = max(4.0, 0.5 * n ** 0.5)
    p = configs.abp_config(n=n, L=L)
    x, y, th = configs.random_state(n, L, seed=5)
    g = np.random.default_rng(n)
    ix = g.integers(-9, 9, n).astype(np.int32) if given in ("x", "both") else None
    iy = g.integers(-9, 9, n).astype(np.int32) if given in ("y", "both") else None
    with System(p) as s:
        for _ in range(2):   # the second upload finds the block used
            s.upload(x, y, th, step0=3, img_x=ix, img_y=iy)
            got = s.download()
            want = (x, y, th, np.zeros(n, np.int32) if ix is None else ix, np.zeros(n, np.int32) if iy is None else iy)
            for a, b in zip(got, want):
                assert np.array_equal(a, b)
            assert s.observables().step == 0
            s.step(3)
        assert s.observables().step == 3


def test_frame_after_a_recovery(gpu_lib):
    """The list overflows behind an unsynchronised frame: the frame and the
    polarization are those of the finished steps."""
    p = configs.abp_config(n=3000, L=22.0)
    st = configs.random_state(p.n, p.L, seed=4)
    out = []
    for cap in (8, 64):
        p.list_capacity = cap
        with System(p) as s:
            s.upload(*st)
            s.step(60)
            frame = s.download()
            s.step(30)
            o = s.observables()
            out.append((frame, o.polarization, o.step, s.download()))
    (fa, pa, sa, ea), (fb, pb, sb, eb) = out
    assert pa == pb and sa == sb == 90
    for a, b in zip(fa + ea, fb + eb):
        assert np.array_equal(a, b)
