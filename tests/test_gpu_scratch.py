"""Sums of a call in scratch that the system keeps: series, histograms, ring
shapes and motions in any order use it again, and a series does not pay for an
allocation."""
import time

import numpy as np
import pytest

from spp_gb300 import System, configs

pytestmark = pytest.mark.gpu


def test_scratch_is_shared_in_any_order(gpu_lib):
    p = configs.vesicle_config(n_rings=30, swimmers_per_ring=6)
    state = configs.vesicle_state(p)
    with System(p) as s:
        def shapes():
            return np.stack(list(s.ring_shapes().values()))

        def motion():
            s.upload(*state)
            s.ring_motion_mark()
            s.step(3)
            return np.stack(list(s.ring_motion().values()))

        def series(frames):
            s.upload(*state)
            return np.concatenate(s.polarization_series(frames, 1))
        calls = {"shapes": shapes, "motion": motion, "g": lambda: s.radial_distribution(3.0, 40),
                 "body": lambda: s.pair_distribution(2.0, 2.0, 30, 30), "short": lambda: series(2), "long": lambda: series(300)}
        s.upload(*state)
        want = {}
        for order in (list(calls), list(calls)[::-1], ["long", "g", "short", "shapes", "body", "motion"]):
            for name in order:
                s.upload(*state)
                got = calls[name]()
                assert np.array_equal(want.setdefault(name, got), got), name


def test_series_longer_than_the_scratch(gpu_lib):
    p = configs.vicsek_config(n=16, L=3.0, eta=0.5, seed=1)
    frames = (1 << 19) + 3
    state = configs.random_state(16, p.L, seed=1)
    with System(p) as s, System(p) as t:
        s.upload(*state)
        t.upload(*state)
        P = s.polarization_series(frames, 1)[0]
        t.step(frames - 1)
        assert t.polarization_series(1, 1)[0][0] == P[-1]


def test_cost_of_a_series(gpu_lib):
    """Frames of a series against steps and waits alone (1.6 of them; 2.5 with an
    allocation per call)."""
    p = configs.abp_config(n=60001, L=0.5 * 60001 ** 0.5)
    with System(p) as s:
        s.upload(*configs.random_state(p.n, p.L, seed=1))
        s.polarization_series(5, 1)

        def steps():
            for _ in range(5):
                s.step(1)
                s.sync()

        def best(call):
            r = []
            for _ in range(30):
                t = time.perf_counter()
                call()
                r.append(time.perf_counter() - t)
            return min(r)
        assert best(lambda: s.polarization_series(5, 1)) < 2.0 * best(steps)
