"""Batches whose cells end at the edges of a scan tile (4,096 cells), whose
particles end at the edges of a block (256) and whose launch space changes or
finishes within a run, for one model and for mixed ones, bit for bit against
the oracle's systems run alone; the step shape of large batches; refused
uploads."""
import numpy as np
import pytest

from oracle import oracle as O
from spp_gb300 import Batch, abi, configs
from spp_gb300.abi import SppError

pytestmark = pytest.mark.gpu

V, A, W = abi.MODEL_VICSEK, abi.MODEL_VICSEK_REF_ANGLE, abi.MODEL_VICSEK_REF_VECTOR


def point(s, n, D, model, push=False):
    p = configs.vicsek_config(n=n, L=0.5 * 1.001 * D + 0.01, eta=0.2, seed=6)
    p.v0, p.model, p.system_id = 0.5, model, s
    if push:
        p.r_push, p.beta_push = 0.8, 0.3
    return p


def same(b, pts, state, got, steps):
    for s, p in enumerate(pts):
        sl = slice(b.offsets[s], b.offsets[s + 1])
        if steps[s] is None:
            continue
        m = O.run32(p, O.State32(*(a[sl] for a in state)), steps[s])
        for g, want in zip(got, (m.x, m.y, m.th, m.ix, m.iy)):
            assert np.array_equal(g[sl], want), s


# (n, D) of the systems: one cell tile exactly, one more, one less, a system
# of one particle, mostly empty grids, crowded ones
SHAPES = {
    "tile": [(700, 64)],
    "tile+9": [(256, 64), (257, 3)],
    "tile-1": [(1, 63), (255, 9), (3000, 6), (40, 3)],   # 3969 + 81 + 36 + 9 cells
    "two tiles": [(513, 90), (2000, 9), (1, 3)],
}


@pytest.mark.parametrize("models", [(V,), (A,), (W,), (V, A, W)], ids=["vicsek", "angle", "vector", "mixed"])
@pytest.mark.parametrize("shape", SHAPES)
def test_edges_of_tiles_and_blocks(gpu_lib, shape, models):
    pts = [point(s, n, D, models[s % len(models)], push=s % 2 == 1) for s, (n, D) in enumerate(SHAPES[shape])]
    state = configs.sweep_state(pts, seed=6)
    with Batch(pts) as b:
        b.upload(*state)
        b.step(3)
        b.step(18)
        same(b, pts, state, b.download(), [21] * len(pts))
        b.upload(*state)                    # a new state starts from its own counts
        b.step(2)
        same(b, pts, state, b.download(), [2] * len(pts))


@pytest.mark.parametrize("models", [(V,), (V, W)], ids=["vicsek", "mixed"])
def test_systems_finish_retire_and_resume_within_runs(gpu_lib, models):
    pts = [point(s, n, D, models[s % len(models)]) for s, (n, D) in enumerate([(300, 12), (1000, 20), (90, 64), (5, 7)])]
    state = configs.sweep_state(pts, seed=6)
    with Batch(pts) as b:
        b.set_windows(5, 10, 40)
        b.upload(*state)
        b.step(7)
        b.retire([1, 3])
        b.step(9)
        b.resume([3])
        b.step(30)                          # 0 and 2 finish at 40 inside this call
        assert [s.steps for s in b.poll()] == [40, 7, 40, 37]
        b.resume([1])
        b.step(1)
        same(b, pts, state, b.download(), [40, 8, 40, 38])
        b.step(50)
        assert [s.active for s in b.poll()] == [0, 0, 0, 0]
        same(b, pts, state, b.download(), [40] * 4)


def test_large_batch(gpu_lib):
    """Above three million active particles Vicsek batches step with another
    shape; retiring systems brings the others below it."""
    pts = [point(s, 50021 if s % 2 else 50000, 150 + s, V) for s in range(61)]
    state = configs.sweep_state(pts, seed=6)
    with Batch(pts) as b:
        b.upload(*state)
        b.step(3)
        b.retire(np.arange(5, 40))
        b.step(2)
        steps = [None] * len(pts)
        steps[0], steps[7], steps[60] = 5, 3, 5
        same(b, pts, state, b.download(), steps)


@pytest.mark.parametrize("i,value,status", [(0, np.nan, "NUMERIC"), (1255, np.inf, "NUMERIC"), (256, 99.0, "INVALID")])
def test_refused_uploads_change_nothing(gpu_lib, i, value, status):
    pts = [point(0, 256, 12, V), point(1, 1000, 20, V)]
    state = configs.sweep_state(pts, seed=6)
    bad = [a.copy() for a in state]
    bad[0][i] = value
    bad[1][min(i + 1, 1255)] = np.nan       # a later particle is not the one named
    with Batch(pts) as b:
        with pytest.raises(SppError, match=f"{status}.*particle {i}$"):
            b.upload(*bad)
        b.upload(*state)
        b.step(4)
        with pytest.raises(SppError, match=f"{status}.*particle {i}$"):
            b.upload(*bad)
        b.step(4)
        same(b, pts, state, b.download(), [8, 8])
