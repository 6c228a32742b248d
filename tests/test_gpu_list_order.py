"""Neighbour lists of every length around the limits of the in-register sort
(8, 12, 16 entries) and of the queue for longer ones, ids in any order, in the
interior and across the box edges: the trajectory must be the oracle's, whose
sums run over the neighbours in id order, bit for bit."""
import numpy as np
import pytest

from oracle import oracle as O
from spp_gb300 import System, abi, configs

pytestmark = pytest.mark.gpu


def groups(sizes, L, seed):
    """Groups of the given sizes, each within the list radius of itself only,
    on a lattice whose first point is the box corner; ids shuffled."""
    g = np.random.default_rng(seed)
    side = int(2 * L / 4)
    at = [(-L + 4 * (q % side), -L + 4 * (q // side)) for q in range(len(sizes))]
    xy = np.concatenate([np.array(c) + 0.5 * (g.random((m, 2)) - 0.5) for c, m in zip(at, sizes)])
    xy = ((xy + L) % (2 * L) - L).astype(np.float32)
    xy[xy >= L] = -L
    xy = xy[g.permutation(len(xy))]
    return xy[:, 0].copy(), xy[:, 1].copy(), (6.28 * g.random(len(xy)) - 3.14).astype(np.float32)


@pytest.mark.parametrize("resident", [1, 0])
@pytest.mark.parametrize("lanes", [1, 4])
@pytest.mark.parametrize("sizes", [
    tuple(range(1, 20)) + (33, 34),          # lengths 0 .. 18, 32, 33
    (9,) * 60,                               # a whole warp at 8
    (10,) * 60, (13,) * 40, (14,) * 40,      # at 9, 12, 13
    (17,) * 30, (18,) * 30,                  # at 16 and one beyond
], ids=["mixed", "8", "9", "12", "13", "16", "17"])
def test_list_lengths(gpu_lib, monkeypatch, sizes, lanes, resident):
    monkeypatch.setenv("SPP_RESIDENT", str(resident))
    L = 16.0
    state = groups(sizes, L, seed=len(sizes))
    p = configs.abp_config(n=len(state[0]), L=L)
    p.gather_lanes, p.k_rep = lanes, 0.5
    with System(p) as s:
        s.upload(*state)
        assert s.observables().max_neighbors == max(sizes) - 1
        s.step(40)
        got = s.download()
    m = O.run32(p, O.State32(*state), 40)
    for g, want in zip(got, (m.x, m.y, m.th, m.ix, m.iy)):
        assert np.array_equal(g, want)
