"""Short lives of systems: created, used and destroyed one after the other and
by several threads at once.  Destroyed systems leave their pinned block to the
next ones; no two may ever hold the same."""
import threading

import numpy as np
import pytest

from spp_gb300 import System, abi, configs

pytestmark = pytest.mark.gpu

SIZES = (1, 50, 190, 200, 1000, 3000, 6500, 16384, 16385)   # blocks of several sizes, and none


def life(n, keep=None):
    p = configs.vicsek_config(n=n, L=max(4.0, 0.5 * n ** 0.5), eta=0.3, seed=n) if n % 2 else \
        configs.abp_config(n=n, L=max(4.0, 0.5 * n ** 0.5), seed=n)
    s = System(p)
    s.upload(*configs.random_state(n, p.L, seed=n))
    s.step(3)
    out = s.download() + (np.float64(s.observables().polarization),)
    if keep is None:
        s.close()
    else:
        keep.append(s)
    return out


def test_lives_in_threads(gpu_lib):
    want = {n: life(n) for n in SIZES}
    wrong = []

    def work(seed):
        g = np.random.default_rng(seed)
        try:
            kept = []
            for _ in range(40):
                n = int(g.choice(SIZES))
                got = life(n, kept if g.random() < 0.3 else None)
                if not all(np.array_equal(a, b) for a, b in zip(got, want[n])):
                    wrong.append(n)
                if len(kept) > 4:
                    s = kept.pop(int(g.integers(len(kept))))
                    m = int(s.params.n)
                    if not all(np.array_equal(a, b) for a, b in zip(s.download(), want[m])):
                        wrong.append(m)
                    s.close()
            for s in kept:
                s.close()
        except Exception as e:   # a thread's failure is the test's
            wrong.append(repr(e))
    threads = [threading.Thread(target=work, args=(q,)) for q in range(8)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong


def test_more_systems_than_spare_blocks(gpu_lib):
    for _ in range(2):
        kept = []
        outs = [life(700, kept) for _ in range(90)]
        assert all(np.array_equal(a, b) for o in outs for a, b in zip(o, outs[0]))
        for s in kept:
            assert np.array_equal(s.download()[0], outs[0][0])
            s.close()


def test_a_refused_system_gives_its_block_back(gpu_lib):
    p = configs.abp_config(n=4096, L=32.0)
    for _ in range(5):
        with pytest.raises(abi.SppError):
            System(p.replace(list_capacity=1 << 30))
        life(4096)
