"""A refused call leaves nothing behind: the next call, on the same or another
handle, does not meet its error again."""
import numpy as np
import pytest

from spp_gb300 import Batch, System, abi, configs

pytestmark = pytest.mark.gpu


def test_failed_allocation(gpu_lib):
    n = 4096
    p = configs.abp_config(n=n, L=32.0)
    state = configs.random_state(n, p.L, seed=1)
    pts = [configs.vicsek_config(n=512, L=12.0, eta=0.2, seed=1)]
    with System(p) as s, Batch(pts) as b:
        s.upload(*state)
        b.upload(*configs.random_state(512, 12.0, seed=1))
        q = p.replace(list_capacity=1 << 30)   # 17 TB of list
        for call in (lambda: s.step(3), s.sync, s.observables, s.download, lambda: s.pairs(1.0),
                     lambda: s.radial_distribution(2.0, 10), lambda: b.step(2), b.poll):
            with pytest.raises(abi.SppError) as e:
                System(q)
            assert e.value.status == 2   # SPP_ERR_ALLOC
            call()
        assert s.observables().step == 3
