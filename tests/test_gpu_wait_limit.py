"""A grid barrier of a resident run that gives up: the launch ends, the next
call that waits reports SPP_ERR_TIMEOUT, further steps end at once, and an
upload makes the handle good again.  Tested with a library whose barriers poll
zero times, so that every wait of a resident run gives up at once."""
import os
import subprocess
import sys
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]

CHILD = """
import os
import numpy as np
from spp_gb300 import System, abi, configs

TIMEOUT = 5


def status(call, *a):
    try:
        call(*a)
    except abi.SppError as e:
        return e.status
    return 0


def cases():
    for n in (1, 4096, 65537, 120000):
        L = max(4.0, 0.5 * n ** 0.5)
        yield configs.abp_config(n=n, L=L), "step"
        for model in (abi.MODEL_VICSEK, abi.MODEL_VICSEK_REF_ANGLE, abi.MODEL_VICSEK_REF_VECTOR):
            yield configs.vicsek_config(n=n, L=L, eta=0.3, seed=1, model=model), "step"
        yield configs.vicsek_config(n=n, L=L, eta=0.3, seed=1), "series"
    for n in (150, 16384):
        yield configs.lyapunov_config(n=n), "lyap"


for p, kind in cases():
    state = configs.random_state(p.n, p.L, seed=2)
    with System(p) as s:
        for _ in range(2):                       # and again after the recovery
            s.upload(*state)
            if kind == "lyap":
                s.lyap_init(3, seed=1)
                call = lambda: s.lyap_step(12, 5)
            elif kind == "series":
                call = lambda: s.polarization_series(4, 3)
            else:
                call = lambda: s.step(300)       # two launches
            assert status(call) == (TIMEOUT if kind == "series" else 0)
            assert s.resident_launches() > 0
            assert status(s.sync) == TIMEOUT
            assert status(s.step, 5) == 0        # ends at once
            assert status(s.download) == TIMEOUT
            assert status(s.observables) == TIMEOUT
        s.upload(*state)
        assert status(s.sync) == 0
        got = s.download()
        assert all(np.array_equal(a, b) for a, b in zip(got, state))
    os.environ["SPP_RESIDENT"] = "0"             # the step graphs have no such waits
    with System(p) as s:
        s.upload(*state)
        s.step(3)
        assert s.observables().step == 3
    del os.environ["SPP_RESIDENT"]
print("all cases ended")
"""


@pytest.mark.gpu
def test_waits_that_give_up(tmp_path):
    env = dict(os.environ)
    env.update(SPP_NVCC_DEFINES="SPP_RUN_WAIT_LIMIT=0", SPP_LIB_OUT=str(tmp_path / "libspp_wait.so"),
               SPP_BUILD_DIR=str(tmp_path / "build"))
    r = subprocess.run([sys.executable, "-m", "spp_gb300.build", "-f"], cwd=ROOT, env=env, capture_output=True, text=True,
                       timeout=900)
    assert r.returncode == 0, r.stdout + r.stderr
    env["SPP_GB300_LIB"] = str(tmp_path / "libspp_wait.so")
    r = subprocess.run([sys.executable, "-c", CHILD], cwd=ROOT, env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout[-3000:] + r.stderr[-3000:]
    assert "all cases ended" in r.stdout
