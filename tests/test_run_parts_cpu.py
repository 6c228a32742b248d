"""How a call's steps are cut into resident launches (spp_parts.h): no launch is
longer than its bound, whatever the distance between frames or
renormalisations (so the grid barrier's 32-bit arrival count cannot wrap), and
every event falls into one launch, at its step.  And when the owners of a
resident Vicsek run are put in order again, whatever the length of the calls."""
import ctypes as C
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

SRC = Path(__file__).resolve().parent / "cpp" / "run_parts.cpp"


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not available")
    so = tmp_path_factory.mktemp("parts") / "parts.so"
    r = subprocess.run([gxx, "-std=c++17", "-O1", "-Wall", "-shared", "-fPIC", "-I", str(SRC.parents[2] / "include"),
                        str(SRC), "-o", str(so)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    lib = C.CDLL(str(so))
    lib.sort_due.argtypes = [C.c_uint32, C.c_uint32]
    lib.parts.argtypes = [C.c_int64, C.c_int, C.POINTER(C.c_int32), C.c_int]
    return lib


def parts(lib, nsteps, every):
    room = nsteps // lib.run_chunk() + 2
    out = np.zeros((room, 4), np.int32)
    n = lib.parts(nsteps, every, out.ctypes.data_as(C.POINTER(C.c_int32)), room)
    assert n >= 0
    return out[:n].tolist()


@pytest.mark.parametrize("every", [0, 1, 3, 1000, "c-1", "c", "c+1", "2c", "2c+5", 1 << 30])
@pytest.mark.parametrize("nsteps", [0, 1, 2, 999, "c-1", "c", "c+1", "3c", "5c+7"])
def test_launches_are_short_and_meet_every_event(lib, nsteps, every):
    c = lib.run_chunk()
    nsteps = eval(str(nsteps).replace("2c", "2*c").replace("3c", "3*c").replace("5c", "5*c"), {"c": c})
    every = eval(str(every).replace("2c", "2*c"), {"c": c})
    at, events = 0, []
    got = parts(lib, nsteps, every)
    for steps, first, count, last in got:
        assert 1 <= steps <= c
        here = list(range(first, steps + 1, every)) if every else []
        assert len(here) == count
        events += [at + e for e in here]
        at += steps
        assert last == (at == nsteps)
    assert at == nsteps
    assert events == (list(range(every, nsteps + 1, every)) if every else [])


def test_frames_further_apart_than_the_barrier_counts(lib):
    """Two frames 2^30 steps apart (every step one arrival per block): no launch
    comes near 2^32 arrivals."""
    got = parts(lib, 1 << 31, 1 << 30)
    assert max(q[0] for q in got) * lib.run_arrivals() * lib.run_max_blocks() < 1 << 31
    assert sum(q[2] for q in got) == 2


@pytest.mark.parametrize("start", [0, 5, (1 << 32) - 600])
@pytest.mark.parametrize("calls", [1, 2, 3, 4, 8, 15, 16, 17, 32, 100])
def test_owners_are_sorted_again_over_calls(lib, start, calls):
    """A launch sorts before the first of its steps at which the rule says so;
    the word that it reads is carried from call to call."""
    sorted_at, last, gaps = start, start, []
    step = start
    while step < start + 500:
        for _ in range(calls):
            if lib.sort_due(step, sorted_at):
                sorted_at = step
                gaps.append(step - last)
                last = step
            step += 1
    assert gaps and set(gaps) == {lib.sort_steps()}
