"""The ring of tile buffers of the two-round pass (csrc/team_ring.cuh), run by
CPU threads (team_ring_model.cpp): no team touches a buffer whose load has not
landed, in whatever order the loads land, and every warp ends when one never does."""
import os
import random
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "omr-ntt_gb300", "csrc")
TILES = 14


@pytest.fixture(scope="module")
def model(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("ring") / "model")
    cxx = shutil.which("g++") or pytest.skip("no g++")
    subprocess.run([cxx, "-std=c++20", "-O1", "-pthread", "-I", CSRC, os.path.join(HERE, "team_ring_model.cpp"), "-o", exe],
                   check=True)
    return exe


def _all(model, ring, limit_ms, delays, flag_ms=0):
    runs = [subprocess.Popen([model, *map(str, [*ring, TILES, limit_ms, flag_ms, *d])], stdout=subprocess.PIPE, text=True)
            for d in delays]
    return [(d, r.communicate(timeout=60)[0].strip()) for d, r in zip(delays, runs)]


@pytest.mark.parametrize("ring", [(3, 2), (1, 1)], ids=["two-teams-three-buffers", "one-team-one-buffer"])
def test_late_loads(model, ring):
    """Every load late by itself and with each of the next four, and random delays."""
    late = [[60 if j in pair else 0 for j in range(TILES)]
            for j0 in range(9) for pair in [(j0,)] + [(j0, j0 + s) for s in range(1, 5)]]
    rng = random.Random(1)
    late += [[rng.choice([0, 0, 1, 3, 9]) for _ in range(TILES)] for _ in range(40)]
    for i in range(0, len(late), 12):
        assert [x for x in _all(model, ring, 20000, late[i:i + 12]) if x[1]] == []


@pytest.mark.parametrize("ring", [(3, 2), (1, 1)], ids=["two-teams-three-buffers", "one-team-one-buffer"])
@pytest.mark.parametrize("flag_ms", [0, 20, 130])
def test_load_that_never_lands(model, ring, flag_ms):
    """The waits give up after 100 ms, and no warp is left at a barrier, at whatever time its team reads the flag."""
    lost = [[-1 if k == j else 0 for k in range(TILES)] for j in range(8)]
    assert [x for x in _all(model, ring, 100, lost, flag_ms) if x[1]] == []
