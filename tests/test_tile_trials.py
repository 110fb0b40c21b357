"""Choice of the sweeps' tiles (pick_sweep_tiles, host/fc_schedule.cpp): trials
estimated from the tiles alone give the choice and, to the last bit, the estimate
of whole schedules; the trials run on no more threads than there are cores."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
HOST = os.path.join(os.path.dirname(HERE), "freecappuccino-dev_gb300", "host")


@pytest.fixture(scope="module")
def trials(tmp_path_factory):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("g++ not available")
    exe = str(tmp_path_factory.mktemp("trials") / "tile_trials")
    subprocess.run([gxx, "-std=c++17", "-O2", "-pthread", "-I", HOST, os.path.join(HERE, "replay", "tile_trials_replay.cpp"),
                    os.path.join(HOST, "fc_schedule.cpp"), "-o", exe], check=True)
    return exe


@pytest.mark.parametrize("case", ["40 38 36 1 152", "24 30 28 2 80", "9 8 7 3 152", "60 5 4 4 40", "3 1 1 5 8", "48 44 40 6 33"])
def test_trials_match_whole_schedules(trials, case):
    out = subprocess.run([trials] + case.split(), capture_output=True, text=True, check=True, timeout=120).stdout
    whole, picked, threads = [line.split() for line in out.splitlines()]
    assert whole == picked, out
    assert int(threads[0]) <= int(threads[1]) + 2, out  # the caller and the watching thread
