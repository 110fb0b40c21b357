"""Levels wider than a step (chunk rows): the replay of the schedule-ordered
sweeps (tests/replay/schedule_replay.cpp) on structures whose wide levels take
several consecutive steps, with the ring depth the builder chose for them,
against plain substitution, bit for bit.  Chunks of one row, of one below and
one above a multiple of the widest level, and chunks no level reaches."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
HOST = os.path.join(os.path.dirname(HERE), "freecappuccino-dev_gb300", "host")

# the builder's deeper ring replaces the replay's R (the call is the only use of the name)
WRAP = """#include "fc_schedule.hpp"
#include <cstdlib>
#define build_ordered_sweep(...) \\
  (build_ordered_sweep(__VA_ARGS__, std::atoi(std::getenv("CHUNK"))) && ((R = O.R), true))
"""


@pytest.fixture(scope="module")
def replay(tmp_path_factory):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("g++ not available")
    d = tmp_path_factory.mktemp("chunks")
    wrap = d / "wrap.hpp"
    wrap.write_text(WRAP)
    exe, obj = str(d / "chunk_replay"), str(d / "replay.o")
    flags = [gxx, "-std=c++17", "-O2", "-pthread", "-I", HOST]
    subprocess.run(flags + ["-include", str(wrap), "-c", os.path.join(HERE, "replay", "schedule_replay.cpp"), "-o",
                            obj], check=True)
    subprocess.run(flags + [obj, os.path.join(HOST, "fc_schedule.cpp"), "-o", exe], check=True)
    return exe


@pytest.mark.parametrize("args", ["16 16 16 2", "12 10 8 16", "20 7 5 40 1", "30 30 30 1", "7 3 1 2 1"])
@pytest.mark.parametrize("chunk", [1, 8, 31, 32, 128])
def test_chunked_levels_match_substitution(replay, args, chunk):
    out = subprocess.run([replay] + args.split(), capture_output=True, text=True, timeout=120,
                         env=dict(os.environ, CHUNK=str(chunk)))
    assert out.returncode == 0 and out.stdout.strip().endswith("OK"), out.stdout + out.stderr
    assert int(out.stdout.split("maxW=")[1].split()[0]) <= chunk
