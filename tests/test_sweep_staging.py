"""Hand-over of the ordered sweeps' stage buffers (host/fc_stage.hpp), played on
the CPU by tests/replay/stage_replay.cpp in random orders of its actors, for
every number of buffers and of steps in a buffer; the groups and descriptors of
the structures that tests/test_gpu_sweep_staging.py solves."""
import os
import shutil
import subprocess

import pytest

import sweep_cases as cases

HERE = os.path.dirname(os.path.abspath(__file__))
HOST = os.path.join(os.path.dirname(HERE), "freecappuccino-dev_gb300", "host")


@pytest.fixture(scope="module")
def replay(tmp_path_factory):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("g++ not available")
    exe = str(tmp_path_factory.mktemp("stage") / "stage_replay")
    subprocess.run([gxx, "-std=c++17", "-O2", "-pthread", "-I", HOST, os.path.join(HERE, "replay", "stage_replay.cpp"),
                    os.path.join(HOST, "fc_stage.cpp"), os.path.join(HOST, "fc_schedule.cpp"), "-o", exe], check=True)
    return lambda *args: subprocess.run([exe] + [str(a) for a in args], capture_output=True, text=True, timeout=120)


@pytest.mark.parametrize("G", [1, 2, 4])
@pytest.mark.parametrize("K", [4, 8, 16])
def test_no_buffer_is_taken_early(replay, K, G):
    out = replay("model", K, G, "code")
    assert out.returncode == 0 and out.stdout.strip() == "OK", out.stdout + out.stderr


@pytest.mark.parametrize("G", [1, 2])
def test_the_model_tells_a_wait_by_parity_that_passes_early(replay, G):
    out = replay("model", 4, G, "parity")
    assert out.returncode == 1 and "over unread ones" in out.stdout, out.stdout + out.stderr


@pytest.mark.parametrize("name", sorted(cases.STAGED))
def test_groups_of_wide_steps(replay, tmp_path, name):
    box, tiles, g, g_gs = cases.STAGED[name]
    path = tmp_path / "pattern.bin"
    cases.write_pattern(path, *cases.red_black(**box)[:3])
    out = replay("groups", path, tiles, 128)
    assert out.returncode == 0, out.stdout + out.stderr
    first, solve, gs = [line.split() for line in out.stdout.splitlines()]
    assert first[1] == str(tiles) and first[-1] == "0"
    assert solve[3] == str(g) and gs[3] == str(g_gs)
    # DILU setup, backward sweep with the dot product; Gauss-Seidel
    buffers = lambda w: {w[i]: int(w[i + 1]) for i in range(4, len(w), 3)}
    assert buffers(solve)["K1"] == 4 and buffers(solve)["K4"] == 4 and buffers(gs)["K5"] == 4


@pytest.mark.parametrize("name", sorted(cases.DENSE))
def test_densely_coupled_rows_get_their_buffers(replay, tmp_path, name):
    make, tiles = cases.DENSE[name]
    path = tmp_path / "pattern.bin"
    cases.write_pattern(path, *make()[:3])
    out = replay("fits", path, tiles)
    assert out.returncode == 0 and out.stdout.startswith("rows "), out.stdout + out.stderr
