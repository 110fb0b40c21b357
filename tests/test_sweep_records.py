"""Row records of the ordered sweeps as the kernels read them, replayed on the CPU
(tests/replay/record_replay.cpp) against plain substitution, bit for bit: rows of
few and of several hundred entries, served by the ring, by the exchange and by
both, on one tile and on several, with steps of several widths."""
import os
import shutil
import subprocess

import pytest

import sweep_cases as cases

HERE = os.path.dirname(os.path.abspath(__file__))
HOST = os.path.join(os.path.dirname(HERE), "freecappuccino-dev_gb300", "host")

PATTERNS = {
    "red_black": lambda: cases.red_black(9, 8, 7),
    "hubs": lambda: cases.red_black(12, 11, 10, 12, 150),
    "blocks": lambda: cases.blocks_coupled(300, 64, 0),
    "blocks_chain": lambda: cases.blocks_coupled(300, 64, 12),
    "blocks_600": lambda: cases.blocks_coupled(600, 40, 0),
    "blocks_256": lambda: cases.blocks_coupled(256, 9, 3),
}


@pytest.fixture(scope="module")
def replay(tmp_path_factory):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("g++ not available")
    exe = str(tmp_path_factory.mktemp("records") / "record_replay")
    subprocess.run([gxx, "-std=c++17", "-O2", "-pthread", "-ffp-contract=off", "-I", HOST,
                    os.path.join(HERE, "replay", "record_replay.cpp"), os.path.join(HOST, "fc_schedule.cpp"), "-o", exe],
                   check=True)
    return lambda *args: subprocess.run([exe] + [str(a) for a in args], capture_output=True, text=True, timeout=120)


@pytest.mark.parametrize("chunk", [32, 128])
@pytest.mark.parametrize("tiles", [1, 2, 7])
@pytest.mark.parametrize("name", sorted(PATTERNS))
def test_records_match_substitution(replay, tmp_path, name, tiles, chunk):
    path = tmp_path / "pattern.bin"
    cases.write_pattern(path, *PATTERNS[name]()[:3])
    out = replay(path, tiles, chunk)
    assert out.returncode == 0, out.stdout + out.stderr
    # on several tiles the long rows have more exchanged entries than a record holds
    assert out.stdout.startswith("tiles") or (tiles > 1 and "exchanged entries" in out.stdout), out.stdout


@pytest.mark.parametrize("name,most", [("blocks", 300), ("blocks_chain", 300), ("blocks_600", 600), ("blocks_256", 256)])
def test_long_rows_from_the_ring(replay, tmp_path, name, most):
    path = tmp_path / "pattern.bin"
    cases.write_pattern(path, *PATTERNS[name]()[:3])
    out = replay(path, 1, 128)
    assert out.returncode == 0 and " most %d " % most in out.stdout, out.stdout + out.stderr
    assert int(out.stdout.split("ring ")[1].split()[0]) > 0


def test_rows_of_more_entries_than_a_record_counts(replay, tmp_path):
    path = tmp_path / "pattern.bin"
    cases.write_pattern(path, *cases.blocks_coupled(8192, 2, 0)[:3])
    out = replay(path, 1, 2048)
    assert out.returncode == 0 and out.stdout.startswith("refused"), out.stdout + out.stderr


@pytest.mark.parametrize("where", ["same", "nan", "inf"])
def test_rows_without_distinct_coordinates_get_their_tiles(replay, tmp_path, where):
    path = tmp_path / "pattern.bin"
    cases.write_pattern(path, *cases.red_black(16, 16, 16)[:3])
    plain, out = replay(path, 12, 128), replay(path, 12, 128, where)
    assert out.returncode == 0 and out.stdout == plain.stdout, out.stdout + out.stderr
    assert int(out.stdout.split()[1]) == 12
