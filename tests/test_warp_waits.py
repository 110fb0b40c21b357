"""Waits in which one lane polls for its warp (csrc/*.cuh, *_wait_warp): the answer
travels by a shuffle, which orders no memory, so each of them has to end with a
__syncwarp() before the other lanes read what was waited for."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "freecappuccino-dev_gb300", "csrc")


def test_waits_of_one_lane_order_the_others():
    waits = {}
    for path in glob.glob(os.path.join(CSRC, "*.cu*")):
        with open(path) as f:
            for m in re.finditer(r"bool (\w+_wait_warp)\([^{]*\{(.*?)\n\}", f.read(), re.S):
                waits[m.group(1)] = m.group(2)
    assert set(waits) >= {"mbar_wait_warp", "word_wait_warp"}
    for name, body in waits.items():
        assert re.search(r"__shfl_sync\([^;]*;\s*__syncwarp\(\);[^;]*\s*return ok;\s*$", body), name
