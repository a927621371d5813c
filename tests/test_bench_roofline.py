"""The benchmark's roofline (CPU): the bytes it says the acceptance cannot do
without are no more than what the profiled kernels moved, but for what they
wrote and the cache kept."""

import os
import re
import sys

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, REPO)


def test_algorithmic_bytes_are_moved():
    import bench
    text = open(os.path.join(REPO, "profiles", "accept_hotspots-5M_poisson.md")).read()
    moved = sum(float(b) for b in re.findall(r"DRAM bytes per candidate \| \*\*([0-9.]+)\*\*", text))
    candidates = int(re.search(r"candidates / list entries \| ([0-9,]+)", text).group(1).replace(",", ""))
    assert round(moved, 1) == bench.ACCEPT_DRAM_BYTES_PER_CANDIDATE
    assert bench.acceptance_bytes(candidates) / candidates - bench.ACCEPT_WRITTEN_PER_CANDIDATE <= moved
