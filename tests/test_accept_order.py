"""The acceptance kernel's warps wait for one another's decisions in shared
memory, their own block's or a cluster's. A wait that ends only by luck shows
in no test run, so the source is looked at instead: every such access names its
order and scope, and those that reach another block name the cluster."""

import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "potreeconverter_b200", "csrc")


def test_shared_memory_that_warps_poll_is_strongly_ordered():
    text = open(os.path.join(CSRC, "accept.cu")).read()
    ops = re.findall(r'asm volatile\("((?:ld|st)\.[a-z0-9_.:]*shared[a-z0-9_.:]*)', text)
    assert len(ops) >= 10
    for op in ops:
        assert re.match(r"(ld\.(relaxed|acquire)|st\.(relaxed|release))\.(cta|cluster)\.", op), op
        if "shared::cluster" in op:
            assert ".cluster.shared::cluster" in op, op
    # and nothing is polled by way of a volatile pointer
    assert not re.search(r"\*\s*\(volatile", text)
