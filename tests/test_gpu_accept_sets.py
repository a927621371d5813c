"""Clusters of every size decide nodes of one cloud: uneven hot-spots, whose
levels have nodes of one block and of clusters of two, four and eight, some
with more candidates than a batch, as the trace of the levels tells. The files
are those of the plain form, which has no clusters."""

import os
import re
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CONVERT = """
import sys
import potreeconverter_b200 as pc
from potreeconverter_b200 import synth
las = synth.generate("hotspots", 10_000_000, 7)
files = []
for form in ("batched", "plain"):
    with pc.Context(form=form) as ctx:
        c = ctx.convert(las, method=sys.argv[1], name="sets")
        files.append((c.octree, c.hierarchy, c.metadata))
assert files[0] == files[1]
"""


@pytest.mark.parametrize("method", ["poisson", "poisson_average"])
def test_clusters_of_every_size(method):
    r = subprocess.run([sys.executable, "-c", CONVERT, method], cwd=REPO, env=dict(os.environ, PCG_TRACE_LEVELS="1"), capture_output=True,
                       text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-2000:]
    sizes, large = set(), set()
    for line in r.stderr.splitlines():
        found = [int(c) for c in re.findall(r" by \d+ x (\d+)", line)]
        sizes.update(found)
        if found and int(re.search(r"largest (\d+)", line).group(1)) > 81_920:
            large.update(found[:1])  # the first set holds the largest node
    assert sizes == {1, 2, 4, 8}
    assert 8 in large
