"""Which nodes the lookup kernels of the plain form give a block of their own:
on a level of few nodes those of 1,024 candidates and more, as the trace of the
levels tells; the decisions are the oracle's on both sides of the line."""

import os
import re
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

ACCEPT = """
import sys
import numpy as np
import potreeconverter_b200 as pc
from tests.oracle_lib import Oracle
from tests.test_gpu_accept import OFFSET, SCALE, SIDE, node
with pc.Context(form="plain") as ctx:
    for n in (1_023, 1_024, 4_095):
        q, child = node("sheet", n, 21)
        args = ("poisson", q[:, 0], q[:, 1], q[:, 2], child, SCALE, OFFSET, np.zeros(3), np.full(3, SIDE), 1.0, None)
        assert (ctx.accept(*args)[0] == Oracle().accept(*args)[0]).all(), n
"""


def test_blocks_from_1024_candidates_on_levels_of_few_nodes():
    r = subprocess.run([sys.executable, "-c", ACCEPT], cwd=REPO, env=dict(os.environ, PCG_TRACE_LEVELS="1"), capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    assert [int(b) for b in re.findall(r"lookup by blocks (\d+)", r.stderr)] == [0, 1, 1]
