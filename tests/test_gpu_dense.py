"""Nodes whose conflict lists find no room keep the lookup kernels, beside
nodes of the same level that have lists: one node with more list entries than
the budget of all long lists, and whole clouds with the room lowered, so that
the pool, the long lists or their entries run out. Results are the oracle's."""

import json
import os
import re
import subprocess
import sys

import numpy as np
import pytest

from tests.test_gpu_accept import OFFSET, SCALE, SIDE, node

pytestmark = pytest.mark.gpu
REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.parametrize("method", ["poisson", "poisson_average"])
@pytest.mark.parametrize("beside", [0, 20_000])
def test_node_over_the_budget(gpu_ctx, oracle, method, beside):
    # 60,000 candidates within a spacing: 1.8 billion entries, 2^28 are kept
    rng = np.random.default_rng(beside)
    q = np.round((64 + rng.uniform(-0.25, 0.25, (60_000, 3))) / 0.001).astype(np.int32)
    if beside:
        q = np.concatenate([q, node("sheet", beside, 2)[0]])
    x = q * 0.001
    child = ((x[:, 0] >= 64).astype(np.uint8) << 2) | ((x[:, 1] >= 64).astype(np.uint8) << 1) | (x[:, 2] >= 64).astype(np.uint8)
    o = np.argsort(child, kind="stable")
    q, child = q[o], child[o]
    rgb = rng.integers(0, 65536, (len(q), 3), dtype=np.uint16) if method == "poisson_average" else None
    args = (method, q[:, 0], q[:, 1], q[:, 2], child, SCALE, OFFSET, np.zeros(3), np.full(3, SIDE), 1.0, rgb)
    want, want_rgb = oracle.accept(*args)
    got, got_rgb = gpu_ctx.accept(*args)
    assert int((got != want).sum()) == 0
    if rgb is not None:
        assert (got_rgb == want_rgb).all()


CONVERT = """
import hashlib, json, sys
import potreeconverter_b200 as pc
from potreeconverter_b200 import synth
from tests.test_gpu_dense import cloud
with pc.Context() as ctx:
    for kind in ("lattice", "clumps"):
        c = ctx.convert(cloud(kind), method=sys.argv[1], name="dense")
        print(json.dumps([hashlib.md5(c.octree).hexdigest(), hashlib.md5(c.hierarchy).hexdigest()]))
"""


def cloud(kind):
    """A lattice, and a terrain with clumps of points far closer than the
    spacings of the upper levels."""
    from potreeconverter_b200 import synth
    if kind == "lattice":
        return synth.generate("lattice", 150_000, 8)
    las = bytearray(synth.terrain(120_000, 9))
    off, rec = int.from_bytes(las[96:100], "little"), int.from_bytes(las[105:107], "little")
    points = np.frombuffer(bytes(las[off:]), dtype=np.uint8).reshape(-1, rec).copy()
    xyz = points[:, :12].copy().view("<i4")
    rng = np.random.default_rng(4)
    for c in range(30):  # 30 clumps of 2,000 points around one of their own
        mine = slice(2_000 * c, 2_000 * (c + 1))
        centre = xyz[2_000 * c]
        near = centre + np.round(rng.normal(0, 300, (2_000, 3))).astype(np.int32)
        xyz[mine] = np.clip(near, xyz.min(0), xyz.max(0))
    points[:, :12] = xyz.view(np.uint8)
    las[off:] = points.tobytes()
    return bytes(las)


@pytest.mark.parametrize("method", ["poisson", "poisson_average"])
@pytest.mark.parametrize("limits", ["5000,1000000,1000000000", "1000000000,200,1000000000", "1000000000,1000000,20000", "1,1,1"])
def test_clouds_with_less_room(oracle, method, limits):
    import hashlib
    env = dict(os.environ, PCG_LIST_LIMITS=limits, PCG_TRACE_LEVELS="1")
    r = subprocess.run([sys.executable, "-c", CONVERT, method], cwd=REPO, env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    got = [json.loads(line) for line in r.stdout.splitlines()]
    for kind, files in zip(("lattice", "clumps"), got):
        want = oracle.convert(cloud(kind), method, name="dense")
        assert files == [hashlib.md5(want[f]).hexdigest() for f in ("octree.bin", "hierarchy.bin")], kind
    levels = [(int(n), int(d)) for n, d in re.findall(r"nodes (\d+) \(dense (\d+)", r.stderr)]
    assert any(d > 0 for n, d in levels)
    if limits != "1,1,1":
        assert any(0 < d < n for n, d in levels), levels


FULL = """
import hashlib, sys
import torch
import potreeconverter_b200 as pc
from tests.test_gpu_estimate import clumps
las = clumps(1_000_000, 250)
leave = float(sys.argv[1])
torch.zeros(1, device="cuda")
with pc.Context() as ctx:
    held = torch.empty(int(torch.cuda.mem_get_info()[0] - leave * 2 ** 30), dtype=torch.uint8, device="cuda") if leave else None
    c = ctx.convert(las, method="poisson", name="full")
    print(hashlib.md5(c.octree + c.hierarchy).hexdigest())
"""


def test_device_that_something_else_fills():
    # 1.2 GiB are left for a conversion that takes 1.2 when it can have them:
    # neither the long lists nor the grids of the nodes without any find the
    # room they ask for
    def convert(leave):
        r = subprocess.run([sys.executable, "-c", FULL, str(leave)], cwd=REPO, capture_output=True, text=True, timeout=300)
        assert r.returncode == 0, r.stderr[-500:]
        return r.stdout

    assert convert(1.2) == convert(0)
