"""Poisson decisions of nodes that clusters of blocks decide, against the
oracle: around the 65,536 candidates from which a node gets one, words and
batches that do not divide among the blocks, long lists, and the 10,001-check
cap."""

import numpy as np
import pytest

from tests.test_gpu_accept import OFFSET, SCALE, SIDE, node

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("method", ["poisson", "poisson_average"])
@pytest.mark.parametrize("kind,n", [("sheet", 65_535), ("sheet", 65_536), ("sheet", 65_537), ("sheet", 65_569), ("sheet", 300_001),
                                    ("shell", 66_000), ("shell", 200_003), ("volume", 65_536), ("volume", 250_007)])
def test_cluster_decisions(gpu_ctx, oracle, method, kind, n):
    q, child = node(kind, n, 11)
    rgb = np.random.default_rng(n).integers(0, 65536, (n, 3), dtype=np.uint16) if method == "poisson_average" else None
    args = (method, q[:, 0], q[:, 1], q[:, 2], child, SCALE, OFFSET, np.zeros(3), np.full(3, SIDE), 1.0, rgb)
    want, want_rgb = oracle.accept(*args)
    got, got_rgb = gpu_ctx.accept(*args)
    assert int((got != want).sum()) == 0
    if rgb is not None:
        assert (got_rgb == want_rgb).all()


def test_clusters_of_several_sizes_in_a_level(gpu_ctx, oracle):
    # clumps of very different sizes: nodes of one level with and without clusters
    from potreeconverter_b200 import synth
    las = synth.generate("hotspots", 900_000, 77)
    want = oracle.convert(las, "poisson", name="mixed")
    got = gpu_ctx.convert(las, method="poisson", name="mixed")
    assert got.octree == want["octree.bin"] and got.hierarchy == want["hierarchy.bin"]
