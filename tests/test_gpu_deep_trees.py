"""Whole conversions of trees deeper than the 21 and the 42 levels at which the
form of a node's number in the hierarchy writer changes, against the oracle."""

import pytest

from tests.test_hierarchy_host import long_box

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("method", ["poisson", "random"])
@pytest.mark.parametrize("length", [1e7, 2e13, 4e13, 1e18])
def test_deep_trees(gpu_ctx, oracle, length, method):
    las = long_box(length)
    want = oracle.convert(las, method, name="deep")
    got = gpu_ctx.convert(las, method=method, name="deep")
    assert got.hierarchy == want["hierarchy.bin"]
    assert got.octree == want["octree.bin"] and got.metadata.encode() == want["metadata.json"]
