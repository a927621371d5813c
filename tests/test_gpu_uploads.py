"""Host records reach the device the same way through the pinned pieces
(pageable memory, 8 MiB and more in all) and directly (page-locked memory, or
less): piece remainders and several sources. And a hierarchy deeper than the
21 levels that 64 bits name."""

import numpy as np
import pytest

from potreeconverter_b200 import synth

pytestmark = pytest.mark.gpu
MIB = 1 << 20


def outputs(conv):
    return conv.octree, conv.hierarchy, conv.metadata


def pinned(las):
    import torch
    t = torch.empty(len(las), dtype=torch.uint8, pin_memory=True)
    t.numpy()[:] = np.frombuffer(las, np.uint8)
    return t


@pytest.mark.parametrize("sizes", [[8 * MIB // 26 - 1], [8 * MIB // 26 + 1], [9 * MIB // 26 + 3], [700_001],
                                   [150_000, 200_001, 30], [100_000, 100_000]])
def test_pageable_as_page_locked(gpu_ctx, sizes):
    files = [synth.generate("terrain", n, 50 + k) for k, n in enumerate(sizes)]
    locked = [pinned(f) for f in files]
    one = len(files) == 1
    got = gpu_ctx.convert(files[0] if one else files, method="poisson", name="up")
    want = gpu_ctx.convert((locked[0].data_ptr(), locked[0].numel()) if one else [(t.data_ptr(), t.numel()) for t in locked],
                           method="poisson", name="up")
    assert outputs(got) == outputs(want)


def test_names_of_more_than_21_levels(gpu_ctx, oracle):
    rng = np.random.default_rng(5)
    near = rng.choice(32**3, 12_000, replace=False)
    base = (1 << 29) + 7
    X, Y, Z = (np.concatenate([[0, 1 << 30], base + v]).astype(np.int32) for v in (near % 32, near // 32 % 32, near // 1024))
    las = synth.write_las(X, Y, Z, synth._common_attrs(rng, len(X), Z.astype(np.float64)), pdrf=2, version_minor=2)
    want = oracle.convert(las, "poisson", name="deep")
    got = gpu_ctx.convert(las, method="poisson", name="deep")
    assert max(len(n[0]) for n in got.nodes) > 22
    assert got.octree == want["octree.bin"] and got.hierarchy == want["hierarchy.bin"]
