"""The distribution of points to chunks against a stable sort: tiles of 2,048
points and groups of 64 tiles and their remainders, one digit of chunk numbers
and two."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
G = 16
CELLS = G**3


@pytest.mark.parametrize("chunks", [1, 2, 256, 257, 3000])
@pytest.mark.parametrize("n", [1, 2047, 2048, 2049, 131_071, 131_072, 131_073, 262_145, 1_000_001])
def test_scatter_sizes(gpu_ctx, chunks, n):
    rng = np.random.default_rng([chunks, n])
    lut = (np.arange(CELLS) % chunks).astype(np.int32)
    # half of the points in one cell: a digit with most of a tile
    cell = np.where(rng.random(n) < 0.5, 17, rng.integers(0, CELLS, n)).astype(np.uint32)
    ids, start = gpu_ctx.scatter(cell, lut, G, chunks)
    of = lut[cell]
    assert (ids == np.argsort(of, kind="stable")).all()
    assert (start == np.searchsorted(of[ids], np.arange(chunks + 1))).all()
