"""The GPU-wide rounds of the std::sort replay against std::sort: segments
around the 1,024 elements from which they go round by round, tiles of 4,096
and their remainders, and partitions that stay lopsided for many rounds."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def keys(kind, n):
    rng = np.random.default_rng([n, len(kind)])
    if kind == "few":  # every key many times
        return rng.integers(0, 7, n).astype(np.float64)
    if kind == "pairs":
        return rng.integers(0, max(n // 2, 1), n).astype(np.float64)
    if kind == "equal":
        return np.full(n, 2.5)
    if kind == "one pair":  # all but two keys distinct: most of it is written from the sorted keys
        k = rng.permutation(n).astype(np.float64)
        k[n // 3] = k[n // 2]
        return k
    pipe = np.minimum(np.arange(n), np.arange(n)[::-1]).astype(np.float64)  # rising, then falling
    return pipe


@pytest.mark.parametrize("kind", ["few", "pairs", "equal", "one pair", "pipe"])
@pytest.mark.parametrize("n", [1023, 1024, 1025, 4096, 4097, 4098, 8193, 8194, 300_001])
def test_replay(gpu_ctx, oracle, kind, n):
    k = keys(kind, n)
    assert (gpu_ctx.sort_keys(k) == oracle.sort_perm(k)).all()
