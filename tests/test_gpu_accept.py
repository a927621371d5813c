"""One node's poisson decisions against the oracle where the acceptance from
conflict lists can go wrong: words of 32 candidates and their remainders,
batches of 81,920, lists around the 4 inline entries and the cap of 32, long
lists, and nodes where the 10,001-check cap decides."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
SCALE = np.full(3, 0.001)
OFFSET = np.zeros(3)
SIDE = 128.0  # node box: 128 spacings of 1


def node(kind, n, seed):
    """Quantized points of a node's box in child order."""
    rng = np.random.default_rng([seed, n])
    if kind == "volume":
        p = rng.uniform(0, SIDE, (n, 3))
    elif kind == "sheet":  # up to n / 128^2 candidates per square spacing
        p = np.stack([rng.uniform(0, SIDE, n), rng.uniform(0, SIDE, n), 64 + rng.normal(0, 0.2, n)], 1)
    elif kind == "shell":  # equal distances: the early exit rarely ends a scan
        v = rng.normal(0, 1, (n, 3))
        p = 64 + 60 * v / np.linalg.norm(v, axis=1, keepdims=True)
    else:  # clumps far denser than the spacing
        c = rng.uniform(10, 118, (4, 3))
        p = c[rng.integers(0, 4, n)] + rng.normal(0, 0.8, (n, 3))
    q = np.clip(np.round(p / 0.001), 0, SIDE / 0.001 - 1).astype(np.int32)
    x = q * 0.001
    child = ((x[:, 0] >= 64).astype(np.uint8) << 2) | ((x[:, 1] >= 64).astype(np.uint8) << 1) | (x[:, 2] >= 64).astype(np.uint8)
    o = np.argsort(child, kind="stable")
    return q[o], child[o]


@pytest.mark.parametrize("method", ["poisson", "poisson_average"])
@pytest.mark.parametrize("kind,n", [("sheet", n) for n in (1, 2, 31, 32, 33, 63, 65, 1023, 8191, 8192, 40_000, 81_920, 81_921, 164_000)]
                         + [("clumps", 500), ("clumps", 3_000), ("clumps", 12_345), ("shell", 30_000), ("shell", 100_000),
                            ("volume", 10_002), ("volume", 150_000)])
def test_node_decisions(gpu_ctx, oracle, method, kind, n):
    q, child = node(kind, n, 3)
    rgb = np.random.default_rng(n).integers(0, 65536, (n, 3), dtype=np.uint16) if method == "poisson_average" else None
    args = (method, q[:, 0], q[:, 1], q[:, 2], child, SCALE, OFFSET, np.zeros(3), np.full(3, SIDE), 1.0, rgb)
    want, want_rgb = oracle.accept(*args)
    got, got_rgb = gpu_ctx.accept(*args)
    assert int((got != want).sum()) == 0
    if rgb is not None:
        assert (got_rgb == want_rgb).all()
