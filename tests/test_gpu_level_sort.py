"""The order in which a node's candidates are decided, against the oracle,
where the sort by quantised distance can go wrong: tiles of 2,048 and their
remainders, runs of candidates with one quantised distance (put in order one
by one up to 32, sorted again on all 64 bits beyond), and equal distances in
runs short and long."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
SIDE = 128.0  # node box: 128 spacings of 1


def node(kind, n):
    """Positions in units of the scale, and the scale."""
    rng = np.random.default_rng([ord(kind[0]), n])
    scale = 1e-6 if kind in ("line", "knot") else 1e-3
    if kind == "sheet":
        p = np.stack([rng.uniform(0, SIDE, n), rng.uniform(0, SIDE, n), np.full(n, 64.0)], 1)
    elif kind == "line":  # distinct distances, from the centre on: n / 27,000 quantised ones at first
        p = np.full((n, 3), 64.0)
        p[:, 0] += 1e-6 * rng.permutation(n)
    elif kind == "knot":  # far from the centre, a few thousand in one quantised distance
        p = np.array([100.0, 90.0, 80.0]) + rng.uniform(0, 1e-5, (n, 3))
    else:  # copies of few positions: equal distances
        p = rng.uniform(0, SIDE, (max(n // 300, 1), 3))[rng.integers(0, max(n // 300, 1), n)]
        p[: n // 2] = rng.uniform(0, SIDE, (n // 2, 3))
    q = np.clip(np.round(p / scale), 0, SIDE / scale - 1).astype(np.int32)
    x = q * scale
    child = ((x[:, 0] >= 64).astype(np.uint8) << 2) | ((x[:, 1] >= 64).astype(np.uint8) << 1) | (x[:, 2] >= 64).astype(np.uint8)
    o = np.argsort(child, kind="stable")
    return q[o], child[o], np.full(3, scale)


@pytest.mark.parametrize("method", ["poisson", "poisson_average"])
@pytest.mark.parametrize("kind,n", [("sheet", 2047), ("sheet", 2048), ("sheet", 2049), ("sheet", 4097), ("sheet", 70_000),
                                    ("line", 40), ("line", 20_000), ("line", 60_000), ("knot", 33), ("knot", 5_000),
                                    ("copies", 90), ("copies", 700), ("copies", 20_000)])
def test_order_of_decisions(gpu_ctx, oracle, method, kind, n):
    q, child, scale = node(kind, n)
    rgb = np.random.default_rng(n).integers(0, 65536, (n, 3), dtype=np.uint16) if method == "poisson_average" else None
    args = (method, q[:, 0], q[:, 1], q[:, 2], child, scale, np.zeros(3), np.zeros(3), np.full(3, SIDE), 1.0, rgb)
    want, want_rgb = oracle.accept(*args)
    got, got_rgb = gpu_ctx.accept(*args)
    assert int((got != want).sum()) == 0
    if rgb is not None:
        assert (got_rgb == want_rgb).all()
