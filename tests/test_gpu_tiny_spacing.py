"""Spacings whose reciprocal is infinite, and an infinite one: a candidate on
the node's lower planes has no cell number then (0 times infinity), and must
get a cell all the same. Decisions are the oracle's."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# (the reference's window of poisson_average is undefined for the huge ones)
@pytest.mark.parametrize("method,spacing", [(m, s) for m in ("poisson", "poisson_average") for s in (5e-324, 1e-310, 5e-309, 6e-309, 1e-200)]
                         + [("poisson", 1e300), ("poisson", np.inf)])
@pytest.mark.parametrize("n", [3, 40, 3_000])
def test_cells_of_extreme_spacings(gpu_ctx, oracle, method, spacing, n):
    rng = np.random.default_rng(n)
    q = rng.integers(0, 200, (n, 3), dtype=np.int32)
    q[: n // 3] = 0  # on the lower corner
    child = ((q[:, 0] >= 100).astype(np.uint8) << 2) | ((q[:, 1] >= 100).astype(np.uint8) << 1) | (q[:, 2] >= 100).astype(np.uint8)
    o = np.argsort(child, kind="stable")
    q, child = q[o], child[o]
    rgb = rng.integers(0, 65536, (n, 3), dtype=np.uint16) if method == "poisson_average" else None
    args = (method, q[:, 0], q[:, 1], q[:, 2], child, np.full(3, 0.01), np.zeros(3), np.zeros(3), np.full(3, 2.0), spacing, rgb)
    want, want_rgb = oracle.accept(*args)
    got, got_rgb = gpu_ctx.accept(*args)
    assert int((got != want).sum()) == 0
    if rgb is not None:
        assert (got_rgb == want_rgb).all()
