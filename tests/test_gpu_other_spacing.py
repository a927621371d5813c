"""Acceptance of a node whose box does not measure 128 spacings, as a caller of
the single entry point may ask: positions many thousand spacings from the
node's corner have no room for the FP32 test's error."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("method", ["poisson", "poisson_average"])
@pytest.mark.parametrize("spacing", [2.0, 1.0, 0.1, 0.001, 0.0003])
def test_small_spacings(gpu_ctx, oracle, method, spacing):
    rng = np.random.default_rng(1)
    n, scale = 20_000, spacing / 1000
    q = np.round((np.array([120.0, 110.0, 100.0]) + rng.uniform(0, min(20 * spacing, 8.0), (n, 3))) / scale).astype(np.int32)
    rgb = rng.integers(0, 65536, (n, 3), dtype=np.uint16) if method == "poisson_average" else None
    args = (method, q[:, 0], q[:, 1], q[:, 2], np.full(n, 7, np.uint8), np.full(3, scale), np.zeros(3), np.zeros(3), np.full(3, 128.0), spacing, rgb)
    want, want_rgb = oracle.accept(*args)
    got, got_rgb = gpu_ctx.accept(*args)
    assert int((got != want).sum()) == 0
    if rgb is not None:
        assert (got_rgb == want_rgb).all()
