"""The warp decoder of LAZ chunks against the scalar decoder of laz.cuh on
chunks of long runs of one byte, which drive the coder into its first and last
symbols: some are decoded and some (cut short) refused, by both alike."""

import numpy as np
import pytest

from perf import cases
from tests.test_gpu_laz_warp import device_decode, host_decode, image  # noqa: F401 - host_decode is a fixture

pytestmark = pytest.mark.gpu


def chunks(pdrf, extra):
    """(LAZ image, whether it is cut short), of 24 chunks of runs."""
    rec = cases.REC_LEN[pdrf] + extra
    for seed in range(24):
        rng = np.random.default_rng([seed, pdrf, extra, 2])
        count = int(rng.integers(2, 900 if seed % 2 else 12))
        cut = seed % 4 == 3
        size = rec + 4 + (int(rng.integers(0, 8)) if cut else count * (rec + 24))
        runs = size // 20 + 1
        body = np.repeat(rng.choice(np.array([0, 255, 128, 1], np.uint8), runs), rng.integers(20, 200, runs))[:size - rec]
        data = np.concatenate([rng.integers(0, 256, rec, dtype=np.uint8), body])
        assert data.size == size
        yield image([data.tobytes()], [count], count, pdrf, extra), cut


@pytest.mark.parametrize("pdrf", [0, 1, 2, 3])
@pytest.mark.parametrize("extra", [0, 1, 7, 64])
def test_chunks_of_runs(gpu_ctx, host_decode, pdrf, extra):  # noqa: F811
    decoded = refused = 0
    for laz, cut in chunks(pdrf, extra):
        want, got = host_decode(laz), device_decode(gpu_ctx, laz)
        assert got == want
        decoded += want is not None
        refused += want is None
    assert decoded >= 4 and refused >= 1, (decoded, refused)
