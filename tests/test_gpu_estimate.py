"""The request loop admits jobs by an estimate of their device memory; it
covers clouds whose conflict lists are as long as they get: points that all lie
within a spacing of one another in a few clumps."""

import numpy as np
import pytest

from potreeconverter_b200 import synth

pytestmark = pytest.mark.gpu


def clumps(n, number):
    """n points in `number` clumps 0.1 m wide, in a cube of 1,000 m."""
    las = bytearray(synth.terrain(n, 3, extent=1000.0))
    off, rec = int.from_bytes(las[96:100], "little"), int.from_bytes(las[105:107], "little")
    points = np.frombuffer(bytes(las[off:]), dtype=np.uint8).reshape(-1, rec).copy()
    xyz = points[:, :12].copy().view("<i4")
    rng = np.random.default_rng(6)
    lo, hi = xyz.min(0), xyz.max(0)
    centres = rng.integers(lo + 100, hi - 100, (number, 3))
    xyz[:] = centres[np.arange(n) % number] + rng.integers(-50, 51, (n, 3))
    points[:, :12] = xyz.view(np.uint8)
    las[off:] = points.tobytes()
    return bytes(las)


@pytest.mark.parametrize("n,number", [(3_000, 2), (20_000, 4), (100_000, 20), (200_000, 28), (1_000_000, 90), (1_000_000, 250), (3_000_000, 300)])
def test_estimate_covers_clumps(gpu_ctx, n, number):
    las = clumps(n, number)
    st = gpu_ctx.convert_stats(las, method="poisson", name="clumps")
    assert st["device_estimate_bytes"] >= st["device_peak_bytes"], st["device_peak_bytes"]
