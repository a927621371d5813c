"""The parallel std::shuffle against libstdc++'s: lengths around the block of
draws settled at once (1,024 draws, two swaps each), both parities, and both
sides of 46,340 elements, where one draw starts to serve one swap."""

import pytest

from potreeconverter_b200 import PINNED_SEED

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 3, 4, 1023, 2047, 2048, 2049, 2050, 9_999, 20_007, 46_339, 46_340, 46_341, 46_342, 250_001])
@pytest.mark.parametrize("seed", [PINNED_SEED, 0, 1, 2_147_483_647, 4_294_967_295])
def test_shuffle(gpu_ctx, oracle, n, seed):
    assert (gpu_ctx.shuffle(n, seed) == oracle.shuffle(n, seed)).all()
