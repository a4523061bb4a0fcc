"""How many block slots a tiled sheet stores for its blocks: the padding that the assembly and every
product read.  Rows of 9 and of 13 blocks alternate on a grid of alternating diagonals (1.21 slots a block
if each slice mixed them); boundary rows and the ends of the tiles' segments leave a few percent.
"""
import pytest

pytestmark = pytest.mark.gpu

from clothsimulator_b200 import scenes


@pytest.mark.parametrize("make,most", [(lambda: scenes.hang(64, 1), 1.06), (lambda: scenes.windy_batch(3, 45, seed=2), 1.08),
                                       (lambda: scenes.precision_sheet(150, seed=3), 1.03), (lambda: scenes.precision_sheet(256, seed=4), 1.03),
                                       (lambda: scenes.large_irregular(200, seed=5), 1.06)])
def test_tiled_rows_are_stored_with_little_padding(ctx_factory, make, most):
    ctx = ctx_factory(make().sheets)
    assert ctx.sizes[3] <= most * ctx.sizes[6]
