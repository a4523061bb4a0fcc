"""How many block slots a tiled sheet stores for its blocks: the padding that the assembly and every
product read.  Rows of 9 and of 13 blocks alternate on a grid of alternating diagonals (1.21 slots a block
if each slice mixed them); boundary rows and the ends of the tiles' segments leave a few percent.  And how much shared memory a cluster's CTAs are launched with.
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


def test_clusters_of_few_sheets_run_one_cta_per_sm(ctx_factory):
    """A tile of 45 x 45 quads leaves room for a second CTA on its SM, which only a batch of many sheets may use:
    two of the lone sheet's CTAs, with the 1 KB the device reserves for each and their static shared memory of
    over 5 KB, exceed an SM's 228 KB; the batch has more clusters of 9 CTAs than 148 SMs hold at one each."""
    lone, many = (ctx_factory(scenes.windy_batch(n, 45, seed=6).sheets).solver_info() for n in (1, 60))
    assert 2 * (lone["smem_bytes"] + 6 * 1024) > 228 * 1024
    assert many["clusters"] * many["ctas_per_cluster"] > 148
