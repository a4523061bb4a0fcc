"""The backward kernels of the learned warm start at the edges of their 128-node tiles: minibatches of
less than a tile, whole tiles, a tile and a remainder, more tiles than thread blocks, and ranges that
start inside the batch, against the FP64 restatement.

Tolerance (norm-wise relative): the gradients pass up to three layers through tensor-core products of
operands rounded to BF16 (relative 2^-9 each, two per product), 6 * 2^-9 in all; the loss is FP32.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

import mlp_oracle
from clothsimulator_b200 import scenes
from test_gpu_mlp import batch_neighbours, recorded_ctx, rel


@pytest.mark.parametrize("sheets,nq,s0,s1", [(3, 2, 0, 3), (2, 2, 1, 2), (1, 15, 0, 1), (2, 10, 0, 2), (5, 16, 1, 4),
                                             (70, 16, 0, 70)])
def test_gradient_at_tile_edges(sheets, nq, s0, s1):
    scene = scenes.windy_batch(sheets, nq, seed=7)
    ctx, _ = recorded_ctx(scene, 2)
    w = ctx.mlp_get_weights()
    feat, target = ctx.mlp_get_record(1)
    n = (nq + 1) ** 2
    nb = [j - n * s0 for j in batch_neighbours(scene)[n * s0:n * s1]]
    g, loss = ctx.mlp_gradient(1, s0, s1)
    loss_ref, g_ref, _ = mlp_oracle.loss_and_grad(w, feat[n * s0:n * s1].astype(np.float64),
                                                  target[n * s0:n * s1].astype(np.float64), nb)
    assert abs(loss - loss_ref) / loss_ref < 1e-4
    assert rel(g, g_ref) < 6 * 2.0 ** -9
    ctx.close()
