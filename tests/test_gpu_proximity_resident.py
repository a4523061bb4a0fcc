"""Sheets whose proximities stay inside the mesh pattern (a vertex of one sheet against a face or an
edge of another couples only neighbours of either sheet) keep the on-chip solvers; a proximity inside
one sheet couples nodes outside its pattern, and that sheet alone goes to the batched loop.

Tolerance: dv of solves to an FP64-checked 1e-10 by two routes, 1e-6 norm-wise relative.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from clothsimulator_b200 import native
from test_gpu_proximity import THICKNESS, make_case, params_for, rel


@pytest.mark.parametrize("nq", [6, 64, 72])  # one-slice strips, a full cluster, a group
@pytest.mark.parametrize("touched", [(), (1,)])
def test_in_pattern_proximities_stay_on_chip(ctx_factory, nq, touched):
    scene, prox = make_case(seed=31, n_sheets=4, nq=nq, touched=touched, pairs=((0, 3), (1, 2)))
    ctx = ctx_factory(scene.sheets)
    free, _ = ctx.step(params_for(scene, advance=0))
    dv0 = ctx.get_dv().copy()
    ctx.set_proximities(prox, THICKNESS)
    out = []
    for kw in (dict(precond_degree=3), dict(), dict(use_graph=0), dict(solver=native.SOLVER_BATCHED)):
        stats, _ = ctx.step(params_for(scene, advance=0, **kw))
        assert stats.converged == 4
        out.append((ctx.get_dv().copy(), stats.loop_trips))
    assert free.loop_trips == 0 and out[3][1] > 1
    if touched:
        assert out[0][1] > 1
    else:
        assert out[0][1] == out[1][1] == 0
    for dv, _ in out[:3]:
        assert rel(dv, out[3][0]) < 1e-6
    assert not np.array_equal(out[0][0], dv0)  # the proximities had an effect
    ctx.set_proximities(None, THICKNESS)
    ctx.step(params_for(scene, advance=0))
    assert np.array_equal(ctx.get_dv(), dv0)


@pytest.mark.parametrize("touched", [(), (1,)])
def test_steps_after_a_change_of_the_proximities_agree(ctx_factory, touched):
    """The first step after a change launches its kernels directly (where no sheet needs the loop), the
    next ones run the graph captured with the new lists: the same bits."""
    scene, prox = make_case(seed=33, n_sheets=4, nq=12, touched=touched, pairs=((0, 3), (1, 2)))
    ctx = ctx_factory(scene.sheets)
    for lists in (prox, {k: v[:-1] for k, v in prox.items()}):
        ctx.set_proximities(lists, THICKNESS)
        out = []
        for graph in (1, 1, 1, 0):
            ctx.step(params_for(scene, advance=0, precond_degree=3, use_graph=graph))
            out.append(ctx.get_dv().copy())
        for dv in out[1:]:
            assert np.array_equal(dv, out[0])
