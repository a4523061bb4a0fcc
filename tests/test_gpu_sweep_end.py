"""Where the on-chip solvers end their last sweep with block-Jacobi: no deeper than the batched loop does,
whose iterations they then take.

The iterations of block-Jacobi CG on one system by two kernels (their sums' orders differ) agree to a few.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from clothsimulator_b200 import native, scenes


@pytest.mark.parametrize("make", [lambda: scenes.hang(16, 1), lambda: scenes.hang(64, 1), lambda: scenes.windy_batch(4, 45, seed=2),
                                  lambda: scenes.precision_sheet(90, seed=3)])
def test_block_jacobi_iterations_as_in_the_loop(ctx_factory, make):
    scene = make()
    ctx = ctx_factory(scene.sheets)
    total = []
    for solver in (native.SOLVER_AUTO, native.SOLVER_BATCHED):
        p = native.step_params(scene.dt, scene.gravity, scene.handle_stiffness, tol=1e-6, max_iters=20000, advance=0,
                               precond_degree=1, coarse=0, solver=solver)
        stats, _ = ctx.step(p)
        assert stats.converged == len(scene.sheets)
        total.append(stats.total_iters)
    assert abs(total[0] - total[1]) <= 0.03 * total[1]
