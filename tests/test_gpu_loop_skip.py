"""The batched solve loop runs only when a sheet needs it: no trip when every sheet is solved on chip, by
the graph or launched from the host, with the same bits; trips as soon as one sheet is not."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from clothsimulator_b200 import native, scenes


def params_for(scene, **kw):
    return native.step_params(scene.dt, scene.gravity, scene.handle_stiffness, tol=1e-8, max_iters=20000, advance=0, **kw)


@pytest.mark.parametrize("scene", [scenes.hang(1), scenes.hang(16), scenes.windy_batch(130, 4, seed=3),
                                   scenes.uneven_batch(5, seed=4, nq_range=(4, 100))], ids=lambda s: s.name)
def test_loop_runs_only_for_sheets_that_need_it(ctx_factory, scene):
    ctx = ctx_factory(scene.sheets)
    out = {}
    for solver in (native.SOLVER_AUTO, native.SOLVER_BATCHED):
        for graph in (1, 0):
            stats, _ = ctx.step(params_for(scene, solver=solver, use_graph=graph))
            assert stats.converged == len(scene.sheets)
            assert (stats.loop_trips > 0) == (solver == native.SOLVER_BATCHED)
            out[solver, graph] = ctx.get_dv().copy()
        assert np.array_equal(out[solver, 1], out[solver, 0])


def test_steps_on_chip_launch_nothing_of_the_loop(ctx_factory):
    """Where every sheet is solved on chip, a step's launches are the assembly's two, the solve set-up's two, the
    solver's and the state update's, whether captured or not; the same steps by the loop take more."""
    scene = scenes.hang(32, 1)
    ctx = ctx_factory(scene.sheets)
    made = {}
    for solver in (native.SOLVER_AUTO, native.SOLVER_BATCHED, native.SOLVER_AUTO):
        for graph in (1, 0):
            p = native.step_params(scene.dt, scene.gravity, scene.handle_stiffness, tol=1e-7, max_iters=20000, advance=0,
                                   precond_degree=3, solver=solver, use_graph=graph)
            c0 = ctx.counters()["launches"]
            stats, _ = ctx.step(p)
            assert stats.converged == 1
            made[solver, graph] = ctx.counters()["launches"] - c0
            dv = ctx.get_dv().copy()
            if solver == native.SOLVER_AUTO:
                assert stats.loop_trips == 0
                assert np.array_equal(dv, made.setdefault("dv", dv))
    assert made[native.SOLVER_AUTO, 0] == made[native.SOLVER_AUTO, 1] == 6
    assert min(made[native.SOLVER_BATCHED, g] for g in (0, 1)) > 50
