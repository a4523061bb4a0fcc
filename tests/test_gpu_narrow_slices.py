"""Sheets with nodes that no face uses: slices of one block per row beside the panels that exceed a CTA's
shared memory.  The on-chip solvers against the batched loop with block-Jacobi alone.

Tolerance: dv of solves to an FP64-checked 1e-10 by two routes, 1e-6 norm-wise relative.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from clothsimulator_b200 import native, scenes


def with_unused(scene, extra, shift):
    """The scene's sheets with rest coordinates moved by `shift` (unused nodes count as at the origin)."""
    for s in scene.sheets:
        s["uv"] = (s["uv"] + np.float32(shift)).astype(np.float32)
        s["x"] = np.concatenate([s["x"], np.zeros((extra, 3), np.float32)])
        s["v"] = np.concatenate([s["v"], np.zeros((extra, 3), np.float32)])
    return scene


SCENES = {"70": lambda: with_unused(scenes.windy_batch(1, 70, seed=1), 33, -1.0),
          "68": lambda: with_unused(scenes.windy_batch(1, 68, seed=2), 160, -0.5),
          "45 at once": lambda: with_unused(scenes.windy_batch(40, 45, seed=3), 64, -0.5),
          "260 irregular": lambda: with_unused(scenes.large_irregular(260, seed=4), 64, -0.5)}


@pytest.mark.parametrize("name", SCENES)
def test_unused_nodes_on_chip(ctx_factory, name):
    scene = SCENES[name]()
    ctx = ctx_factory(scene.sheets)
    used = np.concatenate([np.isin(np.arange(len(s["x"])), s["fx"]) for s in scene.sheets])

    def dv(**kw):
        p = native.step_params(scene.dt, scene.gravity, scene.handle_stiffness, tol=1e-10, max_iters=20000, advance=0, **kw)
        stats, _ = ctx.step(p)
        assert stats.converged == len(scene.sheets)
        return ctx.get_dv().astype(np.float64)[used], stats.loop_trips

    ref, _ = dv(solver=native.SOLVER_BATCHED, coarse=0)
    for kw in (dict(precond_degree=3), dict(precond_degree=3, coarse=0), dict(precond_degree=1)):
        got, trips = dv(**kw)
        assert trips == 0
        assert np.linalg.norm(got - ref) <= 1e-6 * np.linalg.norm(ref)


@pytest.mark.parametrize("name", SCENES)
def test_unused_nodes_stay(ctx_factory, name):
    """A node without a face has an empty row of the system: no preconditioner moves it."""
    scene = SCENES[name]()
    ctx = ctx_factory(scene.sheets)
    unused = np.concatenate([~np.isin(np.arange(len(s["x"])), s["fx"]) for s in scene.sheets])
    for solver in (native.SOLVER_AUTO, native.SOLVER_BATCHED):
        for degree, coarse in ((3, 1), (3, 0), (1, 1), (1, 0)):
            p = native.step_params(scene.dt, scene.gravity, scene.handle_stiffness, tol=1e-7, max_iters=20000, advance=0,
                                   solver=solver, precond_degree=degree, coarse=coarse)
            stats, _ = ctx.step(p)
            assert stats.converged == len(scene.sheets) and not np.any(ctx.get_dv()[unused])
