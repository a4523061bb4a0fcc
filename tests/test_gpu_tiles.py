"""The cluster-resident solver's tiles and levels at the sizes where its plan changes: rows in their own
order (fewer than two slices per CTA), tiles without and with the coarse correction, the largest sheet of
a cluster, mixed batches, two CTAs per SM with panels left in L2; against the batched loop with
block-Jacobi alone.

Tolerance: dv of solves to an FP64-checked 1e-10 by two routes, 1e-6 norm-wise relative.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from clothsimulator_b200 import native, scenes


def rel(a, b):
    a, b = np.asarray(a, np.float64).reshape(-1), np.asarray(b, np.float64).reshape(-1)
    return float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300))


def params_for(scene, **kw):
    kw.setdefault("tol", 1e-10)
    return native.step_params(scene.dt, scene.gravity, scene.handle_stiffness, max_iters=20000, advance=0, **kw)


SCENES = {"1": lambda: scenes.hang(1), "22": lambda: scenes.hang(22), "25": lambda: scenes.hang(25),
          "31": lambda: scenes.windy_batch(3, 31, seed=1), "43": lambda: scenes.windy_batch(2, 43, seed=2),
          "70": lambda: scenes.windy_batch(2, 70, seed=3), "40 at once": lambda: scenes.windy_batch(40, 45, seed=4),
          "uneven": lambda: scenes.uneven_batch(12, seed=5, nq_range=(2, 70))}


@pytest.mark.parametrize("name", SCENES)
def test_tiles_agree_with_batched_loop(ctx_factory, name):
    scene = SCENES[name]()
    ctx = ctx_factory(scene.sheets)
    assert ctx.solver_info()["resident_sheets"] == len(scene.sheets)
    ctx.step(params_for(scene, solver=native.SOLVER_BATCHED, coarse=0))
    ref = ctx.get_dv().copy()
    for kw in (dict(precond_degree=3), dict(precond_degree=3, coarse=0), dict(precond_degree=1), dict(precond_degree=7)):
        stats, _ = ctx.step(params_for(scene, **kw))
        assert stats.converged == len(scene.sheets) and stats.loop_trips == 0
        dv = ctx.get_dv().copy()
        assert rel(dv, ref) < 1e-6
        ctx.step(params_for(scene, use_graph=0, **kw))
        assert np.array_equal(ctx.get_dv(), dv)
    # a wrong warm start is scaled or rejected, the solution itself ends at once
    for factor, scale in ((1.0, 0), (4.0, 1), (4.0, 0)):
        ctx.set_warm_start(factor * ref)
        stats, _ = ctx.step(params_for(scene, precond_degree=3, tol=1e-8, warm_start=native.WARM_GIVEN, warm_scale=scale))
        assert stats.converged == len(scene.sheets)
        assert rel(ctx.get_dv(), ref) < 1e-4
    ctx.step(params_for(scene, precond_degree=3, tol=1e-5, precision=native.PREC_PLAIN_FP32), allow_unconverged=True)
    assert np.all(np.isfinite(ctx.get_dv()))
