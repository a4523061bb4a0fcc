"""Group-resident PCG (a sheet's system held in the shared memory of CTAs across the chip) against
the batched loop on the same state and an FP64 residual computed on the host.

Tolerances (norm-wise relative): dv of solves to an FP64-checked 1e-10 by the two routes, 1e-6 as
for the other solvers; the residual of the FP32-rounded dv in FP64, its rounding bound
|| |A| |dv| || 2^-24 / ||b|| more than the solve's own tolerance.
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
    kw.setdefault("max_iters", 20000)
    kw.setdefault("advance", 0)
    kw.setdefault("precond_degree", 3)
    return native.step_params(scene.dt, scene.gravity, scene.handle_stiffness, **kw)


def both_routes(ctx, scene, **kw):
    """dv by the group-resident route and by the batched loop, and the routes' loop trips."""
    out = []
    for solver in (native.SOLVER_AUTO, native.SOLVER_BATCHED):
        stats, _ = ctx.step(params_for(scene, solver=solver, **kw))
        assert stats.converged == len(scene.sheets)
        out.append((ctx.get_dv().copy(), stats.loop_trips))
    return out


def check_residual(ctx, scene, dv, tol):
    import scipy.sparse as sp

    ctx.assemble(params_for(scene))
    rp, ci, val, b = ctx.system()
    A = sp.bsr_matrix((val.astype(np.float64), ci, rp)).tocsr()
    x = dv.reshape(-1).astype(np.float64)
    bn = np.linalg.norm(b.astype(np.float64))
    bound = np.linalg.norm(abs(A) @ np.abs(x)) * 2.0 ** -24
    assert np.linalg.norm(b - A @ x) <= tol * bn + bound


SCENES = {
    # the smallest sheet beyond a cluster of 10 CTAs (161 slices), an odd size, the panels about
    # filling the chip's shared memory, the largest that is tiled
    "windy 72": lambda: scenes.windy_batch(1, 72, seed=1),
    "precision 101": lambda: scenes.precision_sheet(101, seed=2),
    "precision 256": lambda: scenes.precision_sheet(256, seed=3),
    "precision 274": lambda: scenes.precision_sheet(274, seed=4),
    # rows of up to 17 blocks; panels beyond shared memory
    "irregular 97": lambda: scenes.large_irregular(97, seed=5),
    "irregular 262": lambda: scenes.large_irregular(262, seed=6),
    # several sheets side by side and one after another, with cluster-resident ones
    "uneven": lambda: scenes.uneven_batch(14, seed=7, nq_range=(40, 128)),
}


@pytest.mark.parametrize("name", SCENES)
def test_agrees_with_batched_loop(ctx_factory, name):
    scene = SCENES[name]()
    ctx = ctx_factory(scene.sheets)
    (a, trips_a), (b, trips_b) = both_routes(ctx, scene)
    assert trips_a == 0 < trips_b  # every sheet is solved on chip
    assert rel(a, b) < 1e-6
    check_residual(ctx, scene, a, 1e-10)


@pytest.mark.parametrize("kw", [dict(precond_degree=1), dict(precond_degree=5, coarse=0), dict(precond_degree=1, coarse=0)])
def test_preconditioners(ctx_factory, kw):
    scene = scenes.windy_batch(2, 80, seed=8)
    ctx = ctx_factory(scene.sheets)
    (a, _), (b, _) = both_routes(ctx, scene, **kw)
    assert rel(a, b) < 1e-6


def test_graph_host_loop_and_repeat_give_the_same_bits(ctx_factory):
    scene = scenes.uneven_batch(6, seed=9, nq_range=(72, 128))
    ctx = ctx_factory(scene.sheets)
    out = []
    for graph in (1, 1, 0):
        ctx.step(params_for(scene, use_graph=graph))
        out.append(ctx.get_dv().copy())
    assert np.array_equal(out[0], out[1]) and np.array_equal(out[0], out[2])


def test_warm_starts(ctx_factory):
    """The exact solution ends at once; a worse start than zero is rejected, and accepted once scaled."""
    scene = scenes.windy_batch(2, 90, seed=10)
    ctx = ctx_factory(scene.sheets)
    ctx.step(params_for(scene))
    dv = ctx.get_dv().copy()
    it0 = ctx.instance_stats()[0].copy()
    for factor, scale, rejected in ((1.0, 0, False), (4.0, 0, True), (4.0, 1, False), (-2.0, 1, False)):
        ctx.set_warm_start(factor * dv)
        stats, _ = ctx.step(params_for(scene, warm_start=native.WARM_GIVEN, warm_scale=scale, tol=1e-8))
        assert (stats.warm_rejected == 2) == rejected
        assert rel(ctx.get_dv(), dv) < 1e-5
        if not rejected:
            assert stats.max_iters <= 0.5 * it0.max()


def test_cap_and_plain_precision(ctx_factory):
    """An iteration cap is reported; plain FP32 PCG is the batched loop's."""
    scene = scenes.windy_batch(1, 80, seed=11)
    ctx = ctx_factory(scene.sheets)
    stats, st = ctx.step(params_for(scene, max_iters=5), allow_unconverged=True)
    assert st == native.CS_ERR_NOT_CONVERGED and stats.converged == 0 and stats.max_iters == 5
    stats, _ = ctx.step(params_for(scene, tol=1e-5, precision=native.PREC_PLAIN_FP32, coarse=0), allow_unconverged=True)
    assert stats.loop_trips > 1


def test_too_large_a_sheet_stays_in_the_loop(ctx_factory):
    scene = scenes.precision_sheet(290, seed=12)
    ctx = ctx_factory(scene.sheets)
    stats, _ = ctx.step(params_for(scene, tol=1e-6))
    assert stats.converged == 1 and stats.loop_trips > 1
