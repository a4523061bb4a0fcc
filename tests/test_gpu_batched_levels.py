"""The batched loop's multilevel correction (coarse.cu) at the sizes where its grids change: no finer cells
(a few nodes), fine cells only, middle and fine cells, the largest coarse grid of one CTA and the
smallest that a cluster inverts; uneven batches; the plain FP32 solver.

Tolerances: dv solved to an FP64-checked 1e-10 with and without the correction, 1e-6 norm-wise relative.
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
    return native.step_params(scene.dt, scene.gravity, scene.handle_stiffness, max_iters=20000, advance=0,
                              solver=native.SOLVER_BATCHED, **kw)


CASES = [("4 nodes", lambda: scenes.hang(1), 1.0), ("fine cells", lambda: scenes.hang(15), 1.0),
         ("96", lambda: scenes.windy_batch(2, 96, seed=3), 0.7), ("irregular 240", lambda: scenes.large_irregular(240, seed=4), 0.5),
         ("irregular 515", lambda: scenes.large_irregular(515, seed=5), 0.6),
         ("uneven", lambda: scenes.uneven_batch(9, seed=6, nq_range=(2, 90)), 0.9)]


@pytest.mark.parametrize("name,make,fewer", CASES, ids=[c[0] for c in CASES])
def test_levels_agree_with_block_jacobi(ctx_factory, name, make, fewer):
    scene = make()
    ctx = ctx_factory(scene.sheets)
    out, its = [], []
    for kw in (dict(coarse=0), dict(coarse=1), dict(coarse=1), dict(coarse=1, use_graph=0)):
        stats, _ = ctx.step(params_for(scene, **kw))
        assert stats.converged == len(scene.sheets) and stats.loop_trips > 0
        out.append(ctx.get_dv().copy())
        its.append(stats.max_iters)
    assert rel(out[1], out[0]) < 1e-6
    assert np.array_equal(out[1], out[2]) and np.array_equal(out[1], out[3])
    assert its[1] <= max(fewer * its[0], its[0] + 4 if fewer == 1.0 else 0)
    stats, _ = ctx.step(params_for(scene, tol=1e-4, precision=native.PREC_PLAIN_FP32, coarse=1), allow_unconverged=True)
    assert np.all(np.isfinite(ctx.get_dv())) and stats.max_rel_residual < 1e-2
