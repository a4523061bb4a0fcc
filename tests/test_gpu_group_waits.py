"""Waits of the group-resident solver that run out, and steps of several contexts with such sheets at once.

A wait's limit of zero polls makes the first exchange between CTAs give up: the kernel returns, the step
reports CS_ERR_TIMEOUT, and the device goes on working.
"""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from clothsimulator_b200 import native, scenes


def params_for(scene, **kw):
    return native.step_params(scene.dt, scene.gravity, scene.handle_stiffness, tol=1e-8, max_iters=20000, advance=0,
                              precond_degree=3, **kw)


@pytest.mark.parametrize("use_graph", [0, 1])
def test_wait_that_runs_out_is_reported(monkeypatch, use_graph):
    scene = scenes.precision_sheet(101, seed=1)
    monkeypatch.setenv("CS_GROUP_POLLS", "0")
    ctx = native.Context(0).load(scene.sheets)
    monkeypatch.delenv("CS_GROUP_POLLS")
    for _ in range(2):
        with pytest.raises(native.ClothStepError) as e:
            ctx.step(params_for(scene, use_graph=use_graph))
        assert e.value.status == native.CS_ERR_TIMEOUT
    ctx.step(params_for(scene, solver=native.SOLVER_BATCHED))  # the context goes on: the loop has no such wait
    dv = ctx.get_dv().astype(np.float64)
    ctx.load(scene.sheets)
    ctx.step(params_for(scene, use_graph=use_graph))
    assert np.linalg.norm(ctx.get_dv() - dv) <= 1e-4 * np.linalg.norm(dv)
    ctx.close()


def test_contexts_with_group_sheets_take_turns():
    """Three contexts whose sheets each take most of the chip, stepped from three threads on three streams:
    the bits of a context alone."""
    made = [scenes.precision_sheet(101, seed=1), scenes.precision_sheet(200, seed=2), scenes.large_irregular(150, seed=3)]
    ctxs, alone, got = [native.Context(0).load(s.sheets) for s in made], [], [None] * 3
    for scene, ctx in zip(made, ctxs):
        ctx.step(params_for(scene))
        alone.append(ctx.get_dv().copy())

    def work(k):
        out = []
        for i in range(12):
            stats, _ = ctxs[k].step(params_for(made[k], use_graph=i % 2))
            out.append((stats.converged, stats.loop_trips, ctxs[k].get_dv().copy()))
        got[k] = out

    threads = [threading.Thread(target=work, args=(k,)) for k in range(3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for k in range(3):
        assert got[k] is not None and all(c == 1 and n == 0 and np.array_equal(d, alone[k]) for c, n, d in got[k])
    ctxs[0].close()  # the others go on without it
    stats, _ = ctxs[1].step(params_for(made[1]))
    assert stats.converged == 1 and np.array_equal(ctxs[1].get_dv(), alone[1])
    for c in ctxs[1:]:
        c.close()
