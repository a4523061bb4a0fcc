"""Rows of many blocks: a fan of triangles around one node, whose row couples it to every rim node.  From
182 blocks a row the proximity row kernel takes fewer rows per block; 201 is the most the assembly takes.

Tolerances (norm-wise relative): assembled system with proximities 1e-6 against the oracle's, dv of a
solve to an FP64-checked 1e-10 against the oracle's FP64 solve 1e-6.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

import pyoracle
from clothsimulator_b200 import native, scenes
from proxutil import set_oracle_proximities

THICKNESS = 5e-3


def rel(a, b):
    a, b = np.asarray(a, np.float64).reshape(-1), np.asarray(b, np.float64).reshape(-1)
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


def fan(spokes):
    """A disc of `spokes` triangles around node 0."""
    a = 2 * np.pi * np.arange(spokes) / spokes
    u = np.concatenate([[[0.0, 0.0]], np.stack([np.cos(a), np.sin(a)], 1)])
    f = np.stack([np.zeros(spokes, int), 1 + np.arange(spokes), 1 + (np.arange(spokes) + 1) % spokes], 1).astype(np.int32)
    rng = np.random.default_rng(spokes)
    x = np.concatenate([u, rng.normal(0, 1e-3, (spokes + 1, 1))], 1)
    return {"x": x.astype(np.float32), "v": rng.normal(0, 0.05, x.shape).astype(np.float32), "uv": u.astype(np.float32),
            "fx": f, "fu": f.copy(), "handles": np.array([1, 1 + spokes // 3], np.int32),
            "material": scenes.isotropic_material(50.0, 1e-5), "wind": scenes.no_wind()}


@pytest.mark.parametrize("spokes", [150, 180, 181, 190, 200])
def test_fan_with_proximities(ctx_factory, spokes):
    scene = scenes.Scene("fan", [fan(spokes), scenes.hang(8, 1).sheets[0]], dt=1.0 / 100, steps=1)
    ctx = ctx_factory(scene.sheets)

    def params(**kw):
        return native.step_params(scene.dt, scene.gravity, scene.handle_stiffness, tol=1e-10, max_iters=20000, **kw)

    prox = scenes.synthetic_proximities(scene.sheets[0], np.random.default_rng(1), n_vf=8, n_ee=5, n_ext=4,
                                        thickness=THICKNESS, node_off=0)
    for p in (None, prox):
        ctx.set_proximities(p, THICKNESS)
        ctx.assemble(params())
        rp, ci, val, b = ctx.system()
        n = spokes + 1
        assert p is not None or np.diff(rp).max() == n
        cloth = pyoracle.Cloth(scene.sheets[0], pyoracle.Material(scene.sheets[0]["material"], "float"))
        if p is not None:
            set_oracle_proximities([cloth], prox, np.array([0, n]), THICKNESS)
        orp, oci, oval, ob = cloth.assemble(scenes.step_params(scene, scene.sheets[0]))
        assert np.array_equal(rp[:n + 1], orp) and np.array_equal(ci[:rp[n]], oci)
        assert rel(val[:rp[n]], oval) < 1e-6 and rel(b[:3 * n], ob) < 1e-6
        stats, _ = ctx.step(params(advance=0))
        assert stats.converged == 2
        ref, _ = cloth.solve(pyoracle.METHOD_LLT64)
        assert rel(ctx.get_dv()[:n], ref) < 1e-6
