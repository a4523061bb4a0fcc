"""Rest coordinates that are not finite are refused with CS_ERR_INVALID_ARG, by the faces they give no area, on
the sheets of every solver; where no face uses them they do not matter."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from clothsimulator_b200 import native, scenes


@pytest.mark.parametrize("nq", [6, 40, 90])
@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_rest_coordinates_that_are_not_finite(nq, bad):
    scene = scenes.hang(nq, 1)
    s = scene.sheets[0]
    good = s["uv"].copy()
    s["uv"] = good.copy()
    s["uv"][nq + 2::3] = bad
    ctx = native.Context(0)
    with pytest.raises(native.ClothStepError) as e:
        ctx.load(scene.sheets)
    assert e.value.status == native.CS_ERR_INVALID_ARG
    s["uv"] = np.concatenate([good, np.full((1, 2), bad, np.float32)])
    ctx.load(scene.sheets)
    stats, _ = ctx.step(native.step_params(scene.dt, scene.gravity, scene.handle_stiffness, max_iters=20000, precond_degree=3))
    assert stats.converged == 1
    ctx.close()
