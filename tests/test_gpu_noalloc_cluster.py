"""The allocation-free solve's cluster kernel at the sizes where its split over CTAs, row lanes and
on-chip blocks changes: fewer rows than CTAs, ragged and empty shares, the largest size (blocks
beyond shared memory), against an FP64 solve of the same system."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from clothsimulator_b200 import native


def _spd_system(n, per_row, seed):
    """A seeded symmetric, diagonally dominant block system with rows of 1 to ~2 per_row blocks."""
    import scipy.sparse as sp

    rng = np.random.default_rng(seed)
    k = int(n * per_row / 2)
    i = rng.integers(0, n, k)
    j = np.clip(i + rng.integers(-40, 41, k), 0, n - 1)
    keep = i != j
    i, j = i[keep], j[keep]
    _, first = np.unique(np.minimum(i, j).astype(np.int64) * n + np.maximum(i, j), return_index=True)
    i, j = i[first], j[first]
    blk = rng.normal(0.0, 1.0, (len(i), 3, 3))
    diag = np.zeros((n, 3, 3))
    for r, b in ((i, blk), (j, blk.transpose(0, 2, 1))):
        np.add.at(diag, r, np.abs(b).sum(axis=(1, 2))[:, None, None] * np.eye(3))
    diag += rng.uniform(0.01, 1.0, n)[:, None, None] * np.eye(3)
    rows = np.concatenate([i, j, np.arange(n)])
    cols = np.concatenate([j, i, np.arange(n)])
    val = np.concatenate([blk, blk.transpose(0, 2, 1), diag]).astype(np.float32)
    order = np.lexsort((cols, rows))
    rp = np.zeros(n + 1, np.int32)
    rp[1:] = np.cumsum(np.bincount(rows, minlength=n))
    A = sp.bsr_matrix((val[order].astype(np.float64), cols[order].astype(np.int32), rp), shape=(3 * n, 3 * n))
    return rp, cols[order].astype(np.int32), val[order], A.tocsc(), rng.normal(0.0, 1.0, 3 * n).astype(np.float32)


@pytest.mark.parametrize("n,per_row", [(1, 0), (5, 4), (15, 6), (17, 30), (129, 8), (2049, 11), (2500, 44), (16384, 13)])
def test_sizes_against_fp64(n, per_row):
    import scipy.sparse.linalg as sla
    import torch

    rp, ci, val, A, b = _spd_system(n, per_row, 100 + n)
    d = [torch.from_numpy(a.reshape(-1)).cuda() for a in (rp, ci, val, b)]
    x = torch.full((3 * n + 8,), 7.0, device="cuda")
    torch.cuda.synchronize()
    lib, it, rr = native.load_library(), ctypes.c_int(0), ctypes.c_double(-1.0)
    first = None
    for _ in range(2):  # the second solve finds the scratch as the first left it: the same bits
        st = lib.cs_solve_block_csr_noalloc(n, len(ci), *(t.data_ptr() for t in d), x.data_ptr(), 1e-9, 5000, None,
                                            ctypes.byref(it), ctypes.byref(rr))
        assert st == native.CS_OK and 0 <= rr.value <= 1e-9
        out = x.cpu().numpy()
        assert np.all(out[3 * n:] == 7.0)
        assert first is None or np.array_equal(out, first)
        first = out
    ref = sla.spsolve(A, b.astype(np.float64))
    # the residual's tolerance times the condition of the diagonally dominant system (below 1e3),
    # and the FP32 rounding of x
    assert np.linalg.norm(out[:3 * n] - ref) <= 1e-6 * np.linalg.norm(ref)


@pytest.mark.parametrize("nq,tol", [(40, 1e-7), (64, 1e-8), (100, 1e-8), (120, 1e-6)])
def test_solution_overshoots_the_tolerance(ctx_factory, nq, tol):
    """The last sweep ends at a fifth of the tolerance (and a tenth of that for the recursive residual's
    drift), so that x is as close to the solution as that of a solver that stops anywhere below it."""
    import torch

    from clothsimulator_b200 import scenes

    scene = scenes.hang(nq, 1)
    ctx = ctx_factory(scene.sheets)
    ctx.assemble(native.step_params(scene.dt, scene.gravity, scene.handle_stiffness))
    rp, ci, val, b = ctx.system()
    d = [torch.from_numpy(np.ascontiguousarray(a).reshape(-1)).cuda() for a in (rp, ci, val, b)]
    x = torch.zeros(len(b), device="cuda")
    torch.cuda.synchronize()
    it, rr = ctypes.c_int(0), ctypes.c_double(-1.0)
    st = native.load_library().cs_solve_block_csr_noalloc(len(rp) - 1, len(ci), *(t.data_ptr() for t in d), x.data_ptr(), tol,
                                                          20000, None, ctypes.byref(it), ctypes.byref(rr))
    assert st == native.CS_OK and rr.value <= 0.24 * tol
