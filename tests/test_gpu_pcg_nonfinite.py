"""A PCG that meets a NaN or an infinity reports it: no form of the solve counts it as converged.

Sizes as in test_gpu_pcg_forms: the unscaled PCG as one cluster, with one 32-row slice to a warp and with several; the
scaled PCG as one cluster, as CTAs on every SM and in its looping form.
"""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from andosim_b200 import learned, scenes

pytestmark = pytest.mark.gpu
NOT_SPD = 2


def chain(V):
    """SPD block system of a chain of V vertices: 4 I on the diagonal, -I between neighbours."""
    i = np.arange(V)
    rows = np.concatenate([i, i[1:], i[:-1]]); cols = np.concatenate([i, i[:-1], i[1:]])
    o = np.lexsort((cols, rows))
    rows, cols = rows[o], cols[o]
    vals = np.where(rows == cols, 4.0, -1.0)[:, None, None] * np.eye(3)
    rowptr = np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=V))])
    return rowptr.astype(np.int32), cols.astype(np.int32), vals.astype(np.float32), np.random.default_rng(V).normal(size=3 * V).astype(np.float32)


def solve(abi, rowptr, cols, vals, rhs, tol=1e-4):
    import torch

    V = len(rowptr) - 1
    d = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (rowptr, cols, vals, rhs)]
    x, work = torch.empty(3 * V, device="cuda"), torch.empty(24 * V, device="cuda")
    it, st, rel = C.c_int32(-1), C.c_int32(-1), C.c_double(-1.0)
    rc = abi.lib().ando_pcg_solve_noalloc(0, C.c_void_p(torch.cuda.current_stream().cuda_stream), V, *(t.data_ptr() for t in d), x.data_ptr(),
                                          work.data_ptr(), 24 * V, tol, 200, C.byref(it), C.byref(st), C.byref(rel))
    assert rc == abi.ANDO_OK
    return st.value, rel.value, x.cpu().numpy()


@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("V", [1, 33, 8192, 8193, 120000])
def test_unscaled(abi, V, bad):
    rowptr, cols, vals, rhs = chain(V)
    k = int(rowptr[V // 2])                       # a block of the middle row
    for where in ("rhs", "block", "all of rhs"):
        v, b = vals.copy(), rhs.copy()
        if where == "rhs":
            b[3 * (V // 2) + 1] = bad
        elif where == "block":
            v[k, 0, 0] = bad
        else:
            b[:] = bad
        status, rel, _ = solve(abi, rowptr, cols, v, b)
        assert status == NOT_SPD and not rel < 1e-4, (where, status, rel)
    status, rel, x = solve(abi, rowptr, cols, vals, rhs)      # nothing is left of it
    assert status == 0 and rel < 1e-4 and np.isfinite(x).all()


@pytest.mark.parametrize("precond", ["block_jacobi", "learned"])
@pytest.mark.parametrize("n", [16, 65, 276])
def test_scaled(abi, n, precond):
    """A velocity that is NaN at one vertex: so are the gradient and the right-hand side there."""
    sc = scenes.c4(n=n, size=2.0 * (n - 1) / 255.0)
    S = abi.Scene(sc.vertices, sc.triangles, sc.material)
    if precond == "learned":
        S.set_precond_weights(learned.load_weights())
    p = abi.make_params(dict(sc.params, max_newton_steps=1), semantics="corrected", precond=precond)
    v = np.zeros_like(sc.vertices)
    v[n // 2, 1] = np.nan
    S.upload(sc.vertices, v)
    st = S.step(p, sc.pins_at(0), sc.walls)
    assert st["newton_iters"] > 0 and st["pcg_not_converged"] == st["newton_iters"]
    assert (st["precond_fallbacks"] == st["newton_iters"]) == (precond == "learned")
    x, _ = S.download()
    np.testing.assert_array_equal(x, sc.vertices)      # no direction was found, and nothing moved
    S.close()
