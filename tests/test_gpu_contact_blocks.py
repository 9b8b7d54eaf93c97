"""The contact Hessian's blocks at the key widths of their sort, and after steps that end with and without an assembly."""
from __future__ import annotations

import numpy as np
import pytest

from andosim_b200 import scenes

pytestmark = pytest.mark.gpu


def _blocks(S):
    rows, cols, vals = S.last_contact_blocks()
    assert (np.diff(rows.astype(np.int64) * S.V + cols) > 0).all()   # one block each, by row and column
    assert (rows != cols).all() and np.isfinite(vals).all() and (np.abs(vals).max(axis=(1, 2)) > 0).any()
    # the two blocks of a pair come from the same products, summed in the same order
    order = np.lexsort((rows, cols))
    np.testing.assert_array_equal(cols[order], rows)
    np.testing.assert_array_equal(rows[order], cols)
    np.testing.assert_array_equal(vals[order].transpose(0, 2, 1), vals)
    return rows, cols, vals


def _padded(sc, V):
    """The scene's sheets and, far below, a strip that brings it to V vertices and touches nothing."""
    n = len(sc.vertices)
    k = np.arange(V - n)
    strip = np.stack([0.01 * k, 0.01 * (k % 2), np.full(len(k), -50.0)], axis=1)
    tri = np.arange(max(0, V - n - 2))[:, None] + np.arange(3)[None, :] + n
    return np.concatenate([sc.vertices, strip]), np.concatenate([sc.triangles, tri.astype(np.int32)]) if len(tri) else sc.triangles


# 12 x 12 x 4 vertices alone; keys of 16 + 16 bits up to 65,536 vertices, 17 + 17 above
@pytest.mark.parametrize("V", [65536, 65537, 131073])
def test_blocks_at_key_widths(abi, V):
    sc = scenes.c2(n=12, sheets=4, wave=0.0)
    rng = np.random.default_rng(3)
    x = sc.vertices.copy()
    per = len(x) // 4
    for k in range(4):   # the sheets 0.7 mm apart, slightly rough
        x[k * per:(k + 1) * per, 2] = 0.0007 * k + rng.normal(scale=2e-5, size=per)
    out = []
    for pad in (None, V):
        xv, tri = (sc.vertices, sc.triangles) if pad is None else _padded(sc, pad)
        S = abi.Scene(xv, tri, sc.material)
        xs = xv.copy()
        xs[:len(x)] = x
        S.upload(xs, np.zeros_like(xs), xs)
        S.eval_system(abi.make_params(sc.params, semantics="corrected"))
        rows, cols, vals = _blocks(S)
        g = S.last_gradient()[:3 * len(x)]
        assert rows.max() < len(x)
        out.append((rows, cols, vals, g))
        S.close()
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("tol", [1e-12, 1e12])
def test_blocks_after_a_step(abi, tol):
    sc = scenes.c2(n=12, sheets=3, wave=0.0)
    x = sc.vertices.copy()
    per = len(x) // 3
    for k in range(3):
        x[k * per:(k + 1) * per, 2] = 0.0007 * k
    S = abi.Scene(sc.vertices, sc.triangles, sc.material)
    S.upload(x, np.zeros_like(x), x)
    p = dict(sc.params, pcg_tol=tol)   # 1e12: the second Newton system counts as converged and is not assembled
    S.step(abi.make_params(p, semantics="corrected"), [], sc.walls)
    _blocks(S)
    S.close()
