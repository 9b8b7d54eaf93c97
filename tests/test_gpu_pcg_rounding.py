"""The unscaled PCG rounds a row's product the same way in every form, and as little as a butterfly over eight lanes does.

Block e of a row goes into part e mod 8, and the parts are added ((0 + 4) + (2 + 6)) + ((1 + 5) + (3 + 7)), which keeps the chain
of additions at a row of n blocks to n / 8 + 3. Two iterations are restated here rounding by rounding and must agree in every
bit: with a residual of 1e-4 of terms that cancel, the order of such a sum decides what a solve of a stiff system converges to.
"""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
F, W = np.float32, np.longdouble      # W: 64 bits of mantissa, so that a sum rounds once, to F


def fma(a, b, c):
    return (a.astype(W) * b.astype(W) + c.astype(W)).astype(F)


def dot3(a, b):
    return fma(a[..., 2], b[..., 2], fma(a[..., 0], b[..., 0], (a[..., 1] * b[..., 1]).astype(F)))


def system(nx, ny, reach, seed):
    """SPD blocks between grid vertices at most `reach` apart; 4 I on the diagonal, whose inverse is exact."""
    rng = np.random.default_rng(seed)
    V = nx * ny
    i = np.arange(V)
    x, y = i % nx, i // nx
    a, b = [], []
    for dx in range(-reach, reach + 1):
        for dy in range(0, reach + 1):
            if (dy, dx) > (0, 0) and (reach > 1 or dx + dy != 2):          # reach 1: the grid's triangulation, 7 blocks a row
                ok = (x + dx >= 0) & (x + dx < nx) & (y + dy < ny)
                a.append(i[ok]); b.append(i[ok] + dx + nx * dy)
    a, b = np.concatenate(a), np.concatenate(b)
    B = (rng.normal(size=(len(a), 3, 3)) * 0.4 / (2 * reach + 1) ** 2).astype(F)
    r = np.concatenate([a, b, i]); c = np.concatenate([b, a, i])
    v = np.concatenate([B, B.transpose(0, 2, 1), np.tile(4 * np.eye(3, dtype=F), (V, 1, 1))])
    o = np.lexsort((c, r))
    return np.concatenate([[0], np.cumsum(np.bincount(r, minlength=V))]).astype(np.int32), c[o].astype(np.int32), v[o], \
        rng.normal(size=(V, 3)).astype(F)


def product(rowptr, cols, vals, p):
    n = np.diff(rowptr)
    t = dot3(vals, p[cols][:, None, :])
    parts = np.zeros((8, len(n), 3), F)
    for e in range(n.max()):
        on = e < n
        parts[e % 8, on] += t[rowptr[:-1][on] + e]
    for o in (4, 2, 1):
        parts = parts[:o] + parts[o:2 * o]
    return parts[0]


def two_iterations(rowptr, cols, vals, b):
    total = lambda u, v: float((u.astype(np.float64) * v).sum())
    x, r, p, z = np.zeros_like(b), b.copy(), None, b / F(4)
    rz = total(r, z)
    for _ in range(2):
        p = z if p is None else fma(np.full_like(z, beta), p, z)
        q = product(rowptr, cols, vals, p)
        alpha = F(rz / total(p, q))
        x, r = fma(np.full_like(p, alpha), p, x), fma(np.full_like(q, -alpha), q, r)
        z = r / F(4)
        rz, old = total(r, z), rz
        beta = F(rz / old)
    return x, float(np.abs(r).max()) / float(np.abs(b).max())


@pytest.mark.parametrize("reach", [1, 2])          # 7 and up to 25 blocks a row, which the buffers do not hold whole
@pytest.mark.parametrize("nx,ny", [(40, 30), (90, 89), (91, 100), (323, 300), (350, 340)])    # cluster, cluster; one slice to a warp (20, 24 warps); several
def test_two_iterations(abi, nx, ny, reach):
    import torch

    rowptr, cols, vals, b = system(nx, ny, reach, nx + reach)
    V = nx * ny
    d = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (rowptr, cols, vals, b)]
    x, work = torch.empty(3 * V, device="cuda"), torch.empty(24 * V, device="cuda")
    it, st, rel = C.c_int32(-1), C.c_int32(-1), C.c_double(-1.0)
    rc = abi.lib().ando_pcg_solve_noalloc(0, C.c_void_p(torch.cuda.current_stream().cuda_stream), V, *(t.data_ptr() for t in d), x.data_ptr(),
                                          work.data_ptr(), 24 * V, 1e-30, 2, C.byref(it), C.byref(st), C.byref(rel))
    assert rc == abi.ANDO_OK and (it.value, st.value) == (2, 1)      # stopped by the iteration cap
    want, want_rel = two_iterations(rowptr, cols, vals, b)
    np.testing.assert_array_equal(x.cpu().numpy().reshape(V, 3), want)
    assert rel.value == want_rel
