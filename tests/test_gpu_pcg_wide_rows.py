"""Rows of many blocks in the unscaled PCG: a hub coupled to much of a mesh, and rows that are all wide.

Such rows are summed by their warp. The bound on the time is far above what that takes (3 to 12 times the same mesh without
the hub) and far below what a row summed by one thread took (170 to 490 times).
"""
from __future__ import annotations

import ctypes as C
import time

import numpy as np
import pytest

from test_gpu_pcg_forms import EPS, grid_csr, matvec

pytestmark = pytest.mark.gpu


def solve(abi, rowptr, cols, vals, rhs, tol, repeat=1):
    import torch

    V = len(rowptr) - 1
    d = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (rowptr, cols, vals, rhs)]
    x, work = torch.empty(3 * V, device="cuda"), torch.empty(24 * V, device="cuda")
    it, st, rel = C.c_int32(-1), C.c_int32(-1), C.c_double(-1.0)
    best = 1e9
    for _ in range(repeat):
        t0 = time.perf_counter()
        rc = abi.lib().ando_pcg_solve_noalloc(0, C.c_void_p(torch.cuda.current_stream().cuda_stream), V, *(t.data_ptr() for t in d), x.data_ptr(),
                                              work.data_ptr(), 24 * V, tol, 400, C.byref(it), C.byref(st), C.byref(rel))
        best = min(best, time.perf_counter() - t0)
        assert rc == abi.ANDO_OK and st.value == 0
    return x.cpu().numpy().astype(np.float64).reshape(V, 3), it.value, best


def band(V, half, seed):
    """SPD block system in which every vertex couples with `half` on either side."""
    rng = np.random.default_rng(seed)
    a = np.concatenate([np.arange(V - k) for k in range(1, half + 1)])
    b = a + np.concatenate([np.full(V - k, k) for k in range(1, half + 1)])
    n = rng.normal(size=(len(a), 3))
    B = (np.eye(3) + n[:, :, None] * n[:, None, :] / (n * n).sum(1)[:, None, None]) / half
    D = np.tile(np.eye(3), (V, 1, 1))
    np.add.at(D, a, B)
    np.add.at(D, b, B)
    i = np.arange(V)
    r = np.concatenate([a, b, i]); c = np.concatenate([b, a, i]); v = np.concatenate([-B, -B, D])
    o = np.lexsort((c, r))
    rowptr = np.concatenate([[0], np.cumsum(np.bincount(r, minlength=V))])
    return rowptr.astype(np.int32), r[o], c[o].astype(np.int32), v[o].astype(np.float32), rng.normal(size=3 * V).astype(np.float32)


def check(system, x, it, tol):
    rowptr, rows, cols, vals, rhs = system
    V = len(rowptr) - 1
    y, size = matvec(rows, cols, vals.astype(np.float64), x, V)
    b = rhs.astype(np.float64).reshape(V, 3)
    assert np.abs(b - y).max() <= tol * np.abs(b).max() + (it + 8) * EPS * size.max()


@pytest.mark.parametrize("V,half", [(V, half) for V in (1000, 9000) for half in (15, 16, 31, 32, 70)] + [(120000, 15), (120000, 16)])
def test_wide_rows(abi, V, half):
    """31, 33, 63, 65 and 141 blocks a row; the cluster, one slice to a warp and several."""
    system = band(V, half, V + half)
    x, it, _ = solve(abi, system[0], system[2], system[3], system[4], 1e-5)
    check(system, x, it, 1e-5)


@pytest.mark.parametrize("nx,hub", [(90, 3000), (274, 8000)])
def test_a_hub_does_not_hold_up_the_others(abi, nx, hub):
    plain, with_hub = grid_csr(nx, nx, nx), grid_csr(nx, nx, nx, hub)
    _, it0, t0 = solve(abi, plain[0], plain[2], plain[3], plain[4], 1e-4, repeat=5)
    x, it, t = solve(abi, with_hub[0], with_hub[2], with_hub[3], with_hub[4], 1e-4, repeat=5)
    check(with_hub, x, it, 1e-4)
    assert t / it < 40.0 * t0 / it0
