"""The PCG kernels at the sizes where their form changes.

The unscaled PCG (``ando_pcg_solve_noalloc``) is one cluster up to 8,192 rows, then one CTA per SM
with a 32-row slice to each warp, from 113,665 rows on with several. The
scaled PCG of the CORRECTED step is one cluster (8,192 rows, 1,024 with contact blocks or wide
rows), CTAs of 512 threads, of up to 1,024 on every SM, and a looping form above 151,552 rows.

Each solution is put back into its system in FP64. A PCG that stops at max|r| < tol max|b| has a true
residual of at most that plus the drift of its FP32 recurrence and the rounding of the FP32 result, one
unit in the last place of max(|A| |x|) per iteration and a few for the result.
"""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from andosim_b200 import learned, scenes

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -24


def matvec(rows, cols, vals, x, n):
    """Block rows times x (n, 3), and the same with absolute values."""
    y, a = np.zeros((n, 3)), np.zeros((n, 3))
    p = np.einsum("kab,kb->ka", vals, x[cols])
    q = np.einsum("kab,kb->ka", np.abs(vals), np.abs(x[cols]))
    for c in range(3):
        y[:, c] = np.bincount(rows, p[:, c], n)
        a[:, c] = np.bincount(rows, q[:, c], n)
    return y, a


# ------------------------------------------------------------------ unscaled, a caller's system
def grid_csr(nx, ny, seed, hub=0):
    """SPD 3x3-block system on a triangulated nx by ny grid; the first `hub` vertices also couple with vertex 0."""
    rng = np.random.default_rng(seed)
    V = nx * ny
    i = np.arange(V)
    x, y = i % nx, i // nx
    a, b = [], []
    for dx, dy in ((1, 0), (0, 1), (-1, 1)):
        ok = (x + dx >= 0) & (x + dx < nx) & (y + dy < ny)
        a.append(i[ok]); b.append(i[ok] + dx + nx * dy)
    if hub:
        far = np.setdiff1d(np.arange(2, min(hub, V)), [nx - 1, nx, nx + 1])
        a.append(np.zeros(len(far), int)); b.append(far)
    a, b = np.concatenate(a), np.concatenate(b)
    n = rng.normal(size=(len(a), 3))
    n /= np.linalg.norm(n, axis=1)[:, None]
    B = rng.uniform(2, 6, len(a))[:, None, None] * (0.3 * np.eye(3) + n[:, :, None] * n[:, None, :])
    D = np.tile(np.eye(3), (V, 1, 1))
    np.add.at(D, a, B)
    np.add.at(D, b, B)
    r = np.concatenate([a, b, i]); c = np.concatenate([b, a, i]); v = np.concatenate([-B, -B, D])
    o = np.lexsort((c, r))
    rowptr = np.concatenate([[0], np.cumsum(np.bincount(r, minlength=V))])
    return rowptr.astype(np.int32), r[o], c[o].astype(np.int32), v[o].astype(np.float32), rng.normal(size=3 * V).astype(np.float32)


@pytest.mark.parametrize("nx,ny,hub,shift", [
    (1, 1, 0, 0), (33, 1, 0, 1), (31, 33, 0, 0), (40, 30, 900, 3), (128, 64, 0, 0),      # cluster
    (8193, 1, 0, 2), (300, 250, 3000, 0),                                                 # one slice to a warp
    (400, 300, 0, 1), (500, 460, 0, 0), (600, 575, 0, 0),                                 # several
])
def test_unscaled_pcg(abi, nx, ny, hub, shift):
    """`shift`: the arrays start that many elements past a 16-byte boundary."""
    import torch

    rowptr, rows, cols, vals, rhs = grid_csr(nx, ny, nx + ny, hub)
    V, tol = nx * ny, 1e-4

    def dev(a):
        t = torch.zeros(a.size + 8, dtype=torch.from_numpy(a[:0]).dtype, device="cuda:0")
        t[shift:shift + a.size] = torch.from_numpy(np.ascontiguousarray(a).ravel()).cuda()
        return t, C.c_void_p(t.data_ptr() + 4 * shift)

    (kr, pr), (kc, pc), (kv, pv), (kb, pb) = dev(rowptr), dev(cols), dev(vals), dev(rhs)
    out = []
    for _ in range(2):
        x, px = dev(np.full(3 * V, np.nan, np.float32))
        work, pw = dev(np.full(24 * V, np.nan, np.float32))
        it, st, rel = C.c_int32(-1), C.c_int32(-1), C.c_double(-1.0)
        rc = abi.lib().ando_pcg_solve_noalloc(0, C.c_void_p(torch.cuda.current_stream().cuda_stream), V, pr, pc, pv, pb, px, pw, 24 * V, tol,
                                              2000, C.byref(it), C.byref(st), C.byref(rel))
        assert rc == abi.ANDO_OK and st.value == 0, (rc, st.value, abi.lib().ando_last_error())
        assert 0 <= rel.value < tol
        out.append(x[shift:shift + 3 * V].cpu().numpy())
    np.testing.assert_array_equal(out[0], out[1])
    x = out[0].astype(np.float64).reshape(V, 3)
    y, size = matvec(rows, cols, vals.astype(np.float64), x, V)
    b = rhs.astype(np.float64).reshape(V, 3)
    assert np.abs(b - y).max() <= tol * np.abs(b).max() + (it.value + 8) * EPS * size.max()


# ------------------------------------------------------------------ scaled, the CORRECTED step's system
def solve_step(abi, sc, precond, tol=1e-4):
    """The last Newton system that a step of `sc` solved: statistics of the step, the scaled system, the solution."""
    S = abi.Scene(sc.vertices, sc.triangles, sc.material)
    if precond == "learned":
        S.set_precond_weights(learned.load_weights())
    S.keep_system()
    p = abi.make_params(dict(sc.params, pcg_tol=tol, max_newton_steps=1, pcg_max_iters=2000), semantics="corrected", precond=precond)
    S.apply_gravity(sc.gravity, p.dt)
    p.dt = 1.0 / 600.0      # one sub-step
    st = S.step(p, sc.pins_at(0), sc.walls)
    rowptr, cols, vals, _, d = S.last_system()
    xrow, xcol, xvals = S.last_contact_blocks()
    s = S.last_scaled_system()          # factors and right-hand side; a block-Jacobi step keeps no CSR copy of the scaled blocks
    S.close()
    V = len(rowptr) - 1
    rows = np.concatenate([np.repeat(np.arange(V), np.diff(rowptr)), xrow])
    cols = np.concatenate([cols, xcol])
    M = np.zeros((V, 3, 3))             # L^-1
    for k, (i, j) in enumerate(((0, 0), (1, 0), (1, 1), (2, 0), (2, 1), (2, 2))):
        M[:, i, j] = s["Linv"][:, k]
    vals = np.concatenate([vals, xvals]).astype(np.float64)
    sysm = dict(rows=rows, cols=cols, V=V, contact_blocks=len(xrow), width=int(np.diff(rowptr).max()), M=M,
                vals=np.einsum("kab,kbc,kdc->kad", M[rows], vals, M[cols]),                                   # A^ = L^-1 A L^-T
                size=np.einsum("kab,kbc,kdc->kad", np.abs(M[rows]), np.abs(vals), np.abs(M[cols])),           # with absolute values
                b=s["bhat"].astype(np.float64).reshape(V, 3))
    return st, sysm, d.astype(np.float64).reshape(-1, 3)


def check_scaled(st, s, d, tol=1e-4):
    assert st["pcg_iters"] > 0 and st["precond_fallbacks"] == 0
    V, r, c, v, b = s["V"], s["rows"], s["cols"], s["vals"], s["b"]
    L = np.linalg.inv(s["M"])
    y, _ = matvec(r, c, v, np.einsum("vba,vb->va", L, d), V)                                                  # x^ = L^T d
    size, _ = matvec(r, c, s["size"], np.einsum("vba,vb->va", np.abs(L), np.abs(d)), V)
    stop = tol * np.abs(b).max()
    if st["pcg_not_converged"]:
        # the reference's absolute stop |p^T A p| < 1e-16 (pcg_solver.cpp:8-75), met by a system of tiny forces:
        # |r| <= |p| <= sqrt(1e-16 / smallest eigenvalue)
        A = np.zeros((3 * V, 3 * V))
        for k in range(len(r)):
            A[3 * r[k]:3 * r[k] + 3, 3 * c[k]:3 * c[k] + 3] += v[k]
        stop = 1e-8 / np.sqrt(np.linalg.eigvalsh(A)[0])
    bound = stop + (st["pcg_iters"] + 8) * EPS * size.max()
    assert np.abs(b - y).max() <= bound, (np.abs(b - y).max(), bound)


@pytest.mark.parametrize("n,precond", [
    (4, "block_jacobi"), (11, "learned"), (64, "block_jacobi"), (64, "learned"),          # cluster
    (65, "block_jacobi"), (65, "learned"), (194, "learned"),                               # CTAs of 512 threads
    (195, "block_jacobi"), (257, "learned"), (258, "block_jacobi"), (275, "learned"),      # up to 896, 1,024
    (276, "block_jacobi"),                                                                 # looping
])
def test_scaled_pcg(abi, n, precond):
    sc = scenes.c4(n=n, size=2.0 * (n - 1) / 255.0)
    st, s, d = solve_step(abi, sc, precond)
    assert s["contact_blocks"] == 0
    if precond == "block_jacobi" or n >= 64:          # the shipped weights were trained on larger curtains
        check_scaled(st, s, d)


@pytest.mark.parametrize("n,precond", [(10, "block_jacobi"), (22, "learned"), (40, "block_jacobi"), (100, "learned"), (150, "block_jacobi"),
                                       (200, "block_jacobi")])
def test_scaled_pcg_with_contact_blocks(abi, n, precond):
    """Two curtains 0.8 mm apart: contact blocks at every vertex."""
    sc = scenes.c4(n=n, size=2.0 * (n - 1) / 255.0, spacing=0.0008)
    st, s, d = solve_step(abi, sc, precond)
    assert s["contact_blocks"] > len(d)
    check_scaled(st, s, d)


@pytest.mark.parametrize("n", [9, 40, 130, 200])
def test_scaled_pcg_with_wide_rows(abi, n):
    """Bending doubles the blocks of a row."""
    sc = scenes.c4(n=n, size=2.0 * (n - 1) / 255.0)
    sc.material["bending_stiffness"] = 1e-5
    st, s, d = solve_step(abi, sc, "block_jacobi")
    assert s["width"] > 9
    check_scaled(st, s, d)
