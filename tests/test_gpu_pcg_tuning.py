"""The scaled PCG's launch shapes where they differ: contact blocks, wide rows and the looping form.

Without contact blocks a mesh whose blocks fit on the chip has one launch, whichever candidate is chosen; with them the candidates
keep 22, 15 or 9 of a row's blocks there.
"""
from __future__ import annotations

import numpy as np
import pytest

from andosim_b200 import learned, scenes
from test_gpu_pcg_forms import EPS, matvec, solve_step

pytestmark = pytest.mark.gpu
CLOSE = 0.0008        # metres between the curtains: below the activation distance everywhere


def scene(abi, n, precond, spacing, index=-1, bending=0.0):
    sc = scenes.c4(n=n, size=2.0 * (n - 1) / 255.0, spacing=spacing)
    sc.material["bending_stiffness"] = bending
    S = abi.Scene(sc.vertices, sc.triangles, sc.material)
    if precond == "learned":
        S.set_precond_weights(learned.load_weights())
    S.select_pcg_shape(precond == "learned", index)
    S.select_assembly_tpb(1)      # fixed, so that tune_ms counts the PCG's timing only
    p = abi.make_params(dict(sc.params, max_newton_steps=3), semantics="corrected", precond=precond)
    p.dt = 1.0 / 600.0
    return sc, S, p


@pytest.mark.parametrize("precond", ["block_jacobi", "learned"])
def test_a_mesh_is_tuned_again_on_its_first_contact_blocks(abi, precond):
    sc, S, p = scene(abi, 48, precond, 0.003)
    apart = S.step(p, sc.pins_at(0), sc.walls)
    free = S.pcg_shape(precond == "learned")
    assert apart["contacts"] == 0 and free["tune_ms"] > 0
    x = sc.vertices.copy()
    x[len(x) // 2:, 1] -= 0.003 - CLOSE
    seen = []
    for _ in range(2):
        S.upload(x, np.zeros_like(x), x)
        assert S.step(p, sc.pins_at(0), sc.walls)["contacts"] > len(x)
        seen.append(S.pcg_shape(precond == "learned"))
    S.upload(sc.vertices, np.zeros_like(x), sc.vertices)
    S.step(p, sc.pins_at(0), sc.walls)
    again = S.pcg_shape(precond == "learned")
    S.close()
    assert seen[0]["tune_ms"] > free["tune_ms"] and seen[1] == seen[0]
    assert (seen[0]["tpb"], seen[0]["grid"]) == (256, 18)        # 144 slices, 8 to a CTA: the launch with contact blocks
    assert (free["tpb"], free["grid"]) == (288, 16)              # and the cluster without
    assert {k: again[k] for k in ("tpb", "grid", "unroll")} == {k: free[k] for k in ("tpb", "grid", "unroll")}
    assert again["tune_ms"] == seen[0]["tune_ms"]


def run(abi, n, precond, spacing, index, bending=0.0, frames=2):
    sc, S, p = scene(abi, n, precond, spacing, index, bending)
    iters = 0
    for f in range(frames):
        S.apply_gravity(sc.gravity, p.dt)
        iters += S.step(p, sc.pins_at(f), sc.walls)["pcg_iters"]
    rows = S.last_contact_blocks()[0]
    width = 7 + int(np.bincount(rows).max()) if len(rows) else 13 if bending else 7
    out = (*S.download(), iters, S.pcg_shape(precond == "learned"), width)
    S.close()
    return out


@pytest.mark.parametrize("precond", ["block_jacobi", "learned"])
@pytest.mark.parametrize("n,spacing,bending,wide", [(22, CLOSE, 0.0, 25), (60, CLOSE, 0.0, 25), (60, 0.003, 1e-5, 13), (276, 0.003, 0.0, 0)])
def test_every_shape_gives_the_same_bits(abi, n, spacing, bending, wide, precond):
    """Cluster and grid with contact blocks, wide rows, and the looping form."""
    x0, v0, it0, shape, width = run(abi, n, precond, spacing, 0, bending)
    assert it0 > 0 and shape["candidates"] >= 3 and shape["tune_ms"] == 0
    assert width >= wide        # more of a row's blocks than every candidate keeps on the chip (bending: than the smallest does)
    used = [(shape["tpb"], shape["grid"], shape["unroll"])]
    for k in range(1, shape["candidates"]):
        x, v, it, s, _ = run(abi, n, precond, spacing, k, bending)
        used.append((s["tpb"], s["grid"], s["unroll"]))
        assert it == it0
        np.testing.assert_array_equal(x, x0)
        np.testing.assert_array_equal(v, v0)
    assert len(set(used)) >= 3


def residual(st, s, d):
    L = np.linalg.inv(s["M"])
    y, _ = matvec(s["rows"], s["cols"], s["vals"], np.einsum("vba,vb->va", L, d), s["V"])
    size, _ = matvec(s["rows"], s["cols"], s["size"], np.einsum("vba,vb->va", np.abs(L), np.abs(d)), s["V"])
    return np.abs(s["b"] - y).max(), 1e-4 * np.abs(s["b"]).max() + (st["pcg_iters"] + 8) * EPS * size.max()


@pytest.mark.parametrize("n,precond", [(11, "learned"), (276, "learned"), (276, "block_jacobi")])
def test_solution(abi, n, precond):
    """A curtain the network was not trained for (whichever solve ended it), and the looping form."""
    st, s, d = solve_step(abi, scenes.c4(n=n, size=2.0 * (n - 1) / 255.0), precond)
    assert st["pcg_iters"] > 0 and st["pcg_not_converged"] == 0
    r, bound = residual(st, s, d)
    assert r <= bound


@pytest.mark.parametrize("precond", ["block_jacobi", "learned"])
def test_a_few_rows_with_very_many_contacts(abi, precond):
    """A coarse sheet close under a fine one, a coarse vertex in every slice of 32: the contact blocks' copy by slices would be
    mostly padding, so the solve walks them row by row."""
    nf, nc, size = 62, 8, 0.3
    fine, coarse = scenes.grid_plane(nf, size), scenes.grid_plane(nc, size)
    rng = np.random.default_rng(4)
    fine[:, :2] = fine[:, :2] * 0.98 + 0.003
    v = np.concatenate([fine + [0, 0, 0.5 + CLOSE], coarse + [0, 0, 0.5]]) + rng.uniform(-2e-5, 2e-5, (nf * nf + nc * nc, 3))
    tris = np.concatenate([scenes.grid_triangles(nf, nf), scenes.grid_triangles(nc, nc, offset=nf * nf)])
    place = np.empty(len(v), int)                       # new index of each vertex
    place[nf * nf:] = 32 * np.arange(nc * nc) + 5
    place[:nf * nf] = np.setdiff1d(np.arange(len(v)), place[nf * nf:])
    x = np.empty_like(v)
    x[place] = v
    sc = scenes.c1(n=4)
    sc.vertices, sc.triangles, sc.walls = x, place[tris].astype(np.int32), []
    sc.pins = [(int(place[nf * nf]), x[place[nf * nf]].copy())]
    st, s, d = solve_step(abi, sc, precond)
    count = np.bincount(s["rows"][len(s["rows"]) - s["contact_blocks"]:], minlength=-(-len(x) // 32) * 32)
    assert 32 * count.reshape(-1, 32).max(axis=1).sum() > 6 * s["contact_blocks"] + 65536
    assert st["pcg_iters"] > 0 and st["pcg_not_converged"] == 0
    r, bound = residual(st, s, d)
    assert r <= bound


@pytest.mark.parametrize("m,launch", [(71, (96, 1)), (72, (96, 1)), (200, (224, 1)), (900, (256, 4))])
def test_a_hub_in_a_small_mesh(abi, m, launch):
    """A disc of m triangles about one vertex: up to 72 slots one cluster, above the grid's launch."""
    th = np.linspace(0, 2 * np.pi, m, endpoint=False)
    sc = scenes.c1(n=4)
    sc.vertices = np.concatenate([[[0, 0, 1.0]], np.stack([np.cos(th), np.sin(th), np.ones(m)], 1)])
    i = np.arange(m)
    sc.triangles = np.stack([np.zeros(m, int), 1 + i, 1 + (i + 1) % m], 1).astype(np.int32)
    sc.pins, sc.walls = [(0, sc.vertices[0].copy())], []
    st, s, d = solve_step(abi, sc, "block_jacobi")
    assert s["width"] == m + 1 and st["pcg_iters"] > 0 and st["pcg_not_converged"] == 0
    r, bound = residual(st, s, d)
    assert r <= bound
    S = abi.Scene(sc.vertices, sc.triangles, sc.material)
    S.step(abi.make_params(sc.params, semantics="corrected"), sc.pins, [])
    shape = S.pcg_shape(False)
    S.close()
    assert (shape["tpb"], shape["grid"]) == launch


def test_a_small_mesh_with_few_wide_contact_rows(abi):
    """The same at 909 rows: by slices an iteration took 118 times one without contacts, row by row it takes 50 times."""
    nf, nc, size = 30, 3, 0.145
    fine, coarse = scenes.grid_plane(nf, size), scenes.grid_plane(nc, size)
    rng = np.random.default_rng(4)
    fine[:, :2] = fine[:, :2] * 0.98 + 0.001
    noise = rng.uniform(-2e-5, 2e-5, (nf * nf + nc * nc, 3))
    place = np.empty(nf * nf + nc * nc, int)
    place[nf * nf:] = 96 * np.arange(nc * nc) + 5
    place[:nf * nf] = np.setdiff1d(np.arange(len(place)), place[nf * nf:])
    tris = np.concatenate([scenes.grid_triangles(nf, nf), scenes.grid_triangles(nc, nc, offset=nf * nf)])
    each = []
    for gap in (CLOSE, 0.1):
        x = np.empty((len(place), 3))
        x[place] = np.concatenate([fine + [0, 0, 0.5 + gap], coarse + [0, 0, 0.5]]) + noise
        sc = scenes.c1(n=4)
        sc.vertices, sc.triangles, sc.walls = x, place[tris].astype(np.int32), []
        sc.pins = [(int(place[nf * nf]), x[place[nf * nf]].copy())]
        if gap == CLOSE:
            st, s, d = solve_step(abi, sc, "block_jacobi")
            assert s["contact_blocks"] > 3000 and st["pcg_iters"] > 0 and st["pcg_not_converged"] == 0
            r, bound = residual(st, s, d)
            assert r <= bound
        S = abi.Scene(sc.vertices, sc.triangles, sc.material)
        S.select_pcg_shape(False, 0)
        p = abi.make_params(dict(sc.params, max_newton_steps=1, pcg_tol=1e-30, pcg_max_iters=100), semantics="corrected")
        p.dt = 1.0 / 600.0
        S.step(p, sc.pins, [])
        S.profile_enable(True)
        best = 1e9
        for _ in range(3):
            before = S.profile()["phase_ms"]["pcg"]
            S.upload(x, np.full_like(x, -0.01), x)
            it = S.step(p, sc.pins, [])["pcg_iters"]
            assert it >= 20
            best = min(best, (S.profile()["phase_ms"]["pcg"] - before) / it)
        each.append(best)
        S.close()
    assert each[0] < 80.0 * each[1]
