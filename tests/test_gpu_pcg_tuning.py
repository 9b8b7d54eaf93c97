"""The scaled PCG's launch shapes where they differ: contact blocks, wide rows and the looping form.

Without contact blocks a mesh whose blocks fit on the chip has one launch, whichever candidate is chosen; with them the candidates
keep 22, 15 or 9 of a row's blocks there.
"""
from __future__ import annotations

import numpy as np
import pytest

from andosim_b200 import learned, scenes

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
