"""The captured frame's loop against the host-driven one: every way an iteration, an inner step or the beta loop can end."""
from __future__ import annotations

import numpy as np
import pytest

from andosim_b200 import scenes

pytestmark = pytest.mark.gpu


def _frames(abi, sc, p, profiled, frames=4):
    S = abi.Scene(sc.vertices, sc.triangles, sc.material)
    S.profile_enable(profiled)
    rng = np.random.default_rng(5)
    S.upload(sc.vertices + rng.normal(scale=1e-4, size=sc.vertices.shape), rng.normal(scale=0.2, size=sc.vertices.shape), sc.vertices)
    stats = []
    for f in range(frames):
        S.apply_gravity(sc.gravity, p.dt)
        stats.append(S.step(p, sc.pins_at(f), sc.walls))
    out = S.download()
    S.close()
    return out, stats


@pytest.mark.parametrize("n", [3, 16, 17])   # 9, 256 and 289 vertices: one block of the last kernel, filled, and two
@pytest.mark.parametrize("params", [
    dict(max_newton_steps=1), dict(max_newton_steps=2, beta_max=0.1), dict(max_newton_steps=8, beta_max=0.9),
    dict(beta_max=0.0), dict(pcg_tol=1e3), dict(pcg_max_iters=1, max_newton_steps=3),
    dict(enable_friction=True, friction_mu=0.3), dict(enable_strain_limiting=True, strain_tau=0.001)])
def test_loop(abi, n, params):
    sc = scenes.c1(n=n)
    p = abi.make_params(dict(sc.params, **params), semantics="reference")
    (xg, vg), sg = _frames(abi, sc, p, False)
    (xh, vh), sh = _frames(abi, sc, p, True)
    assert all(s["graph_launched"] for s in sg) and not any(s["graph_launched"] for s in sh)
    np.testing.assert_array_equal(xg, xh)
    np.testing.assert_array_equal(vg, vh)
    for a, b in zip(sg, sh):
        for k in ("newton_iters", "pcg_iters", "pcg_max_per_newton", "pcg_not_converged", "line_search_fail", "strain_active", "beta", "last_alpha"):
            assert a[k] == b[k], k


def test_no_iterations(abi):
    sc = scenes.c1(n=9)
    p = abi.make_params(dict(sc.params, max_newton_steps=0), semantics="reference")
    (x, _), st = _frames(abi, sc, p, False, frames=1)
    assert st[0]["graph_launched"] and st[0]["newton_iters"] == 0 and st[0]["line_search_fail"] == 1 and st[0]["beta"] == 0.0
    assert np.isfinite(x).all()
