"""Batches around the thread count from which a context keeps to one stream: the same states as stepping alone, before and after."""
from __future__ import annotations

import numpy as np
import pytest

from andosim_b200 import scenes

pytestmark = pytest.mark.gpu


def _scene(abi, n, sheets, seed):
    sc = scenes.c2(seed=seed, n=n, sheets=sheets, wave=0.0)
    x = sc.vertices.copy()
    per = len(x) // sheets
    for k in range(sheets):   # 0.8 mm apart: contacts in every frame
        x[k * per:(k + 1) * per, 2] = 0.0008 * k
    S = abi.Scene(sc.vertices, sc.triangles, sc.material)
    S.upload(x, np.zeros_like(x), x)
    return sc, S, abi.make_params(sc.params, semantics="corrected")


@pytest.mark.parametrize("count", [7, 8, 9, 17])
def test_batch_sizes(abi, count):
    make = lambda: [_scene(abi, 5 + k % 4, 2 + k % 3, k) for k in range(count)]
    alone, batch = make(), make()
    touched = 0
    for frame in range(3):
        for sc, S, p in alone:
            S.apply_gravity(sc.gravity, p.dt)
            touched += S.step(p, [], sc.walls)["contacts"] > 0
        for sc, S, p in batch:
            S.apply_gravity(sc.gravity, p.dt)
        if frame < 2:
            abi.step_batch([S for _, S, _ in batch], [p for _, _, p in batch], [[]] * count, [sc.walls for sc, _, _ in batch])
        else:
            for sc, S, p in batch:
                S.step(p, [], sc.walls)
    assert touched > count
    for (_, a, _), (_, b, _) in zip(alone, batch):
        for u, w in zip(a.download(), b.download()):
            np.testing.assert_array_equal(u, w)
        a.close(); b.close()
