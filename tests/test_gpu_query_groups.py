"""The shared descent's groups: queries of a warp that lie together, apart, at one point, far away, or partly nowhere."""
from __future__ import annotations

import numpy as np
import pytest

from andosim_b200 import scenes
from test_gpu_broad_phase import gpu_pairs, oracle_pairs

pytestmark = pytest.mark.gpu


def _check(oracle, abi, sc, x, pad):
    x = x.astype(np.float32).astype(np.float64)
    vo, eo = oracle_pairs(oracle, sc, x, pad)
    vg, eg = gpu_pairs(abi, sc, x, pad)
    np.testing.assert_array_equal(vg, vo)
    np.testing.assert_array_equal(eg, eo)
    return len(vo) + len(eo)


@pytest.mark.parametrize("n", [5, 6, 9, 17])       # 25 to 289 vertices: part of a warp, one warp, several and a rest
@pytest.mark.parametrize("shape", ["rest", "shuffled", "two halves", "one point", "line", "far corner"])
def test_positions(oracle, abi, n, shape):
    sc = scenes.c1(n=n)
    rng = np.random.default_rng(n)
    x = sc.vertices + rng.normal(scale=0.003, size=sc.vertices.shape)
    if shape == "shuffled":            # neighbours of the order lie anywhere
        x = x[rng.permutation(len(x))]
    elif shape == "two halves":        # every other vertex far off: each run spans both
        x[::2] += [3.0, 0.0, 1.0]
    elif shape == "one point":         # boxes without extent, all equal
        x[:] = [0.25, -0.5, 0.125]
    elif shape == "line":
        x[:, 1:] = 0.0
    elif shape == "far corner":        # one vertex makes the hierarchy's box huge
        x[-1] += 1e6
    pairs = _check(oracle, abi, sc, x, 0.01)
    if shape != "far corner":
        assert pairs > 0


@pytest.mark.parametrize("n", [6, 12])
def test_sheets_apart(oracle, abi, n):
    sc = scenes.c2(n=n, sheets=3, wave=0.0)
    x = sc.vertices.copy()
    per = len(x) // 3
    for k, z in enumerate((0.0, 0.004, 50.0)):
        x[k * per:(k + 1) * per, 2] = z
    assert _check(oracle, abi, sc, x, 0.005) > 0
