"""The traversal's leaf queue: queries that overlap more leaves than a warp's queue holds, one step after another."""
from __future__ import annotations

import numpy as np
import pytest

from andosim_b200 import scenes
from test_gpu_broad_phase import gpu_pairs, oracle_pairs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,pad", [(3, 1.0), (6, 0.2), (11, 1.0), (18, 0.12), (18, 1.0)])
def test_dense_overlap(oracle, abi, n, pad):
    sc = scenes.c1(n=n)
    rng = np.random.default_rng(n)
    x = (sc.vertices + rng.normal(scale=0.05, size=sc.vertices.shape)).astype(np.float32).astype(np.float64)
    vo, eo = oracle_pairs(oracle, sc, x, pad)
    vg, eg = gpu_pairs(abi, sc, x, pad)
    if pad == 1.0:          # every vertex meets every triangle that does not hold it
        assert len(vo) == len(x) * sc.num_triangles - 3 * sc.num_triangles
    np.testing.assert_array_equal(vg, vo)
    np.testing.assert_array_equal(eg, eo)


@pytest.mark.parametrize("k", [1, 2, 3, 4, 5, 8, 9, 64, 65])
def test_index_ranges(oracle, abi, k):
    """Strips of k triangles: the sorted keys hold just the bits that the two index ranges need."""
    v = np.array([[0.02 * i, 0.01 * (i % 2), 0.0] for i in range(k + 2)] + [[0.013, 0.004, 5e-5]])
    t = np.array([[i, i + 1, i + 2] for i in range(k)], dtype=np.int32)
    mat = dict(youngs_modulus=1e5, poisson_ratio=0.3, density=200.0, thickness=1e-3)
    sc = scenes.Scene("strip", v, t, mat, scenes.cloth_params(), [], [])
    x = v.astype(np.float32).astype(np.float64)
    for pad in (0.0, 0.5):
        vo, eo = oracle_pairs(oracle, sc, x, pad)
        vg, eg = gpu_pairs(abi, sc, x, pad)
        np.testing.assert_array_equal(vg, vo)
        np.testing.assert_array_equal(eg, eo)
