"""Refit of subtrees by runs of leaves: sizes around a subtree's 1,024 leaves, one CTA's top and the global climb."""
from __future__ import annotations

import numpy as np
import pytest

from andosim_b200 import scenes
from test_gpu_broad_phase import oracle_pairs

pytestmark = pytest.mark.gpu


# a strip of k triangles has 2 k + 1 edges
@pytest.mark.parametrize("k", [1, 2, 15, 16, 511, 512, 1023, 1024, 1025, 2049, 3100])
@pytest.mark.parametrize("shape", ["strip", "folded", "equal"])
def test_sizes(oracle, abi, k, shape):
    i = np.arange(k + 2)
    v = np.stack([0.02 * i, 0.01 * (i % 2), np.zeros(k + 2)], axis=1)
    t = (np.arange(k)[:, None] + np.arange(3)).astype(np.int32)
    mat = dict(youngs_modulus=1e5, poisson_ratio=0.3, density=200.0, thickness=1e-3)
    sc = scenes.Scene("strip", v, t, mat, scenes.cloth_params(), [], [])
    rng = np.random.default_rng(k)
    if shape == "strip":
        x = v + rng.normal(scale=0.002, size=v.shape)
    elif shape == "folded":      # layers over one another: leaves of one place from far apart on the strip
        x = v.copy()
        x[:, 0] = np.abs((x[:, 0] + 1.0) % 2.0 - 1.0)
        x[:, 2] = rng.normal(scale=0.01, size=k + 2)
    else:                        # all codes equal up to 60 places: deep chains of equal keys
        x = v[i % 60]
    x = x.astype(np.float32).astype(np.float64)
    pad = 0.001 if shape == "equal" else 0.004
    vo, eo = oracle_pairs(oracle, sc, x, pad)
    for top in (None, 0):
        S = abi.Scene(sc.vertices, sc.triangles, sc.material)
        if top is not None:
            S.set_refit_top_capacity(top)
        S.upload(x, np.zeros_like(x), sc.vertices, None)
        np.testing.assert_array_equal(S.broad_phase(0, pad).astype(np.int64), vo)
        np.testing.assert_array_equal(S.broad_phase(1, pad).astype(np.int64), eo)
        S.close()
