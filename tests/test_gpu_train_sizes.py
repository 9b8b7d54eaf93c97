"""The training backward's kernels at sizes around their tiles (32 and 64 rows, 148 row ranges), against the FP64 oracle."""
from __future__ import annotations

import numpy as np
import pytest

from andosim_b200 import learned, scenes
from oracle import learned_oracle as lo
from test_gpu_learned import evaluated

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [3, 4, 6, 13, 30])
def test_training_gradient(abi, n):
    """Same tolerance as the gradient's other oracle test: FP32 sums against FP64."""
    S, s = evaluated(abi, scenes.c4(n=n, size=2.0 * (n - 1) / 255.0))
    w = learned.load_weights()
    T = abi.Trainer(w)
    T.add_system(S, max_probes=5, tol=1e-6)
    probes, norms = T.probes(0, S.V)
    loss, grad = T.loss(0, grad=True)
    net = lo.Net(lo.bf16_round(w), s)
    net.forward()
    want = net.loss(probes.astype(np.float64), norms)
    g = net.backward()
    assert abs(loss - want) <= 1e-5 * abs(want)
    parts = [(lo.W_IN, lo.LAYER0), (lo.DV, lo.NPARAM)] + [(lo.LAYER0 + k * lo.L_SIZE, lo.LAYER0 + (k + 1) * lo.L_SIZE) for k in range(3)]
    for a, b in parts:
        assert np.linalg.norm(grad[a:b] - g[a:b]) <= 1e-4 * np.linalg.norm(g[a:b]), (a, b)
    T.close()
    S.close()
