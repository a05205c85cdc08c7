"""The training step's kernels at the edges of their tiles: batches that leave a block of triplets or a row split short
or empty, and dims around the staged chunk, the output tile and the 16-byte rows.  Tolerances as in test_mlp_gpu.py."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import load_package
from test_mlp_gpu import _kink_free_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d", [1, 31, 32, 33, 63, 64, 65, 68, 132])
@pytest.mark.parametrize("B", [2, 8, 9, 43, 130])
def test_gradient(oracle, d, B):
    acknn = load_package()
    rng = np.random.Generator(np.random.PCG64(1000 * d + B))
    p, rows, loss_o, grad_o = _kink_free_case(acknn, oracle, rng, d, B, 4.0)
    loss_g, grad_g = acknn.mlp_loss_grad(p, rows, 4.0)
    assert loss_g == pytest.approx(loss_o, rel=1e-5)
    assert np.linalg.norm(grad_g - grad_o) / np.linalg.norm(grad_o) < 1e-4
    assert np.max(np.abs(grad_g - grad_o)) <= 1e-3 * np.max(np.abs(grad_o))
