"""Rows with infinite values in a tensor-core build: their approximate keys have no order and must not displace the
neighbours of the other rows.  On integer rows every product and sum of the tiles is exact, so wherever a plain FP32
build (the same trees) lists finite distances only, the mixed build lists the same."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import load_package

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [1, 2])
@pytest.mark.parametrize("leaf", [100, 600, 3000])
def test_finite_rows_keep_their_neighbours(leaf, precision):
    acknn = load_package()
    x = acknn.workloads.integer_mixture(seed=5, n=6000, d=48)
    x[::97, 1] = np.inf  # products of one sign: inf - inf in the tiles' key form
    x[1::89, 2] = np.inf
    fi, fd = acknn.knn_build(x, 5, 3, leaf, 0, 0, seed=2)
    mi, md = acknn.knn_build(x, 5, 3, leaf, 0, 0, seed=2, precision=precision)
    rows = np.isfinite(x).all(axis=1) & np.isfinite(fd).all(axis=1)
    assert rows.sum() > 3000
    np.testing.assert_array_equal(mi[rows], fi[rows])
    np.testing.assert_array_equal(md[rows].view(np.uint32), fd[rows].view(np.uint32))
