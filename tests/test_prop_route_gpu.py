"""Propagation with and without the candidate filter: shapes on either side of the rule that chooses between them give the
CPU restatement's lists, in FP32 and from FP16 rows."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import load_package

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("metric", [0, 1, 2])
@pytest.mark.parametrize("d,k", [(8, 5), (9, 5), (8, 6), (40, 3), (41, 3), (128, 8), (129, 8), (190, 6), (190, 5), (200, 8),
                                 (300, 4), (300, 8), (353, 8), (380, 8), (520, 14), (580, 14), (900, 8), (1000, 5), (1000, 9)])
def test_either_side(oracle, metric, d, k):
    acknn = load_package()
    x = acknn.workloads.gaussian_mixture(700, d, 4, seed=d + k)
    for y in (x, x.astype(np.float16)):
        gi, gd = acknn.knn_build(y, k, 2, max(24, 2 * k), 2, metric, seed=1)
        oi, od = oracle.knn_build(y.astype(np.float32), k, 2, max(24, 2 * k), 2, metric, seed=1)
        np.testing.assert_array_equal(gi, oi)
        np.testing.assert_array_equal(gd.view(np.uint32), od.view(np.uint32))
