"""A batch repeated with another launch option does not replay the graph that was captured without it: the call runs the
other kernels, which shows in the scratch that only they need."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import load_package

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("metric,before,after", [
    (0, dict(tile_pairs=-1), dict()),              # dense tiles, then the tensor-core filter
    (0, dict(leaf_tile=64), dict()),
    (1, dict(sparse_dims=-1), dict(sparse_dims=1)),  # all dims, then each tile's non-zero dims
], ids=["tile_pairs", "leaf_tile", "sparse_dims"])
def test_option_changed_after_capture(metric, before, after):
    acknn = load_package()
    sets = [acknn.workloads.gaussian_mixture(n, 64, 8, seed=n) for n in (4000, 3000)]
    ctx = acknn.Context(0)
    try:
        for _ in range(3):  # eager, captured, replayed
            want = acknn.knn_build_batch(sets, 10, 3, 300, 1, metric, context=ctx.handle, **before)
        held = ctx.scratch_bytes
        for _ in range(3):
            got = acknn.knn_build_batch(sets, 10, 3, 300, 1, metric, context=ctx.handle, **after)
            assert ctx.scratch_bytes > held
            for (gi, gd), (wi, wd) in zip(got, want):
                np.testing.assert_array_equal(gi, wi)
                np.testing.assert_array_equal(gd.view(np.uint32), wd.view(np.uint32))
    finally:
        ctx.close()
