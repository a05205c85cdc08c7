"""Trees that the FP32 leaf filter hands over to dense tiles (forced from the host): the same graph as one-sided dense
tiles, where a block takes a whole leaf (leaves of one to five tiles, lists up to its shared memory), a query tile, or several
of them in turn, with either tile size, and in a batch of sets of different depths."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import load_package

pytestmark = pytest.mark.gpu


def _same(got, want):
    for g, w in zip(got, want):
        np.testing.assert_array_equal(g.view(np.uint32), w.view(np.uint32))


@pytest.mark.parametrize("metric", [0, 2])
@pytest.mark.parametrize("n,leaf,k", [
    (26_000, 60, 8),     # 512 leaves of one tile
    (45_001, 120, 10),   # 512 leaves of two tiles
    (80_003, 300, 32),   # 512 leaves of 157: lists of 39.2 KB, over the limit of COSINE
    (149_999, 300, 16),  # 512 leaves of 293, five tiles
    (90_001, 310, 32),   # 512 leaves of 176, 44 KB
    (9_000, 700, 10),    # 16 leaves: query tiles
    (90_001, 800, 10),   # 128 leaves of 11 tiles: more query tiles than blocks
])
def test_handed_over(n, leaf, k, metric):
    acknn = load_package()
    lib = acknn.load_library()
    x = acknn.workloads.gaussian_mixture(n, 20, 12, seed=n)
    want = acknn.knn_build(x, k, 2, leaf, 0, metric, seed=2, tile_pairs=-1)
    ctx = acknn.Context(0)
    try:
        for autotune in (False, True):  # the tuned tile may be 32
            assert lib.knn_test_fail_next_tile_wait(ctx.handle) == 0
            _same(acknn.knn_build(x, k, 2, leaf, 0, metric, seed=2, autotune=autotune, context=ctx.handle), want)
    finally:
        ctx.close()


def test_batch_handed_over():
    acknn = load_package()
    lib = acknn.load_library()
    sets = [acknn.workloads.gaussian_mixture(n, 20, 8, seed=n) for n in (30_000, 17_001, 4_000)]
    ctx = acknn.Context(0)
    try:
        assert lib.knn_test_fail_next_tile_wait(ctx.handle) == 0
        for x, got in zip(sets, acknn.knn_build_batch(sets, 10, 3, 120, 0, 0, context=ctx.handle)):
            _same(got, acknn.knn_build(x, 10, 3, 120, 0, 0, tile_pairs=-1))
    finally:
        ctx.close()
