"""Builds of different shapes in several host threads at once, a context each: every one gives its own graph, whichever
shapes the other threads launch the same kernels with in between."""
from __future__ import annotations

import threading

import numpy as np
import pytest

from conftest import load_package

pytestmark = pytest.mark.gpu

# (n, d, k, trees, leaf, props, metric, precision, hand the filter's trees over)
SHAPES = [
    (45_000, 20, 10, 2, 120, 0, 0, 0, True),   # whole leaves of 88 rows
    (60_000, 20, 16, 2, 130, 0, 0, 0, True),   # whole leaves of 118 rows, longer lists
    (9_000, 24, 10, 2, 700, 0, 0, 0, True),    # query tiles
    (9_000, 20, 10, 2, 300, 1, 0, 1, False),   # re-rank of 20 dims
    (9_000, 250, 10, 2, 300, 1, 0, 1, False),  # and of 250
]


def test_shapes_side_by_side():
    acknn = load_package()
    lib = acknn.load_library()
    xs = [acknn.workloads.gaussian_mixture(s[0], s[1], 8, seed=i) for i, s in enumerate(SHAPES)]

    def build(x, s, ctx, hand):
        if hand:
            assert lib.knn_test_fail_next_tile_wait(ctx) == 0
        return acknn.knn_build(x, s[2], s[3], s[4], s[5], s[6], seed=1, precision=s[7], context=ctx)

    want = []
    for x, s in zip(xs, SHAPES):
        ctx = acknn.Context(0)
        want.append(build(x, s, ctx.handle, False))
        ctx.close()
    failures = []

    def work(i):
        ctx = acknn.Context(0)
        try:
            for _ in range(12):
                gi, gd = build(xs[i], SHAPES[i], ctx.handle, SHAPES[i][8])
                np.testing.assert_array_equal(gi, want[i][0])
                np.testing.assert_array_equal(gd.view(np.uint32), want[i][1].view(np.uint32))
        except BaseException as e:  # noqa: BLE001 (reported below)
            failures.append((i, e))
        finally:
            ctx.close()

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(SHAPES))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failures, failures
