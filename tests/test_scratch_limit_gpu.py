"""Builds where device memory is short: what a build took before the tensor-core filters and the tile kernel's survivor
scratch existed has to be enough.  The limit is the context's own (knn_test_limit_scratch); nothing here fills the device."""
from __future__ import annotations

import ctypes

import numpy as np
import pytest

from conftest import load_package

pytestmark = pytest.mark.gpu


def _same(got, want):
    for g, w in zip(got, want):
        np.testing.assert_array_equal(g.view(np.uint32), w.view(np.uint32))


def _held(acknn, build):
    """Scratch of a build in a context of its own."""
    ctx = acknn.Context(0)
    try:
        build(ctx.handle)
        return ctx.scratch_bytes
    finally:
        ctx.close()


def _limited(acknn, limit, *builds):
    lib = acknn.load_library()
    ctx = acknn.Context(0)
    try:
        assert lib.knn_test_limit_scratch(ctx.handle, limit) == 0
        out = [b(ctx.handle) for b in builds]
        assert ctx.scratch_bytes <= limit
        return out
    finally:
        ctx.close()


@pytest.mark.parametrize("metric", [0, 2])
@pytest.mark.parametrize("leaf", [100, 700])
def test_plain_build_needs_no_more_than_dense_tiles(metric, leaf):
    """The filters' scratch is spare: without it every tree takes dense tiles and every propagation key is exact."""
    acknn = load_package()
    x = acknn.workloads.gaussian_mixture(60_000, 40, 10, seed=leaf)
    build = lambda ctx, **kw: acknn.knn_build(x, 10, 3, leaf, 2, metric, seed=2, context=ctx, **kw)  # noqa: E731
    need = _held(acknn, lambda ctx: acknn.knn_build(x, 10, 3, leaf, 0, metric, context=ctx, tile_pairs=-1))
    full = _held(acknn, build)
    assert full > need
    want = build(None, tile_pairs=-1)
    for limit in (need, (need + full) // 2, full):
        for got in _limited(acknn, limit, build, build):
            _same(got, want)


@pytest.mark.parametrize("precision", [1, 2])
@pytest.mark.parametrize("leaf,d", [(60, 48), (700, 48), (700, 200)])
def test_mixed_build_needs_no_more_than_one_operand_copy(precision, leaf, d):
    """Rows padded to 64 dims, norms, an inverse order and the candidate lists: what the tiles once took."""
    acknn = load_package()
    n, k = 60_000, 10
    x = acknn.workloads.gaussian_mixture(n, d, 10, seed=leaf)
    build = lambda ctx: acknn.knn_build(x, k, 3, leaf, 1, 0, seed=2, precision=precision, context=ctx)  # noqa: E731
    plain = _held(acknn, lambda ctx: acknn.knn_build(x, k, 3, leaf, 0, 0, context=ctx, tile_pairs=-1))
    need = plain + n * (2 * ((d + 63) // 64 * 64) + 4 + 4 + 8 * 2 * k)
    full = _held(acknn, build)
    assert full > need
    want = build(None)
    for limit in (need, (need + full) // 2, full):
        for got in _limited(acknn, limit, build, build):
            _same(got, want)


def test_scratch_of_earlier_calls_is_given_back():
    acknn = load_package()
    x = acknn.workloads.gaussian_mixture(40_000, 64, 10, seed=1)
    y = acknn.workloads.gaussian_mixture(90_000, 24, 10, seed=2)
    a = lambda ctx: acknn.knn_build(x, 10, 3, 300, 1, 0, context=ctx)  # noqa: E731
    b = lambda ctx: acknn.knn_build(y, 12, 2, 60, 1, 2, learned=True, mlp_steps=5, context=ctx)  # noqa: E731
    limit = max(_held(acknn, a), _held(acknn, b))
    for got, f in zip(_limited(acknn, limit, a, b, a, b), (a, b, a, b)):
        _same(got, f(None))


def test_batches_and_their_graphs():
    acknn = load_package()
    sets = [acknn.workloads.gaussian_mixture(n, d, 8, seed=n) for n, d in ((9000, 32), (5000, 64), (30000, 32), (2500, 64))]
    for kw in (dict(), dict(precision=1)):
        build = lambda ctx: acknn.knn_build_batch(sets, 10, 3, 300, 1, 0, context=ctx, **kw)  # noqa: E731
        want = build(None)
        full = _held(acknn, build)
        for limit in (full * 2 // 5, full):
            for got in _limited(acknn, limit, build, build, build, build):
                for g, w in zip(got, want):
                    _same(g, w)


def test_too_little_is_still_an_error():
    acknn = load_package()
    x = acknn.workloads.gaussian_mixture(20_000, 32, 8, seed=1)
    for kw in (dict(), dict(precision=1)):
        with pytest.raises(acknn.KnnError) as e:
            _limited(acknn, 1_000_000, lambda ctx: acknn.knn_build(x, 10, 3, 300, 1, 0, context=ctx, **kw))
        assert e.value.status == -3
