"""Tile pairs of sparse rows that their bound leaves out: graphs equal the one-sided tiles', which compute every key, at
supports that overlap in part, ragged tiles, sums that over- and underflow, mixed signs and non-finite values."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import load_package

pytestmark = pytest.mark.gpu


def _rows(n, d, protos, seed, shared=0.0, scale=1.0, signed=False):
    rng = np.random.Generator(np.random.PCG64(seed))
    sup = rng.random((protos, d)) < 0.2
    sup[:, : int(shared * d)] = True
    x = np.where(sup[rng.integers(0, protos, size=n)], 1.0 - rng.random((n, d)), 0.0)
    if signed:
        x *= rng.choice([-1.0, 1.0], size=(n, d))
    return (x * scale).astype(np.float32)


def _check(x, k, trees, leaf, metric):
    acknn = load_package()
    a = acknn.knn_build(x, k, trees, leaf, 0, metric, seed=3, sparse_dims=1)
    b = acknn.knn_build(x, k, trees, leaf, 0, metric, seed=3, sparse_dims=1, tile_pairs=-1)
    np.testing.assert_array_equal(a[0], b[0])
    np.testing.assert_array_equal(a[1].view(np.uint32), b[1].view(np.uint32))


@pytest.mark.parametrize("metric", [0, 1])
@pytest.mark.parametrize("n,d,k,leaf", [(2000, 31, 5, 1100), (2101, 256, 10, 2101), (3333, 257, 33, 3333),
                                        (2500, 784, 30, 1300), (1500, 1025, 70, 1500)])
@pytest.mark.parametrize("shared", [0.0, 0.15, 0.5])
def test_shapes(metric, n, d, k, leaf, shared):
    _check(_rows(n, d, 5, n, shared), k, 2, leaf, metric)


@pytest.mark.parametrize("metric", [0, 1])
@pytest.mark.parametrize("scale", [1e-42, 1e-23, 1e-19, 1e18, 1e37])
def test_range(metric, scale):
    _check(_rows(2500, 200, 5, 1, 0.1, scale, signed=True), 10, 2, 2500, metric)


@pytest.mark.parametrize("metric", [0, 1])
def test_infinite_values(metric):
    x = _rows(2200, 200, 5, 2)
    x[100, 3] = np.inf  # keys of one row become infinite; no key is NaN
    _check(x, 10, 1, 2200, metric)
