"""Tensor-core leaf tiles at the edges of their shapes: the mixed graph on small integer coordinates (every
product and sum exact) must equal the plain FP32 graph bit for bit, whatever the leaf size (64-column tiles,
128-row query tiles, two of them per block, 1024-column bitmaps, the bounding pass from 1024 columns), the
dims (16-element product steps, 64-element boxes), kq, and the number of rows per launch."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import load_package

pytestmark = pytest.mark.gpu


def _ints(n, d, seed, top=255):
    rng = np.random.Generator(np.random.PCG64(seed))
    centres = rng.uniform(0, top, size=(6, d))
    x = centres[rng.integers(0, 6, n)] + rng.normal(0, top / 12, size=(n, d))
    return np.clip(np.rint(x), 0, top).astype(np.float32)


def _same(x, k, trees, leaf, precision, seed=3):
    acknn = load_package()
    mi, md, st = acknn.knn_build(x, k, trees, leaf, 0, 0, seed=seed, precision=precision, stats=True)
    assert st["leaf_path"] == precision
    pi, pd = acknn.knn_build(x, k, trees, leaf, 0, 0, seed=seed)
    np.testing.assert_array_equal(mi, pi)
    np.testing.assert_array_equal(md.view(np.uint32), pd.view(np.uint32))


# one leaf of exactly `leaf` points and then two trees of two leaves
@pytest.mark.parametrize("leaf", [33, 63, 64, 65, 127, 128, 129, 191, 255, 256, 257, 511, 640, 1023, 1024, 1025,
                                  1100, 2047, 2049, 4097])
def test_leaf_sizes(leaf):
    acknn = load_package()
    _same(_ints(leaf, 32, leaf), 12, 1, leaf, acknn.PREC_BF16_RERANK)
    _same(_ints(2 * leaf - 1, 32, leaf + 1), 16, 3, leaf, acknn.PREC_BF16_RERANK)


@pytest.mark.parametrize("d", [1, 7, 8, 15, 16, 17, 48, 63, 64, 65, 80, 128, 129, 176, 192, 193, 255, 256])
@pytest.mark.parametrize("leaf", [150, 1300])
def test_dims(d, leaf):
    acknn = load_package()
    _same(_ints(3 * leaf + 5, d, d), 10, 3, leaf, acknn.PREC_BF16_RERANK)
    _same(_ints(3 * leaf + 5, d, d + 1), 10, 3, leaf, acknn.PREC_F16_RERANK)


@pytest.mark.parametrize("k", [1, 2, 15, 16, 17, 31, 32])
def test_list_lengths(k):
    acknn = load_package()
    _same(_ints(5000, 24, k), k, 4, 1250, acknn.PREC_BF16_RERANK)
    _same(_ints(3000, 24, k + 50), k, 4, 90, acknn.PREC_BF16_RERANK)


def test_duplicate_points_and_equal_keys():
    """Ties everywhere: every key has many equal ones, ranked by id."""
    acknn = load_package()
    x = _ints(4000, 8, 1, top=3)
    _same(x, 16, 3, 1000, acknn.PREC_BF16_RERANK)
    _same(x, 16, 3, 2000, acknn.PREC_BF16_RERANK)


def test_more_rows_than_one_launch_takes():
    acknn = load_package()
    _same(_ints(1_100_000, 8, 2), 4, 2, 300, acknn.PREC_BF16_RERANK)


def test_block_of_more_than_65536_columns():
    """One leaf of 70,000 points: bitmaps far into the block, every candidate column."""
    acknn = load_package()
    _same(_ints(70_000, 16, 9), 8, 2, 70_000, acknn.PREC_BF16_RERANK)
