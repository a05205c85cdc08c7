"""The FP32 leaf stage behind the tensor-core filter against dense FP32 tiles: the same graph bit for bit at the edges
of its shapes (leaf sizes around tiles, groups of leaves and the bounding pass, dims around product steps and slices, list
lengths) and of the data's range, in batches, and where the filter hands over to dense tiles."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import load_package

pytestmark = pytest.mark.gpu


def _same(x, k, trees, leaf, metric, seed=3):
    acknn = load_package()
    fi, fd, fs = acknn.knn_build(x, k, trees, leaf, 0, metric, seed=seed, stats=True)
    di, dd, ds = acknn.knn_build(x, k, trees, leaf, 0, metric, seed=seed, tile_pairs=-1, stats=True)
    np.testing.assert_array_equal(fi, di)
    np.testing.assert_array_equal(fd.view(np.uint32), dd.view(np.uint32))
    assert fs["leaf_pairs"] == ds["leaf_pairs"]


@pytest.mark.parametrize("metric", [0, 2])
@pytest.mark.parametrize("leaf", [20, 31, 32, 33, 63, 64, 65, 127, 128, 129, 255, 256, 257, 320, 511, 512, 513, 1024, 1025,
                                  2049])
def test_leaf_sizes(metric, leaf):
    acknn = load_package()
    depth = max(1, int(np.ceil(np.log2(1_600_000 / leaf / leaf))))
    x = acknn.workloads.gaussian_mixture((leaf << depth) - 3, 24, 20, seed=leaf)
    _same(x, 4, 3, leaf, metric)


@pytest.mark.parametrize("metric", [0, 2])
@pytest.mark.parametrize("d", [1, 3, 16, 17, 32, 33, 63, 64, 65, 127, 128, 129, 200, 255, 256])
def test_dims(metric, d):
    acknn = load_package()
    _same(acknn.workloads.gaussian_mixture(8000, d, 10, seed=d), 10, 4, 300, metric)
    _same(acknn.workloads.gaussian_mixture(24000, d, 10, seed=d), 10, 3, 100, metric)


@pytest.mark.parametrize("k", [1, 2, 16, 17, 25, 26, 32])
def test_list_lengths(k):
    acknn = load_package()
    _same(acknn.workloads.gaussian_mixture(20000, 40, 10, seed=k), k, 4, 260, 0)
    _same(acknn.workloads.gaussian_mixture(60000, 20, 10, seed=k), k, 3, 80, 2)


@pytest.mark.parametrize("metric", [0, 2])
@pytest.mark.parametrize("leaf", [120, 600])
@pytest.mark.parametrize("kind", ["tiny", "huge", "mixed", "duplicates", "zero_rows", "far_offset", "infinite", "tight"])
def test_values(metric, leaf, kind):
    acknn = load_package()
    n = 20000
    rng = np.random.Generator(np.random.PCG64(1))
    x = acknn.workloads.gaussian_mixture(n, 48, 4, seed=11)
    if kind == "tiny":
        x *= np.float32(1e-12 if metric == 2 else 1e-22)  # squares underflow (EUCLIDEAN)
    elif kind == "huge":
        x *= np.float32(1e12 if metric == 2 else 1e19)    # squares overflow (EUCLIDEAN)
    elif kind == "mixed":
        x *= (10.0 ** rng.uniform(-6, 6, (n, 1))).astype(np.float32)
    elif kind == "duplicates":
        x = np.repeat(x[:n // 20], 20, axis=0)
    elif kind == "zero_rows":
        x[::7] = 0
    elif kind == "far_offset":
        x = (x * np.float32(1e-3) + np.float32(1000.0)).astype(np.float32)
    elif kind == "infinite":
        x[5, 3] = np.inf
    elif kind == "tight":  # clusters far apart, far tighter than the 16-bit rows of a leaf that spans two of them
        x = (rng.integers(0, 50, (n, 1)) * np.float32(1000) + x * np.float32(1e-5)).astype(np.float32)
    _same(np.ascontiguousarray(x), 10, 4, leaf, metric)


def test_sets_with_and_without_the_bounding_pass():
    """One batch whose leaves lie on both sides of the bounding pass's limit, and one whose leaves all lie above it."""
    acknn = load_package()
    for sizes in ([9000, 5000, 300, 4000], [9000, 5000, 2500, 2048]):
        sets = [acknn.workloads.gaussian_mixture(n, 32, 8, seed=n) for n in sizes]
        got = acknn.knn_build_batch(sets, 10, 3, 700, 0, 0)
        for x, (gi, gd) in zip(sets, got):
            di, dd = acknn.knn_build(x, 10, 3, 700, 0, 0, tile_pairs=-1)
            np.testing.assert_array_equal(gi, di)
            np.testing.assert_array_equal(gd.view(np.uint32), dd.view(np.uint32))


def test_more_rows_than_one_launch_takes():
    acknn = load_package()
    _same(acknn.workloads.gaussian_mixture(1_100_000, 8, 30, seed=2), 4, 3, 40, 0)
