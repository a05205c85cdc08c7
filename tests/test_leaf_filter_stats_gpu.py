"""What the statistics say of the FP32 leaf filter: that it ran where the shapes call for it, what ran beside it, that it
handed over where the data defeats it, and, with that seen, that a tree handed over after part of it was merged keeps
the dense tiles' graph."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import load_package

pytestmark = pytest.mark.gpu


def _build(x, k, trees, leaf, metric, **kw):
    acknn = load_package()
    return acknn.knn_build(x, k, trees, leaf, 0, metric, seed=3, stats=True, **kw)


@pytest.mark.parametrize("metric", [0, 2])
@pytest.mark.parametrize("leaf", [20, 31, 32, 33, 63, 64, 65, 127, 128, 129, 255, 256, 257, 320, 511, 512, 513, 1024, 1025,
                                  2049])
def test_leaf_sizes_are_filtered(metric, leaf):
    acknn = load_package()
    depth = max(1, int(np.ceil(np.log2(1_600_000 / leaf / leaf))))
    n = (leaf << depth) - 3
    st = _build(acknn.workloads.gaussian_mixture(n, 24, 20, seed=leaf), 4, 3, leaf, metric)[2]
    whole = (n >> depth) >= 256  # the bounding pass covers the first tree too
    assert (st["leaf_filtered"], st["leaf_handed"]) == (3 if whole else 2, 0)
    assert (st["leaf_tile"], st["tile_pairs"]) == ((128, 0) if whole else (64, 1))
    assert st["leaf_path"] == 0 and st["sparse_dims"] == 0 and st["tc_group"] >= 1


@pytest.mark.parametrize("d", [1, 3, 16, 17, 33, 64, 65, 128, 129, 200, 255, 256, 257])
def test_dims_are_filtered(d):
    acknn = load_package()
    st = _build(acknn.workloads.gaussian_mixture(8000, d, 10, seed=d), 10, 4, 300, 0)[2]
    assert st["leaf_filtered"] == (4 if n_whole(8000, 300) else 3) if d <= 256 else st["leaf_filtered"] == 0
    assert st["leaf_handed"] == 0


def n_whole(n, leaf):
    depth = 0
    while -(-n >> depth) > leaf:
        depth += 1
    return (n >> depth) >= 256


def test_options_and_metrics_without_it():
    acknn = load_package()
    x = acknn.workloads.gaussian_mixture(8000, 32, 10, seed=1)
    for kw in (dict(metric=1), dict(metric=0, tile_pairs=-1), dict(metric=0, leaf_tile=64), dict(metric=0, sparse_dims=1),
               dict(metric=0, precision=1)):
        st = _build(x, 10, 3, 300, **kw)[2]
        assert (st["leaf_filtered"], st["leaf_handed"]) == (0, 0)


@pytest.mark.parametrize("metric", [0, 2])
@pytest.mark.parametrize("leaf", [120, 600])
@pytest.mark.parametrize("kind", ["infinite", "tight"])
def test_hand_over(metric, leaf, kind):
    acknn = load_package()
    n = 20000
    rng = np.random.Generator(np.random.PCG64(1))
    x = acknn.workloads.gaussian_mixture(n, 48, 4, seed=11)
    if kind == "infinite":
        x[5, 3] = np.inf
    else:
        x = (rng.integers(0, 50, (n, 1)) * np.float32(1000) + x * np.float32(1e-5)).astype(np.float32)
    fi, fd, st = _build(x, 10, 4, leaf, metric)
    assert st["leaf_handed"] > 0 and st["leaf_handed"] + st["leaf_filtered"] == (4 if leaf == 600 else 3)
    assert st["leaf_tile"] == 64
    di, dd, _ = _build(x, 10, 4, leaf, metric, tile_pairs=-1)
    np.testing.assert_array_equal(fi, di)
    np.testing.assert_array_equal(fd.view(np.uint32), dd.view(np.uint32))


def test_hand_over_by_a_later_launch():
    """600,000 rows take two launches a tree; a quarter of them, copies that overflow their buffers, lies in the second
    launch's leaves of the first tree, whose first launch is merged by then."""
    acknn = load_package()
    n = 600_000
    x = acknn.workloads.gaussian_mixture(n, 8, 40, seed=2).astype(np.float32)
    tight = slice(3 * n // 4, n)
    x[tight] = np.float32(40.0)
    for seed in range(16):
        where = np.argsort(acknn.build_trees(x, 1, 1024, seed)[0])
        if where[tight].min() > 0.72 * n:
            break
    else:
        pytest.fail("no seed puts the copies last")
    kw = dict(seed=seed, stats=True)
    fi, fd, st = acknn.knn_build(x, 4, 2, 1024, 0, 0, **kw)
    assert st["leaf_handed"] == 2
    di, dd, _ = acknn.knn_build(x, 4, 2, 1024, 0, 0, tile_pairs=-1, **kw)
    np.testing.assert_array_equal(fi, di)
    np.testing.assert_array_equal(fd.view(np.uint32), dd.view(np.uint32))


def test_autotune_leaves_tiles_alone_that_do_not_run():
    acknn = load_package()
    x = acknn.workloads.gaussian_mixture(20000, 32, 10, seed=4)
    ctx = acknn.Context(0)
    try:
        for _ in range(2):
            i, d, st = acknn.knn_build(x, 10, 3, 600, 1, 0, seed=1, autotune=True, stats=True, context=ctx.handle)
            assert (st["leaf_tile"], st["leaf_filtered"]) == (128, 3) and st["prop_warps"] in (2, 4, 8)
    finally:
        ctx.close()
    wi, wd = acknn.knn_build(x, 10, 3, 600, 1, 0, seed=1, tile_pairs=-1)
    np.testing.assert_array_equal(i, wi)
    np.testing.assert_array_equal(d.view(np.uint32), wd.view(np.uint32))
