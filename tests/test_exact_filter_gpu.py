"""The exact search behind its FP32 filter: bit for bit the sequential FP64 brute force, whichever pairs the filter
rejects, at ragged tiles and stages, unaligned rows, every list width, and where FP32 over- or underflows."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import load_package

pytestmark = pytest.mark.gpu


def _check(oracle, x, k, metric, nq, seed=0):
    acknn = load_package()
    rng = np.random.Generator(np.random.PCG64(seed))
    q = np.sort(rng.choice(x.shape[0], size=nq, replace=False)).astype(np.int64)
    gi, gd = acknn.exact_fp64(x, k, q, metric)
    oi, od = oracle.exact(x, k, q, metric)
    np.testing.assert_array_equal(gi, oi)
    np.testing.assert_array_equal(gd.view(np.uint64), od.view(np.uint64))


# 1700 queries: 27 query tiles, 21 slices, so these n give slices past the filter's shortest
@pytest.mark.parametrize("metric", [0, 1, 2])
@pytest.mark.parametrize("d,k,n", [(1, 5, 13001), (4, 8, 14000), (15, 16, 15013), (16, 10, 15013), (17, 30, 17000),
                                   (37, 33, 34000), (64, 64, 55001), (130, 100, 79007)])
def test_shapes(oracle, metric, d, k, n):
    acknn = load_package()
    _check(oracle, acknn.workloads.gaussian_mixture(n, d, 8, seed=d), k, metric, 1700, d)


@pytest.mark.parametrize("metric", [0, 1, 2])
def test_ties_and_copies(oracle, metric):
    """Few distinct rows: most pairs tie with the k-th key, and blocks are left to the dense kernel."""
    rng = np.random.Generator(np.random.PCG64(7))
    x = rng.integers(0, 2, size=(15000, 3)).astype(np.float32)
    _check(oracle, x, 10, metric, 1700)
    y = rng.integers(0, 6, size=(15000, 9)).astype(np.float32)
    y[::7] = 0.0
    _check(oracle, y, 16, metric, 1700)


@pytest.mark.parametrize("metric", [0, 1, 2])
@pytest.mark.parametrize("scale", [1e-42, 1e-23, 1e-15, 1e17, 2e19, 1e38])
def test_range(oracle, metric, scale):
    """Squares and differences past FP32's range on either side."""
    acknn = load_package()
    x = acknn.workloads.gaussian_mixture(14000, 12, 8, seed=3)
    x = (x / np.abs(x).max() * 3.0 * scale).astype(np.float32)
    x[::3] *= np.float32(1e-3)
    _check(oracle, x, 12, metric, 1700)


@pytest.mark.parametrize("metric", [0, 1, 2])
@pytest.mark.parametrize("d", [7, 18])
def test_rows_in_place(oracle, metric, d):
    """The entry point without allocation reads the caller's rows, here off 16-byte boundaries."""
    torch = pytest.importorskip("torch")
    acknn = load_package()
    lib = acknn.load_library()
    n, k, nq = 15000, 10, 1700
    x = acknn.workloads.gaussian_mixture(n, d, 8, seed=d)
    q = np.arange(3, 3 + nq, dtype=np.int64)
    xd, qd = torch.from_numpy(x).cuda(), torch.from_numpy(q).cuda()
    idx = torch.empty((nq, k), dtype=torch.int32, device="cuda")
    dist = torch.empty((nq, k), dtype=torch.float64, device="cuda")
    assert lib.knn_exact_fp64_noalloc(xd.data_ptr(), n, d, k, metric, qd.data_ptr(), nq, idx.data_ptr(),
                                      dist.data_ptr(), None) == 0
    oi, od = oracle.exact(x, k, q, metric)
    np.testing.assert_array_equal(idx.cpu().numpy(), oi)
    np.testing.assert_array_equal(dist.cpu().numpy().view(np.uint64), od.view(np.uint64))
