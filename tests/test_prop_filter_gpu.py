"""Filtered propagation at the edges of its shapes (lanes per candidate row, steps per row, candidates per batch, list
registers, width of the exact slices) and of its value range, against the CPU restatement, which evaluates every key."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import load_package

pytestmark = pytest.mark.gpu


def _check(oracle, x, k, metric, seed):
    acknn = load_package()
    n = x.shape[0]
    rng = np.random.Generator(np.random.PCG64(seed))
    # random distinct neighbours, sorted by (key, id)
    perm = acknn.build_trees(x, 1, max(k + 1, 40), seed)
    idx, key = oracle.leaf_stage(x, k, perm, max(k + 1, 40), metric)
    # a third of the rows start from random neighbours instead: poor lists, many entrants
    for i in range(0, n, 3):
        c = rng.choice(n - 1, size=k, replace=False)
        c = np.where(c >= i, c + 1, c).astype(np.int32)
        kk = np.array([oracle.pair_key(x[i], x[j], metric) for j in c], dtype=np.float32)
        o = np.lexsort((c, kk))
        idx[i], key[i] = c[o], kk[o]
    for _ in range(2):
        gi, gk = acknn.propagate_step(x, idx, key, metric)
        oi, ok = oracle.propagate(x, idx, key, metric)
        np.testing.assert_array_equal(gi, oi)
        np.testing.assert_array_equal(gk.view(np.uint32), ok.view(np.uint32))
        idx, key = oi, ok


@pytest.mark.parametrize("metric", [0, 1, 2])
@pytest.mark.parametrize("d", [1, 7, 8, 9, 16, 17, 33, 64, 65, 127, 256, 257, 512, 513, 784, 1023, 1024, 1025])
def test_dims(oracle, metric, d):
    acknn = load_package()
    _check(oracle, acknn.workloads.gaussian_mixture(400, d, 4, seed=d), 10, metric, d)


@pytest.mark.parametrize("k", [1, 2, 3, 15, 16, 17, 31, 32, 33, 64, 65])
def test_list_lengths(oracle, k):
    acknn = load_package()
    _check(oracle, acknn.workloads.gaussian_mixture(300, 24, 3, seed=k), k, 0, k)
    _check(oracle, acknn.workloads.gaussian_mixture(300, 40, 3, seed=k), k, 1, k)


@pytest.mark.parametrize("metric", [0, 1, 2])
@pytest.mark.parametrize("kind", ["tiny", "huge", "mixed", "sparse", "duplicates", "zero_rows", "far_offset"])
def test_values(oracle, metric, kind):
    acknn = load_package()
    x = acknn.workloads.gaussian_mixture(400, 48, 4, seed=11)
    if kind == "tiny":
        x *= np.float32(1e-12 if metric == 2 else 1e-24)  # squares underflow (EUCLIDEAN)
    elif kind == "huge":
        x *= np.float32(1e12 if metric == 2 else 1e22)    # squares overflow (EUCLIDEAN)
    elif kind == "mixed":
        x *= (10.0 ** np.random.Generator(np.random.PCG64(1)).uniform(-6, 6, (400, 1))).astype(np.float32)
    elif kind == "sparse":
        x[np.random.Generator(np.random.PCG64(2)).random(x.shape) < 0.8] = 0
    elif kind == "duplicates":
        x = np.repeat(x[:100], 4, axis=0)
    elif kind == "zero_rows":
        x[::7] = 0
    elif kind == "far_offset":
        x = (x * np.float32(1e-3) + np.float32(1000.0)).astype(np.float32)  # 16-bit rows nearly all equal
    _check(oracle, np.ascontiguousarray(x), 12, metric, 5)


def test_float16_input_and_steps_of_a_build(oracle):
    acknn = load_package()
    x = acknn.workloads.normalized_mixture(seed=3, n=3000, d=96, clusters=20)
    gi, gd = acknn.knn_build(x, 10, 3, 40, 3, 2, seed=2)
    oi, od = oracle.knn_build(x.astype(np.float32), 10, 3, 40, 3, 2, seed=2)
    np.testing.assert_array_equal(gi, oi)
    np.testing.assert_array_equal(gd.view(np.uint32), od.view(np.uint32))
