"""Column groups of the tensor-core leaf stage's bounding pass (k_leaf_tc, approximate-cuda-knn_b200/csrc/leaf_umma.cu),
restated: 64 groups of 8, 16 or 32 columns by the block's size, wrapping past the 64th.  Where the pass runs, kq groups hold
a column, and the kq-th smallest group minimum is no smaller than the kq-th smallest key; and a list length that the
pass covers at its smallest block is covered at every larger one, which lets the FP32 filter take a first tree."""
from __future__ import annotations

import numpy as np
import pytest

GROUPS, SMALLEST = 64, 256


def width(nb):
    return 8 if nb <= 8 * GROUPS else 16 if nb <= 16 * GROUPS else 32


def applies(nb, kq):
    return nb >= SMALLEST and nb >= width(nb) * (kq + kq // 4)


def covers_first_tree(minleaf, k):
    return minleaf >= SMALLEST and 8 * (k + k // 4) <= SMALLEST


@pytest.mark.parametrize("nb", [256, 257, 511, 512, 513, 520, 1023, 1024, 1025, 1040, 2048, 2049, 5000])
def test_kth_group_minimum_bounds_the_kth_key(nb):
    rng = np.random.Generator(np.random.PCG64(nb))
    group = (np.arange(nb) // width(nb)) % GROUPS
    for kq in (1, 2, 10, 20, 25, 26, 32):
        if not applies(nb, kq):
            continue
        assert len(np.unique(group)) >= kq
        for own in (0, nb // 2, nb - 1):  # the row's own column takes no part
            key = rng.standard_normal(nb).astype(np.float32)
            key[own] = np.inf
            mins = np.full(GROUPS, np.inf, dtype=np.float32)
            np.minimum.at(mins, group, key)
            kth = np.sort(mins)[kq - 1]
            assert np.isfinite(kth) and kth >= np.sort(key)[kq - 1]


def test_first_tree_rule_covers_every_block():
    for k in range(1, 33):
        assert covers_first_tree(SMALLEST, k) == applies(SMALLEST, k)
        if covers_first_tree(SMALLEST, k):
            assert all(applies(nb, k) for nb in range(SMALLEST, 3000))
