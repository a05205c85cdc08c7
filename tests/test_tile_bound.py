"""The tensor-core leaf stage's bounding pass (k_leaf_tc, approximate-cuda-knn_b200/csrc/leaf_umma.cu), restated.

Pass 0 takes, per row, the smallest key' = fma(-2, dot, |y|^2) (EUCLIDEAN) or -dot (COSINE) of each column
group; the kq-th smallest group minimum T, in key units and widened by 2^-21 (|T| + 2 |x|^2 + max|y|^2) (or
2^-21 (|T| + 2)), must not lie below the row's kq-th smallest exact key, whatever the rounding of either.
The float32 operations are in the kernel's order."""
from __future__ import annotations

import numpy as np
import pytest

F = np.float32
SLACK = F(2.0 ** -21)


def fma32(a, b, c):
    return (np.float64(a) * b.astype(np.float64) + c.astype(np.float64)).astype(F)


def bound(keyp, groups, kq):
    """kq-th smallest of the group minima (slice s of 32 columns in group s mod groups)."""
    n = keyp.shape[0]
    slices = [keyp[s:s + 32].min() for s in range(0, n, 32)]
    mins = np.full(groups, np.inf, dtype=F)
    for s, m in enumerate(slices):
        mins[s % groups] = min(mins[s % groups], m)
    return np.sort(mins)[kq - 1]


@pytest.mark.parametrize("scale", [1e-3, 1.0, 1e4])
@pytest.mark.parametrize("near", [False, True])
@pytest.mark.parametrize("columns,kq", [(1024, 32), (1056, 20), (2000, 32), (5000, 12)])
def test_widened_bound_covers_the_kqth_exact_key(scale, near, columns, kq):
    rng = np.random.Generator(np.random.PCG64(columns + kq))
    for _ in range(40):
        xn = F(scale * rng.uniform(0.5, 2.0))
        yn = (scale * rng.uniform(0.5, 2.0, columns)).astype(F)
        if near:  # products that cancel the norms to a few ulps
            dot = (0.5 * (xn.astype(np.float64) + yn) * (1 - rng.uniform(0, 1e-6, columns))).astype(F)
        else:
            dot = (np.sqrt(np.float64(xn) * yn) * rng.uniform(-1, 1, columns)).astype(F)
        keyp = fma32(F(-2.0), dot, yn)
        t = bound(keyp, 64, kq)
        cap = F(t + xn) + F(SLACK * (F(np.abs(t)) + F(2.0) * xn + yn.max()))
        exact = fma32(F(-2.0), dot, (xn + yn).astype(F))
        assert cap >= np.sort(exact)[kq - 1]
        cosd = (dot / np.abs(dot).max()).astype(F)
        t = bound((-cosd).astype(F), 64, kq)
        cap = F(t + F(1.0)) + F(SLACK * (F(np.abs(t)) + F(2.0)))
        assert cap >= np.sort((F(1.0) - cosd).astype(F))[kq - 1]
