"""The propagation's candidate filter (k_propagate_filtered, approximate-cuda-knn_b200/csrc/propagate.cu), restated.

Rows are rounded to FP16 of s * x (EUCLIDEAN, TAXICAB) or of the unit row (COSINE), delta bounds the row's
rounding error, and g = (2 d + 64) 2^-24 covers FP32 rounding.  For any two candidates c and e of a query, if
c's lower bound exceeds e's upper bound (widened as the kernel does), c's exact FP32 key must exceed e's: that is what
lets the filter drop c without changing the step's result.  The same holds against a list's exact key."""
from __future__ import annotations

import numpy as np
import pytest

F = np.float32


def exact_key(q, c, metric, nq, nc):
    """Sequential 256-dim partial sums, as the kernels form every key."""
    total = F(0)
    for s in range(0, q.size, 256):
        part = F(0)
        for a, b in zip(q[s:s + 256], c[s:s + 256]):
            if metric == 0:
                t = F(a - b)
                part = F(np.float64(t) * np.float64(t) + np.float64(part))
            elif metric == 1:
                part = F(part + F(abs(F(a - b))))
            else:
                part = F(np.float64(a) * np.float64(b) + np.float64(part))
        total = F(total + part)
    if metric != 2:
        return total
    return F(1) if nq == 0 or nc == 0 else F(F(1) - F(total / F(nq * nc)))


def rows16(x, metric):
    """(h as float32, delta, s)"""
    if metric == 2:
        nr = np.sqrt((x.astype(np.float64) ** 2).sum(1)).astype(F)
        inv = np.where(nr > 0, F(1) / np.where(nr > 0, nr, F(1)), F(0)).astype(F)
        v, s = (x * inv[:, None]).astype(F), F(1)
    else:
        nr = None
        m = np.abs(x).max()
        s = F(2.0 ** (15 - np.frexp(m)[1])) if m > 0 else F(1)
        v = (x * s).astype(F)
    h = v.astype(np.float16).astype(F)
    e = (v - h).astype(np.float64)
    d = np.abs(e).sum(1) if metric == 1 else np.sqrt((e * e).sum(1))
    return h, (d.astype(F) * F(1 + 2.0 ** -10)).astype(F), s, nr


def bounds(a, dsum, g, metric):
    if metric == 2:
        e = F(dsum * F(1 + 2.0 ** -10) + F(4) * g)
        return F(F(1) - a) - e, F(F(1) - a) + e
    r = F(np.sqrt(a)) if metric == 0 else a
    return F(F(r * F(F(1) - g)) - dsum), F(F(r + dsum) * F(F(1) + g))


def key_units(key, s, g, metric):
    if metric == 0:
        return F(s * F(F(np.sqrt(key)) * F(F(1) + g)))
    return F(s * F(key * F(F(1) + g))) if metric == 1 else key


@pytest.mark.parametrize("metric", [0, 1, 2])
@pytest.mark.parametrize("d,scale", [(3, 1.0), (40, 1e-20), (40, 1e4), (300, 1.0), (784, 0.01)])
def test_bounds_order_exact_keys(metric, d, scale):
    rng = np.random.Generator(np.random.PCG64(d + metric))
    g = F((2 * d + 64) * 2.0 ** -24)
    under = F(0)
    for trial in range(3):
        base = rng.standard_normal(d) * scale
        # candidates at nearly equal distances, so that the bounds are put to use
        x = np.stack([base] + [base + scale * 0.3 * rng.standard_normal(d) * (1 + 1e-4 * i) for i in range(24)]).astype(F)
        x[5] = x[4]
        h, delta, s, nr = rows16(x, metric)
        if metric == 0:
            under = F(s * F(np.sqrt(F(d * 2.0 ** -138))) * F(1.01))
        lo, hi, key = [], [], []
        for c in range(1, 25):
            t = h[0] - h[c]
            a = F((t.astype(np.float64) ** 2).sum()) if metric == 0 else F(np.abs(t).sum(dtype=F)) if metric == 1 \
                else F((h[0] * h[c]).sum(dtype=F))
            b = bounds(a, F(delta[0] + delta[c]), g, metric)
            lo.append(b[0])
            hi.append(b[1])
            key.append(exact_key(x[0], x[c], metric, nr[0] if metric == 2 else 0, nr[c] if metric == 2 else 0))
        used = 0
        for c in range(24):
            for e in range(24):
                widen = F(1) if metric == 2 else F(F(1) + g)
                if lo[c] > F(F(hi[e] * widen) + under):
                    used += 1
                    assert key[c] > key[e]
                if lo[c] > F(F(key_units(key[e], s, g, metric) * widen) + under):
                    assert key[c] > key[e]
        # the bounds do separate candidates (where the keys' squares do not underflow, which nothing can rank)
        assert used > 0 or (metric == 0 and scale < 1e-18)
