"""The FP32 leaf stage's tensor-core filter (k_center_operand, k_leaf_tc and key_distance / minimum_distance of
approximate-cuda-knn_b200/csrc/leaf_umma.cu), restated.

A leaf's rows are rounded to FP16 of s (x - c), c a row of the leaf (COSINE: of s (u - v), unit rows), and delta bounds a
row's rounding error.  A column is dropped where |h_q|^2 + |h_c|^2 - 2 h_q.h_c exceeds (t + delta_q + delta_c)^2 widened by
the products' rounding, t being the scaled distance of an exact key, or a bound on it from another pair's 16-bit rows.
Dropped columns must have larger exact keys than that pair."""
from __future__ import annotations

import numpy as np
import pytest

from test_prop_filter_bounds import F, exact_key


def rows16(x, c, metric, s):
    if metric == 2:
        nr = np.array([np.sqrt(exact_key(np.zeros_like(r), r, 0, 0, 0)) for r in x], dtype=F)
        u = (x * (F(1) / nr)[:, None]).astype(F)
        v = ((u - u[c]).astype(F) * s).astype(F)
        base = F(s * F(2.0 ** -21))
    else:
        nr, v, base = np.zeros(len(x), dtype=F), ((x - x[c]).astype(F) * s).astype(F), F(0)
    h = v.astype(np.float16).astype(F)
    e = (v - h).astype(np.float64)
    sq = (h.astype(np.float64) ** 2).sum(1).astype(F)
    delta = (np.sqrt((e * e).sum(1)) * (1 + 2.0 ** -10) + np.sqrt(sq.astype(np.float64)) * 2.0 ** -23 + base).astype(F)
    return h, sq, delta, nr


@pytest.mark.parametrize("metric", [0, 2])
@pytest.mark.parametrize("d,scale,offset", [(3, 1.0, 0.0), (40, 1e-20, 0.0), (40, 1e4, 0.0), (128, 1.0, 1000.0),
                                            (256, 0.01, 1.0)])
def test_dropped_columns_have_larger_keys(metric, d, scale, offset):
    rng = np.random.Generator(np.random.PCG64(d + metric))
    g, g1 = F((2 * d + 64) * 2.0 ** -24), F((d + 64) * 2.0 ** -21)
    used = 0
    for trial in range(3):
        base = rng.standard_normal(d) * scale + offset
        spread = 0.3 * scale if trial < 2 else 3e-3 * scale
        x = np.stack([base] + [base + spread * (1 + 0.02 * i) * rng.standard_normal(d) for i in range(24)]).astype(F)
        x[5] = x[4]
        m = np.abs(x).max()
        s = F(8192) if metric == 2 else F(2.0 ** (14 - np.frexp(m)[1]))
        h, sq, delta, nr = rows16(x, 12, metric, s)
        key = [exact_key(x[0], x[c], metric, nr[0], nr[c]) for c in range(1, 25)]
        dot = (h[1:] * h[0]).sum(1, dtype=F)
        lower = (sq[1:] - F(2) * dot).astype(F)  # + |h_q|^2 on both sides
        cm, dt = sq.max(), delta.max()

        def threshold(t):
            r = F(F(t + delta[0] + dt) * (F(1) + g))
            return F(F(r * r + g1 * (sq[0] + cm)) - sq[0])

        for e in range(24):
            q = F(2) * max(key[e], F(0)) + F(3) * g if metric == 2 else key[e] + F(d * 2.0 ** -138)
            exact = F(s * F(np.sqrt(F(q))) * (F(1) + g))
            r = F(np.sqrt(max(F(lower[e] + sq[0] + g1 * (sq[0] + cm)), F(0)))) + F(delta[0] + dt)
            slack = F(6) * g if metric == 2 else F(d * 2.0 ** -137)
            rows = F(F(np.sqrt(F(r * r + s * F(s * slack)))) * (F(1) + F(2) * g))
            for t in (threshold(exact), threshold(rows)):
                for c in range(24):
                    if lower[c] > t:
                        used += 1
                        assert key[c] > key[e]
    # the filter does drop columns, except where no FP32 key ranks them: squares that underflow, or COSINE keys (about
    # (0.3 scale / offset)^2 / 2) below their own rounding, 1.5 g
    blind = scale < 1e-18 if metric == 0 else offset > 0 and 0.045 * (scale / offset) ** 2 < 1.5 * g
    assert used > 0 or blind
