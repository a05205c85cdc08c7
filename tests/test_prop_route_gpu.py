"""Propagation with and without the candidate filter: shapes on either side of the rule that chooses between them give the
CPU restatement's lists, in FP32 and from FP16 rows, and the ranges of a sharded step take one route."""
from __future__ import annotations

import ctypes

import numpy as np
import pytest

from conftest import load_package

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("metric", [0, 1, 2])
@pytest.mark.parametrize("d,k", [(8, 5), (9, 5), (8, 6), (40, 3), (41, 3), (128, 8), (129, 8), (190, 6), (190, 5), (200, 8),
                                 (300, 4), (300, 8), (353, 8), (380, 8), (520, 14), (580, 14), (900, 8), (1000, 5), (1000, 9)])
def test_either_side(oracle, metric, d, k):
    acknn = load_package()
    x = acknn.workloads.gaussian_mixture(700, d, 4, seed=d + k)
    for y in (x, x.astype(np.float16)):
        gi, gd = acknn.knn_build(y, k, 2, max(24, 2 * k), 2, metric, seed=1)
        oi, od = oracle.knn_build(y.astype(np.float32), k, 2, max(24, 2 * k), 2, metric, seed=1)
        np.testing.assert_array_equal(gi, oi)
        np.testing.assert_array_equal(gd.view(np.uint32), od.view(np.uint32))


@pytest.mark.parametrize("world", [3, 7, 8, 9, 12])
def test_ranges_of_a_step_take_one_route(world):
    """Ranges of an even split differ by a point; the filter's rows are scratch, so the route shows in the bytes held."""
    torch = pytest.importorskip("torch")
    acknn = load_package()
    lib = acknn.load_library()
    n, d, k = 4003, 24, 16
    x = torch.from_numpy(acknn.workloads.gaussian_mixture(n, d, 8, seed=1)).cuda()
    ctx = acknn.Context(0)
    idx = torch.empty((n, k), dtype=torch.int32, device="cuda")
    key = torch.empty((n, k), dtype=torch.float32, device="cuda")
    opt = acknn.default_options(points_on_device=1, outputs_on_device=1, raw_keys=1)
    assert lib.knn_build_ex(ctx.handle, x.data_ptr(), n, d, k, 2, 60, 0, 0, 1, idx.data_ptr(), key.data_ptr(),
                            ctypes.byref(opt), None) == 0
    ctx.close()
    held, lists = set(), []
    for r in range(world):
        r0, r1 = acknn.sharded.point_range(n, r, world)
        oi, ok, fl = torch.empty_like(idx), torch.empty_like(key), torch.zeros((n, 1), dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()
        ctx = acknn.Context(0)
        assert lib.knn_propagate_range(ctx.handle, x.data_ptr(), n, d, k, 0, r0, r1, idx.data_ptr(), key.data_ptr(), None,
                                       oi.data_ptr(), ok.data_ptr(), fl.data_ptr(), ctypes.byref(opt)) == 0
        held.add(ctx.scratch_bytes)
        lists.append((oi[r0:r1].cpu(), ok[r0:r1].cpu()))
        ctx.close()
    assert len(held) == 1, held
    whole_i, whole_k = torch.empty_like(idx), torch.empty_like(key)
    fl = torch.zeros((n, 1), dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    ctx = acknn.Context(0)
    assert lib.knn_propagate_range(ctx.handle, x.data_ptr(), n, d, k, 0, 0, n, idx.data_ptr(), key.data_ptr(), None,
                                   whole_i.data_ptr(), whole_k.data_ptr(), fl.data_ptr(), ctypes.byref(opt)) == 0
    ctx.close()
    assert torch.equal(torch.cat([i for i, _ in lists]), whole_i.cpu())
    assert torch.equal(torch.cat([q for _, q in lists]), whole_k.cpu())


def test_statistics_name_the_route():
    acknn = load_package()
    for d, k, metric, dtype, want in ((64, 16, 0, np.float32, 1), (300, 8, 0, np.float32, 0), (300, 8, 2, np.float32, 0),
                                      (200, 8, 0, np.float32, 1), (200, 8, 0, np.float16, 0), (8, 5, 1, np.float32, 0),
                                      (1030, 8, 0, np.float32, 0)):
        x = acknn.workloads.gaussian_mixture(600, d, 4, seed=d).astype(dtype)
        assert acknn.knn_build(x, k, 2, 30, 1, metric, stats=True)[2]["prop_filtered"] == want
        assert acknn.knn_build(x, k, 2, 30, 0, metric, stats=True)[2]["prop_filtered"] == 0
