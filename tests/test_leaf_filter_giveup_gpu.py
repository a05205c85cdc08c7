"""A plain FP32 build whose filter tiles give up: the tree goes to dense FP32 tiles and the build succeeds with the same
graph, whether synchronous, asynchronous or a batch, and reports no failure.  The give-up is set from the host
(knn_test_fail_next_tile_wait); no device wait runs out here."""
from __future__ import annotations

import ctypes

import numpy as np
import pytest

from conftest import load_package

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("metric", [0, 2])
@pytest.mark.parametrize("leaf", [40, 120, 600])  # groups of leaves; one tile a leaf; the bounding pass (every tree filtered)
def test_synchronous_build(metric, leaf):
    acknn = load_package()
    lib = acknn.load_library()
    x = acknn.workloads.gaussian_mixture(40_000, 48, 8, seed=leaf)
    ctx = acknn.Context(0)
    try:
        want = acknn.knn_build(x, 10, 3, leaf, 1, metric, seed=2, tile_pairs=-1)
        for _ in range(2):
            assert lib.knn_test_fail_next_tile_wait(ctx.handle) == 0
            gi, gd = acknn.knn_build(x, 10, 3, leaf, 1, metric, seed=2, context=ctx.handle)
            np.testing.assert_array_equal(gi, want[0])
            np.testing.assert_array_equal(gd.view(np.uint32), want[1].view(np.uint32))
        assert lib.knn_context_status(ctx.handle, None) == 0
    finally:
        ctx.close()


def test_asynchronous_build_and_the_one_after():
    import torch

    acknn = load_package()
    lib = acknn.load_library()
    x = acknn.workloads.gaussian_mixture(30_000, 64, 8, seed=1)
    wi, wd = acknn.knn_build(x, 10, 4, 300, 0, 0, seed=3, tile_pairs=-1)
    xd = torch.from_numpy(x).cuda()
    oi = torch.empty((30_000, 10), dtype=torch.int32, device="cuda")
    od = torch.empty((30_000, 10), dtype=torch.float32, device="cuda")
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    ctx = acknn.Context(0)
    opt = acknn.default_options(points_on_device=1, outputs_on_device=1, stream=stream.cuda_stream)
    try:
        for hook in (True, False):
            if hook:
                assert lib.knn_test_fail_next_tile_wait(ctx.handle) == 0
            oi.fill_(-1)
            torch.cuda.synchronize()
            assert lib.knn_build_ex(ctx.handle, xd.data_ptr(), 30_000, 64, 10, 4, 300, 0, 0, 3, oi.data_ptr(),
                                    od.data_ptr(), ctypes.byref(opt), None) == 0
            assert lib.knn_context_status(ctx.handle, ctypes.c_void_p(stream.cuda_stream)) == 0
            np.testing.assert_array_equal(oi.cpu().numpy(), wi)
            np.testing.assert_array_equal(od.cpu().numpy().view(np.uint32), wd.view(np.uint32))
    finally:
        stream.synchronize()
        ctx.close()


def test_batch():
    acknn = load_package()
    lib = acknn.load_library()
    sets = [acknn.workloads.gaussian_mixture(n, 32, 8, seed=n) for n in (9000, 5000, 2500)]
    ctx = acknn.Context(0)
    try:
        want = [acknn.knn_build(x, 10, 3, 300, 1, 0, tile_pairs=-1) for x in sets]
        for hook in (False, True, False, False):  # eager, given up, captured, replayed
            if hook:
                assert lib.knn_test_fail_next_tile_wait(ctx.handle) == 0
            for (gi, gd), (wi, wd) in zip(acknn.knn_build_batch(sets, 10, 3, 300, 1, 0, context=ctx.handle), want):
                np.testing.assert_array_equal(gi, wi)
                np.testing.assert_array_equal(gd.view(np.uint32), wd.view(np.uint32))
    finally:
        ctx.close()
