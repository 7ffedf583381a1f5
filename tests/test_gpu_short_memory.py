"""A movie where device memory is short: smaller capacities serve when the
usual ones do not fit."""
import ctypes

import numpy as np
import pytest

from tracking_optimizations_b200 import synth

pytestmark = pytest.mark.gpu


def test_movie_beside_other_data(gpu):
    import torch

    from tracking_optimizations_b200 import gpu_tracking

    T, H, W = 60, 2048, 2040
    spec = synth.scaled(synth.PLAIN_1000, frames=2, height=H, width=W, spots=2000, seed=1)
    frames = torch.from_numpy(synth.make_movie(spec).view(np.int16)).cuda().repeat(T // 2, 1, 1)
    params = dict(search_range=4.0, memory=3)
    want = gpu_tracking.batch_device(frames, 9, **params)
    out, n = torch.zeros_like(want), ctypes.c_int64()
    ctx, lib, p = ctypes.c_void_p(), gpu.load(), gpu.make_params(9, **params)
    assert lib.gt_ctx_create(0, ctypes.byref(ctx)) == 0
    torch.cuda.empty_cache()
    # the usual capacities want 1 GB and more, half of them 0.8
    free = torch.cuda.mem_get_info()[0]
    data = torch.empty(free - (850 << 20), dtype=torch.uint8, device="cuda")
    try:
        for _ in range(2):
            out.zero_()
            st = lib.gt_batch_device(ctx, frames.data_ptr(), 0, T, H, W, ctypes.byref(p), out.data_ptr(), len(out),
                                     ctypes.byref(n), None)
            assert st == 0, lib.gt_last_error(ctx)
            assert n.value == len(want) and torch.equal(out, want)
            assert lib.gt_last_error(ctx) == b""
        # what does not fit at all is refused, and the next call is not
        large = gpu.make_params(9, search_range=9.0, memory=900)
        st = lib.gt_batch_device(ctx, frames.data_ptr(), 0, 30 * T, H // 30, W, ctypes.byref(large), out.data_ptr(),
                                 len(out), ctypes.byref(n), None)
        assert st == gpu.GT_ERR_OOM
        st = lib.gt_batch_device(ctx, frames.data_ptr(), 0, 2, H, W, ctypes.byref(p), out.data_ptr(), len(out),
                                 ctypes.byref(n), None)
        assert st == 0, lib.gt_last_error(ctx)
    finally:
        lib.gt_ctx_destroy(ctx)
        del data
        torch.cuda.empty_cache()
