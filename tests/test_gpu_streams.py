"""Calls on the context's own stream (NULL) while other streams are captured."""
import ctypes

import numpy as np
import pytest

from tracking_optimizations_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("blocking", [False, True])
def test_call_beside_a_capture(gpu, blocking):
    """A stream that synchronises with the legacy default stream (blocking) or
    does not is being captured: the call runs and the capture goes on.  Waiting
    for the default stream would end the blocking stream's capture."""
    import torch

    from tracking_optimizations_b200 import _native, gpu_tracking

    spec = synth.scaled(synth.PLAIN_1000, frames=4, height=96, width=96, spots=30, seed=4)
    frames = torch.from_numpy(synth.make_movie(spec).view(np.int16)).cuda()
    want = gpu_tracking.batch_device(frames, 7)
    ctx, lib, params = _native.context(0), _native.load(), _native.make_params(7)
    out, n = torch.zeros_like(want), ctypes.c_int64()
    x = torch.zeros(1000, device="cuda")
    cudart = torch.cuda.cudart()
    raw = ctypes.c_void_p()
    if blocking:
        assert int(cudart.cudaStreamCreate(ctypes.addressof(raw))) == 0
        stream = torch.cuda.ExternalStream(raw.value)
    else:
        stream = torch.cuda.Stream()
    graph = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    try:
        with torch.cuda.graph(graph, stream=stream, capture_error_mode="relaxed"):
            x.add_(1.0)
            st = lib.gt_batch_device(ctx, frames.data_ptr(), _native.GT_U16, 4, 96, 96, ctypes.byref(params),
                                     out.data_ptr(), len(out), ctypes.byref(n), None)
            x.mul_(2.0)
        assert st == 0, lib.gt_last_error(ctx)
        assert n.value == len(want) and torch.equal(out, want)
        graph.replay()
        torch.cuda.synchronize()
        assert torch.all(x == 2.0)
    finally:
        torch.cuda.synchronize()
        del graph
        if blocking:
            cudart.cudaStreamDestroy(raw.value)
