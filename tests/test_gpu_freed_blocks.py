"""Freed blocks that a context keeps: not handed out while any stream may use them, whatever another
thread captures meanwhile."""

import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


class _Alias:
    """A device tensor as torch sees it."""

    def __init__(self, t):
        self.__cuda_array_interface__ = {"shape": (t.nbytes,), "typestr": "|u1", "data": (t.ptr, False), "version": 3}


@pytest.mark.parametrize("nbytes", [4096, 3 << 20, 96 << 20])
def test_not_handed_out_under_another_stream(nbytes):
    """A kernel of a stream unknown to the context reads a block some 50 ms after it was freed."""
    import tenetgb
    import torch

    ctx = tenetgb.Context(0)
    rng = np.random.default_rng(0)
    data = rng.integers(0, 256, nbytes, dtype=np.uint8).view(np.float64)
    zeros = np.zeros_like(data)
    t = tenetgb.DeviceTensor.from_numpy(ctx, data)
    out = torch.zeros(nbytes, dtype=torch.uint8, device="cuda")
    alias = torch.as_tensor(_Alias(t), device="cuda")
    torch.cuda.synchronize()
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        torch.cuda._sleep(100_000_000)
        out.copy_(alias)
    del t
    for _ in range(40):  # (as many as are kept undrained, and more)
        u = tenetgb.DeviceTensor(ctx, data.shape, data.dtype)
        ctx.h2d(u.ptr, zeros)
        del u
    torch.cuda.synchronize()
    assert (out.cpu().numpy().view(np.float64).view(np.uint8) == data.view(np.uint8)).all()


def test_freed_while_another_thread_captures():
    """One thread holds a thread-local stream capture open while another allocates and frees."""
    import tenetgb
    import torch

    ctx = tenetgb.Context(0)
    x = torch.zeros(1024, device="cuda")
    errors = []

    def work():
        try:
            for k in range(100):
                tenetgb.DeviceTensor(ctx, (100 + k % 3,), np.complex128)  # (freed at once)
                if k % 20 == 0:
                    tenetgb.DeviceTensor(ctx, (1 << 23,), np.complex128)
        except Exception as e:
            errors.append(e)

    torch.cuda.synchronize()
    graph, stream = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    with torch.cuda.stream(stream):
        graph.capture_begin(capture_error_mode="thread_local")
        x.add_(1)
        thread = threading.Thread(target=work)
        thread.start()
        thread.join()
        x.add_(1)
        graph.capture_end()
    assert not errors
    graph.replay()
    torch.cuda.synchronize()
    assert (x == 2).all()
    # (a tensor's free that failed would have been swallowed: nothing may be left over)
    assert ctx.hbm_in_use() == 0
