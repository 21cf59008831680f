"""Freed blocks that a context keeps: not handed out while any stream may use them, whatever another
thread captures meanwhile, and never beyond the HBM budget."""

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


def _held(before):
    import torch

    return before - torch.cuda.mem_get_info()[0]


@pytest.mark.parametrize("sizes", [(80, 64, 36), (90, 75, 25), (40, 33, 67)])
def test_budget_holds_over_reused_blocks(sizes):
    """A block freed, one up to a quarter smaller taken, then what the budget leaves: the memory held is
    within it, up to the driver's pages of 2 MiB, and nothing within it is refused."""
    import tenetgb
    import torch

    MB = 1 << 20
    ctx = tenetgb.Context(0)
    warm = ctx.alloc(256)
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    ctx.set_hbm_budget(100 * MB + 256)
    first, second, third = (s * MB for s in sizes)
    ctx.free(ctx.alloc(first))
    assert _held(before) <= 100 * MB + 8 * MB
    p, q = ctx.alloc(second), ctx.alloc(third)
    assert ctx.hbm_in_use() == second + third + 256
    assert _held(before) <= 100 * MB + 8 * MB
    with pytest.raises(Exception, match="budget"):
        ctx.alloc(1)
    ctx.free(p)
    ctx.free(q)
    ctx.free(warm)


def test_budget_set_over_kept_blocks():
    import tenetgb
    import torch

    MB = 1 << 20
    ctx = tenetgb.Context(0)
    ctx.alloc(256)
    before = torch.cuda.mem_get_info()[0]
    for p in [ctx.alloc(s * MB) for s in (50, 60, 70)]:
        ctx.free(p)
    ctx.set_hbm_budget(100 * MB)
    assert _held(before) <= 100 * MB + 8 * MB


def test_release_cached():
    import tenetgb
    import torch

    MB = 1 << 20
    ctx = tenetgb.Context(0)
    ctx.alloc(256)
    before = torch.cuda.mem_get_info()[0]
    for p in [ctx.alloc(s * MB) for s in (50, 60, 70)]:
        ctx.free(p)
    ctx.release_cached()
    assert _held(before) <= 8 * MB and ctx.hbm_in_use() == 256
    ctx.free(ctx.alloc(60 * MB))
