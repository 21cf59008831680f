"""Batches of small FP64 SVDs with both factors on both sides of where one CTA per matrix takes less time
than a CTA per column pair.  The route is told by the sweeps reported (−1: one CTA per matrix).

Tolerance: 1e-12, as in the other tests of the two kernels' batches.
"""

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,batch,in_smem", [
    (8, 8, 64, False), (8, 8, 128, True), (8, 8, 200, True), (16, 16, 100, False), (16, 16, 128, True), (24, 16, 303, True),
    (32, 32, 64, False), (32, 32, 128, True), (32, 32, 200, False), (48, 24, 128, False), (64, 24, 303, True),
    (9, 9, 1, False), (31, 8, 152, True), (100, 100, 150, False),
])
def test_batched_svd(m, n, batch, in_smem):
    import tenetgb

    ctx = tenetgb.Context(0)
    rng = np.random.default_rng(m * n + batch)
    A = rng.standard_normal((batch, m, n)) + 1j * rng.standard_normal((batch, m, n))
    dA = tenetgb.DeviceTensor.from_numpy(ctx, np.transpose(A, (1, 2, 0)))
    dU, dV = tenetgb.DeviceTensor(ctx, (m, n, batch), complex), tenetgb.DeviceTensor(ctx, (n, n, batch), complex)
    dS = tenetgb.DeviceTensor(ctx, (n, batch), float)
    ctx.check(ctx.lib.tn_svd_thin(ctx.h, 3, 0, m, n, C.c_void_p(dA.ptr), m, m * n, C.c_void_p(dU.ptr), m * n,
                                  C.c_void_p(dS.ptr), n, C.c_void_p(dV.ptr), n * n, batch))
    f32, f64 = C.c_int32(), C.c_int32()
    ctx.check(ctx.lib.tn_svd_last_sweeps(ctx.h, C.byref(f32), C.byref(f64), None, 0))
    assert (f64.value == -1) == in_smem
    U, S, V = (np.moveaxis(x.numpy(), -1, 0) for x in (dU, dS, dV))
    scale = np.linalg.norm(A, axis=(1, 2))
    assert (np.linalg.norm((U * S[:, None, :]) @ V - A, axis=(1, 2)) <= 1e-12 * scale).all()
    eye = np.eye(n)
    assert np.abs(np.conj(np.transpose(U, (0, 2, 1))) @ U - eye).max() <= 1e-12
    assert np.abs(V @ np.conj(np.transpose(V, (0, 2, 1))) - eye).max() <= 1e-12
    assert (np.diff(S, axis=1) <= 0).all()


@pytest.mark.parametrize("m,n,batch", [(300, 90, 5), (300, 90, 12), (257, 120, 9), (400, 150, 6), (512, 80, 10)])
def test_batches_of_tall_matrices(m, n, batch):
    """More than 256 rows, on both sides of where several launches of pairs take longer than a launch per round."""
    import tenetgb

    ctx = tenetgb.Context(0)
    rng = np.random.default_rng(m * n + batch)
    A = rng.standard_normal((batch, m, n)) + 1j * rng.standard_normal((batch, m, n))
    dA = tenetgb.DeviceTensor.from_numpy(ctx, np.transpose(A, (1, 2, 0)))
    dU, dV = tenetgb.DeviceTensor(ctx, (m, n, batch), complex), tenetgb.DeviceTensor(ctx, (n, n, batch), complex)
    dS = tenetgb.DeviceTensor(ctx, (n, batch), float)
    ctx.check(ctx.lib.tn_svd_thin(ctx.h, 3, 0, m, n, C.c_void_p(dA.ptr), m, m * n, C.c_void_p(dU.ptr), m * n,
                                  C.c_void_p(dS.ptr), n, C.c_void_p(dV.ptr), n * n, batch))
    U, S, V = (np.moveaxis(x.numpy(), -1, 0) for x in (dU, dS, dV))
    scale = np.linalg.norm(A, axis=(1, 2))
    assert (np.linalg.norm((U * S[:, None, :]) @ V - A, axis=(1, 2)) <= 1e-12 * scale).all()
    assert np.abs(np.conj(np.transpose(U, (0, 2, 1))) @ U - np.eye(n)).max() <= 1e-12
    assert np.abs(V @ np.conj(np.transpose(V, (0, 2, 1))) - np.eye(n)).max() <= 1e-12


@pytest.mark.parametrize("m,n,batch", [(128, 120, 1), (128, 128, 19), (128, 128, 20), (126, 126, 40)])
def test_fp32_block_rounds(m, n, batch):
    """ComplexF32 SVDs in blocks of columns, with a row or two per thread.  FP32: 1e-4 (√n·sweeps·u is 1e-5)."""
    import tenetgb

    ctx = tenetgb.Context(0)
    rng = np.random.default_rng(m * n + batch)
    A = (rng.standard_normal((batch, m, n)) + 1j * rng.standard_normal((batch, m, n))).astype(np.complex64)
    dA = tenetgb.DeviceTensor.from_numpy(ctx, np.transpose(A, (1, 2, 0)))
    dU, dV = tenetgb.DeviceTensor(ctx, (m, n, batch), np.complex64), tenetgb.DeviceTensor(ctx, (n, n, batch), np.complex64)
    dS = tenetgb.DeviceTensor(ctx, (n, batch), float)
    ctx.check(ctx.lib.tn_svd_thin(ctx.h, 2, 0, m, n, C.c_void_p(dA.ptr), m, m * n, C.c_void_p(dU.ptr), m * n,
                                  C.c_void_p(dS.ptr), n, C.c_void_p(dV.ptr), n * n, batch))
    U, S, V = (np.moveaxis(x.numpy(), -1, 0) for x in (dU, dS, dV))
    scale = np.linalg.norm(A, axis=(1, 2))
    assert (np.linalg.norm((U * S[:, None, :]) @ V - A, axis=(1, 2)) <= 1e-4 * scale).all()
    assert np.abs(np.conj(np.transpose(U, (0, 2, 1))) @ U - np.eye(n)).max() <= 1e-4
