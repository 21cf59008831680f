"""The QR's tuning table: an entry sets the blocked QR's widths where that kernel runs, and does not take a
shape away from the kernel with one CTA per column.

Tolerance: Householder QR is backward stable, 1e-13 covers the sizes here (√(m·n)·u ≤ 4e-14).
"""

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _qr(ctx, A):
    """A: (batch, m, n); Q, R and the kernels launched"""
    import tenetgb

    batch, m, n = A.shape
    k = min(m, n)
    dA = tenetgb.DeviceTensor.from_numpy(ctx, np.transpose(A, (1, 2, 0)))
    dQ, dR = tenetgb.DeviceTensor(ctx, (m, k, batch), complex), tenetgb.DeviceTensor(ctx, (k, n, batch), complex)
    before = ctx.launches()
    ctx.check(ctx.lib.tn_qr_thin(ctx.h, 3, 0, m, n, C.c_void_p(dA.ptr), m, m * n, C.c_void_p(dQ.ptr), m * k,
                                 C.c_void_p(dR.ptr), k * n, batch))
    launched = ctx.launches() - before
    Q, R = np.transpose(dQ.numpy(), (2, 0, 1)), np.transpose(dR.numpy(), (2, 0, 1))
    for a, q, r in zip(A, Q, R):
        assert np.linalg.norm(q @ r - a) <= 1e-13 * np.linalg.norm(a)
        assert np.abs(q.conj().T @ q - np.eye(k)).max() <= 1e-13
        assert (np.tril(r, -1) == 0).all()
    return launched


def _gauss(batch, m, n):
    rng = np.random.default_rng(m + n + batch)
    return rng.standard_normal((batch, m, n)) + 1j * rng.standard_normal((batch, m, n))


@pytest.mark.parametrize("m,n,batch,bucket", [(64, 64, 1, 1), (300, 77, 3, 4), (512, 256, 1, 1)])
def test_entry_of_a_shape_of_the_column_kernel(m, n, batch, bucket):
    import tenetgb

    ctx = tenetgb.Context(0)
    ctx.load_tuning(f"qr8:{m}:{n}:{bucket} 4 1\n")
    assert _qr(ctx, _gauss(batch, m, n)) == 1


@pytest.mark.parametrize("m,n,batch,bucket", [(513, 20, 1, 1), (600, 77, 3, 4), (64, 64, 40, 64), (8, 64, 40, 64), (4, 2, 900, 64)])
@pytest.mark.parametrize("nb,slab", [(1, 1), (4, 2), (8, 4), (16, 1)])
def test_entry_of_a_shape_of_the_blocked_kernel(m, n, batch, bucket, nb, slab):
    import tenetgb

    ctx = tenetgb.Context(0)
    ctx.load_tuning(f"qr8:{m}:{n}:{bucket} {nb} {slab}\n")
    widths = -(-min(m, n) // nb)  # panels, if the rows leave room for this width
    assert _qr(ctx, _gauss(batch, m, n)) >= 2 * widths
    assert ctx.tuning() == f"qr8:{m}:{n}:{bucket} {nb} {slab}\n"


def test_autotuner():
    import tenetgb

    ctx = tenetgb.Context(0)
    ctx.set_autotune(True)
    _qr(ctx, _gauss(1, 64, 64))
    assert ctx.tuning() == ""
    _qr(ctx, _gauss(1, 600, 40))
    assert ctx.tuning().startswith("qr8:600:40:1 ")
    _qr(ctx, _gauss(1, 600, 40))
