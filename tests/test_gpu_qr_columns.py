"""QR with one CTA per column (k_qr_cols), with and without CTAs for the rows of Q, at the edges of its rows per thread, for tall, square
and wide matrices, batches, rank deficiency and in-place calls, against LAPACK.

Tolerances: Householder QR is backward stable, ‖QR − A‖ and ‖QᴴQ − I‖ are a small multiple of
√(m·k)·u with u = 1.1e-16; 1e-13 covers m = 512.  Q and R themselves follow LAPACK's sign
convention and agree with it to κ(A)·√(m·k)·u, κ ≤ 1e3 here for the tall Gaussian matrices.
"""

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    import tenetgb

    return tenetgb.Context(0)


def _qr(ctx, A, in_place=False, lda_pad=0):
    import tenetgb

    batch, m, n = A.shape
    k, lda = min(m, n), m + lda_pad
    store = np.zeros((batch, n, lda), complex)
    store[:, :, :m] = A.transpose(0, 2, 1)
    dA = tenetgb.DeviceTensor.from_numpy(ctx, store.reshape(-1), ["x"])
    dQ = dA if in_place else tenetgb.DeviceTensor.from_numpy(ctx, np.full(batch * m * k, np.nan + 0j), ["x"])
    dR = tenetgb.DeviceTensor.from_numpy(ctx, np.full(batch * k * n, np.nan + 0j), ["x"])
    sQ = lda * n if in_place else m * k
    ctx.check(ctx.lib.tn_qr_thin(ctx.h, 3, 0, m, n, C.c_void_p(dA.ptr), lda, lda * n, C.c_void_p(dQ.ptr), sQ,
                                 C.c_void_p(dR.ptr), k * n, batch))
    q, r = dQ.numpy(), dR.numpy()
    Q = np.stack([q[b * sQ: b * sQ + m * k].reshape((m, k), order="F") for b in range(batch)])
    return Q, r.reshape(batch, n, k).transpose(0, 2, 1)


def _check(A, Q, R, lapack=True):
    for a, q, r in zip(A, Q, R):
        scale = max(np.linalg.norm(a), 1e-300)
        assert np.linalg.norm(q @ r - a) <= 1e-13 * scale
        assert np.abs(q.conj().T @ q - np.eye(q.shape[1])).max() <= 1e-13
        assert (np.tril(r, -1) == 0).all() and (np.diagonal(r).imag == 0).all()
        if lapack:
            q0, r0 = np.linalg.qr(a)
            assert np.abs(q - q0).max() <= 1e-10 and np.abs(r - r0).max() <= 1e-10 * scale


@pytest.mark.parametrize("m,n,batch", [
    (1, 1, 1), (2, 1, 3), (2, 2, 1), (127, 5, 1), (128, 64, 2), (129, 40, 1), (256, 31, 1), (257, 33, 1), (512, 200, 1),
    (37, 90, 2), (128, 128, 1), (5, 300, 1), (300, 300, 1), (16, 8, 40), (513, 20, 1),
    (152, 152, 1), (153, 152, 1), (19, 19, 8), (19, 20, 8), (300, 4, 1), (300, 5, 1),
])
def test_columns_qr_matches_lapack(ctx, m, n, batch):
    rng = np.random.default_rng(m * 1000 + n)
    A = rng.standard_normal((batch, m, n)) + 1j * rng.standard_normal((batch, m, n))
    Q, R = _qr(ctx, A)
    _check(A, Q, R, lapack=m != n)


@pytest.mark.parametrize("m,n,batch,pad", [(64, 32, 2, 0), (200, 200, 1, 0), (30, 80, 2, 0), (64, 32, 2, 7)])
def test_columns_qr_in_place(ctx, m, n, batch, pad):
    rng = np.random.default_rng(m + n)
    A = rng.standard_normal((batch, m, n)) + 1j * rng.standard_normal((batch, m, n))
    Q, R = _qr(ctx, A, in_place=True, lda_pad=pad)
    _check(A, Q, R, lapack=m != n)


@pytest.mark.parametrize("scale", [1.0, 1e-120, 1e120])
def test_columns_qr_of_special_matrices(ctx, scale):
    """A zero column, repeated columns, a real matrix, an upper triangular one; tiny and huge entries."""
    rng = np.random.default_rng(5)
    g = rng.standard_normal((60, 24)) + 1j * rng.standard_normal((60, 24))
    zero, twice = g.copy(), g.copy()
    zero[:, 3] = 0
    twice[:, 9] = twice[:, 2]
    A = scale * np.stack([zero, twice, g.real + 0j, np.triu(g)])
    Q, R = _qr(ctx, A)
    _check(A, Q, R, lapack=False)


@pytest.mark.parametrize("bad", [np.nan, np.inf])
@pytest.mark.parametrize("m,n", [(60, 24), (200, 40)])
def test_columns_qr_non_finite(ctx, bad, m, n):
    """A column that is not finite spoils its own part of R, and Q from there on, and no column of R
    before it (Q's earlier columns follow all reflectors where its rows are formed)."""
    rng = np.random.default_rng(6)
    A = rng.standard_normal((1, m, n)) + 1j * rng.standard_normal((1, m, n))
    clean = A.copy()
    A[0, m // 2, 7] = bad
    Q, R = _qr(ctx, A)
    assert np.abs(R[0][:, :7] - np.linalg.qr(clean[0])[1][:, :7]).max() <= 1e-9
    assert not np.isfinite(R[0][:8, 7]).all() and not np.isfinite(Q[0][:, 8:]).any()


def test_columns_qr_norms_and_reflectors_to_rounding(ctx):
    """Single columns of three entries from 1e-130 to 1e130, on both sides of where Newton's iteration
    forms the norm and the reflector's scale: R = ∓‖a‖ and Q = a/R.

    With u = 1.1e-16: ‖a‖² is off by 3u, its root by 3u/2 and its own rounding, so R by 4u relative.
    An entry of Q is κ·u·conj(u₁), at most 2 in modulus, from a handful of such roundings: 16u.
    """
    rng = np.random.default_rng(7)
    n = 500
    g = rng.standard_normal((n, 3, 1)) + 1j * rng.standard_normal((n, 3, 1))
    A = g * 10.0 ** np.concatenate([rng.uniform(-130, 130, n - 100), rng.uniform(-91, -89, 50), rng.uniform(89, 91, 50)])[:, None, None]
    Q, R = _qr(ctx, A)
    wide = A[:, :, 0].astype(np.clongdouble)
    r = -np.sign(wide[:, 0].real) * np.sqrt((wide.real**2 + wide.imag**2).sum(axis=1))
    u = 2.0**-53
    assert np.abs(R[:, 0, 0] / r - 1).max() <= 4 * u
    assert np.abs(Q[:, :, 0] - wide / r[:, None]).max() <= 16 * u
