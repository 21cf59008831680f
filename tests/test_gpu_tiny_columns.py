"""FP64 QR and SVD of matrices whose squared column norms, or their inverses, leave FP64's range:
columns of falling scale down to 1e-300, whole matrices of tiny or huge entries, and a tiny
complex residual below columns of ordinary size.

Tolerances: Householder QR and the Jacobi sweeps are backward stable whatever the scale,
‖QR − A‖, ‖UΣVᴴ − A‖ ≤ 1e-13·‖A‖ and |QᴴQ − I| ≤ 1e-13 as for matrices of ordinary size
(√(m·n)·u is 4e-14 at m = n = 400).  The residual of a QR holds column by column, as each column is
reflected by itself; it is asked of the columns down to 1e-150 of the largest.
"""

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(23, 23), (24, 24), (64, 64), (200, 200), (30, 23), (40, 24), (129, 64), (300, 200)]


@pytest.fixture(scope="module")
def ctx():
    import tenetgb

    return tenetgb.Context(0)


def _matrix(kind, m, n):
    """(A / 2^e, e)"""
    rng = np.random.default_rng(m * 1000 + n)
    g = rng.standard_normal((m, n)) + 1j * rng.standard_normal((m, n))
    if kind == "graded":
        return g * 10.0 ** np.linspace(0, -300, n), 0
    if kind == "graded_up":
        return g * 10.0 ** np.linspace(-300, 0, n), 0
    if kind == "residual":  # column 5 is the combination of the columns before it, but for 1e-159
        g[:, :5] = 0
        g[np.arange(5), np.arange(5)] = 1
        g[5:, 5] *= 1e-159
        return g, 0
    return g, {"1e-158": -525, "1e-300": -997, "1e+250": 830}[kind]


KINDS = ["graded", "graded_up", "residual", "1e-158", "1e-300", "1e+250"]


@pytest.mark.parametrize("m,n", SHAPES)
@pytest.mark.parametrize("kind", KINDS)
def test_qr(ctx, m, n, kind):
    import tenetgb

    A, e = _matrix(kind, m, n)
    dA = tenetgb.DeviceTensor.from_numpy(ctx, np.ldexp(A.real, e) + 1j * np.ldexp(A.imag, e))
    dQ = tenetgb.DeviceTensor.from_numpy(ctx, np.full((m, n), np.nan + 0j))
    dR = tenetgb.DeviceTensor.from_numpy(ctx, np.full((n, n), np.nan + 0j))
    ctx.check(ctx.lib.tn_qr_thin(ctx.h, 3, 0, m, n, C.c_void_p(dA.ptr), m, m * n, C.c_void_p(dQ.ptr), m * n,
                                 C.c_void_p(dR.ptr), n * n, 1))
    Q, R = dQ.numpy(), dR.numpy()
    R = np.ldexp(R.real, -e) + 1j * np.ldexp(R.imag, -e)
    assert np.isfinite(Q).all() and np.isfinite(R).all()
    assert np.abs(Q.conj().T @ Q - np.eye(n)).max() <= 1e-13
    assert (np.tril(R, -1) == 0).all() and (np.diagonal(R).imag == 0).all()
    assert np.linalg.norm(Q @ R - A) <= 1e-13 * np.linalg.norm(A)
    size = np.abs(A).max(axis=0)
    big = size > 1e-150 * size.max()
    err = np.linalg.norm((Q @ (R[:, big] / size[big])) - A[:, big] / size[big], axis=0)
    assert (err <= 1e-13 * np.linalg.norm(A[:, big] / size[big], axis=0)).all()


# (matrices of fewer than 24 columns have no QR before the sweeps and are swept as they are)
@pytest.mark.parametrize("m,n,kind", [(m, n, k) for m, n in SHAPES for k in KINDS if n >= 24 or k[0] != "1"])
def test_svd(ctx, m, n, kind):
    import tenetgb

    A, e = _matrix(kind, m, n)
    dA = tenetgb.DeviceTensor.from_numpy(ctx, np.ldexp(A.real, e) + 1j * np.ldexp(A.imag, e), ["r", "c"])
    U, S, V = (x.numpy() for x in tenetgb.tensor_svd_thin(dA, ["r"], ["c"], "s"))
    S = np.ldexp(S, -e)
    for x in (U, S, V):
        assert np.isfinite(x).all()
    assert (np.diff(S) <= 0).all()
    assert np.abs(U.conj().T @ U - np.eye(n)).max() <= 1e-13
    assert np.abs(V @ V.conj().T - np.eye(n)).max() <= 1e-13
    assert np.linalg.norm((U * S) @ V - A) <= 1e-13 * np.linalg.norm(A)


@pytest.mark.parametrize("n", [23, 24, 64, 200])
@pytest.mark.parametrize("kind", ["graded", "graded_up", "residual"])
def test_left_vectors_only(ctx, n, kind):
    """A two-site update that keeps U and S·Vᴴ: the SVD without right vectors."""
    import tenetgb

    A, _ = _matrix(kind, n, n)
    T = lambda x, inds: tenetgb.DeviceTensor.from_numpy(ctx, x, inds)
    a = T(A.reshape(n, 1, n), ["l", "a", "m"])
    b = T(np.eye(n, dtype=complex).reshape(n, 1, n), ["m", "b", "r"])
    one = T(np.ones((1, 1, 1, 1), complex), ["ao", "bo", "a", "b"])
    an, bn = tenetgb.simple_update(a, "a", b, "b", "m", one, "ao", "bo", absorb="v")
    u, sv = an.numpy().reshape(n, -1), bn.numpy().reshape(-1, n)
    assert np.isfinite(u).all() and np.isfinite(sv).all()
    assert np.abs(u.conj().T @ u - np.eye(u.shape[1])).max() <= 1e-13
    assert np.linalg.norm(u @ sv - A) <= 1e-13 * np.linalg.norm(A)
