"""The SVD kernels at the edges of their row and column groups: the column-pair kernel (two
threads per row up to 64 rows, then 1, 2 and 4 rows per thread), the ordered QR before it, and
the tensor-pipe block rounds of the mixed pre-pass (32 columns, 128 rows at a time).

Tolerances: the sweeps end with couplings at rounding level, so ‖UΣVᴴ − A‖ ≤ 1e-13·‖A‖ and
|UᴴU − I|, |VᴴV − I| ≤ 1e-13 in FP64 (√n·sweeps·u is 3e-14 at n = 512); the mixed path's products
are accurate to 1e-14 per entry (8 digit planes), 1e-12 over n of them; values to 1e-12 of the
largest.
"""

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    import tenetgb

    return tenetgb.Context(0)


def _svd(ctx, A, prec):
    """A: (batch, m, n) through tn_svd_thin."""
    import tenetgb

    batch, m, n = A.shape
    k = min(m, n)
    dA = tenetgb.DeviceTensor.from_numpy(ctx, np.concatenate([a.reshape(-1, order="F") for a in A]), ["x"])
    dU, dV = (tenetgb.DeviceTensor(ctx, (batch * k * x,), np.complex128) for x in (m, n))
    dS = tenetgb.DeviceTensor(ctx, (batch * k,), np.float64)
    ctx.check(ctx.lib.tn_svd_thin(ctx.h, 3, prec, m, n, C.c_void_p(dA.ptr), m, m * n, C.c_void_p(dU.ptr), m * k,
                                  C.c_void_p(dS.ptr), k, C.c_void_p(dV.ptr), k * n, batch))
    U = dU.numpy().reshape(batch, k, m).transpose(0, 2, 1)
    Vh = dV.numpy().reshape(batch, n, k).transpose(0, 2, 1)
    return U, dS.numpy().reshape(batch, k), Vh


def _check(A, U, S, Vh, tol):
    for a, u, s, v in zip(A, U, S, Vh):
        scale, k = np.linalg.norm(a), len(s)
        assert np.linalg.norm((u * s) @ v - a) <= tol * scale
        assert np.abs(u.conj().T @ u - np.eye(k)).max() <= tol
        assert np.abs(v @ v.conj().T - np.eye(k)).max() <= tol
        assert (np.diff(s) <= 0).all()
        ref = np.linalg.svd(a, compute_uv=False)
        assert np.abs(s - ref).max() <= 1e-12 * ref[0]


def _gauss(rng, shape):
    return rng.standard_normal(shape) + 1j * rng.standard_normal(shape)


@pytest.mark.parametrize("m,n,batch", [
    (8, 8, 1), (9, 9, 3), (24, 23, 1), (24, 24, 2), (25, 24, 1), (64, 64, 1), (65, 63, 1), (65, 65, 1), (128, 31, 1),
    (128, 128, 2), (129, 129, 1), (256, 90, 1), (257, 100, 1), (300, 256, 1), (512, 33, 1), (40, 100, 2), (500, 499, 1),
    (33, 33, 40), (16, 12, 700),
])
def test_native_svd(ctx, m, n, batch):
    rng = np.random.default_rng(m * 1000 + n)
    A = _gauss(rng, (batch, m, n))
    _check(A, *_svd(ctx, A, 0), 1e-13)


@pytest.mark.parametrize("m,n", [(23, 23), (64, 2), (65, 3), (129, 22), (257, 23), (512, 8), (300, 300)])
@pytest.mark.parametrize("kind", ["parallel", "repeated", "zero"])
def test_large_rotations(ctx, m, n, kind):
    """Columns that are almost one another, equal or zero: angles of 45° round after round, which the
    columns' scales take up, and pairs that must be left alone."""
    rng = np.random.default_rng(m * 1000 + n)
    A = _gauss(rng, (m, n))
    if kind == "parallel":
        A = A[:, :1] * np.exp(2j * np.pi * rng.random(n)) + 1e-3 * A
    elif kind == "repeated":
        A = A[:, rng.integers(0, (n + 1) // 2, n)] * rng.choice([1, -1, 1j], n)
    else:
        A[:, rng.permutation(n)[: n // 2]] = 0
    U, S, Vh = _svd(ctx, A[None], 0)
    _check(A[None], U, S, Vh, 1e-13)


@pytest.mark.parametrize("m,n,batch", [(128, 128, 1), (129, 128, 2), (200, 150, 1), (256, 255, 1), (385, 130, 3), (512, 512, 1)])
def test_mixed_svd(ctx, m, n, batch):
    rng = np.random.default_rng(m * 1000 + n)
    A = _gauss(rng, (batch, m, n))
    _check(A, *_svd(ctx, A, 1), 1e-12)


@pytest.mark.parametrize("m,n", [(128, 128), (256, 200), (512, 512)])
@pytest.mark.parametrize("coupling", [0.0, 1e-15, 1e-20, 1e-22, 1e-25, 1e-40])
def test_mixed_svd_of_nearly_orthogonal_columns(ctx, m, n, coupling):
    """Couplings whose squares are no normal FP32 numbers must not turn into rotations."""
    rng = np.random.default_rng(m + n)
    A = coupling * _gauss(rng, (m, n))
    A[np.arange(n), rng.permutation(n)] += np.linspace(1.0, 2.0, n) * np.exp(2j * np.pi * rng.random(n))
    _check(A[None], *_svd(ctx, A[None], 1), 1e-12)


@pytest.mark.parametrize("m,n", [(32, 32), (100, 40)])
@pytest.mark.parametrize("scale", [1.0, 1e-130, 1e130])
def test_columns_of_different_scale(ctx, m, n, scale):
    """A·D with D over twelve decades, unsorted: one-sided Jacobi finds the small values to their
    own relative accuracy, and the ordering before the QR keeps that.  κ of the unscaled factor
    is below 1e3, so 1e-11 relative."""
    rng = np.random.default_rng(m + n)
    d = 10.0 ** rng.permutation(np.linspace(0, -12, n))
    q, _ = np.linalg.qr(_gauss(rng, (m, n)))
    B = q @ (np.eye(n) + 0.3 * _gauss(rng, (n, n)) / np.sqrt(n))
    A = (scale * B * d)[None]
    U, S, Vh = _svd(ctx, A, 0)
    # reference: the same values from the graded Gram factor, in extended precision by the QR of
    # the sorted columns
    order = np.argsort(-d)
    r = np.linalg.qr((B * d)[:, order])[1]
    ref = _graded_values(r)
    assert np.abs(S[0] / scale - ref).max() <= 1e-12 * ref[0]
    assert (np.abs(S[0] / scale - ref) <= 1e-11 * ref).all()
    assert np.abs(U[0].conj().T @ U[0] - np.eye(n)).max() <= 1e-12


def _graded_values(r):
    """Singular values of a triangular matrix with graded rows, by one-sided Jacobi on its adjoint."""
    w = r.conj().T.astype(np.clongdouble)
    n = w.shape[1]
    for _ in range(30):
        worst = 0
        for i in range(n - 1):
            for j in range(i + 1, n):
                a, b = (np.abs(w[:, i]) ** 2).sum(), (np.abs(w[:, j]) ** 2).sum()
                g = (w[:, i].conj() * w[:, j]).sum()
                rho = abs(g) / np.sqrt(a * b)
                if rho < 1e-17:
                    continue
                worst = max(worst, rho)
                z = (b - a) / (2 * abs(g))
                t = (1 if z >= 0 else -1) / (abs(z) + np.sqrt(1 + z * z))
                c = 1 / np.sqrt(1 + t * t)
                s = c * t * g / abs(g)
                w[:, i], w[:, j] = c * w[:, i] - np.conj(s) * w[:, j], s * w[:, i] + c * w[:, j]
        if worst < 1e-15:
            break
    return np.sort(np.sqrt((np.abs(w) ** 2).sum(0)).astype(float))[::-1]
