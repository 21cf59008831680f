"""The fine-grained complex GEMM (k_gemm_fine) at the edges of its tiles, K stages, K groups
and cluster ranks, against numpy in extended precision.

Tolerance: every output is a sum of 4k rounded products in some order, so
|ΔC| ≤ 2·(4k + 8)·u·(|A|·|B|) elementwise, with u the unit roundoff of the type.
"""

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    import tenetgb

    return tenetgb.Context(0)


def _gemm(ctx, A, B, opa, opb, alpha=1.0, beta=0.0, C0=None):
    """A: (batch, rows, cols) as stored; returns alpha op(A) op(B) + beta C0."""
    import tenetgb

    nb = A.shape[0]
    m, k = A.shape[1:] if opa == "N" else A.shape[:0:-1]
    n = B.shape[2] if opb == "N" else B.shape[1]
    flat = lambda X: np.concatenate([x.reshape(-1, order="F") for x in X])
    dA, dB = (tenetgb.DeviceTensor.from_numpy(ctx, flat(X), ["x"]) for X in (A, B))
    c0 = np.zeros((nb, m, n), A.dtype) if C0 is None else C0
    dC = tenetgb.DeviceTensor.from_numpy(ctx, flat(c0), ["x"])
    al, be = ((C.c_double * 2)(complex(x).real, complex(x).imag) for x in (alpha, beta))
    code = 3 if A.dtype == np.complex128 else 2
    ctx.check(ctx.lib.tn_gemm(ctx.h, code, 0, opa.encode(), opb.encode(), m, n, k, al, C.c_void_p(dA.ptr), A.shape[1],
                              A.shape[1] * A.shape[2], C.c_void_p(dB.ptr), B.shape[1], B.shape[1] * B.shape[2], be,
                              C.c_void_p(dC.ptr), m, m * n, nb))
    return np.stack([v.reshape((m, n), order="F") for v in dC.numpy().reshape(nb, m * n)])


def _op(X, op):
    return X if op == "N" else X.transpose(0, 2, 1) if op == "T" else X.conj().transpose(0, 2, 1)


def _gauss(rng, shape, dtype):
    return (rng.standard_normal(shape) + 1j * rng.standard_normal(shape)).astype(dtype)


@pytest.mark.parametrize("dtype", [np.complex128, np.complex64])
@pytest.mark.parametrize("m,n,k,batch", [
    (1, 1, 1, 1), (1, 16, 32, 1), (1, 17, 33, 2), (2, 31, 15, 1), (3, 40, 64, 1), (4, 16, 16, 3), (5, 9, 31, 1),
    (8, 8, 512, 1), (9, 7, 63, 1), (64, 128, 64, 1), (65, 33, 257, 2), (24, 24, 12, 1), (250, 510, 100, 1),
])
@pytest.mark.parametrize("opa,opb", [("N", "N"), ("C", "N"), ("N", "C"), ("T", "T")])
def test_fine_gemm_within_rounding(ctx, dtype, m, n, k, batch, opa, opb):
    rng = np.random.default_rng(m * 1000 + n * 10 + k)
    A = _gauss(rng, (batch, m, k) if opa == "N" else (batch, k, m), dtype)
    B = _gauss(rng, (batch, k, n) if opb == "N" else (batch, n, k), dtype)
    C0 = _gauss(rng, (batch, m, n), dtype)
    alpha, beta = 0.5 - 0.25j, -0.75
    got = _gemm(ctx, A, B, opa, opb, alpha, beta, C0)
    a, b = _op(A, opa), _op(B, opb)
    ref = alpha * np.matmul(a.astype(np.clongdouble), b.astype(np.clongdouble)) + beta * C0
    bound = abs(alpha) * np.matmul(np.abs(a).astype(float), np.abs(b).astype(float)) + abs(beta) * np.abs(C0)
    u = np.finfo(dtype).eps / 2
    assert (np.abs(got - ref) <= 2 * (4 * k + 8) * u * bound).all()


@pytest.mark.parametrize("dtype", [np.complex128, np.complex64])
@pytest.mark.parametrize("n,k", [(128, 64), (48, 300), (512, 256)])
def test_rows_do_not_depend_on_their_number(ctx, dtype, n, k):
    """A row's product is the same bits with 1, 2, 3, 8 or 40 rows (what a served query relies on)."""
    rng = np.random.default_rng(n + k)
    A, B = _gauss(rng, (1, 40, k), dtype), _gauss(rng, (1, k, n), dtype)
    full = _gemm(ctx, A, B, "N", "N")
    for m in (1, 2, 3, 8):
        np.testing.assert_array_equal(_gemm(ctx, A[:, :m], B, "N", "N"), full[:, :m])

