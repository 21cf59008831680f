"""The split-BF16 GEMM at the edges of its 128×64 tiles and 32-wide K stages, for every number of
digit planes, and its epilogue's forms (alpha ±1 or not, beta 0, 1 or not, sums over chunks of k).

Tolerances: integers below 2^11 whose digits fit the planes give exact products, so C must be equal
to the integer result (all sums are below 2^53 and alpha, beta, C are small dyadic numbers).  With S < 8
planes on Gaussian data the error is bounded by ~S·2^{1−7S} per product of row and column
maxima (dropped pairs and digit remainders): 4·S·2^{1−7S}·2k·max|a_i|·max|b_j|, plus FP64 rounding.
"""

import numpy as np
import pytest

from test_gpu_split_gemm import cgauss, ctx, run_gemm  # noqa: F401  (ctx is a fixture)

pytestmark = pytest.mark.gpu


def _ints(rng, shape, top):
    return (rng.integers(-top, top + 1, shape) + 1j * rng.integers(-top, top + 1, shape)).astype(complex)


@pytest.mark.parametrize("m,n,k,batch", [
    (128, 64, 32, 1), (64, 129, 33, 2), (65, 127, 47, 1), (129, 65, 255, 3), (256, 33, 257, 2), (63, 192, 300, 1),
    (97, 100, 64, 40), (512, 512, 40, 3), (1000, 41, 512, 1),
])
@pytest.mark.parametrize("alpha,beta", [(1, 0), (-1, 1), (1, 1), (0.5 - 2j, 0), (1, 1 - 1j)])
def test_tiles_and_epilogue_exact(ctx, m, n, k, batch, alpha, beta):  # noqa: F811
    rng = np.random.default_rng(m + 3 * n + 7 * k)
    A, B, C0 = _ints(rng, (batch, m, k), 1000), _ints(rng, (batch, k, n), 1000), _ints(rng, (batch, m, n), 9)
    A[:, m // 2] = 0
    B[:, :, n // 3] = 0
    got, _ = run_gemm(ctx, A, B, C0, "N", "N", complex(alpha), complex(beta))
    assert np.array_equal(got, alpha * (A @ B) + beta * C0)


@pytest.mark.parametrize("n,k,batch", [(96, 32, 2), (128, 300, 1), (129, 64, 3), (191, 33, 1), (320, 600, 2), (512, 40, 1)])
@pytest.mark.parametrize("alpha,beta", [(1, 0), (-1, 0), (2, 0), (1, 1), (1 + 1j, 0)])
def test_gram_products_exact(ctx, n, k, batch, alpha, beta):  # noqa: F811
    """AᴴA of one operand (its planes cut once, with a real alpha and beta = 0 the tiles above the
    diagonal only) against the integer result; for Gaussian data it is Hermitian
    to the last bit off the diagonal blocks."""
    import ctypes as C

    import tenetgb

    rng = np.random.default_rng(n + k)
    al, be = (C.c_double * 2)(complex(alpha).real, complex(alpha).imag), (C.c_double * 2)(beta, 0)
    for exact in (True, False):
        A = _ints(rng, (batch, k, n), 1000) if exact else cgauss(rng, (batch, k, n))
        C0 = _ints(rng, (batch, n, n), 9)
        dA = tenetgb.DeviceTensor.from_numpy(ctx, np.transpose(A, (1, 2, 0)))
        dC = tenetgb.DeviceTensor.from_numpy(ctx, np.transpose(C0, (1, 2, 0)))
        ctx.check(ctx.lib.tn_gemm(ctx.h, 3, 3, b"C", b"N", n, n, k, al, C.c_void_p(dA.ptr), k, k * n, C.c_void_p(dA.ptr), k,
                                  k * n, be, C.c_void_p(dC.ptr), n, n * n, batch))
        got = np.transpose(dC.numpy(), (2, 0, 1))
        ref = alpha * (A.conj().transpose(0, 2, 1) @ A) + beta * C0
        if exact:
            assert np.array_equal(got, ref)
        else:
            assert np.linalg.norm(got - ref) <= 1e-13 * np.linalg.norm(ref)
            if beta == 0 and complex(alpha).imag == 0:  # (64 × 64 blocks on the diagonal are computed in full)
                h = got.conj().transpose(0, 2, 1)
                off = np.arange(n)[:, None] // 64 != np.arange(n)[None] // 64
                assert np.array_equal(got[:, off], h[:, off])


@pytest.mark.parametrize("ea,eb", [(-400, 300), (-500, -480), (500, 450), (-600, 0)])
def test_scales_are_exact(ctx, ea, eb):  # noqa: F811
    """Rows and columns scaled by powers of two: the products scale exactly, also where the sum of
    exponents leaves the range that the epilogue adds to (2^-980 and below)."""
    rng = np.random.default_rng(3)
    A, B = _ints(rng, (1, 130, 40), 1000), _ints(rng, (1, 40, 70), 1000)
    got, _ = run_gemm(ctx, A * 2.0**ea, B * 2.0**eb, np.zeros((1, 130, 70), complex), "N", "N", 1 + 0j, 0j)
    assert np.array_equal(got, np.ldexp(1.0, ea + eb) * (A @ B))


@pytest.mark.parametrize("S", [2, 3, 4, 5, 6, 7, 8])
def test_every_plane_count(ctx, S):  # noqa: F811
    rng = np.random.default_rng(S)
    m, n, k = 130, 100, 90
    A, B = cgauss(rng, (2, m, k)), cgauss(rng, (2, k, n))
    ctx.check(ctx.lib.tn_set_split_slices(ctx.h, S))
    try:
        got, _ = run_gemm(ctx, A, B, np.zeros((2, m, n), complex), "N", "N", 1 + 0j, 0j)
    finally:
        ctx.check(ctx.lib.tn_set_split_slices(ctx.h, 8))
    row = np.maximum(np.abs(A.real), np.abs(A.imag)).max(2)[:, :, None]
    col = np.maximum(np.abs(B.real), np.abs(B.imag)).max(1)[:, None, :]
    bound = (4 * S * 2.0 ** (1 - 7 * S) * 2 * k + 1e-15 * k) * row * col
    assert (np.abs(got - A @ B) <= bound).all()
