"""ComplexF64 products on both sides of where the fine-grained GEMM takes less time than the register tiles:
short contractions, many tiles, batches.

Tolerance: 4k rounded products per part in some order, |Δ| ≤ 2·(4k + 8)·u·(|A|·|B|) with u = 2⁻⁵³.
"""

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k,batch", [
    (64, 1000, 1, 10), (64, 1000, 9, 10), (2000, 64, 4, 1), (2000, 64, 64, 1), (16, 64, 8, 200), (16, 64, 65, 200),
    (64, 128, 200, 40), (256, 256, 512, 1), (8, 300, 33, 50), (5, 128, 64, 60), (4, 40, 3, 90), (2, 300, 4, 1), (1, 1000, 200, 3),
    (20, 20, 1, 1), (300, 7, 2, 5), (33, 1, 31, 200),
])
def test_products(m, n, k, batch):
    import tenetgb

    ctx = tenetgb.default_context()
    rng = np.random.default_rng(m + n + k)
    g = lambda *s: rng.standard_normal(s) + 1j * rng.standard_normal(s)
    A, B = g(m, k, batch), g(k, n, batch)
    dA, dB = tenetgb.DeviceTensor.from_numpy(ctx, A), tenetgb.DeviceTensor.from_numpy(ctx, B)
    dC = tenetgb.DeviceTensor.from_numpy(ctx, np.full((m, n, batch), np.nan + 0j))
    one, zero = (C.c_double * 2)(1, 0), (C.c_double * 2)(0, 0)
    ctx.check(ctx.lib.tn_gemm(ctx.h, 3, 0, b"N", b"N", m, n, k, one, C.c_void_p(dA.ptr), m, m * k, C.c_void_p(dB.ptr), k, k * n,
                              zero, C.c_void_p(dC.ptr), m, m * n, batch))
    got = np.moveaxis(dC.numpy(), -1, 0)
    A, B = np.moveaxis(A, -1, 0), np.moveaxis(B, -1, 0)
    assert (np.abs(got - A @ B) <= 2 * (4 * k + 8) * 2.0**-53 * (np.abs(A) @ np.abs(B))).all()
