"""ComplexF32 contractions whose operands are read in place through strided views, at the edges of
the tiles (128 rows, 64 columns, stages of K) and over the leg orders the rule accepts, against
the same contraction in double precision.

Tolerance: 4k rounded products per part in index order, |Δ| ≤ 2·(4k + 8)·u·(|A|·|B|) with
u = 2⁻²⁴; the tensor-pipe modes add their documented 16× (3×TF32) and one TF32 rounding of each
operand (2⁻¹¹ each) for tf32.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CASES = [
    # (a labels, a dims, b labels, b dims, contracted)
    ("abxcy", (40, 30, 5, 33, 7), "xyuv", (5, 7, 6, 9), "xy"),      # legs inside and at the end
    ("xabcy", (6, 50, 31, 20, 5), "xyuv", (6, 5, 8, 8), "xy"),      # K first: rows not contiguous
    ("abcxy", (37, 41, 27, 3, 4), "xyu", (3, 4, 65), "xy"),         # plain matrix
    ("axbyc", (64, 9, 32, 2, 20), "xyuv", (9, 2, 5, 7), "xy"),      # three runs of rows: permuted copy
    ("abxcy", (40, 30, 5, 33, 7), "uyvx", (6, 7, 9, 5), "xy"),      # b's legs interleaved
    ("axb", (300, 130, 150), "xu", (130, 33), "x"),
    ("axb", (200, 300, 200), "xu", (300, 56), "x"),                 # k over more than one table of offsets
    ("abx", (200, 210, 1), "xu", (1, 40), "x"),                     # k = 1
    ("xab", (4, 128, 304), "ux", (32, 4), "x"),                     # exactly the smallest columns
    ("ayxb", (129, 8, 8, 310), "xyu", (8, 8, 64), "xy"),            # K order differs between a and b
]


@pytest.mark.parametrize("la,da,lb,db,con", CASES)
@pytest.mark.parametrize("precision", ["native", "mixed", "tf32"])
def test_contraction_through_views(la, da, lb, db, con, precision):
    import tenetgb

    ctx = tenetgb.default_context()
    rng = np.random.default_rng(sum(da) * 7 + sum(db))
    A, B = ((rng.standard_normal(d) + 1j * rng.standard_normal(d)).astype(np.complex64) for d in (da, db))
    tA, tB = tenetgb.DeviceTensor.from_numpy(ctx, A, list(la)), tenetgb.DeviceTensor.from_numpy(ctx, B, list(lb))
    out = [c for c in la if c not in con] + [c for c in lb if c not in con]
    got = tenetgb.binary_einsum(tA, tB, dims=list(con), precision=precision)
    assert got.inds == out
    spec = f"{la},{lb}->{''.join(out)}"
    ref = np.einsum(spec, A.astype(complex), B.astype(complex), optimize=True)
    k = int(np.prod([da[la.index(c)] for c in con]))
    mag = np.einsum(spec, np.abs(A).astype(float), np.abs(B).astype(float), optimize=True)
    u = 2.0**-24
    rel = {"native": 2 * (4 * k + 8) * u, "mixed": 16 * 2 * (4 * k + 8) * u, "tf32": 2.0**-9 + 2 * (4 * k + 8) * u}[precision]
    assert (np.abs(got.numpy() - ref) <= rel * mag).all()


@pytest.mark.parametrize("m,n,k", [(20000, 64, 64), (19457, 49, 49), (30000, 100, 33), (9800, 130, 40), (128 * 152, 64, 32)])
@pytest.mark.parametrize("precision", ["mixed", "tf32"])
def test_tall_tensor_pipe_products(m, n, k, precision):
    """The tall TF32 kernel at ragged rows, columns and contraction lengths, with alpha and beta."""
    import ctypes as C

    import tenetgb

    ctx = tenetgb.default_context()
    rng = np.random.default_rng(m + n + k)
    g = lambda *s: (rng.standard_normal(s) + 1j * rng.standard_normal(s)).astype(np.complex64)
    A, B, C0 = g(m, k), g(n, k), g(m, n)
    dA, dB, dC = (tenetgb.DeviceTensor.from_numpy(ctx, x) for x in (A, B, C0))
    al, be = (C.c_double * 2)(0.5, 0), (C.c_double * 2)(-0.25, 0)
    code = tenetgb.core.precision_code(precision)
    ctx.check(ctx.lib.tn_gemm(ctx.h, 2, code, b"N", b"C", m, n, k, al, C.c_void_p(dA.ptr), m, 0, C.c_void_p(dB.ptr), n, 0, be,
                              C.c_void_p(dC.ptr), m, 0, 1))
    ref = 0.5 * A.astype(complex) @ B.astype(complex).conj().T - 0.25 * C0
    mag = 0.5 * np.abs(A).astype(float) @ np.abs(B).astype(float).T + 0.25 * np.abs(C0)
    u = 2.0**-24
    rel = {"mixed": 32 * (4 * k + 8) * u, "tf32": 2.0**-9 + 2 * (4 * k + 8) * u}[precision]
    assert (np.abs(dC.numpy() - ref) <= rel * mag).all()
