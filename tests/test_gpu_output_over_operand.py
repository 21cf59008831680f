"""ComplexF32 products whose output lies over an operand that the general path copies first: they are
not read in place.  Against the same product in double precision.

Tolerance: 4k rounded products per part, |Δ| ≤ 2·(4k + 8)·u·(|A|·|B|) with u = 2⁻²⁴ (16× that for
3×TF32).
"""

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

REL = {"native": lambda k: 2 * (4 * k + 8) * 2.0**-24, "mixed": lambda k: 32 * (4 * k + 8) * 2.0**-24}


def _data(rng, shape):
    return (rng.standard_normal(shape) + 1j * rng.standard_normal(shape)).astype(np.complex64)


@pytest.mark.parametrize("la,da,lb,db,con", [
    ("abxcy", (40, 30, 5, 33, 7), "xyu", (5, 7, 33), "xy"),
    ("ayxb", (129, 8, 8, 310), "xyu", (8, 8, 64), "xy"),
])
@pytest.mark.parametrize("precision", ["native", "mixed"])
def test_contraction_into_its_operand(la, da, lb, db, con, precision):
    import tenetgb
    from tenetgb import core

    ctx = tenetgb.default_context()
    rng = np.random.default_rng(sum(da) + sum(db))
    A, B = _data(rng, da), _data(rng, db)
    tA, tB = (tenetgb.DeviceTensor.from_numpy(ctx, x, list(l)) for x, l in ((A, la), (B, lb)))
    out = [c for c in la if c not in con] + [c for c in lb if c not in con]
    shape = [dict(zip(la + lb, da + db))[c] for c in out]
    tC = tenetgb.DeviceTensor(ctx, shape, np.complex64, out, ptr=tA.ptr)
    assert tC.nbytes <= tA.nbytes
    ids = core._modes(tA.inds, tB.inds, out)
    a, b, c = core._desc(tA, ids), core._desc(tB, ids), core._desc(tC, ids)
    ctx.check(ctx.lib.tn_contract(ctx.h, tA.code, core.precision_code(precision), C.byref(a), C.byref(b), C.byref(c)))
    spec = f"{la},{lb}->{''.join(out)}"
    ref = np.einsum(spec, A.astype(complex), B.astype(complex), optimize=True)
    mag = np.einsum(spec, np.abs(A).astype(float), np.abs(B).astype(float), optimize=True)
    k = int(np.prod([da[la.index(x)] for x in con]))
    assert (np.abs(tC.numpy() - ref) <= REL[precision](k) * mag).all()


@pytest.mark.parametrize("batch", [1, 2])
@pytest.mark.parametrize("over", ["A", "B"])
def test_tall_product_into_its_operand(over, batch):
    import tenetgb
    from tenetgb import core

    ctx = tenetgb.default_context()
    m, k = 20000, 64
    n = k
    rng = np.random.default_rng(8 + batch)
    A, B = _data(rng, (m, k, batch)), _data(rng, (k, n, batch))
    dA = tenetgb.DeviceTensor.from_numpy(ctx, A)
    pad = np.zeros((m * n, batch), np.complex64)  # B at the head of a buffer that has room for C
    pad[: k * n] = B.reshape((k * n, batch), order="F")
    dB = tenetgb.DeviceTensor.from_numpy(ctx, pad)
    dC = dA if over == "A" else dB
    one, zero = (C.c_double * 2)(1, 0), (C.c_double * 2)(0, 0)
    ctx.check(ctx.lib.tn_gemm(ctx.h, 2, core.precision_code("mixed"), b"N", b"N", m, n, k, one, C.c_void_p(dA.ptr), m, m * k,
                              C.c_void_p(dB.ptr), k, m * n, zero, C.c_void_p(dC.ptr), m, m * n, batch))
    got = dC.numpy().reshape(-1, order="F").reshape((m, n, batch), order="F")
    for b in range(batch):
        ref = A[..., b].astype(complex) @ B[..., b].astype(complex)
        mag = np.abs(A[..., b]).astype(float) @ np.abs(B[..., b]).astype(float)
        assert (np.abs(got[..., b] - ref) <= REL["mixed"](k) * mag).all()
