"""The SVD's scratch: a HBM budget that leaves room for the matrices and the general kernels is enough, and
a sweep of SVDs uses one reservation.

Tolerance: the general kernels rotate down to couplings of 4·√m·ε (2e-14 at m = 512), which over n columns
leaves √n·4·√m·ε = 4.5e-13: 1e-12, as in the other tests of these kernels.
"""

import ctypes as C

import numpy as np
import pytest

from oracle import tenet_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,precision,budget", [
    (200, 200, "native", 4_900_000),    # matrices 1.9 MB, W and V 1.3 MB with a margin 2.7
    (300, 100, "native", 3_400_000),    # 1.1 and 0.65: 1.9
    (512, 512, "native", 25_000_000),   # 12.6 and 8.4: 11.6
    (256, 256, "mixed", 24_000_000),    # 3.1 and 7.9: 11, digit planes 6.4
])
def test_svd_within_a_budget(m, n, precision, budget):
    import tenetgb

    ctx = tenetgb.Context(0)
    ctx.set_hbm_budget(budget)
    rng = np.random.default_rng(m + n)
    A = rng.standard_normal((m, n)) + 1j * rng.standard_normal((m, n))
    dA = tenetgb.DeviceTensor.from_numpy(ctx, A)
    dU, dV = tenetgb.DeviceTensor(ctx, (m, n), complex), tenetgb.DeviceTensor(ctx, (n, n), complex)
    dS = tenetgb.DeviceTensor(ctx, (n,), float)
    for _ in range(2):  # (the second call keeps the reservation of the first)
        ctx.check(ctx.lib.tn_svd_thin(ctx.h, 3, tenetgb.core.precision_code(precision), m, n, C.c_void_p(dA.ptr), m, m * n,
                                      C.c_void_p(dU.ptr), m * n, C.c_void_p(dS.ptr), n, C.c_void_p(dV.ptr), n * n, 1))
        assert ctx.hbm_in_use() <= budget
    U, S, V = dU.numpy(), dS.numpy(), dV.numpy()
    tol = 1e-12
    assert np.linalg.norm((U * S) @ V - A) <= tol * np.linalg.norm(A)
    assert np.abs(U.conj().T @ U - np.eye(n)).max() <= tol and np.abs(V @ V.conj().T - np.eye(n)).max() <= tol


@pytest.mark.parametrize("L", [20, 40])
def test_zip_up_over_many_sites(L):
    """The largest block has 1024 rows, the sites' own 64."""
    import tenetgb

    rng = np.random.default_rng(L)
    bonds = [min(2**i, 2 ** (L - i), 32) for i in range(L + 1)]
    ws = [1] + [8] * (L - 1) + [1]
    g = lambda *s: rng.standard_normal(s) + 1j * rng.standard_normal(s)
    sites = [g(a, 2, b) / np.sqrt(4 * a) for a, b in zip(bonds, bonds[1:])]
    mpo = [g(a, 2, 2, b) / np.sqrt(4 * a) for a, b in zip(ws, ws[1:])]
    psi = tenetgb.MPS([s.copy() for s in sites], ctx=tenetgb.Context(0))
    ref = O.OMPS([s.copy() for s in sites])
    tenetgb.evolve_mpo_(psi, mpo, algorithm="zipup", maxdim=32)
    O.evolve_mpo_zipup(ref, mpo, maxdim=32)
    assert psi.bondsizes() == ref.bondsizes()
    both = tenetgb.MPS([s.copy() for s in ref.sites], ctx=psi.ctx)
    n2, r2, o = abs(psi.overlap(psi)), abs(both.overlap(both)), psi.overlap(both)
    assert abs(n2 / r2 - 1) <= 1e-11 and abs(abs(o) / np.sqrt(n2 * r2) - 1) <= 1e-11
