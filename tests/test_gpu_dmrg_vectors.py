"""The Lanczos orthogonalisation on one CTA up to a cluster of 16 per instance, for each of its
basis sizes, and the fibre products, against the oracle's energy after every half sweep.

Tolerance: an untruncated local ground-state energy is an eigenvalue of a Hermitian matrix of
norm ≤ 5L; Lanczos on vectors orthogonal to a few u resolves it to a small multiple of
‖H‖·u ≈ 1e-14, and a restart carries the error of the vector only quadratically into it.  1e-9
leaves room for steps that stop unconverged, where the same Krylov space gives the same Ritz value
up to ‖H‖·u times the condition of the basis.
"""

import numpy as np
import pytest

from oracle import tenet_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,krylovdim,method", [
    (4, 3, 2), (8, 3, 2), (10, 3, 1), (12, 3, 2), (10, 6, 2), (12, 10, 2), (12, 10, 1),
])
def test_lanczos_vectors_match_oracle(n, krylovdim, method):
    import tenetgb

    rng = np.random.default_rng(100 + n)
    bonds = [min(2**i, 2**(n - i)) for i in range(n + 1)]
    sites = [(rng.standard_normal((bonds[i], 2, bonds[i + 1])) + 1j * rng.standard_normal((bonds[i], 2, bonds[i + 1])))
             / np.sqrt(4 * bonds[i]) for i in range(n)]
    H, ref = O.heisenberg_mpo(n, 1.0, 0.6, 0.1), []
    opts = dict(maxdim=2**(n // 2), krylovdim=krylovdim, maxiter=2)
    psi = tenetgb.MPS([s.copy() for s in sites])
    _, _, hist = tenetgb.dmrg_(psi, H, 1, method=tenetgb.Dmrg1 if method == 1 else tenetgb.Dmrg2, history=True, **opts)
    O.dmrg(O.OMPS([s.copy() for s in sites]), H, 1, method=f"dmrg{method}", history=ref, **opts)
    assert len(hist) == len(ref) and np.allclose(hist, ref, rtol=0, atol=1e-9)
