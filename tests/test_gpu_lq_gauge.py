"""Right-to-left gauge moves: sites factored in place as L·Qᴴ where the column kernel takes them (square,
wide, batched, up to 512 rows of the adjoint), and by way of the adjoint otherwise, against the
state they started from.

Tolerance: n Householder factorisations and products, n·√(χd)·u ≲ 1e-14 relative; 1e-12.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d,bonds,batch", [
    (2, [2, 4, 2], 1), (2, [2, 4, 8, 16, 8, 4, 2], 3), (3, [3, 7, 20, 9, 3], 2), (16, [16, 16], 1), (16, [3, 31, 32], 2),
    (16, [16, 64, 32], 1), (16, [40, 33, 33], 1), (2, [2, 9, 30, 8], 2),
])
def test_move_to_the_left(d, bonds, batch):
    import tenetgb

    rng = np.random.default_rng(sum(bonds) + d)
    b = [1] + bonds + [1]
    insts = [[(rng.standard_normal((b[i], d, b[i + 1])) + 1j * rng.standard_normal((b[i], d, b[i + 1])))
              / np.sqrt(2 * d * b[i]) for i in range(len(b) - 1)] for _ in range(batch)]
    psi = tenetgb.MPS.batched([[s.copy() for s in x] for x in insts], max_bond=max(b))
    psi.canonize_(tenetgb.MixedCanonical(1))
    for k, sites in enumerate(insts):
        got = psi.sites(k)
        e = f = np.ones((1, 1), complex)
        for a, q in zip(sites, got):
            e = np.einsum("xy,xpk,ypl->kl", e, a.conj(), a, optimize=True)
            f = np.einsum("xy,xpk,ypl->kl", f, a.conj(), q, optimize=True)
        assert abs(f[0, 0] - e[0, 0]) <= 1e-12 * abs(e[0, 0])
        for q in got[1:]:
            w = q.reshape(q.shape[0], -1)
            assert np.abs(w @ w.conj().T - np.eye(len(w))).max() <= 1e-12
