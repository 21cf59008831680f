"""The group's QR with one CTA per column, for instances of different sizes in one launch at the
edges of its rows per thread, and the blocked QR beyond them, against a dense QR sweep.

Tolerance: a chain of n Householder QRs and products is backward stable, its error n·√(χd)·u ≲ 1e-14
relative to the norm of the state; 1e-12.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d,bonds", [
    (2, [[2, 4, 2]]),
    (2, [[1, 2, 1], [2, 4, 8, 4, 2], [2, 1, 2]]),
    (16, [[8, 16], [9, 16], [16, 15], [1, 1], [7]]),
    (16, [[16, 17, 16], [3, 2]]),
    (16, [[16, 32, 16], [16, 31, 5], [16, 16]]),
    (16, [[16, 33, 16], [3, 2]]),
    (2, [[2, 4, 8, 16, 32, 64, 100, 64, 32, 16, 8, 4, 2], [2, 4, 8, 16, 31, 16, 8, 4, 2]]),
])
def test_group_qr_sweeps(d, bonds):
    from tenetgb.group import MPSGroup

    rng = np.random.default_rng(sum(map(sum, bonds)))
    data = []
    for b in bonds:
        b = [1] + b + [1]
        data.append([(rng.standard_normal((b[i], d, b[i + 1])) + 1j * rng.standard_normal((b[i], d, b[i + 1])))
                     / np.sqrt(2 * d * b[i]) for i in range(len(b) - 1)])
    g = MPSGroup.from_arrays(data)
    norms = g.canonize_compress_norm([1 << 20] * len(data))
    for k, sites in enumerate(data):
        e = np.ones((1, 1), complex)
        for a in sites:
            e = np.einsum("xy,xpk,ypl->kl", e, a.conj(), a, optimize=True)
        ref = np.sqrt(e[0, 0].real)
        assert abs(norms[k] - ref) <= 1e-12 * ref
        f = np.ones((1, 1), complex)  # <before|after>: the same state
        for a, q in zip(sites, g.sites(k)):
            f = np.einsum("xy,xpk,ypl->kl", f, a.conj(), q, optimize=True)
        assert abs(f[0, 0] - ref**2) <= 1e-12 * ref**2
        for q in g.sites(k)[:-1]:
            m = q.reshape(-1, q.shape[2])
            assert np.abs(m.conj().T @ m - np.eye(m.shape[1])).max() <= 1e-12
