"""Shifted real factorizations without their imaginary planes, at the edges of
the tile sizes (32, 64 and 128 wide tiles; ragged last tiles): inertia against
block elimination in float64 at shifts that lie in gaps of the spectrum, and
solves by their backward error.

Tolerances: pivoting stays inside the tiles, and among the few hundred to few
thousand eigenvalues (norm 3) of the diagonal Schur complements the smallest is
about 2^-10, by which entries may grow: 2^-24 * 2^10 * 2^5 = 2^-9 of backward
error (a product left out gives order one).  A shift counts as in a gap when the
count is the same 2e-3 to either side; at 6001 rows, where there is none, the
count may be off by the two eigenvalues nearest to the shift.
"""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _band_matrix(n, w, rng):
    """Random symmetric band of half width w, CSR."""
    from scipy import sparse

    diags = [rng.standard_normal(n - d) / np.sqrt(2.0 * w) for d in range(w + 1)]
    diags[0] = 4.0 * rng.random(n) - 2.0
    offsets = list(range(w + 1)) + [-d for d in range(1, w + 1)]
    return sparse.diags(diags + diags[1:], offsets, format="csr").astype(np.float32)


def _negatives(a, shift, w):
    """Eigenvalues of the band matrix below the shift, by block elimination."""
    n = a.shape[0]
    d = a.astype(np.float64).tocsr() - shift * _eye(n)
    count, prev = 0, None
    for k in range(0, n, w):
        e = min(k + w, n)
        block = d[k:e, k:e].toarray()
        if prev is not None:
            couple = d[k:e, k - w:k].toarray()
            block -= couple @ np.linalg.solve(prev, couple.T)
        count += int((np.linalg.eigvalsh(block) < 0).sum())
        prev = block
    return count


def _eye(n):
    from scipy import sparse

    return sparse.eye(n, format="csr")


@pytest.mark.parametrize("n,width", [(97, 40), (512, 70), (513, 150), (577, 200), (1024, 90),
                                     (6001, 300)])
def test_real_factor_counts_and_solves(n, width):
    from scipy import sparse

    from aospectrum_b200.gamma import GammaShiftFactor

    rng = np.random.default_rng(n)
    h = _band_matrix(n, width, rng)
    h.sort_indices()
    s = sparse.csr_matrix(((h.indices == np.repeat(np.arange(n), np.diff(h.indptr)))
                           .astype(np.float32), h.indices, h.indptr), shape=(n, n))
    shift, below = next((x, c) for x in np.float32(0.11) + 0.037 * np.arange(40, dtype=np.float32)
                        for c in [_negatives(h, float(x), width)]
                        if n > 2000 or c == _negatives(h, float(x) + 2e-3, width)
                        == _negatives(h, float(x) - 2e-3, width))
    rhs = rng.standard_normal((n, 3)).astype(np.float32)
    import torch

    with GammaShiftFactor(n, h.indptr, h.indices, torch.tensor(h.data, device="cuda"),
                          torch.tensor(s.data, device="cuda"), float(shift)) as f:
        assert abs(f.inertia.below - below) <= (2 if n > 2000 else 0)
        assert f.inertia.zero == 0 and f.inertia.above == n - f.inertia.below
        x = f.solve(rhs).double().cpu().numpy()
    m = h.astype(np.float64) - float(shift) * _eye(n)
    r = rhs - m @ x
    scale = 4.0 * np.linalg.norm(x) + np.linalg.norm(rhs)
    assert np.linalg.norm(r) <= 2.0 ** -9 * scale
