"""Diagonal-tile LU: inverse triangles and pivots of dense one-tile pencils.

A plan whose matrix fits one tile holds, after a plain factorization, exactly
what the diagonal kernel made of it: inv(L) strictly below, inv(U) on and
above the diagonal, and the row order of P A = L U.  Standard rounding bounds
of an LU with explicit triangle inverses (Higham, Accuracy and Stability of
Numerical Algorithms, ch. 9 and 14) give
|| inv(U) inv(L) P A - I || <= c T u || inv(U) || || inv(L) || || A ||
in FP32 (u = 2^-24); c = 8 covers the complex products.  The multipliers obey
|re| + |im| pivoting: |l| <= sqrt(2).
"""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _one_tile(mats, tile):
    import torch

    from aospectrum_b200 import native
    from aospectrum_b200.engine import SymbolicPlan

    dev = torch.device("cuda", 0)
    P, n, _ = mats.shape
    indptr = np.arange(n + 1, dtype=np.int64) * n
    indices = np.tile(np.arange(n, dtype=np.int32), n)
    plan = SymbolicPlan(n, indptr, indices, tile=tile, ordering="natural", device=dev)
    try:
        assert plan.info.n_tiles == 1
        perm = plan.perm()
        h = torch.from_numpy(mats.reshape(P, n * n).astype(np.complex64)).to(dev)
        s = torch.zeros_like(h)
        pk = torch.arange(P, dtype=torch.int32, device=dev)
        z = torch.zeros(P, dtype=torch.complex128, device=dev)
        factor = torch.empty((P, 2, tile, tile), dtype=torch.float32, device=dev)
        piv = torch.empty((P, tile), dtype=torch.int32, device=dev)
        status = torch.zeros(P, dtype=torch.int32, device=dev)
        fa = native.FactorArgs(native.ABI_VERSION, native.C.sizeof(native.FactorArgs), P,
                               native.PRECISION_PLAIN, h.data_ptr(), s.data_ptr(), pk.data_ptr(),
                               z.data_ptr(), factor.data_ptr(), piv.data_ptr(),
                               status.data_ptr(), None, torch.cuda.current_stream().cuda_stream)
        native.call("aosb_factor", plan.handle, native.C.byref(fa))
        torch.cuda.synchronize()
        f = factor.cpu().numpy().astype(np.float64)
        padded = np.zeros((P, tile, tile), dtype=np.complex128)
        for i in range(tile):
            if perm[i] < 0:
                padded[:, i, i] = 1.0
                continue
            for j in range(tile):
                if perm[j] >= 0:
                    padded[:, i, j] = mats[:, perm[i], perm[j]].astype(np.complex64)
        return f[:, 0] + 1j * f[:, 1], piv.cpu().numpy(), status.cpu().numpy(), padded
    finally:
        plan.close()


def _matrices(n, seed):
    rng = np.random.default_rng(seed)
    a = rng.standard_normal((4, n, n)) + 1j * rng.standard_normal((4, n, n))
    a[1] = np.diag(rng.uniform(1, 2, n))[rng.permutation(n)]   # every row moves
    a[2] = np.where(rng.random((n, n)) < 0.5, 1.0, -1.0)       # ties in every column
    a[2] += np.diag(rng.uniform(0.0, 1.0, n))
    a[3] = a[3] + a[3].conj().T - 0.3j * np.eye(n)             # a shifted Hermitian pencil
    return a


@pytest.mark.parametrize("tile,n", [(32, 32), (32, 9), (64, 64), (64, 61), (128, 128), (128, 100),
                                    (128, 65)])
def test_one_tile_inverse_triangles(tile, n):
    f, piv, status, a = _one_tile(_matrices(n, tile + n), tile)
    assert np.all(status == 0)
    eye = np.eye(tile)
    for p in range(a.shape[0]):
        assert np.array_equal(np.sort(piv[p]), np.arange(tile))
        linv, uinv = np.tril(f[p], -1) + eye, np.triu(f[p])
        err = np.linalg.norm(uinv @ (linv @ a[p][piv[p]]) - eye)
        bound = 8 * tile * 2.0 ** -24 * np.linalg.norm(uinv) * np.linalg.norm(linv) \
            * np.linalg.norm(a[p])
        assert err <= bound, (p, err, bound)
        multipliers = np.abs(np.linalg.inv(linv))
        assert multipliers.max() <= np.sqrt(2.0) * (1 + 1e-3)


def test_singular_and_nonfinite_tiles_are_reported():
    a = _matrices(64, 5)
    a[0][:, 17] = 0.0
    a[1][3, 4] = np.inf
    _, _, status, _ = _one_tile(a, 64)
    assert status[0] == 50 and status[1] == 51 and status[2] == 0 and status[3] == 0
