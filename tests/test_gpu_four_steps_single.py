"""A plan with more than 10,000 tile products a step takes four steps at a time
for one pencil too, and keeps no two-step lists on the device; the two-CTA form
still runs two steps from its own lists.  Both are held to the backward error of
2^-13 that split-BF16 products (2^-16 each, no growth: the shift lies outside the
spectrum) leave room for; a product left out shows as about 2^-10."""

from __future__ import annotations

from types import SimpleNamespace

import numpy as np
import pytest

from test_gpu_parity import _factor_solve
from test_native_cpu import _plan

pytestmark = pytest.mark.gpu

T, NB = 128, 175


def test_one_pencil_of_a_large_dense_plan():
    import torch
    from scipy import sparse

    from aospectrum_b200 import native

    rng = np.random.default_rng(2)
    n = NB * T - 51
    rows = np.repeat(np.arange(n), NB)
    cols = rng.integers(0, T, rows.size) + T * np.tile(np.arange(NB), n)
    keep = cols < n
    a = sparse.csr_matrix((np.ones(int(keep.sum())), (rows[keep], cols[keep])), shape=(n, n))
    a = (a + a.T + sparse.eye(n)).tocsr()
    a.sort_indices()
    values = (rng.standard_normal(a.nnz) + 1j * rng.standard_normal(a.nnz)) / np.sqrt(a.nnz / n)
    h = sparse.csr_matrix((values.astype(np.complex64), a.indices, a.indptr), shape=(n, n))
    s = sparse.csr_matrix(((a.indices == np.repeat(np.arange(n), np.diff(a.indptr)))
                           .astype(np.complex64), a.indices, a.indptr), shape=(n, n))
    rc, handle, msg = _plan(a.indptr, a.indices, n, T, 0)
    assert rc == 0, msg
    lib = native.library()
    info = native.PlanInfo()
    pairs = lib.aosb_factor_set_schur_pairs(0)
    try:
        native.call("aosb_plan_upload", handle)
        lib.aosb_plan_info(handle, native.C.byref(info))
        assert info.n_tiles == NB and info.schur_tile_updates >= 10000 * NB
        plan = SimpleNamespace(handle=handle, info=SimpleNamespace(n_pad=info.n_pad))
        hv, sv = (torch.tensor(m.data[None], device="cuda") for m in (h, s))
        rhs = rng.standard_normal((n, 2)) + 1j * rng.standard_normal((n, 2))
        z = 2.0 + 0.1j
        m = (h - z * s).astype(np.complex128)
        for on in (0, 1):
            lib.aosb_factor_set_schur_pairs(on)
            x = _factor_solve(SimpleNamespace(n=n), plan, hv, sv, [z], rhs, torch,
                              precision=native.PRECISION_BF16X3)
            r = rhs - m @ x[0]
            scale = abs(z) * np.linalg.norm(x[0]) + np.linalg.norm(rhs)
            assert np.linalg.norm(r) <= 2.0 ** -13 * scale, on
    finally:
        lib.aosb_factor_set_schur_pairs(pairs)
        lib.aosb_plan_destroy(handle)
