"""Factorizations by four tile steps at a time (K up to 512 per target).

Tile counts of every remainder modulo four, a ragged last tile, and a pattern
whose first tiles couple to different parts of the rest, so that items lack some
of their steps.  Each pencil's unrefined solve is held to a backward error of
2^-13: the split-BF16 products are good to 2^-16 each and the shifts lie outside
the spectrum (no growth).  One 128-deep product left out or added twice shows: a
coupled tile acts with about 0.2 on a vector, so the product with about
0.2 * 0.2 / 2 on one of forty tiles, 2^-10 of the scale."""

from __future__ import annotations

from types import SimpleNamespace

import numpy as np
import pytest

from test_gpu_parity import _factor_solve
from test_native_cpu import _plan

pytestmark = pytest.mark.gpu

T = 128


def _mask(core, leaves):
    """Tile pattern: `leaves` leading tiles, tile t coupled to every third core
    tile, and a dense core."""
    nb = core + leaves
    m = np.eye(nb, dtype=bool)
    m[leaves:, leaves:] = True
    for t in range(leaves):
        m[t, leaves + t % 3::3] = m[leaves + t % 3::3, t] = True
    return m


@pytest.mark.parametrize("core,leaves,pencils", [(40, 0, 20), (41, 0, 20), (42, 0, 19), (43, 0, 18),
                                                 (46, 6, 17)])
def test_four_step_factor_solves(core, leaves, pencils):
    import torch
    from scipy import sparse

    from aospectrum_b200 import native

    rng = np.random.default_rng(core)
    mask = _mask(core, leaves)
    nb = core + leaves
    n = nb * T - 37
    ti, tj = np.nonzero(mask)
    per = 3  # entries per row of a coupled tile
    rows = (ti[:, None, None] * T + np.arange(T)[None, :, None] + np.zeros((1, 1, per), int)).ravel()
    cols = (tj[:, None, None] * T + rng.integers(0, T, (ti.size, T, per))).ravel()
    keep = (rows < n) & (cols < n)
    a = sparse.csr_matrix((np.ones(int(keep.sum())), (rows[keep], cols[keep])), shape=(n, n))
    a = (a + a.T + sparse.eye(n)).tocsr()
    a.sort_indices()
    values = (rng.standard_normal(a.nnz) + 1j * rng.standard_normal(a.nnz)) / np.sqrt(a.nnz / n)
    h = sparse.csr_matrix((values.astype(np.complex64), a.indices, a.indptr), shape=(n, n))
    s = sparse.csr_matrix(((a.indices == np.repeat(np.arange(n), np.diff(a.indptr)))
                           .astype(np.complex64), a.indices, a.indptr), shape=(n, n))
    offsets = np.append(np.arange(nb) * T, n).astype(np.int64)
    rc, handle, msg = _plan(a.indptr, a.indices, n, T, 0, offsets)
    assert rc == 0, msg
    lib = native.library()
    info = native.PlanInfo()
    try:
        native.call("aosb_plan_upload", handle)
        lib.aosb_plan_info(handle, native.C.byref(info))
        assert info.n_tiles == nb
        assert info.schur_tile_updates >= 500 * nb  # the plan takes four steps
        assert info.schur_tile_updates * pencils >= 10000 * nb
        plan = SimpleNamespace(handle=handle, info=SimpleNamespace(n_pad=info.n_pad))
        dev = SimpleNamespace(n=n)
        shifts = 2.0 + 0.1j * np.arange(1, pencils + 1)
        rhs = rng.standard_normal((n, 2)) + 1j * rng.standard_normal((n, 2))
        x = _factor_solve(dev, plan, torch.tensor(h.data[None], device="cuda"),
                          torch.tensor(s.data[None], device="cuda"), shifts, rhs, torch,
                          precision=native.PRECISION_BF16X3)
        for p, z in enumerate(shifts):
            m = (h - z * s).astype(np.complex128)
            r = rhs - m @ x[p]
            scale = abs(z) * np.linalg.norm(x[p]) + np.linalg.norm(rhs)
            assert np.linalg.norm(r) <= 2.0 ** -13 * scale, p
    finally:
        lib.aosb_plan_destroy(handle)
