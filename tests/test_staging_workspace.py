"""Staging workspace of the tensor-core factorization by batch size: four
buffers of split panel tiles where a batch takes two steps at a time, eight from
10,000 tile products a step on."""

from __future__ import annotations

from types import SimpleNamespace

import numpy as np
import pytest
from scipy import sparse

from aospectrum_b200 import native
from test_native_cpu import _plan

T, NB = 128, 40
TILE = 4 * T * T * 2                       # one staged tile: four BF16 planes
STEP = (2 * (NB - 1) + 2) * TILE           # the longest step's tiles and two inverses


@pytest.fixture(scope="module")
def dense_plan():
    """All 40 x 40 tiles filled: one entry a tile."""
    at = np.arange(NB) * T
    rows, cols = (x.ravel() for x in np.meshgrid(at, at))
    a = (sparse.csr_matrix((np.ones(rows.size), (rows, cols)), shape=(NB * T, NB * T))
         + sparse.eye(NB * T)).tocsr()
    a.sort_indices()
    rc, handle, msg = _plan(a.indptr, a.indices, NB * T, T, 0)
    assert rc == 0, msg
    info = native.PlanInfo()
    native.library().aosb_plan_info(handle, native.C.byref(info))
    assert info.schur_tile_updates == sum(k * k for k in range(NB)) >= 500 * NB
    yield SimpleNamespace(handle=handle, info=info)
    native.library().aosb_plan_destroy(handle)


def _bytes(plan, pencils):
    return native.library().aosb_factor_workspace_bytes(plan.handle, pencils,
                                                        native.PRECISION_BF16X3)


def test_buffers_follow_the_batch(dense_plan):
    line = -(-10000 * NB // dense_plan.info.schur_tile_updates)
    assert line > 2
    for pencils in (1, 2, line - 1, line, line + 1, 64):
        buffers = 8 if pencils >= line else 4
        assert _bytes(dense_plan, pencils) == buffers * pencils * STEP + 256
    # the workspace of a batch serves any smaller one
    sizes = [_bytes(dense_plan, p) for p in range(1, 3 * line)]
    assert sizes == sorted(sizes)


def test_pencils_that_fit_the_memory(dense_plan, monkeypatch):
    """max_pencils is the largest batch whose own need fits the budget."""
    import torch

    from aospectrum_b200 import engine
    from aospectrum_b200.engine import BandEngine

    monkeypatch.setattr(engine, "_torch", lambda: torch)
    eng = BandEngine.__new__(BandEngine)
    eng.plan, eng.n, eng.device = dense_plan, NB * T, "cuda:0"
    eng.engine = SimpleNamespace(max_pencils=0, memory_fraction=0.5)
    line = -(-10000 * NB // dense_plan.info.schur_tile_updates)
    need = [0] + [eng.pencil_bytes(32, p) for p in range(1, 4 * line)]
    for free in [n + d for n in need[1:] for d in (-1, 0)]:
        monkeypatch.setattr(torch.cuda, "mem_get_info", lambda _, f=free: (2 * f, 2 * f))
        monkeypatch.setattr(torch.cuda, "memory_reserved", lambda _: 0)
        monkeypatch.setattr(torch.cuda, "memory_allocated", lambda _: 0)
        fits = max(1, max(p for p, n in enumerate(need) if n <= free))
        assert eng.max_pencils(32, 4 * line - 1) == fits
    eng.engine.max_pencils = 3
    assert eng.max_pencils(32) == 3 and eng.max_pencils(32, 2) == 2
