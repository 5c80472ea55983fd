"""Cluster form of the tensor-core solves (whole sweeps in one launch).

Column counts at the edges of the 8-column blocks and 32-column strips, odd
ones (8-byte X accesses) and pencil counts that select different cluster sizes,
both directions, against the FP32 SIMT sweeps on the same factors: the updates
drop lo x lo and round lo, 2^-16 relative per product, which the pencil's
condition amplifies to the 1e-3 that unrefined split-BF16 solves are held to.
A solve adds each element of X once per step, so repeating it must give the same
bits."""

from __future__ import annotations

import numpy as np
import pytest

import bundles
from test_gpu_parity import _factor_solve, _pencil_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("adjoint", [0, 1])
@pytest.mark.parametrize("pencils,columns", [(1, 1), (1, 8), (2, 9), (8, 16), (12, 17), (20, 24),
                                             (25, 25), (30, 32), (13, 33), (40, 31), (60, 6)])
def test_cluster_solves_match_simt_sweeps(pencils, columns, adjoint):
    import torch

    from aospectrum_b200 import native

    dev, plan, h, s = _pencil_case(bundles.small2d(), bundles.KPOINTS[1], torch, 128)
    try:
        rng = np.random.default_rng(pencils + columns)
        rhs = rng.standard_normal((dev.n, columns)) + 1j * rng.standard_normal((dev.n, columns))
        shifts = np.linspace(-2.6, 0.5, pencils) + 1j * np.linspace(0.05, 0.6, pencils)
        kw = dict(precision=native.PRECISION_BF16X3, adjoint=adjoint)
        ref = _factor_solve(dev, plan, h, s, shifts, rhs, torch, **kw)
        got = _factor_solve(dev, plan, h, s, shifts, rhs, torch, flags=native.SOLVE_TENSOR_CORES,
                            **kw)
        again = _factor_solve(dev, plan, h, s, shifts, rhs, torch,
                              flags=native.SOLVE_TENSOR_CORES, **kw)
        for p in range(pencils):
            err = np.linalg.norm(got[p] - ref[p]) / np.linalg.norm(ref[p])
            assert err < 1e-3, (p, err)
        assert np.array_equal(got, again)
    finally:
        dev.close()
        plan.close()
